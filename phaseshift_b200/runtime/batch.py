"""Per-step batch descriptor (the analogue of the reference's DeviceBatchContext,
include/phaseshift/runtime/batch/device_batch_context.h:14-85).

The host describes a step by *requests* (slot, first position, number of rows, which rows need logits);
the per-row arrays the kernels index (token id, slot, position) are expanded into ONE packed int32
buffer that goes to the device with ONE pinned host-to-device copy.  The device buffers are allocated
once per row bucket, so a captured CUDA graph can be replayed after refreshing them.
"""
from __future__ import annotations

from dataclasses import dataclass, field
from typing import List, Optional, Sequence

import numpy as np
import torch

from ..core.native import runtime

ROW_BUCKETS = (1, 2, 4, 8, 16, 32, 64, 128, 256, 512, 1024, 2048)


def resolve_row_bucket(rows: int) -> int:
    """Smallest bucket holding `rows` (reference: include/phaseshift/runtime/execution/row_bucket.h:7-68,
    extended downwards: on B200 decode steps are graph-captured per small bucket)."""
    for b in ROW_BUCKETS:
        if rows <= b:
            return b
    raise ValueError(f"{rows} rows exceed the largest row bucket {ROW_BUCKETS[-1]}")


@dataclass
class SeqRows:
    slot: int
    pos_start: int
    token_ids: Sequence[int]
    output_rows: Sequence[int] = ()        # indices into token_ids whose logits are sampled
    temperature: float = 0.0
    top_p: float = 1.0
    top_k: int = 0
    seed: int = 0
    sample_index: int = 0                  # tokens generated so far (first output row); +1 per further row


SAMPLING_ROW_DTYPE = np.dtype([("mode", "<u4"), ("temperature", "<f4"), ("top_p", "<f4"), ("top_k", "<u4"),
                               ("seed", "<u8"), ("sample_index", "<u8")])


class StepBatch:
    """Host-side packed step + its device mirror."""
    SHORT_SEQ_ROWS = 16          # = CudaOps.ATTN_PREFILL_MIN_ROWS: sequences with more rows take the tiled attention kernel

    def __init__(self, max_rows: int, max_seqs: int, device, pinned: Optional[bool] = None):
        self.max_rows, self.max_seqs, self.device = max_rows, max_seqs, device
        use_pin = (device.type == "cuda") if pinned is None else pinned
        n_int = 3 * max_rows + 4 * max_seqs + 2 * max_rows    # ids, slot, pos | seq descs | output rows | pos of short sequences' rows
        # one buffer for the integers and the sampling rows behind them, so that a step's description is one copy
        ints, samp = -(-n_int * 4 // 16) * 16, max_rows * SAMPLING_ROW_DTYPE.itemsize
        self.h_all = torch.zeros(ints + samp, dtype=torch.uint8, pin_memory=use_pin)
        self.d_all = torch.zeros(ints + samp, dtype=torch.uint8, device=device)
        self.h_int, self.h_samp = self.h_all[:n_int * 4].view(torch.int32), self.h_all[ints:]
        self.d_int, self.d_samp = self.d_all[:n_int * 4].view(torch.int32), self.d_all[ints:]
        self.n_rows = self.n_seqs = self.n_out = 0
        self.max_visible = 1
        # graph_static: the step is replayed from a captured CUDA graph, so launch geometry must not
        # depend on this step's contents (attention covers max_context, GDN covers max_seqs descriptors)
        self.graph_static = False
        self.identity_out = False
        self.several_rows = False        # some sequence has more than one row in the step
        # More than three rows a sequence: the delta rule's kernel that prepares rows together is sooner from there on (us with 48 heads, row after
        # row / together: two rows 6.1 / 7.0, three 7.9 / 8.0, four 9.7 / 8.9, eight 17.1 / 12.0; three sequences of two rows 7.6 / 8.9)
        self.multi_rows = False
        self.max_context = 1
        o = 0
        self.ids = self.d_int[o:o + max_rows]; o += max_rows
        self.row_slot = self.d_int[o:o + max_rows]; o += max_rows
        self.row_pos = self.d_int[o:o + max_rows]; o += max_rows
        self.seq_desc = self.d_int[o:o + 4 * max_seqs].view(max_seqs, 4); o += 4 * max_seqs
        self.out_rows = self.d_int[o:o + max_rows]; o += max_rows
        # positions of the rows of sequences with at most SHORT_SEQ_ROWS rows in the step, -2 for the rows of longer sequences
        # (the per-row attention kernel leaves those rows' outputs alone: the tiled kernel of the same step wrote them) and
        # -1 for padding rows
        self.row_pos_short = self.d_int[o:o + max_rows]
        self._np_samp = self.h_samp.numpy().view(SAMPLING_ROW_DTYPE)
        self._fill = runtime().fill_step
        self.seqs: List[SeqRows] = []

    def fill(self, seqs: Sequence[SeqRows]) -> None:
        self.n_rows, self.n_out, self.max_visible, self.identity_out = self._fill(
            self.h_int.data_ptr(), self.h_samp.data_ptr(), self.max_rows, self.max_seqs, self.SHORT_SEQ_ROWS, seqs)
        # (identity_out: output row i is step row i for every i -- a pure decode batch -- so the output gather is the identity)
        self.n_seqs = len(seqs)
        self.seqs = list(seqs)
        self.several_rows, self.multi_rows = self.n_rows > self.n_seqs, self.n_rows > 3 * self.n_seqs

    @property
    def max_visible_launch(self) -> int:
        return self.max_context if self.graph_static else self.max_visible

    def upload(self) -> None:
        self.d_all.copy_(self.h_all, non_blocking=True)

    def h2d_bytes(self) -> int:
        return self.h_all.numel()
