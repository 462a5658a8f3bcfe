"""Which bf16 GEMM a projection calls: weights that the launch before expands into the shared scratch must not be read ahead of the wait for
that launch, the model's own may be (csrc/kernels/gemm_tc.cu: ps_gemm_bf16_tc, ps_gemm_bf16_tc_resident)."""
import types

import pytest
import torch

from phaseshift_b200.ops import cuda_ops
from phaseshift_b200.ops.cuda_ops import CudaOps


@pytest.mark.parametrize("M", [9, 64, 129, 600])
@pytest.mark.parametrize("resident", [False, True])
def test_scratch_is_not_read_ahead_of_its_writer(monkeypatch, M, resident):
    calls = []
    monkeypatch.setattr(cuda_ops._lib, "call", lambda name, *args: calls.append((name, [getattr(x, "value", None) for x in args])))
    o = object.__new__(CudaOps)
    o.device, o.wscratch, o.status, o.launches = torch.device("cpu"), None, torch.zeros(1, dtype=torch.int32), 0
    o._smallm_splits, o.ws = {(256, 64): 1}, {}
    own = torch.zeros(256, 64, dtype=torch.bfloat16)
    w = types.SimpleNamespace(fmt="nvfp4", N=256, k_padded=64, tensor_scale=1.0, tiled=torch.zeros(64), rowmajor_bf16=own if resident else None)
    out = torch.empty(M, 256, dtype=torch.bfloat16)
    o.linear_large(torch.zeros(M, 64, dtype=torch.bfloat16), w, norm_w=None, eps=0.0, residual=None, epi=cuda_ops.EPI_STORE, out_f32=False, out=out)
    name, args = calls[-1]
    if resident:
        assert len(calls) == 1 and own.data_ptr() in args
        assert name == ("ps_gemm_smallm_normed" if M <= 64 else "ps_gemm_bf16_tc_resident")
    else:                                              # (the few-row GEMM reads early as well)
        assert [n for n, _ in calls] == ["ps_dequant_tiled", "ps_gemm_bf16_tc"] and o.wscratch.data_ptr() in args
