"""Decode attention with even shares where neighbouring pieces of a CTA have few and many rows (softmax spread over the accumulator's
quadrants or not, idle warps, queries loaded once or four times), distance biases, and partials by SM instead of by tile."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
HQ, HKV = 12, 3


def check(seqs_rows, dim, page, shared, options, max_splits, max_visible):
    """``seqs_rows``: (tokens with the step's rows, rows) of each sequence."""
    from phaseshift_b200.ops import _lib
    from phaseshift_b200.ops.cuda_ops import AttnOptions, c_float, c_int, ptr
    from phaseshift_b200.ops.specs import AttnSpec
    need = [-(-n // page) for n, _ in seqs_rows]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(dim)) + 1           # page 0 is nobody's
    table = torch.zeros(len(need), max(need), dtype=torch.int32)
    for i, pages in enumerate(torch.split(order, need)):
        table[i, :len(pages)] = pages
    seqs, pos, at = [], [], 0
    for i, (n, r) in enumerate(seqs_rows):
        seqs.append((at, r, i, n - r))
        pos += range(n - r, n)
        at += r
    rows, n_pages = at + 1, sum(need) + 1                        # and a padding row
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, k = rand(rows, HQ, dim), rand(n_pages, HKV, page, dim)
    v = k if shared else rand(n_pages, HKV, page, dim)
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    table_d, seqs_d, pos_d = table.cuda(), dev(seqs), dev(pos + [-1])
    acc = torch.full((rows, HQ, max_splits, dim), float("nan"), device="cuda")
    ml = torch.full((rows, HQ, max_splits, 2), float("nan"), device="cuda")
    part_n = torch.full((rows, HKV), 1 << 30, dtype=torch.int32, device="cuda")
    out = torch.full((rows, HQ * dim), 7.0, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    spec = AttnSpec(HQ, HKV, dim, dim ** -0.5, **options)
    opts = AttnOptions.of(spec)
    _lib.call("ps_attn_decode_tc_even", ptr(q), c_int(rows), ptr(k), ptr(v), ptr(table_d), c_int(table.shape[1]), c_int(page), c_int(n_pages),
              ptr(seqs_d), c_int(len(seqs)), c_int(16), c_int(HQ), c_int(HKV), c_int(dim), c_float(spec.scale), c_int(max_splits), c_int(max_visible),
              ptr(acc), ptr(ml), ptr(part_n), ptr(status), ctypes.byref(opts))
    _lib.call("ps_paged_attention_merge_even", ptr(acc), ptr(ml), ptr(part_n), ptr(pos_d), c_int(rows), c_int(HQ), c_int(HKV), c_int(dim),
              c_int(max_splits), ptr(None), c_int(0), c_int(0), c_int(0), ptr(out), ctypes.byref(opts))
    torch.cuda.synchronize()
    assert status.item() == 0 and bool((out[-1] == 0).all()) and int(part_n[:-1].max()) <= max_splits
    worst = (0.0,)
    for at, r, slot, start in seqs:
        pages = table[slot, :need[slot]].long().cuda()
        ks, vs = (p[pages].double().transpose(1, 2).reshape(-1, HKV, dim) for p in (k, v))
        for i in range(r):
            p = start + i
            s = torch.einsum("hgd,thd->hgt", q[at + i].double().view(HKV, HQ // HKV, dim), ks[:p + 1]) * spec.scale
            if spec.bias is not None:
                far = p - torch.arange(p + 1, device="cuda")
                s = s + spec.bias.double().view(HKV, HQ // HKV, -1)[:, :, far.clamp(max=spec.bias.shape[1] - 1)]
            want, size = (torch.einsum("hgt,thd->hgd", s.softmax(-1), x[:p + 1]).reshape(-1) for x in (vs, vs.abs()))
            # probabilities are rounded to 8 significant bits before the product: each moves by up to 2^-8 of itself, and so does the
            # sum of sizes; the result is rounded likewise; scores in 32 bits and the hardware's exponential add less than 2^-12
            err, tol = (out[at + i].double() - want).abs(), (2 ** -8 + 2 ** -12) * size + 2 ** -8 * want.abs() + 1e-6
            worst = max(worst, (float((err / tol).max()), slot, p, int((err > tol).sum())))
    assert worst[0] <= 1, worst


ROWS = [1, 4, 5, 8, 13, 16, 2, 3, 12]


@pytest.mark.parametrize("dim,page,shared,biased", [(256, 16, False, False), (256, 64, True, False), (64, 32, False, True), (128, 16, False, True)])
@pytest.mark.parametrize("n,longest", [(90, 200), (25, 900)])
def test_pieces_of_few_and_many_rows(dim, page, shared, biased, n, longest):
    g = torch.Generator().manual_seed(n)
    lens = torch.randint(16, longest, (n,), generator=g).tolist()
    bias = torch.randn(HQ, 100, generator=g).cuda() if biased else None
    check([(m, ROWS[i % len(ROWS)]) for i, m in enumerate(lens)], dim, page, shared, dict(bias=bias), -(-longest // 64), longest)


def test_a_partial_for_every_sm_suffices():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    check([(40000, 2), (17, 16), (12345, 5), (1, 1)], 256, 64, False, {}, sms, 131073)
