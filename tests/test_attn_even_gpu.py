"""Decode attention with even shares of a batch's tiles (csrc/kernels/attn_tc.cuh, `part_n`): sequences from one tile to many, shares that
begin and end inside them, several rows, masks, keys that are the values, sequences and rows that belong to others."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
LENS = [[1, 64, 65, 3000, 129, 1500, 7, 640, 2000, 63], [5], list(range(1, 41)), [4000] * 40]


def pages_of(lens, page, seed):
    """Scattered pages; page 0 is nobody's."""
    n_pages, used = sum(-(-n // page) for n in lens) + 1, 0
    order = torch.randperm(n_pages - 1, generator=torch.Generator().manual_seed(seed)) + 1
    table = torch.zeros(len(lens) + 1, -(-4100 // page), dtype=torch.int32)
    for i, n in enumerate(lens):
        b = -(-n // page)
        table[i, :b] = order[used:used + b]
        used += b
    return n_pages, table


def partials(rows, hq, hkv, dim):
    splits = -(-4100 // 64)
    acc = torch.full((rows, hq, splits, dim), float("nan"), device="cuda")
    ml = torch.full((rows, hq, splits, 2), float("nan"), device="cuda")
    return splits, acc, ml, torch.full((rows, hkv), 1 << 30, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("lens", LENS, ids=["ragged", "one", "short", "many"])
@pytest.mark.parametrize("dim,page,shared,options", [(256, 16, False, {}), (256, 64, True, dict(chunk=1024)), (64, 32, False, dict(window=300, keep_first=70)),
                                                     (128, 16, False, dict(temp_coef=0.1, temp_every=512.0))])
def test_even_shares(lens, dim, page, shared, options):
    from phaseshift_b200.ops import _lib
    from phaseshift_b200.ops.cuda_ops import AttnOptions, c_float, c_int, ptr
    from phaseshift_b200.ops.specs import AttnSpec
    hq, hkv = 12, 3
    n_pages, table = pages_of(lens, page, dim)
    seqs, pos, at = [], [], 0
    for i, n in enumerate(lens):                    # up to three rows each, the last of which sees n positions
        r = min(1 + i % 3, n)
        seqs.append((at, r, i, n - r))
        pos += range(n - r, n)
        at += r
    rows = at + 2                                   # a row of another kernel of the step and a padding row
    pos += [-2, -1]
    seqs.insert(len(seqs) // 2, (0, 17, 0, 50))     # more rows than this kernel takes
    seqs.append((0, 0, -1, 0))                      # unused
    g = torch.Generator(device="cuda").manual_seed(1)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, k = rand(rows, hq, dim), rand(n_pages, hkv, page, dim)
    v = k if shared else rand(n_pages, hkv, page, dim)
    dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    table_d, seqs_d, pos_d = table.cuda(), dev(seqs), dev(pos)
    splits, acc, ml, part_n = partials(rows, hq, hkv, dim)
    out = torch.full((rows, hq * dim), 7.0, device="cuda", dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    spec = AttnSpec(hq, hkv, dim, dim ** -0.5, **options)
    opts = AttnOptions.of(spec)
    for _ in range(2):
        _lib.call("ps_attn_decode_tc_even", ptr(q), c_int(rows), ptr(k), ptr(v), ptr(table_d), c_int(table.shape[1]), c_int(page), c_int(n_pages),
                  ptr(seqs_d), c_int(len(seqs)), c_int(16), c_int(hq), c_int(hkv), c_int(dim), c_float(spec.scale), c_int(splits), c_int(4100),
                  ptr(acc), ptr(ml), ptr(part_n), ptr(status), ctypes.byref(opts))
        _lib.call("ps_paged_attention_merge_even", ptr(acc), ptr(ml), ptr(part_n), ptr(pos_d), c_int(rows), c_int(hq), c_int(hkv), c_int(dim),
                  c_int(splits), ptr(None), c_int(0), c_int(0), c_int(0), ptr(out), ctypes.byref(opts))
    torch.cuda.synchronize()
    assert status.item() == 0
    assert (out[-2] == 7).all() and (out[-1] == 0).all()
    q64, worst = q.double().view(rows, hkv, hq // hkv, dim), (0.0,)
    for at, r, slot, start in seqs:
        if not 0 < r <= 16:
            continue
        pages = table[slot, :-(-(start + r) // page)].long().cuda()
        ks, vs = (p[pages].double().transpose(1, 2).reshape(-1, hkv, dim) for p in (k, v))
        for i in range(r):
            p = start + i
            seen = torch.arange(p + 1, device="cuda")
            lo = p // spec.chunk * spec.chunk if spec.chunk else max(0, p - spec.window + 1) if spec.window else 0
            seen = seen[(seen >= lo) | (seen < spec.keep_first)]
            s = torch.einsum("hgd,thd->hgt", q64[at + i], ks[seen]) * spec.scale
            if spec.temp_coef:
                s = s * (1 + spec.temp_coef * torch.log(torch.floor(torch.tensor((p + 1) / spec.temp_every, dtype=torch.float64, device="cuda")) + 1))
            want, size = (torch.einsum("hgt,thd->hgd", s.softmax(-1), x[seen]).reshape(-1) for x in (vs, vs.abs()))
            # probabilities are rounded to 8 significant bits before the product: each moves by up to 2^-8 of itself, and so does the
            # sum of sizes; the result is rounded likewise; scores in 32 bits and the hardware's exponential add less than 2^-12
            err, tol = (out[at + i].double() - want).abs(), (2 ** -8 + 2 ** -12) * size + 2 ** -8 * want.abs() + 1e-6
            worst = max(worst, (float((err / tol).max()), slot, p, int((err > tol).sum())))
    assert worst[0] <= 1, worst
