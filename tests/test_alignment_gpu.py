"""Rows that begin at any element: kernels with wide loads and stores take them by narrower ones and leave the same bytes."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
ci, cf = ctypes.c_int, ctypes.c_float


def _vp(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else None)


def _shifted(t, by):
    """A copy of `t` that begins `by` elements into its allocation."""
    raw = torch.zeros(t.numel() + by, dtype=t.dtype, device=t.device)
    raw[by:].copy_(t.reshape(-1))
    return raw[by:].view(t.shape)


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("rows", [3, 70])
def test_rotation_and_append_to_rows_at_odd_addresses(fmt, rows):
    from phaseshift_b200.ops import _lib
    hq, hkv, D, rot, page, pages = 6, 2, 128, 64, 16, 8
    g = torch.Generator(device="cuda").manual_seed(rows)
    qkv = torch.randn(rows, (2 * hq + 2 * hkv) * D, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2, D, device="cuda", generator=g) * 0.1).bfloat16()
    freq = 1e4 ** (-torch.arange(rot // 2, dtype=torch.float64, device="cuda") / (rot // 2))
    slot = torch.zeros(rows, dtype=torch.int32, device="cuda")
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    table = torch.arange(1, pages, dtype=torch.int32, device="cuda").view(1, -1)
    got = []
    for by in (0, 1):
        q = _shifted(torch.zeros(rows, hq * D, dtype=torch.bfloat16, device="cuda"), by)
        pool = torch.zeros(pages, hkv, page, D, dtype=torch.uint8 if fmt else torch.bfloat16, device="cuda")
        k, v = _shifted(pool, by), _shifted(pool, by)
        scale = torch.zeros(2, pages, hkv, page, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("ps_attn_prep", _vp(_shifted(qkv, by)), ci(qkv.shape[1]), ci(rows), ci(hq), ci(hkv), ci(D), ci(rot), _vp(w[0]), _vp(w[1]), cf(1e-6), _vp(freq),
                  _vp(slot), _vp(pos), _vp(q), _vp(k), _vp(v), _vp(scale[0]), _vp(scale[1]), _vp(table), ci(pages - 1), ci(page), ci(pages), ci(fmt), _vp(status))
        torch.cuda.synchronize()
        assert int(status[0]) == 0
        got.append([q.clone(), k.clone(), v.clone(), scale])
    assert all(torch.equal(a, b) for a, b in zip(*got)) and bool(got[0][1].float().abs().sum() > 0)


@pytest.mark.parametrize("H,rows", [(32, 1), (2560, 5)])
def test_quantised_embedding_rows_at_odd_addresses(H, rows):
    from phaseshift_b200.ops import _lib
    vocab = 40
    g = torch.Generator(device="cuda").manual_seed(H)
    codes = torch.randint(0, 256, (vocab, H), device="cuda", generator=g, dtype=torch.uint8)
    codes[(codes & 0x7F) == 0x7F] = 0                       # (the two NaN codes)
    scales = torch.randint(100, 140, (vocab, H // 32), device="cuda", generator=g, dtype=torch.uint8)
    ids = torch.randint(0, vocab, (rows,), device="cuda", generator=g, dtype=torch.int32)
    want = (codes.view(torch.float8_e4m3fn).float().view(vocab, -1, 32) * torch.exp2(scales.float() - 127)[..., None]).view(vocab, H).bfloat16()[ids.long()]
    for c_by, o_by, pad in ((0, 0, 0), (1, 0, 0), (4, 1, 0), (0, 4, 8), (3, 0, 1)):
        c = _shifted(codes, c_by)
        out = _shifted(torch.full((rows, H + pad), 7.0, dtype=torch.bfloat16, device="cuda"), o_by)
        ssq = torch.zeros(rows, device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("ps_embedding_mxfp8", _vp(ids), _vp(c), _vp(scales), ci(rows), ci(vocab), ci(H), _vp(out), ci(H + pad), _vp(status), _vp(ssq), ci(1))
        torch.cuda.synchronize()
        assert int(status[0]) == 0 and torch.equal(out[:, :H], want) and bool((out[:, H:] == 7).all())
        # a 32-bit sum of H squares: H 2^-24 of it at most
        assert torch.allclose(ssq.double(), want.double().pow(2).sum(1), rtol=H * 2.0 ** -24, atol=0)


@pytest.mark.parametrize("by", [0, 1])
def test_residual_projection_before_a_norm_whose_weights_lie_anywhere(by):
    """The norm joins the projection's reduction where it can; other weights leave it to the next projection, which gives the same rows."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import LinearW
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.ops.specs import NextNorm
    from phaseshift_b200.quant.formats import quantize
    dev = torch.device("cuda:0")
    ops = CudaOps(tiny_config(), dev)
    g = torch.Generator(device="cuda").manual_seed(1)
    W, V = (LinearW(quantize(torch.randn(256, 256, device="cuda", generator=g) / 16, "bf16")) for _ in range(2))
    x, res = (torch.randn(4, 256, device="cuda", generator=g).bfloat16() for _ in range(2))
    nxt = NextNorm(_shifted((torch.randn(256, device="cuda", generator=g) * 0.1).bfloat16(), by), 1e-6, "xn")
    r = ops.linear(x, W, name="r", residual=res, norm_next=nxt)
    assert (nxt.rows is None) == bool(by)
    y = ops.linear(r, V, name="y", norm_w=nxt.weight, eps=1e-6, x_normed=nxt.rows, out_f32=True)
    rd = (x.double() @ W.q.codes.double().T).bfloat16().double() + res.double()
    assert float((r.double() - rd).norm() / rd.norm()) < 2.0 ** -7          # the product and the sum, each rounded to bf16 (2^-8)
    rd = r.double()
    want = (rd * torch.rsqrt(rd.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + nxt.weight.double())) @ V.q.codes.double().T
    assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -8      # the normed rows, rounded to bf16
