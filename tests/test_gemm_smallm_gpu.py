"""Few-row bf16 products (csrc/kernels/gemm_smallm.cu): their reductions at the edges of tiles and splits, and the one that norms the
rows for the next projection."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
ci, cf = ctypes.c_int, ctypes.c_float
EPS = 1e-6


def _vp(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else None)


def _run(a, w, out, epi=0, residual=None, norm_w=None, normed=None):
    from phaseshift_b200.ops import _lib
    M, K = a.shape
    N = w.shape[0]
    part = torch.empty(_lib.lib().ps_gemm_smallm_splits(ci(N), ci(K)) * M * N, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("ps_gemm_smallm_normed", _vp(a), ci(a.stride(0)), _vp(w), ci(w.stride(0)), ci(M), ci(N), ci(K), ci(epi), _vp(residual),
              ci(residual.stride(0) if residual is not None else 0), _vp(out), ci(out.stride(0)), ci(int(out.dtype == torch.float32)),
              _vp(norm_w), cf(EPS), _vp(normed), ci(normed.stride(0) if normed is not None else 0), _vp(part), _vp(status))
    torch.cuda.synchronize()
    assert int(status[0]) == 0


@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (2, 130, 2560), (8, 2560, 4096), (9, 132, 9216), (33, 5120, 1032), (64, 16384, 256)])
def test_smallm_products_and_normed_rows(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()
    res = torch.randn(M, N + 4, device="cuda", generator=g).bfloat16()[:, :N]
    ref = a.double() @ w.double().T
    # 32-bit sums (K additions of at most 2^-24 of the largest term) and roundings to bf16 (8 significant bits) of at most 2^-8 of a value
    acc, rnd = K * 2.0 ** -24, 2.0 ** -8
    rel = lambda x, y: float((x.double() - y).norm() / y.norm())
    out = torch.empty(M, N, device="cuda")
    _run(a, w, out)
    assert rel(out, ref) < acc
    half = torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda")
    _run(a, w, half, 2)
    assert rel(half, torch.nn.functional.silu(ref[:, 0::2]) * ref[:, 1::2]) < 4 * acc + 4 * rnd
    buf = torch.full((M + 1, N + 4), 7.0, dtype=torch.bfloat16, device="cuda")
    _run(a, w, buf[:M, :N], 1, res)
    assert rel(buf[:M, :N], ref + res.double()) < acc + 2 * rnd
    assert bool((buf[M] == 7).all()) and bool((buf[:, N:] == 7).all())
    if N % 4 == 0:
        nw = (torch.randn(N, device="cuda", generator=g) * 0.1).bfloat16()
        x = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        y = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
        _run(a, w, x, 1, res, nw, y[:M])
        assert torch.equal(x, buf[:M, :N])
        xd = x.double()
        want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + EPS) * (1 + nw.double())
        assert rel(y[:M], want) < rnd + 1e-5 and bool((y[M] == 7).all())


@pytest.mark.parametrize("rows,H,pad", [(1, 8, 0), (3, 2560, 8), (2, 4104, 0), (5, 8200, 8), (2, 16384, 0), (3, 20, 0), (2, 16392, 0), (4, 2560, 1)])
def test_rmsnorm_rows(rows, H, pad):
    """Vector and scalar kernels; rows and pitches that are no multiple of 16 bytes take the latter."""
    from phaseshift_b200.ops import _lib
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(rows, H + pad, device="cuda", generator=g).bfloat16()[:, :H]
    w = (torch.randn(H, device="cuda", generator=g) * 0.1).bfloat16()
    for one_plus in (0, 1):
        out = torch.full((rows + 1, H + pad), 7.0, dtype=torch.bfloat16, device="cuda")
        _lib.call("ps_rmsnorm", _vp(x), ci(x.stride(0)), _vp(None), ci(0), _vp(None), ci(0), _vp(w), cf(EPS), ci(rows), ci(H), _vp(out),
                  ci(out.stride(0)), ci(one_plus))
        xd = x.double()
        want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + EPS) * (one_plus + w.double())
        assert float((out[:rows, :H].double() - want).norm() / want.norm()) < 2.0 ** -8 + 1e-5
        assert bool((out[rows] == 7).all()) and bool((out[:, H:] == 7).all())


@pytest.mark.parametrize("M,N,K", [(32, 34816, 5120), (8, 18432, 2560), (2, 37888, 2560), (64, 20480, 5184), (5, 4096, 128), (3, 131, 64)])
def test_smallm_sums_lose_no_more_than_half_a_run(M, N, K):
    """Error against 64 bits of products whose CTAs have long runs of K, and of ones with a single step or none to spare."""
    from phaseshift_b200.ops import _lib
    g = torch.Generator(device="cuda").manual_seed(N + K)
    N += N & 1
    a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=g) * 0.02).bfloat16()
    out = torch.empty(M, N, device="cuda")
    _run(a, w, out)
    ref = torch.cat([a.double() @ p.double().T for p in w.split(8192)], 1)
    # an addition to the accumulator drops half a last place on average, 2^-25 to 2^-24 of its value; over a run the sum grows as the
    # square root of its length, so n additions cost about n 2^-25 of the result.  A run is what a CTA adds up, or half of it where that
    # is more than eight steps, at 4 additions per step; below that the 32-bit sum of a few runs and the stored result are left (2^-24 each).
    steps = -(-(-(-K // 64)) // _lib.lib().ps_gemm_smallm_splits(ci(N), ci(K)))
    run = steps if steps <= 8 else -(-steps // 2)
    assert float((out.double() - ref).norm() / ref.norm()) < 4 * run * 2.0 ** -25 + 4 * 2.0 ** -24


def test_runs_of_k_fit_the_device_at_once():
    from phaseshift_b200.ops import _lib
    room = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    for N in (8, 130, 2560, 5120, 12352, 18432, 34816, 151936):
        for K in (64, 520, 2560, 5120, 17408):
            splits = _lib.lib().ps_gemm_smallm_splits(ci(N), ci(K))
            assert splits == 1 or (splits <= 16 and splits * -(-N // 128) <= room)
