"""Epilogue of the streamed block-scaled projections (csrc/kernels/gemm_bs.cu) at the edges of its blocks of rows, its pieces of columns and
cut tiles: every epilogue, rows of the output and the residual at any address, and nothing written beside them."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
@pytest.mark.parametrize("N,K,grid", [(200, 512, 0), (1030, 520, 7), (384, 5120, 148)])
@pytest.mark.parametrize("pad", [0, 8, 3])
def test_streamed_rows(fmt, N, K, grid, pad):
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import LinearW
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.quant.act_quant import fake_quant
    from phaseshift_b200.quant.formats import quantize
    ops = CudaOps(tiny_config(), torch.device("cuda:0"))
    ops.BS_RESIDENT_MAX_ROWS, ops.bs_grid_override = 0, grid
    g = torch.Generator(device="cuda").manual_seed(N + K)
    W = LinearW(quantize(torch.randn(N, K, device="cuda", generator=g) * 0.05, fmt)).make_umma()
    W.act_scale = 0.02
    wd = W.dense().double()
    for M in (1, 31, 33, 64, 65, 127, 129, 191, 193, 256, 257, 320):
        x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        y = fake_quant(x.float(), W.fmt, W.act_scale).double() @ wd.T
        yb = y.float().bfloat16().double()
        res = torch.randn(M, N + pad, device="cuda", generator=g).bfloat16()[:, pad:]
        for kind, n, want in (("store", N, y), ("residual", N, yb + res.double()), ("swiglu", N // 2, F.silu(yb[:, 0::2]) * yb[:, 1::2]), ("f32", N, y)):
            whole = torch.full((M + 1, n + pad + 1), 7.0, dtype=torch.float32 if kind == "f32" else torch.bfloat16, device="cuda")
            out = whole[:M, pad:pad + n]
            ops.linear_bs(x, W, name="y", norm_w=None, eps=1e-6, residual=res if kind == "residual" else None, swiglu=kind == "swiglu",
                          out_f32=kind == "f32", out=out)
            torch.cuda.synchronize()
            assert int(ops.status[0]) == 0
            # exact products of codes in 32-bit sums; a rounding to bf16 of the product, of the activation and of the result (2^-9 of each, and
            # a product on the edge between two bf16 values may fall to either)
            assert float((out.double() - want).norm() / want.norm()) < (1e-5 if kind == "f32" else 4 * 2.0 ** -9), (M, kind)
            assert bool((whole[M] == 7).all()) and bool((whole[:, :pad] == 7).all()) and bool((whole[:, pad + n:] == 7).all()), (M, kind)


@pytest.mark.parametrize("fmt,N,K", [("nvfp4", 1032, 5120), ("mxfp8", 640, 4096)])
def test_rows_of_a_tile_do_not_depend_on_how_many_are_live(fmt, N, K):
    """The last blocks of a 128-row tile are left out where they have no rows: what is computed has the bits of the full tile, in
    whole and in cut tiles."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import LinearW
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.quant.formats import quantize
    ops = CudaOps(tiny_config(), torch.device("cuda:0"))
    ops.BS_RESIDENT_MAX_ROWS = 0
    g = torch.Generator(device="cuda").manual_seed(N)
    W = LinearW(quantize(torch.randn(N, K, device="cuda", generator=g) * 0.05, fmt)).make_umma()
    W.act_scale = 0.02
    x, res = (torch.randn(128, c, device="cuda", generator=g).bfloat16() for c in (K, N))
    for grid in (3, 148):
        ops.bs_grid_override = grid
        for kind, n in (("store", N), ("residual", N), ("swiglu", N // 2), ("f32", N)):
            def rows(M):
                out = torch.full((128, n), 7.0, dtype=torch.float32 if kind == "f32" else torch.bfloat16, device="cuda")
                ops.linear_bs(x[:M], W, name="y", norm_w=None, eps=1e-6, residual=res[:M] if kind == "residual" else None, swiglu=kind == "swiglu",
                              out_f32=kind == "f32", out=out[:M])
                return out
            full = rows(128)
            for M in (1, 9, 16, 31, 32, 33, 48, 63, 64, 65, 95, 96, 97, 127):
                part = rows(M)
                assert torch.equal(part[:M], full[:M]) and bool((part[M:] == 7).all()), (grid, kind, M)
    torch.cuda.synchronize()
    assert int(ops.status[0]) == 0
