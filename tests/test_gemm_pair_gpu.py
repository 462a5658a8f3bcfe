"""The bf16 GEMM on CTA pairs (csrc/kernels/gemm_tc.cu) at the edges of its tiles: row and column remainders, depths that are no
multiple of a stage, tile widths below 256, more tiles than pairs, every epilogue; and rows of an output that it must not touch."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

STORE, RESIDUAL, SWIGLU, REGLU, GELU, GEGLU = range(6)


def _gemm(a, w, out, epi=STORE, residual=None):
    from phaseshift_b200.ops import _lib
    vp = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else None)
    ci = ctypes.c_int
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("ps_gemm_bf16_tc", vp(a), ci(a.stride(0)), vp(w), ci(w.stride(0)), ci(a.shape[0]), ci(w.shape[0]), ci(a.shape[1]), ci(epi),
              vp(residual), ci(residual.stride(0) if residual is not None else 0), vp(out), ci(out.stride(0)),
              ci(int(out.dtype == torch.float32)), vp(status))
    torch.cuda.synchronize()
    assert int(status[0]) == 0


@pytest.mark.parametrize("M,N,K", [(129, 256, 1032), (255, 330, 1088), (256, 2560, 1096), (257, 264, 2560), (777, 4104, 1032), (1300, 12352, 1088)])
def test_pair_gemm_edges(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    # operands and outputs inside larger buffers: pitches beyond the extents, and canaries around the rows
    a = torch.randn(M, K + 8, device="cuda", generator=g).bfloat16()[:, :K]
    w = (torch.randn(N, K + 16, device="cuda", generator=g) * K ** -0.5).bfloat16()[:, :K]
    ref = a.double() @ w.double().T
    # one rounding to bf16 (8 significant bits) is at most 2^-8 of a value; the sums are kept in 32 bits, K additions of at most 2^-24 of the largest term each
    acc = K * 2.0 ** -24
    rel = lambda x, y: float((x.double() - y).norm() / y.norm())
    for dtype, tol in ((torch.float32, acc), (torch.bfloat16, acc + 2.0 ** -8)):
        buf = torch.full((M + 2, N + 8), 7.0, dtype=dtype, device="cuda")
        _gemm(a, w, buf[1:-1, :N])
        assert rel(buf[1:-1, :N], ref) < tol
        assert bool((buf[0] == 7).all()) and bool((buf[-1] == 7).all()) and bool((buf[:, N:] == 7).all())
    res = torch.randn(M, N, device="cuda", generator=g).bfloat16()
    out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    _gemm(a, w, out, RESIDUAL, res)
    assert rel(out, ref + res.double()) < acc + 2 * 2.0 ** -8
    _gemm(a, w, out, GELU)
    assert rel(out, torch.nn.functional.gelu(ref, approximate="tanh")) < 2 * acc + 2 * 2.0 ** -8
    gate, up = ref[:, 0::2], ref[:, 1::2]
    for epi, y in ((SWIGLU, torch.nn.functional.silu(gate) * up), (REGLU, torch.relu(gate) * up),
                   (GEGLU, torch.nn.functional.gelu(gate, approximate="tanh") * up)):
        out = torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda")
        _gemm(a, w, out, epi)                    # gate, up and their product are rounded
        assert rel(out, y) < 4 * acc + 4 * 2.0 ** -8


def test_pair_gemm_row_does_not_depend_on_the_others():
    """Padding rows and the number of rows of a step change no other row."""
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(900, 1088, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2560, 1088, device="cuda", generator=g) * 0.03).bfloat16()
    full, part = (torch.empty(n, 2560, dtype=torch.bfloat16, device="cuda") for n in (900, 300))
    _gemm(a, w, full)
    _gemm(a[:300], w, part)
    assert torch.equal(full[:300], part)


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp8"])
@pytest.mark.parametrize("M", [129, 600])
def test_weights_expanded_into_one_scratch_in_turn(fmt, M):
    """Block-quantised weights without tensor-core scales go through one scratch matrix, written by the launch before the product:
    every product has its own weights, whatever the scratch held before."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import LinearW
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.quant.formats import quantize
    ops = CudaOps(tiny_config(), torch.device("cuda:0"))
    N, K = 1536, 2048
    g = torch.Generator(device="cuda").manual_seed(M)
    ws = [LinearW(quantize(torch.randn(N, K, device="cuda", generator=g) * 0.03, fmt)) for _ in range(2)]
    x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(8)]
    for i, out in enumerate(outs):                     # nothing between the launches
        ops.linear(x, ws[i % 2], name="y", out=out)
    torch.cuda.synchronize()
    assert int(ops.status[0]) == 0
    for i, out in enumerate(outs):
        # the expanded weights and the result are rounded to bf16 (2^-8 at most each); 32-bit sums of K products
        want = x.double() @ ws[i % 2].dense().double().T
        assert float((out.double() - want).norm() / want.norm()) < K * 2.0 ** -24 + 2 * 2.0 ** -8, i
        assert torch.equal(out, outs[i % 2])
