"""Buffers that captured steps of few rows write to outlive larger steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_partial_sums_of_small_steps_keep_their_buffer():
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import LinearW
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.quant.formats import quantize
    dev = torch.device("cuda:0")
    ops = CudaOps(tiny_config(), dev)
    held = lambda: {k: t.data_ptr() for k, t in ops.ws.items() if k[0] == "smallm_partial"}
    for N, M in ((2560, 8), (5120, 64), (151936, 64)):
        before = held()
        W = LinearW(quantize(torch.randn(N, 512, device="cuda") * 0.02, "bf16"))
        ops.linear(torch.randn(M, 512, device="cuda").bfloat16(), W, name="y%d" % N)
        after = held()
        assert after and all(after.get(k) == p for k, p in before.items())


def test_products_that_are_stored_directly_hold_no_partial_sums():
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import LinearW
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.quant.formats import quantize
    ops = CudaOps(tiny_config(), torch.device("cuda:0"))
    W = LinearW(quantize(torch.randn(40000, 64, device="cuda") * 0.1, "bf16"))           # more column tiles than run at once: one run of K
    x = torch.randn(64, 64, device="cuda").bfloat16()
    y = ops.linear(x, W, name="logits", out_f32=True)
    want = x.double() @ W.q.codes.double().T
    assert float((y.double() - want).norm() / want.norm()) < 64 * 2.0 ** -24             # 32-bit sums of 64 terms
    assert not any(k[0] == "smallm_partial" for k in ops.ws) and ops.launches == 1
    ops.linear(x, W, name="rows")                                                        # bf16: through the reduction
    assert any(k[0] == "smallm_partial" for k in ops.ws) and ops.launches == 3
