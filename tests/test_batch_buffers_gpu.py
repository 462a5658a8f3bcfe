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
