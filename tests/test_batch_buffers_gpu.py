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


def test_joined_projection_belongs_to_the_tensor_cores():
    """With the tensor-core GEMM switched off its weights must not be laid out a second time for the streaming kernel."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.models.qwen35.weights import build_engine_weights, random_getter
    from phaseshift_b200.runtime.batch import SeqRows
    from phaseshift_b200.runtime.engine import Engine
    from phaseshift_b200.runtime.state import StateConfig
    dev, cfg = torch.device("cuda:0"), tiny_config()
    logits = []
    for on in (True, False):
        w = build_engine_weights(cfg, random_getter(cfg, 0, dev), "bf16", dev)
        eng = Engine(w, dev, StateConfig(max_slots=2, max_seq_len=64, page_tokens=16))
        eng.ops.use_tc_gemm = on
        eng.apply_block_updates([(0, 0, 1), (1, 0, 2)])
        _, out, status = eng.run_rows([SeqRows(0, 0, [5], (0,)), SeqRows(1, 0, [9], (0,))], want_logits=True)
        assert status == 0
        logits.append(out.logits.double().clone())
        assert all(L.mixer.in_ba.tiled is None for L in w.layers if L.kind == 0)
    # bf16 activations through four layers
    assert float((logits[0] - logits[1]).norm() / logits[0].norm()) < 3e-2
