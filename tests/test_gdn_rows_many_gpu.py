"""The delta-rule kernel for sequences with several rows in a step (csrc/kernels/gdn_recurrent.cu: gdn_rows_many_kernel) has the bits of the one
that takes row after row: outputs, state, history and log, at the edges of its eight rows and of the history ring."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [128, 64])
@pytest.mark.parametrize("ring,logged,projected", [(4, False, False), (11, True, True), (19, True, False)])
def test_rows_have_the_same_bits(dim, ring, logged, projected):
    from phaseshift_b200.models.qwen35.config import Qwen35Config
    from phaseshift_b200.models.qwen35.weights import build_engine_weights, random_hf_weights
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    dev, hk, hv = torch.device("cuda:0"), 2, 4
    cfg = Qwen35Config(vocab_size=1024, hidden_size=256, intermediate_size=256, num_hidden_layers=4, linear_num_key_heads=hk, linear_num_value_heads=hv,
                       linear_key_head_dim=dim, linear_value_head_dim=dim)
    hf = random_hf_weights(cfg, seed=4, device="cuda")
    gw = build_engine_weights(cfg, lambda n: hf[n], "bf16", "cuda").layers[0].mixer
    lens = [[1, 2, 3, 8], [9, 4, 16, 7], [1, 13, 5, 1]]
    got = []
    for many in (False, True):
        ops = CudaOps(cfg, dev, max_seq_len=512)
        st = ModelState(cfg, StateConfig(max_slots=4, max_seq_len=512, conv_ring=ring), dev)
        g = torch.Generator(device="cuda").manual_seed(ring)
        for t in (st.gdn[0].rec, st.gdn[0].conv):
            t.copy_(torch.randn(t.shape, device="cuda", generator=g) * 0.3)
        pos, res = [0, 0, 5, 700], []
        for rows in lens:
            n = sum(rows)
            proj = (torch.randn(n, gw.in_proj.N + gw.ba_proj.N, device="cuda", generator=g) * 0.7).bfloat16()
            xn = torch.randn(n, 256, device="cuda", generator=g).bfloat16() if projected else None
            b = StepBatch(64, 4, dev)
            b.fill([SeqRows(s, pos[s], [0] * k, ()) for s, k in enumerate(rows)])
            b.upload()
            b.multi_rows = many
            log = tuple(torch.zeros(n, hv, *e, device="cuda") for e in ((dim,), (dim,), ())) if logged else None
            out = ops.gdn(proj, gw, hk, hv, b, st.gdn[0], st, log=log, xn=xn)
            torch.cuda.synchronize()
            res += [out.clone(), st.gdn[0].rec.clone(), st.gdn[0].conv.clone(), *(log or ())]
            pos = [p + k for p, k in zip(pos, rows)]
        got.append(res)
    assert len(got[0]) == len(got[1]) and all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("hidden", [128, 520, 1288])
def test_projected_gates_have_the_same_bits(hidden):
    """Beta and decay projected in the kernel, for widths below, beside and above a pass of the CTA's threads (512 columns)."""
    from phaseshift_b200.models.qwen35.config import Qwen35Config
    from phaseshift_b200.models.qwen35.weights import build_engine_weights, random_hf_weights
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    dev, hk, hv, lens = torch.device("cuda:0"), 2, 4, [1, 5, 8, 9]
    cfg = Qwen35Config(vocab_size=1024, hidden_size=hidden, intermediate_size=256, num_hidden_layers=4, linear_num_key_heads=hk, linear_num_value_heads=hv)
    hf = random_hf_weights(cfg, seed=4, device="cuda")
    gw = build_engine_weights(cfg, lambda n: hf[n], "bf16", "cuda").layers[0].mixer
    n, got = sum(lens), []
    for many in (False, True):
        ops, st = CudaOps(cfg, dev, max_seq_len=512), ModelState(cfg, StateConfig(max_slots=4, max_seq_len=512), dev)
        g = torch.Generator(device="cuda").manual_seed(hidden)
        proj = (torch.randn(n, gw.in_proj.N + gw.ba_proj.N, device="cuda", generator=g) * 0.7).bfloat16()
        xn = torch.randn(n, hidden, device="cuda", generator=g).bfloat16()
        b = StepBatch(64, 4, dev)
        b.fill([SeqRows(s, 0, [0] * k, ()) for s, k in enumerate(lens)])
        b.upload()
        b.multi_rows = many
        out = ops.gdn(proj, gw, hk, hv, b, st.gdn[0], st, xn=xn)
        torch.cuda.synchronize()
        got.append((out.clone(), st.gdn[0].rec.clone(), st.gdn[0].conv.clone()))
    assert all(torch.equal(x, y) for x, y in zip(*got))
