"""The chunked delta rule with its scan on tcgen05 (csrc/kernels/gdn_chunked.cu) at the edges of its chunks, against the same
recurrence row by row in 64 bits: single and ragged chunks, several sequences, a prompt that continues, fast and slow decays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(proj, gw, hk, hv, history, state, eps):
    """(outputs, new state) of one sequence: proj [n, ...] in 64 bits, history: the three raw inputs before it."""
    n, qk = len(proj), hk * 128
    ch = 2 * qk + hv * 128
    x = torch.cat([history, proj[:, :ch]])
    taps = gw.conv_w.double()
    x = torch.nn.functional.silu(sum(x[j:j + n] * taps[:, j] for j in range(4)))
    q, k, v = (t.reshape(n, -1, 128) for t in x.split([qk, qk, hv * 128], 1))
    q, k = ((t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(hv // hk, 1) for t in (q, k))
    z, b, a = proj[:, ch:].split([hv * 128, hv, hv], 1)
    decay = torch.exp(-torch.exp(gw.A_log.double()) * torch.nn.functional.softplus(a + gw.dt_bias.double()))
    beta, S, out = torch.sigmoid(b), state.clone(), []
    for t in range(n):
        S = S * decay[t][:, None, None]
        d = (v[t] - torch.einsum("hkv,hk->hv", S, k[t])) * beta[t][:, None]
        S = S + k[t][:, :, None] * d[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]) * 128 ** -0.5)
    o = torch.stack(out)
    o = o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + eps) * gw.norm_w.double() * torch.nn.functional.silu(z.reshape(n, hv, 128))
    return o.reshape(n, -1), S


@pytest.mark.parametrize("steps,rate", [([[17]], 0.0), ([[64], [64]], -6.0), ([[65, 130], [63, 20]], 0.0), ([[300]], 2.0), ([[128, 17, 193]], -2.0)])
def test_chunked_delta_rule(steps, rate):
    from phaseshift_b200.models.qwen35.config import Qwen35Config
    from phaseshift_b200.models.qwen35.weights import build_engine_weights, random_hf_weights
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    dev = torch.device("cuda:0")
    cfg = Qwen35Config(vocab_size=1024, hidden_size=256, intermediate_size=256, num_hidden_layers=4, linear_num_key_heads=2, linear_num_value_heads=4)
    hf = random_hf_weights(cfg, seed=4, device="cuda")
    gw = build_engine_weights(cfg, lambda n: hf[n], "bf16", "cuda").layers[0].mixer
    gw.A_log += rate                                     # from hardly any decay to a factor of e^-20 per row
    ops, hk, hv = CudaOps(cfg, dev, max_seq_len=512), 2, 4
    slots = len(steps[0])
    st = ModelState(cfg, StateConfig(max_slots=slots, max_seq_len=512), dev)
    g = torch.Generator(device="cuda").manual_seed(sum(steps[0]))
    st.gdn[0].rec.normal_(0, 0.3, generator=g)
    state = st.gdn[0].rec.double().clone()
    history = torch.zeros(slots, 3, (2 * hk + hv) * 128, dtype=torch.float64, device="cuda")
    pos = [0] * slots
    for rows in steps:
        proj = (torch.randn(sum(rows), gw.in_proj.N + gw.ba_proj.N, device="cuda", generator=g) * 0.7).bfloat16()
        b = StepBatch(512, slots, dev)
        b.fill([SeqRows(s, pos[s], [0] * n, ()) for s, n in enumerate(rows)])
        b.upload()
        got = ops.gdn(proj, gw, hk, hv, b, st.gdn[0], st)
        torch.cuda.synchronize()
        assert int(ops.status[0]) == 0
        at = 0
        for s, n in enumerate(rows):
            p = proj[at:at + n].double()
            want, state[s] = _exact(p, gw, hk, hv, history[s], state[s], cfg.rms_norm_eps)
            history[s] = torch.cat([history[s], p[:, :history.shape[2]]])[-3:]
            # operands of TF32 (2^-11 of a value) in sums of up to 128 terms; the head norm divides by small outputs: 1e-2 of the rows'
            # norm, as the mixed test of both kernels allows; the state has no such division
            assert float((got[at:at + n].double() - want).norm() / want.norm()) < 1e-2
            assert float((st.gdn[0].rec[s].double() - state[s]).norm() / state[s].norm()) < 2e-3
            pos[s] += n
            at += n
