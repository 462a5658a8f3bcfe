"""Split-KV attention over FP8-E4M3 pages on tensor-core fragments (csrc/kernels/attn_fp8_decode.cu) against the same codes in 64 bits,
and against the kernel that takes the other geometries: ends of runs, pages and splits, head counts, scales far from one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,D,page,positions,spread", [
    (24, 4, 256, 16, [0, 15, 16, 63, 64, 200, 1000], 0.0), (16, 2, 128, 32, [5, 31, 700], 0.0), (8, 8, 256, 64, [300, 2047], 0.0),
    (12, 2, 256, 16, [900, 131], 12.0), (16, 4, 256, 16, list(range(40, 1240, 40)), 0.0)])
def test_fp8_rows(hq, hkv, D, page, positions, spread):
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.ops.specs import AttnSpec
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    dev, n, longest = torch.device("cuda:0"), len(positions), max(positions) + 1
    cfg = tiny_config(num_attention_heads=hq, num_key_value_heads=hkv, head_dim=D)
    st = ModelState(cfg, StateConfig(max_slots=n, max_seq_len=longest, page_tokens=page, kv_dtype="fp8_e4m3"), dev)
    kv = next(x for x in st.kv if x is not None)
    g = torch.Generator(device="cuda").manual_seed(D + n)
    pages, at = [], torch.randperm(st.num_pages - 1, generator=torch.Generator().manual_seed(n)) + 1
    for s, p in enumerate(positions):
        m = p // page + 1
        pages.append(at[:m].to(dev))
        st.block_table[s, :m] = at[:m].to(torch.int32).to(dev)
        at = at[m:]
    kv.k.view(torch.float8_e4m3fn).copy_((torch.randn(kv.k.shape, device="cuda", generator=g) * 100).clamp(-448, 448).to(torch.float8_e4m3fn))
    kv.v.view(torch.float8_e4m3fn).copy_((torch.randn(kv.v.shape, device="cuda", generator=g) * 100).clamp(-448, 448).to(torch.float8_e4m3fn))
    for scale in (kv.k_scale, kv.v_scale):
        scale.copy_(0.01 * torch.exp2(torch.randn(scale.shape, device="cuda", generator=g) * (spread if scale is kv.v_scale else 0.3)))
    q = (torch.randn(n, hq * D, device="cuda", generator=g) * torch.exp2(torch.randn(n, 1, device="cuda", generator=g))).bfloat16()
    b = StepBatch(n, n, dev)
    b.fill([SeqRows(s, p, [0], (0,)) for s, p in enumerate(positions)])
    b.upload()
    spec = AttnSpec(hq, hkv, D, D ** -0.5)
    want = torch.empty(n, hq, D, dtype=torch.float64, device="cuda")
    for s, p in enumerate(positions):
        k, v = ((pool.view(torch.float8_e4m3fn)[pages[s]].double() * scale[pages[s]].double()[..., None]).transpose(1, 2).reshape(-1, hkv, D)[:p + 1]
                for pool, scale in ((kv.k, kv.k_scale), (kv.v, kv.v_scale)))
        for h in range(hq):
            w = torch.softmax(q[s].double().reshape(hq, D)[h] @ k[:, h * hkv // hq].T * D ** -0.5, 0)
            want[s, h] = w @ v[:, h * hkv // hq]
    err = {}
    for name, on in (("fragments", True), ("other", False)):
        ops = CudaOps(cfg, dev, max_seq_len=longest)
        ops.attn_decode_tc = on
        got = ops.attention(q, spec, b, kv, st, longest)
        torch.cuda.synchronize()
        assert int(st.status[0]) == 0
        err[name] = float((got.double().reshape(n, hq, D) - want).norm() / want.norm())
    # one rounding of the output to bf16 (at most 2^-8 of a value) and 32-bit sums; no less exact than the kernel beside it
    assert err["fragments"] < 2.0 ** -8 and err["fragments"] < 1.05 * err["other"] + 1e-6


def test_fp8_rows_beyond_the_position_do_not_count():
    """NaN codes and scales after a row's position, in its own last page, change nothing."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.ops.specs import AttnSpec
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    dev = torch.device("cuda:0")
    cfg = tiny_config(num_attention_heads=12, num_key_value_heads=2, head_dim=256)
    st = ModelState(cfg, StateConfig(max_slots=1, max_seq_len=128, page_tokens=16, kv_dtype="fp8_e4m3"), dev)
    kv = next(x for x in st.kv if x is not None)
    st.block_table[0, :6] = torch.arange(1, 7, dtype=torch.int32, device=dev)
    for pool in (kv.k, kv.v):
        pool.view(torch.float8_e4m3fn).copy_((torch.randn(pool.shape, device="cuda") * 50).to(torch.float8_e4m3fn))
    q = torch.randn(1, 12 * 256, device="cuda").bfloat16()
    b = StepBatch(1, 1, dev)
    b.fill([SeqRows(0, 74, [0], (0,))])
    b.upload()
    ops = CudaOps(cfg, dev, max_seq_len=128)
    first = ops.attention(q, AttnSpec(12, 2, 256, 1 / 16), b, kv, st, 75).clone()
    for pool, scale in ((kv.k, kv.k_scale), (kv.v, kv.v_scale)):
        pool[5, :, 11:] = 0x7f
        scale[5, :, 11:] = float("nan")
    assert torch.equal(first, ops.attention(q, AttnSpec(12, 2, 256, 1 / 16), b, kv, st, 75)) and bool(torch.isfinite(first.float()).all())


@pytest.mark.parametrize("hq,hkv,D,positions,split,scale_q,spread", [
    (24, 4, 256, [500, 1000, 4000], 64, 1.0, 0.0), (16, 4, 256, list(range(64, 4096, 500)), 256, 1.0, 0.0), (16, 2, 128, [100, 3000], 512, 1.0, 0.0),
    (24, 4, 256, [500, 8000], 2048, 6.0, 0.0), (12, 2, 256, list(range(5, 1000, 40)), 64, 1.0, 3.0), (24, 4, 256, [8000], 4096, 0.05, 0.0)])
def test_fp8_partials_are_as_exact_as_those_of_the_other_kernel(hq, hkv, D, positions, split, scale_q, spread, monkeypatch):
    """The partial sums in 32 bits, merged in 64: short and long splits, peaked and flat weights, row scales far apart."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.ops.specs import AttnSpec
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    monkeypatch.setenv("PS_ATTN_SPLIT_TOKENS", str(split))
    dev, n, longest = torch.device("cuda:0"), len(positions), max(positions) + 1
    cfg = tiny_config(num_attention_heads=hq, num_key_value_heads=hkv, head_dim=D)
    st = ModelState(cfg, StateConfig(max_slots=n, max_seq_len=longest, page_tokens=16, kv_dtype="fp8_e4m3"), dev)
    kv = next(x for x in st.kv if x is not None)
    g = torch.Generator(device="cuda").manual_seed(split)
    pages = torch.split(torch.arange(1, 1 + sum(p // 16 + 1 for p in positions), device=dev), [p // 16 + 1 for p in positions])
    for s, at in enumerate(pages):
        st.block_table[s, :len(at)] = at.to(torch.int32)
    for pool, scale in ((kv.k, kv.k_scale), (kv.v, kv.v_scale)):
        x = torch.randn(pool.shape, device="cuda", generator=g) + (0.3 if scale is kv.v_scale else 0.0)
        top = x.abs().amax(-1) / 448
        pool.view(torch.float8_e4m3fn).copy_((x / top[..., None]).to(torch.float8_e4m3fn))
        scale.copy_(top * torch.exp2(torch.randn(top.shape, device="cuda", generator=g) * (spread if scale is kv.v_scale else 0.0)))
    q = (torch.randn(n, hq * D, device="cuda", generator=g) * scale_q).bfloat16()
    b = StepBatch(n, n, dev)
    b.fill([SeqRows(s, p, [0], (0,)) for s, p in enumerate(positions)])
    b.upload()
    want = torch.empty(n, hq, D, dtype=torch.float64, device="cuda")
    for s, p in enumerate(positions):
        k, v = ((pool.view(torch.float8_e4m3fn)[pages[s]].double() * scale[pages[s]].double()[..., None]).transpose(1, 2).reshape(-1, hkv, D)[:p + 1]
                for pool, scale in ((kv.k, kv.k_scale), (kv.v, kv.v_scale)))
        for h in range(hq):
            want[s, h] = torch.softmax(q[s].double().reshape(hq, D)[h] @ k[:, h * hkv // hq].T * D ** -0.5, 0) @ v[:, h * hkv // hq]
    err = []
    for on in (True, False):
        ops = CudaOps(cfg, dev, max_seq_len=longest)
        ops.attn_decode_tc, ops.exact_rows = on, True             # (the split length as it is set)
        ops.attention(q, AttnSpec(hq, hkv, D, D ** -0.5), b, kv, st, longest)
        torch.cuda.synchronize()
        assert int(st.status[0]) == 0 and ops.split_tokens == split
        part = {key: t.double().reshape(n, hq, ops.max_splits, -1) for (name, _), t in ops.ws.items() for key in ("attn_part_acc", "attn_part_ml") if name.startswith(key)}
        got = torch.empty_like(want)
        for s, p in enumerate(positions):
            ml, acc = (part[key][s, :, :p // split + 1] for key in ("attn_part_ml", "attn_part_acc"))
            w = torch.exp(ml[..., 0] - ml[..., 0].amax(1, keepdim=True))
            got[s] = (w[..., None] * acc).sum(1) / (w * ml[..., 1]).sum(1)[:, None]
        err.append(float((got - want).norm() / want.norm()))
    # the same inputs and splits on both sides: 32-bit sums in another order, no less exact (0.2 to 0.95 of the other's error)
    assert err[0] <= err[1]


def test_fp8_rows_with_query_entries_of_very_different_sizes():
    """Small query entries that decide the scores because the keys are zero where the large ones are: 2^-24 to 2^-45 of the largest."""
    from phaseshift_b200.models.qwen35.config import tiny_config
    from phaseshift_b200.ops.cuda_ops import CudaOps
    from phaseshift_b200.ops.specs import AttnSpec
    from phaseshift_b200.runtime.batch import SeqRows, StepBatch
    from phaseshift_b200.runtime.state import ModelState, StateConfig
    dev, hq, hkv, D, last = torch.device("cuda:0"), 8, 2, 256, 200
    cfg = tiny_config(num_attention_heads=hq, num_key_value_heads=hkv, head_dim=D)
    st = ModelState(cfg, StateConfig(max_slots=1, max_seq_len=last + 1, page_tokens=16, kv_dtype="fp8_e4m3"), dev)
    kv = next(x for x in st.kv if x is not None)
    pages = torch.arange(1, 2 + last // 16, device=dev)
    st.block_table[0, :len(pages)] = pages.to(torch.int32)
    g = torch.Generator(device="cuda").manual_seed(3)
    for pool in (kv.k, kv.v):
        x = torch.randn(pool.shape, device="cuda", generator=g) * 50
        if pool is kv.k:
            x[..., ::64] = 0
        pool.view(torch.float8_e4m3fn).copy_(x.to(torch.float8_e4m3fn))
    size = torch.exp2(-torch.tensor([24., 28, 30, 32, 34, 37, 40, 45], device="cuda"))[:, None]
    q = torch.randn(hq, D, device="cuda", generator=g) * size * 2.0 ** 20
    q[:, ::64] = 2.0 ** 20
    # scores of about one for every head of a KV head: its heads' sizes differ, so the keys' scale suits the middle one
    kv.k_scale.fill_(1.0)
    kv.k_scale[:, 0], kv.k_scale[:, 1] = 2.0 ** 6, 2.0 ** 14
    kv.v_scale.fill_(0.01)
    q = q.reshape(1, -1).bfloat16()
    b = StepBatch(1, 1, dev)
    b.fill([SeqRows(0, last, [0], (0,))])
    b.upload()
    k, v = ((pool.view(torch.float8_e4m3fn)[pages].double() * scale[pages].double()[..., None]).transpose(1, 2).reshape(-1, hkv, D)[:last + 1]
            for pool, scale in ((kv.k, kv.k_scale), (kv.v, kv.v_scale)))
    ops = CudaOps(cfg, dev, max_seq_len=last + 1)
    got = ops.attention(q, AttnSpec(hq, hkv, D, D ** -0.5), b, kv, st, last + 1).double().reshape(hq, D)
    assert int(st.status[0]) == 0
    for h in range(hq):
        s = q.double().reshape(hq, D)[h] @ k[:, h * hkv // hq].T * D ** -0.5
        want = torch.softmax(s, 0) @ v[:, h * hkv // hq]
        # the output's rounding to bf16, and scores in 32 bits (2^-24 each for the products, their sums and the scale's factor: 2^-20 of one)
        assert float((got[h] - want).norm() / want.norm()) < 2.0 ** -8 + 2.0 ** -20 * float(s.abs().max()), h
