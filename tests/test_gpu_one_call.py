"""The decode step in one library call against the calls it stands for, and the attention without an index list."""
import sys
import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _hash(heads, gen, dtype):
    from spotlight_b200 import ops
    return ops.HashParams([(torch.randn((heads, 128, 128), generator=gen, device="cuda") * 0.05).to(dtype)])


def _session(seed, batch, qh, kh, layers, n, dtype, lru_slots=0, fused=True, mask_out=0.9):
    from spotlight_b200.session import DecodeSession, SessionConfig
    gen = torch.Generator(device="cuda").manual_seed(seed)
    hq, hk = [_hash(qh, gen, dtype) for _ in range(layers)], [_hash(kh, gen, dtype) for _ in range(layers)]
    s = DecodeSession(SessionConfig(batch, qh, kh, layers, n + 8, dtype, mask_out, lru_slots=lru_slots, fused_kv=fused), hq, hk)
    for l in range(layers):
        s.load_context(l, *(torch.randn((batch, n, kh, 128), generator=gen, device="cuda").to(dtype) for _ in range(2)))
    return s, gen


@pytest.mark.parametrize("batch,qh,kh,layers,n,dtype,lru_slots,fused", [
    (1, 8, 8, 1, 700, torch.float32, 0, True), (2, 8, 2, 3, 3000, torch.bfloat16, 0, False), (1, 16, 4, 2, 3000, torch.bfloat16, 800, True),
    (2, 4, 4, 2, 900, torch.float32, 400, True), (1, 8, 8, 2, 900, torch.float16, 0, True)])
def test_step_is_the_layer_steps(batch, qh, kh, layers, n, dtype, lru_slots, fused):
    a, gen = _session(5, batch, qh, kh, layers, n, dtype, lru_slots, fused)
    b, _ = _session(5, batch, qh, kh, layers, n, dtype, lru_slots, fused)
    for t in range(3):
        for x, h in (("q_in", qh), ("k_in", kh), ("v_in", kh)):
            value = torch.randn((layers, batch, h, 128), generator=gen, device="cuda").to(dtype)
            getattr(a, x).copy_(value)
            getattr(b, x).copy_(value)
        for s in (a, b):
            s.set_position(n + t, 10000.0)
        assert a._one_call(n + t)
        a.step(n + t)
        for l in range(layers):
            b.layer_step(l, n + t)
        assert torch.equal(a.out, b.out)
        for l in range(layers):
            assert torch.equal(a.k_cache[l][:, : n + t + 1], b.k_cache[l][:, : n + t + 1])
            assert torch.equal(a.codes[l].view(torch.int32)[:, : n + t + 1], b.codes[l].view(torch.int32)[:, : n + t + 1])
            if lru_slots:
                assert a.lru[l].step == b.lru[l].step == t + 1
                for x in ("tok2slot", "slot2tok", "last_used", "stats", "status"):
                    assert torch.equal(getattr(a.lru[l], x), getattr(b.lru[l], x)), x


def test_step_takes_the_layer_steps_where_one_call_does_not_serve():
    s, _ = _session(6, 1, 4, 4, 2, 300, torch.bfloat16)
    assert s._one_call(300) and not s._one_call(308) and not s._one_call(-1)
    with pytest.raises(AssertionError, match="full"):
        s.step(308)
    s.k_cache[1], s.v_cache[1] = s.k_cache[1].contiguous(), s.v_cache[1].contiguous()      # another geometry than layer 0
    assert not s._one_call(300)
    s.step(300)
    s.layer_step = lambda *a: None                               # a caller's own layer loop
    assert not s._one_call(300)


# buffers a caller exchanged: what the calls of layer_step refuse (or serve with another geometry) is left to them
@pytest.mark.parametrize("what", ["codes", "heads", "batch", "idx", "cnt", "list", "slots", "table", "shape"])
def test_one_call_leaves_exchanged_buffers_to_the_layer_steps(what):
    from spotlight_b200 import ops
    n = 300
    s, _ = _session(10, 2, 4, 4, 1, n, torch.bfloat16, lru_slots=200)
    s.set_position(n, 10000.0)
    assert s._one_call(n)
    if what == "codes":
        s.codes = [s.codes[0][:1].clone()]                         # one batch row for two
    elif what == "heads":
        s.k_cache, s.v_cache = ([x[0][:, :, :2].contiguous()] for x in (s.k_cache, s.v_cache))
    elif what == "batch":
        s.k_cache, s.v_cache = ([x[0][:1].contiguous()] for x in (s.k_cache, s.v_cache))
    elif what == "idx":
        s.idx = s.idx.long()
    elif what == "cnt":
        s.cnt = s.cnt.long()
    elif what == "list":
        s.idx = s.idx[:, :, :0]
    elif what == "slots":
        s.slots = s.slots[:, :, :5].contiguous()
    elif what == "table":
        s.lru = [ops.LruTable(1, 4, n + 8, 200, torch.bfloat16, "cuda", fused=True)]
    elif what == "shape":
        s.codes = [s.codes[0].flatten(2)]
    assert not s._one_call(n)
    if what in ("codes", "idx"):
        with pytest.raises(AssertionError):
            s.step(n)


# what Python's budget rule takes: integers beyond 32 bits ("never prune"), a budget above and below the other term, numbers that
# are no int, a mask_out that leaves more than every key
@pytest.mark.parametrize("mask_out,min_remain", [(0.9, sys.maxsize), (0.9, 2 ** 31), (0.9, 2 ** 32 + 5), (0.9, 20.5), (np.float32(0.9), 20), (1, 33), (0, 20),
                                                 (-0.5, 20), (1.25, 40)])
def test_step_keeps_pythons_budget(mask_out, min_remain):
    n = 700
    a, gen = _session(8, 1, 8, 2, 2, n, torch.bfloat16)
    b, _ = _session(8, 1, 8, 2, 2, n, torch.bfloat16)
    for s in (a, b):
        s.cfg.mask_out, s.cfg.min_remain = mask_out, min_remain
        s.idx = torch.empty((1, 2, n + 8), dtype=torch.int32, device="cuda")
        s.set_position(n, 10000.0)
    for x in ("q_in", "k_in", "v_in"):
        getattr(a, x).copy_(torch.randn(getattr(a, x).shape, generator=gen, device="cuda"))
        getattr(b, x).copy_(getattr(a, x))
    assert a._one_call(n)
    a.step(n)
    for l in range(2):
        b.layer_step(l, n)
    assert torch.equal(a.cnt, b.cnt) and torch.equal(a.out, b.out)
    if min_remain >= 2 ** 31:
        assert a.cnt.tolist() == [[n + 1] * 2]
        b.step_native(n)
        assert b.cnt.tolist() == [[n + 1] * 2] and torch.equal(a.out, b.out)


def _hook_layer(qh, kh, gen, **draft):
    """An attention layer as self_attn_forward meets it, its projections given: (layer, a function that sets q, k and v)."""
    layer = types.SimpleNamespace(config=types.SimpleNamespace(num_attention_heads=qh, num_key_value_heads=kh, hidden_size=qh * 128, rope_theta=10000.0),
                                  draft_kwargs={"enable": True, "mask_out": 0.9, **draft}, is_fix_layer=False, o_proj=lambda o: o)
    hq, hk = _hash(qh, gen, torch.bfloat16), _hash(kh, gen, torch.bfloat16)
    layer._hash_q_params, layer._hash_k_params = lambda: hq, lambda: hk

    def give(q, k, v):
        layer.q_proj, layer.k_proj, layer.v_proj = lambda h: q, lambda h: k, lambda h: v
    return layer, give


@pytest.mark.parametrize("min_remain,mask_out", [(sys.maxsize, 0.9), (2 ** 31, 0.9), (2 ** 32 + 5, 0.9), (20, np.float32(0.9)), (30, 0.98)])
def test_hook_keeps_pythons_budget(min_remain, mask_out):
    from spotlight_b200.modifiers.spotlight_generation import budget, self_attn_forward
    gen = torch.Generator(device="cuda").manual_seed(9)
    layer, give = _hook_layer(8, 2, gen, min_remain=min_remain, mask_out=mask_out, sink=0, recent=0)
    state = None
    for T in (900, 1, 1):
        x = [torch.randn((1, T, h * 128), generator=gen, device="cuda").bfloat16() for h in (8, 2, 2)]
        give(*x)
        with torch.no_grad():
            _, state = self_attn_forward(layer, x[0], state)
    keep = budget(902, mask_out, min_remain)
    assert state.last_cnt.tolist() == [[keep] * 2] and (min_remain < 2 ** 31 or keep == 902)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("B,n,QH,KH", [(1, 1, 8, 8), (1, 16, 8, 2), (2, 17, 4, 4), (1, 1000, 32, 8), (3, 4097, 10, 2), (1, 20001, 7, 1), (2, 500, 4, 1)])
def test_dense_attention_is_the_attention_over_a_list_of_all_keys(B, n, QH, KH, dtype):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(n)
    q = torch.randn((B, QH, 128), generator=gen, device="cuda").to(dtype)
    kv = torch.randn((B, n + 5, KH, 2, 128), generator=gen, device="cuda").to(dtype)
    idx = torch.arange(n, dtype=torch.int32, device="cuda").expand(B, KH, n).contiguous()
    cnt = torch.full((B, KH), n, dtype=torch.int32, device="cuda")
    got = ops.dense_attn_decode(q, kv[:, :, :, 0], kv[:, :, :, 1], n)
    assert torch.equal(got, ops.sparse_attn_decode(q, kv[:, :, :, 0], kv[:, :, :, 1], idx, cnt))


def test_the_hooks_state_names_the_keys_of_a_dense_layer_when_asked():
    from spotlight_b200.modifiers.spotlight_generation import LayerState
    st = LayerState(2, 3, 20, torch.bfloat16, "cuda")
    assert st.last_idx is None and st.last_cnt is None
    st._last = 7
    assert torch.equal(st.last_idx, torch.arange(7, dtype=torch.int32, device="cuda").expand(2, 3, 7)) and st.last_cnt.tolist() == [[7] * 3] * 2
    st.last_cnt = None
    assert st.last_cnt is None and st.last_idx.shape == (2, 3, 7)


@pytest.mark.parametrize("dtype,lru_slots", [(torch.bfloat16, 100), (torch.float32, 100), (torch.bfloat16, 2100)])
def test_an_overfull_lru_table_raises_its_status_and_the_attention_stays_in_bounds(dtype, lru_slots):
    """More attended keys than slots: the update gives out none, and the list it leaves is one the attention can read. In bf16
    (the attention fetches what is missing itself) the step's output is the one without the table."""
    from spotlight_b200 import ops
    n = 20 * lru_slots // 9                                       # half of it attended: 1.1 times the slots, in one CTA and in several
    s, gen = _session(7, 1, 4, 4, 2, n, dtype, lru_slots=lru_slots, mask_out=0.5)
    for x in ("q_in", "k_in", "v_in"):
        getattr(s, x).copy_(torch.randn(getattr(s, x).shape, generator=gen, device="cuda"))
    s.set_position(n, 10000.0)
    s.slots.fill_(2 ** 30)                                        # an entry the update does not write would show, and be read, as this
    s.step(n)
    torch.cuda.synchronize()
    assert [int(t.status) for t in s.lru] == [3, 3]
    assert all(int(t.slot2tok.max()) == -1 and int(t.tok2slot.max()) == -1 and not t.k.any() and not t.v.any() for t in s.lru)
    left = s.slots[torch.arange(s.slots.shape[2], device="cuda") < s.cnt[..., None]]
    assert bool((left == (0 if dtype == torch.float32 else -2 ** 31)).all())       # any slot, or a miss without one
    ops.check_status(torch.device("cuda", 0))
    out = s.out.clone()
    s.use_lru = False
    s.step(n)
    if dtype == torch.bfloat16:
        assert torch.equal(s.out, out)


@pytest.mark.parametrize("multi", [1, 0])
def test_one_lru_workspace_serves_lists_of_any_capacity(multi):
    """Long and short lists in turn (several CTAs per pair and one): the table whose workspace stays is the table that gets a new one."""
    from spotlight_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(30)
    B, KH, n = 1, 4, 20000
    k, v = (torch.randn((B, n, KH, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    a, b = (ops.LruTable(B, KH, n, 9000, torch.bfloat16, "cuda") for _ in range(2))
    ops.configure(_lib.SL_OPT_LRU_MULTI_CTA, multi)
    try:
        for keep in (6000, 700, 6000, 3100, 2049, 8192, 40):
            idx = torch.stack([torch.randperm(n, generator=gen, device="cuda")[:keep].sort().values for _ in range(KH)])[None].int()
            cnt = torch.full((B, KH), keep, dtype=torch.int32, device="cuda")
            b.ws = None
            sa, sb = (ops.lru_update(t, idx, cnt, k, v) for t in (a, b))
            assert torch.equal(sa, sb)
            for x in ("k", "v", "tok2slot", "slot2tok", "last_used", "stats", "status"):
                assert torch.equal(getattr(a, x), getattr(b, x)), (keep, x)
            assert torch.equal(a.slot2tok.gather(2, sa.long()), idx)
    finally:
        ops.configure(_lib.SL_OPT_LRU_MULTI_CTA, 1)
