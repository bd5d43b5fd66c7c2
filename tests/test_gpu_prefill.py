"""RoPE + append and the causal attention of a prompt (tcgen05) against plain PyTorch, and against the general path."""
import subprocess
import sys
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, pos):
    B, T, QH, _ = q.shape
    n, KH = k.shape[1], k.shape[2]
    kk, vv = k.float().repeat_interleave(QH // KH, dim=2), v.float().repeat_interleave(QH // KH, dim=2)
    s = torch.einsum("bthd,bnhd->bhtn", q.float(), kk) / 128 ** 0.5
    later = torch.arange(n, device=q.device)[None] > pos + torch.arange(T, device=q.device)[:, None]
    return torch.einsum("bhtn,bnhd->bthd", s.masked_fill(later, float("-inf")).softmax(-1), vv)


def _caches(B, cap, KH, fused, gen):
    if fused:
        kv = torch.randn((B, cap, KH, 2, 128), generator=gen, device="cuda").bfloat16()
        return kv[:, :, :, 0], kv[:, :, :, 1]
    return tuple(torch.randn((B, cap, KH, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))


# tokens per tile are 128 / group: tile and block edges for groups of 1, 4, 5 and 7 (which leave rows of a tile unused), a
# context before the tokens, several batch rows, and rows of the cache past the context that hold NaN
@pytest.mark.parametrize("B,T,pos,QH,KH,fused", [
    (1, 2, 0, 8, 8, True), (1, 255, 0, 4, 4, False), (2, 129, 127, 8, 2, True), (1, 64, 0, 8, 2, True), (1, 65, 63, 8, 2, False),
    (3, 37, 200, 10, 2, True), (1, 50, 0, 5, 1, True), (1, 36, 1, 14, 2, True), (1, 37, 511, 7, 1, False), (1, 1000, 333, 32, 8, True),
    (1, 3, 5000, 16, 1, True), (1, 700, 0, 2, 2, True)])
def test_prefill_attention(B, T, pos, QH, KH, fused):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(T * 1000 + pos)
    k, v = _caches(B, pos + T + 130, KH, fused, gen)
    k[:, 0] *= 4.0                                    # one key with large scores, so that the running maximum moves
    if pos + T > 300:
        k[:, 290] *= 9.0
    k[:, pos + T:], v[:, pos + T:] = float("nan"), float("nan")
    q = torch.randn((B, T, QH, 128), generator=gen, device="cuda").bfloat16()
    got = ops.prefill_attention(q, k, v, pos).float()
    ref = _reference(q, k[:, : pos + T], v[:, : pos + T], pos)
    # p and the result are rounded to bf16 (2^-9 each, the first averaged over the keys): a few parts in a thousand
    assert torch.isfinite(got).all()
    assert (got - ref).norm() <= 5e-3 * ref.norm()
    assert (got - ref).abs().max() <= 2.0 ** -7 * max(1.0, ref.abs().max().item())
    ops.check_status(torch.device("cuda", 0))


# groups that leave much of a tile unused: one token per 128 rows, up to 63 of them without a query head
@pytest.mark.parametrize("B,T,pos,QH,KH", [(1, 5, 130, 71, 1), (1, 3, 0, 128, 1), (2, 40, 300, 65, 1), (1, 2, 127, 200, 2), (1, 33, 0, 43, 1)])
def test_prefill_attention_of_wide_groups(B, T, pos, QH, KH):
    test_prefill_attention(B, T, pos, QH, KH, True)


# what a row may meet besides numbers: rows that see nothing but scores of -inf up to some key (all of it, a whole tile, part of one), a key of
# NaN or +inf scores, infinite values: the same entries are NaN or infinite as in plain softmax, the others within its tolerance
@pytest.mark.parametrize("what", ["-inf first", "-inf tile", "-inf some", "nan key", "+inf key", "inf value", "nan value"])
def test_prefill_attention_of_infinities_and_nan(what):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(17)
    T, pos, QH, KH = 300, 40, 8, 2
    k, v = _caches(1, pos + T, KH, True, gen)
    q = torch.randn((1, T, QH, 128), generator=gen, device="cuda").bfloat16()
    q[..., 0] = 1.0
    inf = float("inf")
    if what == "-inf first":
        k[:, :pos + 1, :, 0] = -inf
    elif what == "-inf tile":
        k[:, :140, :, 0] = -inf
    elif what == "-inf some":
        k[:, 30:260:3, :, 0] = -inf
    elif what in ("nan key", "+inf key"):
        k[:, 200, 1, 0] = float("nan") if what == "nan key" else inf
    else:
        v[:, 150, 0, 5] = inf if what == "inf value" else float("nan")
    got, ref = ops.prefill_attention(q, k, v, pos).float(), _reference(q, k, v, pos)
    if "value" in what:                               # a masked weight is an exact 0, and 0 times that value NaN, only where its tile is visited at all
        seen = torch.arange(T, device="cuda") + pos >= 150
        got, ref = got[:, seen], ref[:, seen]
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got.isinf(), ref.isinf())
    a, b = (x.masked_fill(~ref.isfinite(), 0.0) for x in (got, ref))
    assert (a - b).norm() <= 5e-3 * b.norm()
    assert ref.isfinite().any() and (what == "-inf some" or not ref.isfinite().all())
    ops.check_status(torch.device("cuda", 0))


@pytest.mark.parametrize("B,T,pos,QH,KH,fused", [(1, 2, 0, 8, 8, True), (2, 131, 7, 28, 4, True), (3, 5, 100, 32, 8, False)])
def test_rope_append_is_torchs_operator_sequence(B, T, pos, QH, KH, fused):
    from spotlight_b200 import ops
    from spotlight_b200.modifiers.spotlight_generation import _rope_rows, _rotate
    gen = torch.Generator(device="cuda").manual_seed(T)
    kc, vc = _caches(B, pos + T + 3, KH, fused, gen)
    k0, v0 = kc.clone(), vc.clone()
    q, k, v = (torch.randn((B, T, h, 128), generator=gen, device="cuda").bfloat16() for h in (QH, KH, KH))
    cos, sin = _rope_rows(torch.arange(pos, pos + T, device="cuda"), 500000.0, torch.bfloat16)
    qr = ops.rope_append(q, k, v, cos, sin, pos, kc, vc)
    k0[:, pos:pos + T], v0[:, pos:pos + T] = _rotate(k, cos[None, :, None], sin[None, :, None]), v
    assert torch.equal(qr, _rotate(q, cos[None, :, None], sin[None, :, None]))
    assert torch.equal(kc, k0) and torch.equal(vc, v0)


def test_the_hook_keeps_the_general_path_for_what_autograd_sees():
    from spotlight_b200 import ops
    q = torch.randn((1, 4, 8, 128), device="cuda").bfloat16()
    k, v = (torch.randn((1, 4, 2, 128), device="cuda").bfloat16() for _ in range(2))
    kv = torch.zeros((1, 16, 2, 2, 128), device="cuda", dtype=torch.bfloat16)
    kc, vc = kv[:, :, :, 0], kv[:, :, :, 1]
    assert ops.prefill_covers(q, k, v, kc, vc)
    assert not ops.prefill_covers(q.requires_grad_(True), k, v, kc, vc)
    with torch.no_grad():
        assert ops.prefill_covers(q, k, v, kc, vc)
    q = q.detach()
    assert not ops.prefill_covers(q.float(), k, v, kc, vc)
    assert not ops.prefill_covers(q, k, v, kc.cpu(), vc.cpu())
    with torch.autograd.forward_ad.dual_level():
        assert not ops.prefill_covers(q, k, v, kc, vc)
    two = kv.expand(2, -1, -1, -1, -1)               # batch rows that share memory
    assert not ops.prefill_covers(q.expand(2, -1, -1, -1), k.expand(2, -1, -1, -1), v.expand(2, -1, -1, -1), two[:, :, :, 0], two[:, :, :, 1])


def _dense_layer(qh, kh, q, k, v):
    """A layer that attends to every key, as the hook meets it, with its projections given."""
    return types.SimpleNamespace(config=types.SimpleNamespace(num_attention_heads=qh, num_key_value_heads=kh, hidden_size=qh * 128, rope_theta=10000.0),
                                 draft_kwargs={"enable": True}, is_fix_layer=True, q_proj=lambda h: q, k_proj=lambda h: k, v_proj=lambda h: v, o_proj=lambda o: o)


@torch.no_grad()
@pytest.mark.parametrize("which", ["q", "k", "v"])
def test_a_prompt_takes_projections_that_start_between_16_byte_boundaries(which):
    from spotlight_b200 import ops
    from spotlight_b200.modifiers.spotlight_generation import self_attn_forward
    gen = torch.Generator(device="cuda").manual_seed(11)
    x = {n: torch.randn((1, 70, h * 128), generator=gen, device="cuda").bfloat16() for n, h in (("q", 8), ("k", 2), ("v", 2))}
    want, st0 = self_attn_forward(_dense_layer(8, 2, **x), x["q"])
    x[which] = torch.empty(x[which].numel() + 1, dtype=torch.bfloat16, device="cuda")[1:].view(x[which].shape).copy_(x[which])
    got, st = self_attn_forward(_dense_layer(8, 2, **x), x["q"])
    assert (got.float() - want.float()).norm() <= 5e-3 * want.float().norm()              # the general path's own roundings
    assert torch.equal(st.k[:, :70], st0.k[:, :70]) and torch.equal(st.v[:, :70], st0.v[:, :70])
    strided = torch.empty((1, 70, 9, 128), dtype=torch.bfloat16, device="cuda")[:, :, 1:]   # not contiguous: copied, the copy is aligned
    kc, vc = _caches(1, 80, 2, True, gen)
    assert ops.prefill_covers(strided, *(torch.zeros((1, 70, 2, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2)), kc, vc)


def _hash(kind, heads, gen, dtype=torch.bfloat16):
    from spotlight_b200 import ops
    dims, residue = {"linear": ((128, 128), False), "mlp256": ((128, 256, 128), False), "mlp128": ((128, 128, 128), False),
                     "mlp128_residual": ((128, 128, 128), True)}[kind]
    ws = [(torch.randn((heads, i, o), generator=gen, device="cuda") * 0.5 / i ** 0.5).to(dtype) for i, o in zip(dims[:-1], dims[1:])]
    bs = [None if kind == "linear" else (0.1 * torch.randn((heads, o), generator=gen, device="cuda")).to(dtype) for o in dims[1:]]
    return ops.HashParams(ws, bs, residue)


# tile edges (127 .. 129 rows), one tile in flight only, more tiles than CTAs, several batch rows, both cache layouts,
# a transposed source; kernel 0: the tensor-core kernel moves the rows itself, 1: the copy kernel and the warp-level code build
@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("kind", ["linear", "mlp256", "mlp128", "mlp128_residual"])
@pytest.mark.parametrize("B,T,start,KH,fused", [(1, 127, 0, 8, True), (2, 129, 5, 4, False), (3, 128, 1, 2, True), (1, 5001, 77, 8, True),
                                                (2, 64, 0, 40, True)])
def test_load_rows_moves_rows_and_builds_the_codes_of_hash_encode(B, T, start, KH, fused, kind, kernel):
    from spotlight_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(B * T + KH)
    kc, vc = _caches(B, start + T + 9, KH, fused, gen)
    codes = torch.zeros((B, start + T + 9, KH, 4), dtype=torch.int32, device="cuda").view(torch.uint32)
    k = torch.randn((B, KH, T, 128), generator=gen, device="cuda").bfloat16().transpose(1, 2)       # head-major source
    v = torch.randn((B, T, KH, 128), generator=gen, device="cuda").bfloat16()
    h = _hash(kind, KH, gen)
    k0, v0 = kc.clone(), vc.clone()
    k0[:, start:start + T], v0[:, start:start + T] = k, v
    rows = slice(start, start + T)
    assert ops.load_rows_covers(k, v, kc[:, rows], vc[:, rows])
    ops.configure(_lib.SL_OPT_HASH_KERNEL, kernel)
    try:
        ops.load_rows(k, v, kc[:, rows], vc[:, rows], h, codes[:, rows])
        want = ops.hash_encode(k0[:, rows], h)
    finally:
        ops.configure(_lib.SL_OPT_HASH_KERNEL, 0)
    torch.cuda.synchronize()
    assert torch.equal(kc, k0) and torch.equal(vc, v0)
    got = codes.view(torch.int32)
    assert torch.equal(got[:, rows], want.view(torch.int32))
    assert int(got[:, :start].abs().max() if start else 0) == 0 and int(got[:, start + T:].abs().max()) == 0
    ops.check_status(torch.device("cuda", 0))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_load_rows_other_types(dtype):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(3)
    k, v = (torch.randn((2, 131, 3, 128), generator=gen, device="cuda").to(dtype) for _ in range(2))
    kv = torch.zeros((2, 140, 3, 2, 128), dtype=dtype, device="cuda")
    codes = torch.zeros((2, 140, 3, 4), dtype=torch.int32, device="cuda").view(torch.uint32)
    h = _hash("mlp128", 3, gen, dtype)
    ops.load_rows(k, v, kv[:, 2:133, :, 0], kv[:, 2:133, :, 1], h, codes[:, 2:133])
    assert torch.equal(kv[:, 2:133, :, 0], k) and torch.equal(kv[:, 2:133, :, 1], v) and int((kv[:, 133:] != 0).sum()) == 0
    assert torch.equal(codes[:, 2:133].view(torch.int32), ops.hash_encode(k, h).view(torch.int32))


def test_load_context_keeps_torchs_copy_for_the_rest():
    from spotlight_b200.session import DecodeSession, SessionConfig
    gen = torch.Generator(device="cuda").manual_seed(4)
    h = [_hash("linear", 2, gen)]
    s = DecodeSession(SessionConfig(1, 2, 2, 1, 64), h, h)
    k, v = (torch.randn((1, 20, 2, 128), generator=gen, device="cuda") for _ in range(2))
    s.load_context(0, k.cpu(), v, 3)                                             # a host tensor, and fp32 into a bf16 cache
    assert torch.equal(s.k_cache[0][:, 3:23], k.bfloat16()) and torch.equal(s.v_cache[0][:, 3:23], v.bfloat16())
    s.load_context(0, s.k_cache[0][:, 3:13], s.v_cache[0][:, 3:13], 30)          # a view of the cache itself
    assert torch.equal(s.k_cache[0][:, 30:40], k.bfloat16()[:, :10]) and torch.equal(s.codes[0][:, 30:40].view(torch.int32), s.codes[0][:, 3:13].view(torch.int32))
    s.load_context(0, k[:, :1, :1].bfloat16(), v[:, :1].bfloat16(), 50)          # one head for both
    assert torch.equal(s.k_cache[0][:, 50, 1], s.k_cache[0][:, 50, 0])


@pytest.mark.parametrize("B,T", [(0, 20), (2, 0), (65537, 2)])
def test_load_context_of_nothing_and_of_very_many_batch_rows(B, T):
    from spotlight_b200.session import DecodeSession, SessionConfig
    gen = torch.Generator(device="cuda").manual_seed(12)
    h = [_hash("linear", 1, gen)]
    s = DecodeSession(SessionConfig(B, 1, 1, 1, max(T, 1)), h, h)
    k, v = (torch.randn((B, T, 1, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    s.load_context(0, k, v, 0, codes=False)
    assert torch.equal(s.k_cache[0][:, :T], k) and torch.equal(s.v_cache[0][:, :T], v)


@pytest.mark.parametrize("T,codes,one_call", [(50, False, False), (6655, False, False), (6656, False, True), (50, True, True)])
def test_load_context_leaves_few_rows_without_codes_to_torchs_copies(T, codes, one_call, monkeypatch):
    from spotlight_b200 import ops
    from spotlight_b200.session import DecodeSession, SessionConfig
    gen = torch.Generator(device="cuda").manual_seed(14)
    h = [_hash("linear", 8, gen)]
    s = DecodeSession(SessionConfig(1, 8, 8, 1, T + 7), h, h)
    calls, load_rows = [], ops.load_rows
    monkeypatch.setattr(ops, "load_rows", lambda *a: (calls.append(1), load_rows(*a)))
    k, v = (torch.randn((1, T, 8, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    s.load_context(0, k, v, 3, codes=codes)
    assert bool(calls) == one_call
    assert torch.equal(s.k_cache[0][:, 3:3 + T], k) and torch.equal(s.v_cache[0][:, 3:3 + T], v)


@pytest.mark.parametrize("call", ["hash", "attention", "load"])
def test_the_first_call_of_a_process_may_be_inside_a_capture(call):
    """In a process of its own: the library's first tensor-core call allocates its status word."""
    code = f"""
import torch
from spotlight_b200 import ops
torch.manual_seed(0)
r = lambda *s: torch.randn(s, device="cuda").bfloat16()
h, x, q, kv, codes = ops.HashParams([r(4, 128, 128)]), r(1, 300, 4, 128), r(1, 300, 8, 128), r(1, 300, 4, 2, 128), torch.zeros((1, 300, 4, 4), dtype=torch.int32, device="cuda")
rows = kv[:, :, :, 0], kv[:, :, :, 1]
run = dict(hash=lambda: ops.hash_encode(x, h).view(torch.int32), attention=lambda: ops.prefill_attention(q, *rows, 0),
           load=lambda: (ops.load_rows(x, x, *rows, h, codes), codes)[1])["{call}"]
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    out = run()
g.replay()
got = out.clone()
assert torch.equal(got, run())
ops.check_status()
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("apart", [True, False])
def test_load_rows_covers_a_source_apart_from_the_rows(apart):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(15)
    kc, vc = _caches(2, 100, 4, True, gen)
    src = slice(0, 40) if apart else slice(21, 61)
    one = [x[:1] for x in (kc, vc)]                            # of several batch rows the address ranges cross
    assert ops.load_rows_covers(one[0][:, src], one[1][:, src], one[0][:, 60:100], one[1][:, 60:100]) == apart
    assert not ops.load_rows_covers(kc[:, src], vc[:, src], kc[:, 60:100], vc[:, 60:100])


def test_load_context_fills_codes_held_as_signed_words():
    from spotlight_b200.session import DecodeSession, SessionConfig
    gen = torch.Generator(device="cuda").manual_seed(13)
    h = [_hash("linear", 8, gen)]
    s = DecodeSession(SessionConfig(1, 8, 8, 1, 5000), h, h)
    k, v = (torch.randn((1, 5000, 8, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    s.load_context(0, k, v)
    want = s.codes[0].view(torch.int32).clone()
    s.codes[0] = torch.zeros_like(want)
    s.load_context(0, k, v)
    assert torch.equal(s.codes[0], want)


def test_the_hash_kernels_silu_is_the_accurate_formula_for_every_bf16():
    """Every finite bf16 through the tcgen05 kernel's activation: with an identity first layer, hidden value j of a row is
    silu(x_j); +-identity in the second layer and torch's value (fp32 x / (1 + exp(-x)), rounded once) taken off as the bias
    leave a sign bit exactly where the hidden value is larger (smaller) than that."""
    from spotlight_b200 import _lib, ops
    bits = torch.arange(65536, dtype=torch.int32)
    x = bits.to(torch.int16).view(torch.bfloat16).view(512, 128).cuda()
    x = torch.where(torch.isfinite(x), x, torch.zeros_like(x))
    ref = torch.nn.functional.silu(x)
    rows = x[None, None].expand(1, 64, -1, -1).contiguous()
    eye = torch.eye(128, device="cuda").bfloat16().expand(512, 128, 128)
    ops.configure(_lib.SL_OPT_HASH_KERNEL, 2)
    try:
        for sign in (1, -1):
            codes = ops.hash_encode(rows, ops.HashParams([eye, sign * eye], [None, -sign * ref]))
            assert int(codes.view(torch.int32).ne(0).sum()) == 0, f"sign {sign}"
        codes = ops.hash_encode(rows, ops.HashParams([eye, eye], [None, -ref + 2.0 ** -120]))        # the test does see a difference
        assert int(codes.view(torch.int32).ne(0).sum()) > 0
    finally:
        ops.configure(_lib.SL_OPT_HASH_KERNEL, 0)
