"""RoPE + append and the causal attention of a prompt (tcgen05) against plain PyTorch, and against the general path."""
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
