"""Top-k over given scores on the one-barrier kernel against the general kernel and a stable sort, and the two-cache gather."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(scores, k, sink, recent):
    """Ascending indices of the k best scores (lowest index wins a tie) and the window, per batch row and head."""
    B, N, KH = scores.shape
    out = {}
    for b in range(B):
        for h in range(KH):
            top = np.argsort(-scores[b, :, h].astype(np.int64), kind="stable")[: min(k, N)]
            out[b, h] = np.union1d(np.union1d(top, np.arange(min(sink, N))), np.arange(max(0, N - recent), N))
    return out


# batch rows whose scores do not start on a 16-byte boundary, chunks that end inside a group of eight scores, one head and 32, a
# single chunk (general kernel), heads that are no power of two (general kernel), windows, ties everywhere, k = 0 and k = N
@pytest.mark.parametrize("B,N,KH,max_score,k,sink,recent", [
    (1, 4097, 8, 512, 400, 0, 0), (3, 5003, 1, 128, 500, 4, 64), (8, 9001, 4, 896, 181, 0, 0), (2, 3333, 2, 256, 3333, 0, 0),
    (2, 2049, 32, 128, 0, 4, 60), (1, 20011, 16, 256, 2000, 0, 90), (1, 100, 8, 512, 10, 0, 0), (2, 6001, 6, 384, 77, 4, 64), (1, 70000, 8, 3, 9999, 0, 0)])
def test_topk_from_scores(B, N, KH, max_score, k, sink, recent):
    from spotlight_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(N)
    mean = max_score / 2
    s = (mean + max_score ** 0.5 / 2 * torch.randn((B, N, KH), generator=gen, device="cuda")).round().clamp(0, max_score).to(torch.int16)
    ref = _reference(s.cpu().numpy(), k, sink, recent)
    got = {}
    for kernel in (1, 0):
        ops.configure(_lib.SL_OPT_SCAN_KERNEL, kernel)
        try:
            for _ in range(3):                               # the coarse histogram's two buffers take turns
                idx, cnt = ops.topk_from_scores(s, k, max_score, sink, recent)
        finally:
            ops.configure(_lib.SL_OPT_SCAN_KERNEL, 1)
        got[kernel] = idx.cpu().numpy(), cnt.cpu().numpy()
    ops.check_status(torch.device("cuda", 0))
    for idx, cnt in got.values():
        for (b, h), want in ref.items():
            assert cnt[b, h] == len(want)
            np.testing.assert_array_equal(idx[b, h, : cnt[b, h]], want)


# score ranges of one coarse bin of eight scores and the first of two and three, over heads that share a warp's bins
@pytest.mark.parametrize("KH", [1, 2, 8, 32])
@pytest.mark.parametrize("max_score", [0, 1, 2, 3, 4, 5, 6, 7, 8, 15, 16])
def test_topk_from_scores_of_a_small_range(KH, max_score):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(100 * max_score + KH)
    s = torch.randint(0, max_score + 1, (2, 1501, KH), generator=gen, device="cuda", dtype=torch.int32).to(torch.int16)
    s[1] = max_score                                         # every key a tie
    for k, sink, recent in ((150, 0, 0), (700, 4, 60)):
        ref = _reference(s.cpu().numpy(), k, sink, recent)
        for _ in range(2):
            idx, cnt = (x.cpu().numpy() for x in ops.topk_from_scores(s, k, max_score, sink, recent))
            for (b, h), want in ref.items():
                assert cnt[b, h] == len(want)
                np.testing.assert_array_equal(idx[b, h, : cnt[b, h]], want)
    ops.check_status(torch.device("cuda", 0))


@pytest.mark.parametrize("values", [(0,), (0, 1), (0, 5), (7, 7)])
def test_topk_and_gather_reads_its_range_from_the_scores(values):
    from spotlight_b200.modifiers.gpu_cache import topk_and_gather
    gen = torch.Generator(device="cuda").manual_seed(len(values))
    pick = torch.randint(0, len(values), (2, 900, 8), generator=gen, device="cuda")
    s = torch.tensor(values, device="cuda", dtype=torch.int16)[pick]
    k, v = (torch.randn((2, 900, 8, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
    at = torch.stack([torch.tensor(np.stack([np.sort(np.argsort(-s[b, :, h].cpu().numpy().astype(np.int64), kind="stable")[:90]) for h in range(8)], 1)) for b in range(2)])
    at = at.cuda()[..., None].expand(-1, -1, -1, 128)
    for got, src in zip(topk_and_gather(s, k, v, 90), (k, v)):
        assert torch.equal(got, src.gather(1, at))


def test_topk_from_scores_clamps_to_the_given_range():
    from spotlight_b200 import ops
    s = torch.randint(0, 100, (2, 3001, 4), device="cuda", dtype=torch.int16)
    s[0, 17, 2], s[1, 2999, 0] = 3000, -5
    c = s.clamp(0, 128)
    for a, b in zip(ops.topk_from_scores(s, 300, 128), ops.topk_from_scores(c, 300, 128)):
        assert torch.equal(a, b)


def test_a_context_whose_scores_spill_leaves_the_workspace_to_a_shorter_one():
    """The workspace of a shape serves every length: scores that do not fit on chip must not land where a shorter context's launch
    keeps its counts."""
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(21)
    B, KH, N, short = 37, 32, 13500, 3000                        # four CTAs per batch row, 3375 keys of 32 heads each: 216 KB of scores
    words = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, generator=gen, device="cuda").to(torch.int32).view(torch.uint32)
    q, codes = words(B, KH, 4), words(B, N, KH, 4)
    ops.workspaces.reset()
    want = [x.clone() for x in ops.scan_topk(q, codes[:, :short], 300)]
    ops.workspaces.reset()
    for _ in range(2):
        ops.scan_topk(q, codes, 1350)
        idx, cnt = ops.scan_topk(q, codes[:, :short], 300)
        assert torch.equal(cnt, want[1])
        valid = torch.arange(idx.shape[2], device="cuda") < cnt[..., None]
        assert torch.equal(idx[valid], want[0][valid])
    ops.check_status(torch.device("cuda", 0))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,N,KH,budget", [(1, 50, 3, 1), (2, 300, 4, 63), (3, 1000, 8, 129), (1, 65, 1, 65)])
def test_gather_kv(B, N, KH, budget, dtype):
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(N)
    k, v = (torch.randn((B, N + 7, KH, 128), generator=gen, device="cuda").to(dtype)[:, :N] for _ in range(2))
    idx = torch.randint(0, N, (B, KH, budget + 2), generator=gen, device="cuda", dtype=torch.int32)
    at = idx[:, :, :budget].long().transpose(1, 2)[..., None].expand(-1, -1, -1, 128)
    for got, src in zip(ops.gather_kv(k, v, idx, budget), (k, v)):
        assert torch.equal(got, src.gather(1, at))
    assert torch.equal(ops.gather_rows(k, idx, budget), k.gather(1, at))
