"""Calls of one shape on several streams: each stream has workspaces of its own, and a graph those of its warm-up."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_workspace_belongs_to_a_stream():
    from spotlight_b200.ops import _Workspaces
    w, dev = _Workspaces(), torch.device("cuda")
    streams = [torch.cuda.Stream() for _ in range(w.MAX_STREAMS + 3)]

    def get(stream, nbytes=1000, shape=(1, 2, 3), **kw):
        with torch.cuda.stream(stream):
            return w.get("x", dev, nbytes, shape, **kw)

    a, b = get(streams[0]), get(streams[1])
    assert a[0].data_ptr() != b[0].data_ptr() and a[1].data_ptr() != b[1].data_ptr()
    assert get(streams[0])[0] is a[0] and get(streams[1])[0] is b[0]
    assert get(streams[0], 500)[0] is a[0] and get(streams[0], shape=(1, 2, 4))[0] is not a[0]
    assert {key[1] for key, _ in w.status_words()} == {torch.device("cuda", 0)} == {key[1] for key, _ in w.status_words("cuda")}
    kept = get(streams[0], keep=True)[0]
    grown = get(streams[0], 5000)[0]                            # the outgrown buffer stays: a graph may replay with it
    assert kept is a[0] and grown.numel() >= 5000 and any(s is a[1] for _, s in w.status_words())
    for s in streams[1:]:
        get(s)
    assert len(w._bufs["x", torch.device("cuda", 0), (1, 2, 3)]) <= w.MAX_STREAMS + 1 and get(streams[0])[0] is grown
    last = get(streams[2])                                      # a capture on a stream without a buffer takes the one used last
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        took = w.get("x", dev, 800, (1, 2, 3))
    assert took[0] is last[0]
    for s in streams[3:]:
        get(s)
    assert get(streams[2])[0] is took[0]
    took[0].fill_(1)
    took[1].fill_(3)
    (bad,) = [key for key, s in w.status_words() if int(s)]
    w.clean(bad)
    assert get(streams[2])[0] is took[0] and not took[0].any() and not took[1].any()       # cleaned where the graph expects it
    w.reset()
    assert not w.status_words()


# few CTAs per call (four to eight), so that the calls of both streams are resident together
def test_two_streams_at_once():
    from spotlight_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    B, N, QH, KH, k = 2, 1000, 8, 4, 100
    streams, inputs, want, got = [torch.cuda.Stream() for _ in range(2)], [], [], [[], []]
    for _ in streams:
        words = lambda *s: torch.randint(-2 ** 31, 2 ** 31, s, generator=gen, device="cuda").to(torch.int32).view(torch.uint32)
        inputs.append((words(B, QH, 4), words(B, N, KH, 4), torch.randint(0, 257, (B, N, KH), generator=gen, device="cuda", dtype=torch.int32).to(torch.int16),
                       *(torch.randn((B, n, h, 128), generator=gen, device="cuda").bfloat16() for n, h in ((1, QH), (N, KH), (N, KH)))))

    def run(q_codes, codes, scores, q, keys, vals):
        idx, cnt = ops.scan_topk(q_codes, codes, k)
        out = ops.sparse_attn_decode(q[:, 0], keys, vals, idx, cnt)
        return idx, cnt, out, *ops.topk_from_scores(scores, k, 256), ops.dense_attn_decode(q[:, 0], keys, vals, N)

    for x in inputs:
        want.append([t.clone() for t in run(*x)])
    torch.cuda.synchronize()
    for _ in range(100):
        for s, x, g in zip(streams, inputs, got):
            with torch.cuda.stream(s):
                g.append(run(*x))
    torch.cuda.synchronize()
    ops.check_status(torch.device("cuda", 0))
    for w, g in zip(want, got):
        cnt = w[1]
        valid = torch.arange(w[0].shape[2], device="cuda") < cnt[..., None]
        for r in g:
            assert torch.equal(r[0][valid], w[0][valid])
            assert all(torch.equal(a, b) for a, b in zip(r[1:], w[1:]))
