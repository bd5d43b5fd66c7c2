"""The work a user of this library has it do, as cases that can be timed: what each one stands for is said
beside it in ``listed``; ``draw`` gives more of the same ranges. Shapes are the repository's own workloads
(``spotlight_b200.workloads.CONFIGS``: Llama-3-8B, Llama-2-7B, Qwen2.5-7B, Qwen2.5-14B head shapes).

Inputs are made on the GPU from the seed alone: K, V ~ N(0,1) with four outlier key channels and a large
key 0, RoPE applied, a query near none of them in particular, hash parameters of the size a trained
hash has (pre-sign values spread over SiLU's whole range, biases that are not zero)."""
import types

import torch

from spotlight_b200 import ops
from spotlight_b200.kernel import attn_cuda_func, pack_cuda_func
from spotlight_b200.modifiers.gpu_cache import topk_and_gather
from spotlight_b200.modifiers.spotlight_generation import Spotlight
from spotlight_b200.session import DecodeSession, SessionConfig
from spotlight_b200.workloads import apply_rope, budget, rope_tables, torch_dtype

DEV = "cuda"
SINK, RECENT, MIN_REMAIN, THETA = 4, 64, 20, 500000.0
HASHES = {"linear": ((128, 128), False), "mlp256": ((128, 256, 128), False), "mlp128_residual": ((128, 128, 128), True)}
HEADS = ((8, 8), (32, 8), (32, 32), (28, 4), (40, 8))          # query heads, kv heads
DRIFT = 0.25                                                    # new part of the query from token to token


def listed():
    def decode(name, batch, heads, context, layers, hash, mask_out, position="host", dtype="bf16"):
        return {"name": name, "kind": "decode", "batch": batch, "q_heads": heads[0], "kv_heads": heads[1], "context": context,
                "layers": layers, "hash": hash, "mask_out": mask_out, "position": position, "dtype": dtype}

    def lru(name, batch, heads, context, layers, hash, mask_out):
        return {"name": name, "kind": "lru", "batch": batch, "q_heads": heads[0], "kv_heads": heads[1], "context": context,
                "layers": layers, "hash": hash, "mask_out": mask_out, "dtype": "bf16"}

    def load(name, batch, kv_heads, start, tokens, hash):
        return {"name": name, "kind": "load", "batch": batch, "kv_heads": kv_heads, "start": start, "tokens": tokens, "hash": hash,
                "dtype": "bf16"}

    def hook(name, batch, heads, context, tokens, layers, fixed, hash, gqa_mode, mask_out):
        return {"name": name, "kind": "hook", "batch": batch, "q_heads": heads[0], "kv_heads": heads[1], "context": context,
                "tokens": tokens, "layers": layers, "fixed": fixed, "hash": hash, "gqa_mode": gqa_mode, "mask_out": mask_out,
                "dtype": "bf16"}

    return [
        # one layer-step of a small fp32 model, called layer by layer: the smallest call, three launches and the host work before them
        decode("decode_fp32_4k", 1, (8, 8), 4096, 1, "linear", 0.9, "eager", "fp32"),
        # every layer of an 8B model for one token of a generation at 32K: one graph for every token, position on the device
        decode("decode_8b_32k", 1, (32, 8), 32769, 32, "mlp256", 0.9, "device"),
        # the same model at 128K, the workload bench.py reports (one graph for a known position)
        decode("decode_8b_128k", 1, (32, 8), 131072, 32, "mlp256", 0.9),
        # a batch of eight long contexts (Qwen2.5-7B heads), 98 % pruned: short lists, a large code stream
        decode("decode_7b_128k_b8", 8, (28, 4), 131072, 4, "linear", 0.98),
        # a million keys on one GPU (Qwen2.5-14B heads)
        decode("decode_14b_1m", 1, (40, 8), 1048576, 2, "linear", 0.98),
        # four stages, multi-head attention: the attended keys stay resident while the query drifts from token to token
        lru("lru_7b_mha_16k_b8", 8, (32, 32), 16384, 4, "linear", 0.98),
        # four stages at the 128K shape: long lists, a quarter of them new in each token
        lru("lru_8b_128k", 1, (32, 8), 131072, 8, "mlp256", 0.9),
        # a prefill's keys and values into the caches of one layer, with their codes: a whole 128K prompt
        load("load_8b_128k", 1, 8, 0, 131072, "mlp256"),
        # the next chunk of a prompt of odd length, with the hash of the reference's shipped configurations
        load("load_7b_mha_chunk", 1, 32, 8191, 4999, "mlp128_residual"),
        # one token through the attention hook of a model's layers, projections included; the first two layers attend to every key
        hook("hook_decode_32k", 1, (32, 8), 32000, 1, 4, 2, "mlp128_residual", "kv_head", 0.98),
        # a prompt through the same hook
        hook("hook_prefill_4k", 1, (32, 8), 0, 4001, 2, 1, "mlp128_residual", "kv_head", 0.98),
        # the reference's kernel entry points one by one: pack, scores, top-k and gather of the selected rows
        {"name": "kernels_7b_128k_b8", "kind": "kernels", "batch": 8, "q_heads": 28, "kv_heads": 4, "context": 131072,
         "mask_out": 0.98, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "lru", "load", "hook", "kernels"))
    qh, kh = rng.choice(HEADS)
    hash = rng.choice(tuple(HASHES))
    mask_out = rng.choice((0.9, 0.95, 0.98))
    batch = rng.choice((1, 1, 2, 3, 4, 8))
    if kind == "load":
        tokens = min(_log(rng, 100, 131072), 8 * 131072 // (batch * kh))
        return {"kind": kind, "batch": batch, "kv_heads": kh, "start": rng.choice((0, rng.randint(1, 4095))), "tokens": tokens,
                "hash": hash, "dtype": "bf16"}
    if kind == "hook":
        tokens = rng.choice((1, 1, _log(rng, 64, 4096)))
        context = rng.choice((0, rng.randint(1, 512))) if tokens > 1 else _log(rng, 500, 32768)
        layers = rng.choice((1, 2))
        return {"kind": kind, "batch": 1 if tokens > 1024 else min(batch, 4), "q_heads": qh, "kv_heads": kh, "context": context,
                "tokens": tokens, "layers": layers, "fixed": rng.randint(0, layers), "hash": hash,
                "gqa_mode": rng.choice(("kv_head", "query_head")), "mask_out": mask_out, "dtype": "bf16"}
    rows = {"decode": 16 * 1048576, "lru": 4 * 1048576, "kernels": 4 * 1048576}[kind]      # keys x kv heads over the batch
    context = max(1000, min(_log(rng, 1000, 1048576 if kind == "decode" else 131072), rows // (batch * kh)))
    case = {"kind": kind, "batch": batch, "q_heads": qh, "kv_heads": kh, "context": context, "mask_out": mask_out, "dtype": "bf16"}
    if kind == "kernels":
        return case
    case["hash"] = hash
    case["layers"] = max(1, min(rng.randint(1, 8), 2 * rows // (batch * kh * context)))
    if kind == "decode":
        case["position"] = rng.choice(("host", "device", "eager"))
        if 32 * 1048576 // 5 < batch * kh * context:            # the one-graph form is for shapes whose scores stay on chip
            case["position"] = "host"
        if context <= 16384 and rng.random() < 0.25:
            case["dtype"] = "fp32"
    return case


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(shape, gen, dtype):
    return torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32).to(dtype)


def _keys(batch, lo, hi, kv_heads, gen, channels, dtype):
    """Post-RoPE keys of positions [lo, hi)."""
    k = torch.randn((batch, hi - lo, kv_heads, 128), generator=gen, device=DEV)
    k[..., channels] *= 8.0
    if lo == 0:
        k[:, 0] *= 4.0
    cos, sin = rope_tables(torch.arange(lo, hi, device=DEV).cpu(), THETA)
    return apply_rope(k, cos.to(DEV)[None, :, None, :], sin.to(DEV)[None, :, None, :]).to(dtype)


def _hash(kind, heads, gen, dtype):
    dims, residue = HASHES[kind]
    ws = [_randn((heads, i, o), gen, torch.float32) * (0.5 / i ** 0.5) for i, o in zip(dims[:-1], dims[1:])]
    bs = [None if kind == "linear" else (0.1 * _randn((heads, o), gen, torch.float32)).to(dtype) for o in dims[1:]]
    return ops.HashParams([w.to(dtype) for w in ws], bs, residue)


def _session(case, seed, extra, lru_slots=0):
    dtype, gen = torch_dtype(case["dtype"]), _gen(seed)
    B, QH, KH, L, n = case["batch"], case["q_heads"], case["kv_heads"], case["layers"], case["context"]
    hq = [_hash(case["hash"], QH, gen, dtype) for _ in range(L)]
    hk = hq if QH == KH else [_hash(case["hash"], KH, gen, dtype) for _ in range(L)]
    s = DecodeSession(SessionConfig(B, QH, KH, L, n + extra, dtype, case["mask_out"], MIN_REMAIN, SINK, RECENT, lru_slots=lru_slots),
                      hq, hk, DEV)
    channels = torch.randperm(128, generator=gen, device=DEV)[:4]
    step = max(1, (1 << 22) // (B * KH * 8))
    for layer in range(L):
        for lo in range(0, n - 1, step):
            hi = min(n - 1, lo + step)
            s.load_context(layer, _keys(B, lo, hi, KH, gen, channels, dtype), _randn((B, hi - lo, KH, 128), gen, dtype), lo)
    s.set_position(n - 1, THETA)
    token = {x: _randn((L, B, h, 128), gen, dtype) for x, h in (("q", QH), ("k", KH), ("v", KH))}
    return s, token, gen


# ------------------------------------------------------------------------------------------ the five kinds
def _prepare_decode(case, seed):
    s, token, _ = _session(case, seed, 16)
    pos, graph = case["context"] - 1, None
    if case["position"] == "host":
        graph = s.capture(pos)
    elif case["position"] == "device":
        s.set_position_table(0, s.cfg.capacity, THETA)
        s.pos_dev.fill_(pos)
        graph = s.capture_dev()
    return {"case": case, "s": s, "token": token, "graph": graph, "pos": pos}


def _run_decode(st):
    """One token: its q / k / v into the session, every layer's hash, append, selection and attention."""
    s, pos = st["s"], st["pos"]
    s.q_in.copy_(st["token"]["q"])
    s.k_in.copy_(st["token"]["k"])
    s.v_in.copy_(st["token"]["v"])
    if st["graph"] is None:
        s.step(pos)
    else:
        if st["case"]["position"] == "device":
            s.pos_dev.fill_(pos)
        st["graph"].replay()
    last = s.cfg.layers - 1
    return [s.out, s.codes[last][:, pos].view(torch.int32), s.k_cache[last][:, pos], s.v_cache[last][:, pos]]


def _prepare_lru(case, seed):
    keep = budget(case["context"], case["mask_out"], MIN_REMAIN) + SINK + RECENT
    s, token, gen = _session(case, seed, 16, lru_slots=2 * keep)
    queries = [(token["q"].float() + DRIFT * _randn(token["q"].shape, gen, torch.float32)).to(token["q"].dtype) for _ in range(8)]
    return {"case": case, "s": s, "token": token, "queries": queries, "at": 0, "pos": case["context"] - 1}


def _run_lru(st):
    """One token of a drifting query through all four stages, layer by layer. Which slot a key has is the table's own
    business; that the resident rows are the right ones shows in the outputs of the tokens that follow."""
    s = st["s"]
    s.q_in.copy_(st["queries"][st["at"] % len(st["queries"])])
    s.k_in.copy_(st["token"]["k"])
    s.v_in.copy_(st["token"]["v"])
    st["at"] += 1
    s.step(st["pos"])
    last = s.cfg.layers - 1
    return [s.out, s.codes[last][:, st["pos"]].view(torch.int32), s.k_cache[last][:, st["pos"]], s.v_cache[last][:, st["pos"]]]


def _prepare_load(case, seed):
    dtype, gen = torch_dtype(case["dtype"]), _gen(seed)
    B, KH, lo, T = case["batch"], case["kv_heads"], case["start"], case["tokens"]
    h = _hash(case["hash"], KH, gen, dtype)
    s = DecodeSession(SessionConfig(B, KH, KH, 1, lo + T + 1, dtype), [h], [h], DEV)
    channels = torch.randperm(128, generator=gen, device=DEV)[:4]
    return {"case": case, "s": s, "k": _keys(B, lo, lo + T, KH, gen, channels, dtype), "v": _randn((B, T, KH, 128), gen, dtype)}


def _run_load(st):
    """A layer's new keys and values into the caches, and the codes of the keys."""
    s, lo = st["s"], st["case"]["start"]
    hi = lo + st["case"]["tokens"]
    s.load_context(0, st["k"], st["v"], lo)
    return [s.codes[0][:, lo:hi].view(torch.int32), s.k_cache[0][:, lo:hi], s.v_cache[0][:, lo:hi]]


def _attention_model(case, gen, dtype):
    """The attention layers of a Llama-shaped model, as the hook meets them."""
    QH, KH = case["q_heads"], case["kv_heads"]
    hidden = QH * 128

    def linear(i, o):
        m = torch.nn.Linear(i, o, bias=False, device=DEV, dtype=dtype)
        m.weight.data.copy_(_randn((o, i), gen, torch.float32) / i ** 0.5)
        return m

    class Attention(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.q_proj, self.k_proj, self.v_proj = linear(hidden, hidden), linear(hidden, KH * 128), linear(hidden, KH * 128)
            self.o_proj = linear(hidden, hidden)

    class Layer(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.self_attn = Attention()

    model = torch.nn.Module()
    model.config = types.SimpleNamespace(num_attention_heads=QH, num_key_value_heads=KH, hidden_size=hidden, rope_theta=THETA)
    model.model = torch.nn.Module()
    model.model.layers = torch.nn.ModuleList(Layer() for _ in range(case["layers"]))
    return model.requires_grad_(False)


def _prepare_hook(case, seed):
    dtype, gen = torch_dtype(case["dtype"]), _gen(seed)
    dims, residue = HASHES[case["hash"]]
    kw = {"enable": True, "fix_layers": list(range(case["fixed"])), "mask_out": case["mask_out"], "min_remain": MIN_REMAIN,
          "num_mlp_layers": len(dims) - 1, "mlp_dims": list(dims), "mlp_residue": residue, "gqa_mode": case["gqa_mode"],
          "max_seq_len": case["context"] + case["tokens"] + 16}
    model = Spotlight(_attention_model(case, gen, dtype), config={"draft_kwargs": kw},
                      hash_kind="linear" if case["hash"] == "linear" else "mlp").requires_grad_(False)
    for p in model.ft_params():
        is_bias = p.dim() == 4 and p.shape[2] == 1
        p.data.copy_(_randn(p.shape, gen, torch.float32) * (0.1 if is_bias else 0.5 / p.shape[2] ** 0.5))
    caches, attns = [None] * case["layers"], [l.self_attn for l in model.model.layers]
    context, new = _hidden_states(case, seed, dtype)
    with torch.no_grad():
        for h in context:
            for i, attn in enumerate(attns):
                caches[i] = attn(h, caches[i])[1]
    return {"case": case, "model": model, "attns": attns, "caches": caches, "h": new,
            "lengths": [0 if c is None else c.length for c in caches]}


def _hidden_states(case, seed, dtype):
    """The context so far, a chunk at a time, and the new tokens of every layer."""
    gen, B, hidden = _gen(seed + (1 << 32)), case["batch"], case["q_heads"] * 128
    chunks = (min(512, case["context"] - lo) for lo in range(0, case["context"], 512))
    context = [_randn((B, n, hidden), gen, dtype) for n in chunks if n > 1]
    return context, [_randn((B, case["tokens"], hidden), gen, dtype) for _ in range(case["layers"])]


@torch.no_grad()
def _run_hook(st):
    """New tokens (one: a decode step; more: a prompt or its next chunk) through every layer's attention, each layer on
    hidden states of its own (what the MLPs between them make of an output is not this library's)."""
    caches, outs = list(st["caches"]), []
    for i, attn in enumerate(st["attns"]):
        if caches[i] is not None:
            caches[i].length = st["lengths"][i]
        o, caches[i] = attn(st["h"][i], caches[i])
        outs.append(o)
    return outs + [x for c, n in zip(caches, st["lengths"]) for x in (c.k[:, n:c.length], c.v[:, n:c.length])]


def _prepare_kernels(case, seed):
    dtype, gen = torch_dtype(case["dtype"]), _gen(seed)
    B, QH, KH, n = case["batch"], case["q_heads"], case["kv_heads"], case["context"]
    codes = torch.randint(-2 ** 31, 2 ** 31, (B, n, KH, 4), generator=gen, device=DEV, dtype=torch.int64).to(torch.int32).view(torch.uint32)
    return {"case": case, "codes": codes, "q": _randn((B, 1, QH, 128), gen, dtype), "k": _randn((B, n, KH, 128), gen, dtype),
            "v": _randn((B, n, KH, 128), gen, dtype)}


def _run_kernels(st):
    """A layer's selection through the reference's entry points: pack the query, score every key, take the best rows."""
    case = st["case"]
    scores = attn_cuda_func(pack_cuda_func(st["q"]), st["codes"])
    keys, vals = topk_and_gather(scores, st["k"], st["v"], budget(case["context"], case["mask_out"], MIN_REMAIN),
                                 128 * (case["q_heads"] // case["kv_heads"]))
    return [scores, keys, vals]


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    """Where an output depends on which keys a hash picked, or is a code or a score, there is no value in 64 bits: a key
    whose score is the threshold may go either way. What is left is the hook's dense attention (a prompt, and the
    layers that attend to every key) and the rows that go into the caches."""
    if case["kind"] == "load":
        st = _prepare_load(case, seed)
        return [None, st["k"].double(), st["v"].double()]
    if case["kind"] != "hook":
        return None
    dtype, B, T, QH, KH = torch_dtype(case["dtype"]), case["batch"], case["tokens"], case["q_heads"], case["kv_heads"]
    layers = _attention_model(case, _gen(seed), dtype).model.layers
    context, new = _hidden_states(case, seed, dtype)
    n, G, outs, rows = sum(h.shape[1] for h in context), QH // KH, [], []
    angle = torch.arange(n + T, device=DEV, dtype=torch.float64)[:, None] / THETA ** (torch.arange(0, 128, 2, device=DEV, dtype=torch.float64) / 128)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def heads(h, linear, rotate):
        x = (h.double() @ linear.weight.double().T).view(B, h.shape[1], -1, 128)
        if rotate is None:
            return x
        a, b = x[..., :64], x[..., 64:]
        c, s = cos[rotate:rotate + h.shape[1]], sin[rotate:rotate + h.shape[1]]
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1)

    for i, layer in enumerate(layers):
        at = layer.self_attn
        h = torch.cat(context + [new[i]], dim=1)
        k, v = heads(h, at.k_proj, 0), heads(h, at.v_proj, None)
        rows += [k[:, n:], v[:, n:]]
        if T == 1 and i >= case["fixed"]:
            outs.append(None)
            continue
        q, o = heads(new[i], at.q_proj, n), torch.empty((B, T, QH, 128), device=DEV, dtype=torch.float64)
        later = torch.arange(n + T, device=DEV)[None] > n + torch.arange(T, device=DEV)[:, None]
        for b in range(B):
            for j in range(QH):
                s = (q[b, :, j] @ k[b, :, j // G].T / 128 ** 0.5).masked_fill_(later, float("-inf"))
                o[b, :, j] = s.softmax(dim=-1) @ v[b, :, j // G]
        outs.append(o.view(B, T, QH * 128) @ at.o_proj.weight.double().T)
    return outs + rows


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _hash_size(kind):
    dims, _ = HASHES[kind]
    return sum(i * o + o for i, o in zip(dims[:-1], dims[1:]))


def _attended(n, mask_out):
    k = budget(n, mask_out, MIN_REMAIN)
    return min(n, k + round((SINK + RECENT) * (1 - k / n)))


def work(case):
    kind, size = case["kind"], 4 if case["dtype"] == "fp32" else 2
    B, KH = case["batch"], case["kv_heads"]
    if kind == "load":                      # K and V in and out, codes out
        rows = B * case["tokens"] * KH
        return {"bytes": rows * (4 * 128 * size + 16) + KH * _hash_size(case["hash"]) * size, "flops": 2 * rows * _hash_size(case["hash"])}
    QH, n = case["q_heads"], case["context"]
    if kind == "kernels":                   # codes in, scores out and in, the selected K and V rows in and out
        k = budget(n, case["mask_out"], MIN_REMAIN)
        return {"bytes": B * KH * (n * (16 + 2 + 2) + k * 4 * 128 * size) + B * QH * 128 * size, "flops": 0}
    if kind in ("decode", "lru"):           # codes, attended K and V rows, hash weights, the token's q, k, v and outputs
        m, hp = _attended(n, case["mask_out"]), _hash_size(case["hash"])
        layer = B * KH * (n * 16 + m * 2 * 128 * size) + (QH + (KH if QH != KH else 0)) * hp * size + B * (2 * QH + 4 * KH) * 128 * size
        flops = B * QH * m * 4 * 128 + 2 * B * (QH + KH) * hp
        return {"bytes": case["layers"] * layer, "flops": case["layers"] * flops}
    T, hidden, out = case["tokens"], QH * 128, {"bytes": 0, "flops": 0}
    weights = hidden * (2 * hidden + 2 * KH * 128)
    for layer in range(case["layers"]):
        pruned = layer >= case["fixed"]
        heads = QH if case["gqa_mode"] == "query_head" else KH                 # heads of the code cache
        hp = (QH + (KH if heads == KH else 0)) * _hash_size(case["hash"]) if pruned else 0
        out["bytes"] += (weights + hp) * size + 2 * B * T * hidden * size + B * T * KH * 2 * 128 * size
        out["flops"] += 2 * B * T * weights
        if T > 1:                           # causal attention over everything so far, codes of the new keys
            out["bytes"] += B * n * KH * 2 * 128 * size + (B * T * heads * 16 if pruned else 0)
            out["flops"] += B * QH * 4 * 128 * (T * n + T * (T + 1) // 2) + (2 * B * T * heads * _hash_size(case["hash"]) if pruned else 0)
        else:
            m = _attended(n + 1, case["mask_out"]) if pruned else n + 1
            rows = m * (heads if pruned else KH)
            out["bytes"] += B * rows * 2 * 128 * size + (B * (n + 1) * heads * 16 if pruned else 0)
            out["flops"] += B * QH * m * 4 * 128
    return out


def tolerance(case):
    """About four times what was seen on a B200. fp32: one layer against 64 bits, 3.7e-7 (largest difference 8e-7). bf16:
    attention against 64 bits 1.7e-3 (largest 4e-3), with its sums split another way 8e-4 (largest 8e-3), and 3e-3
    (largest 1e-2) after the hook's output projection; a prompt's dense attention by another kernel 8e-4 (largest 1.6e-2, the last bit of a large value). Codes: 1e-6 of the words
    hold another bit when the products of the hash are summed in another order (a sum within rounding of zero)."""
    if case["dtype"] == "fp32":
        return {"rel": 2e-6, "max": 1e-5, "differ": 4e-6}
    return {"rel": 1e-2, "max": 0.04, "differ": 4e-6}
