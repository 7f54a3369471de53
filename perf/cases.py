"""The work that programs on this framework have it do, as cases to time: spiking attention layers in decode and prefill, the LIF
operator, and the two dense designs through their engine, prompts and decode steps.  Shapes are the ones ``bench.py`` and its
workloads run (0.5b: 24 layers of width 896, 14 heads of 64; 7b: 28 heads of 128), data is random.

A case is a dict; ``kind`` says which path it takes:

``spike_decode``   ``layers`` x ``fused_qkv_attention`` over decode rows, one CUDA graph replay, as a decode step holds them.
``spike_prefill``  one ``fused_qkv_attention`` over prompt portions, called eagerly, as an engine's prefill does.
``lif``            ``lif_multistep`` with the final membrane, the operator form.
``prefill``        ``extend`` of new requests + logits of each last token + ``release`` (Manirax or Gotunex).
``decode``         continuations of a batch of contexts: ``restore`` and some ``feed`` steps with given tokens, logits of each."""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from spikeinfer_b200.attention import AttentionMetadata, fused_qkv_attention
from spikeinfer_b200.kernels import lif_multistep
from spikeinfer_b200.modeling_gotunex import GotunexConfig, GotunexModel
from spikeinfer_b200.modeling_manirax import ManiraxConfig, ManiraxModel
from spikeinfer_b200.registry import new_engine

DEV = "cuda"
T = 4        # timesteps of the spiking model
PAGE = 16
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def listed() -> list[dict]:
    return [
        # a few interactive users: short contexts, the step is a chain of launches
        dict(name="spike_decode_8", kind="spike_decode", layers=24, rows=8, low=96, high=224, heads=14, kv_heads=2, dim=64, dtype="bf16"),
        # a full serving batch with contexts of every length (14/2 heads of 64)
        dict(name="spike_decode_64", kind="spike_decode", layers=8, rows=64, low=128, high=4096, heads=14, kv_heads=2, dim=64, dtype="bf16"),
        # one GPU's heads of the 7b shape cut four ways, long contexts
        dict(name="spike_decode_256", kind="spike_decode", layers=1, rows=256, low=1024, high=32768, heads=7, kv_heads=1, dim=128, dtype="bf16"),
        # a group of prompts of one length, from their first token
        dict(name="spike_prefill_16x512", kind="spike_prefill", portions=16, tokens=512, ragged=False, cached=0, heads=14, kv_heads=2, dim=64,
             dtype="bf16"),
        # unequal portions of long prompts behind cached tokens, the 7b shape's heads
        dict(name="spike_prefill_chunks", kind="spike_prefill", portions=3, tokens=1531, ragged=True, cached=700, heads=28, kv_heads=4, dim=128,
             dtype="bf16"),
        # the LIF operator on a prefill batch's feed-forward currents
        dict(name="lif_8192", kind="lif", tokens=8192, width=4864, dtype="bf16"),
        # dense designs: groups of prompts (throughput), a long prompt (time to its first token)
        dict(name="manirax_prefill_16x512", kind="prefill", design="Manirax", shape="0.5b", prompts=16, tokens=512, ragged=False),
        dict(name="manirax_prefill_7b", kind="prefill", design="Manirax", shape="7b4", prompts=1, tokens=4096, ragged=False),
        dict(name="gotunex_prefill_ragged", kind="prefill", design="Gotunex", shape="0.5b", prompts=13, tokens=901, ragged=True),
        # dense designs: a full batch, and one user
        dict(name="manirax_decode_64", kind="decode", design="Manirax", shape="0.5b", rows=64, context=1024, steps=4),
        dict(name="gotunex_decode_64", kind="decode", design="Gotunex", shape="0.5b", rows=64, context=1024, steps=4),
        dict(name="gotunex_decode_1", kind="decode", design="Gotunex", shape="0.5b", rows=1, context=333, steps=4),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("spike_decode", "spike_decode", "spike_prefill", "spike_prefill", "lif", "prefill", "prefill", "decode", "decode"))
    if kind.startswith("spike"):
        heads, kv_heads, dim = rng.choice(((14, 2, 64), (7, 1, 128), (28, 4, 128), (4, 2, 64)))
        common = dict(heads=heads, kv_heads=kv_heads, dim=dim, dtype=rng.choice(("bf16", "bf16", "bf16", "fp16", "fp32")))
        if kind == "spike_decode":
            rows = _log(rng, 1, 256)
            high = _log(rng, 100, 32768 if rows * kv_heads <= 64 else 4096)
            return dict(kind=kind, layers=max(1, min(24, 40000 // (rows * high * kv_heads // 64 + 1))), rows=rows, low=max(1, high // rng.choice((2, 8, 32))), high=high, **common)
        portions = _log(rng, 1, 16)
        tokens = _log(rng, 16, max(17, min(4096, 8192 // portions)))
        return dict(kind=kind, portions=portions, tokens=tokens, ragged=rng.random() < 0.5, cached=rng.choice((0, 0, _log(rng, 16, 2048))), **common)
    if kind == "lif":
        return dict(kind=kind, tokens=_log(rng, 64, 8192), width=rng.choice((896, 1000, 4736, 4864)), dtype=rng.choice(("bf16", "bf16", "fp16", "fp32")))
    design, shape = rng.choice((("Manirax", "0.5b"), ("Manirax", "0.5b"), ("Manirax", "7b4"), ("Gotunex", "0.5b"), ("Gotunex", "0.5b")))
    if kind == "prefill":
        prompts = _log(rng, 1, 16)
        return dict(kind=kind, design=design, shape=shape, prompts=prompts, tokens=_log(rng, 40, min(4096, 8192 // prompts)), ragged=rng.random() < 0.5)
    return dict(kind=kind, design=design, shape=shape, rows=_log(rng, 1, 64), context=_log(rng, 32, 1024), steps=4)


# ---- sizes that follow from a case alone ------------------------------------------------------------------------------------

def _lengths(c: dict) -> list[int]:
    """Decode rows: evenly spread from ``low`` to ``high``.  Portions and prompts: all ``tokens``, or down to a quarter of it."""
    if c["kind"] == "spike_decode":
        n, lo, hi = c["rows"], c["low"], c["high"]
        return [lo + (hi - lo) * i // max(1, n - 1) if n > 1 else hi for i in range(n)]
    n = c["portions"] if c["kind"] == "spike_prefill" else c["prompts"]
    return [max(1, c["tokens"] - (3 * c["tokens"] * i // (4 * n) if c["ragged"] else 0)) for i in range(n)]


def _spike_sizes(c: dict) -> tuple[list[int], list[int]]:
    """``(new tokens, tokens cached before them)`` of every row or portion."""
    if c["kind"] == "spike_decode":
        return [1] * c["rows"], [n - 1 for n in _lengths(c)]
    return _lengths(c), [c["cached"]] * c["portions"]


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


# ---- spiking attention ------------------------------------------------------------------------------------------------------

def _spike_inputs(c: dict, seed: int) -> dict:
    g = _gen(seed)
    new, before = _spike_sizes(c)
    layers, n = c.get("layers", 1), sum(new)
    hq, hkv, d = c["heads"], c["kv_heads"], c["dim"]
    dtype = DTYPES[c["dtype"]]
    need = [-(-(a + b) // PAGE) for a, b in zip(new, before)]
    blocks = sum(need) + 1
    order = torch.randperm(blocks - 1, generator=g, device=DEV).to(torch.int32)  # pages lie anywhere in the pool
    tables = torch.full((len(need), max(need)), blocks - 1, dtype=torch.int32, device=DEV)
    at = 0
    for i, k in enumerate(need):
        tables[i, :k] = order[at: at + k]
        at += k
    rows = torch.repeat_interleave(torch.arange(len(new), device=DEV), torch.tensor(new, device=DEV))
    positions = torch.cat([torch.arange(b, a + b, device=DEV) for a, b in zip(new, before)])
    slots = tables[rows, positions // PAGE].to(torch.int64) * PAGE + positions % PAGE
    shape = (layers, T, hkv, blocks * PAGE, d // 32)
    word = lambda: torch.randint(-2 ** 31, 2 ** 31, shape, generator=g, device=DEV, dtype=torch.int32)
    pool = lambda: word() & word() & (word() | word())  # spikes at about 19 %
    k, v = pool(), pool()
    x = torch.randn((layers, T, n, (hq + 2 * hkv) * d), generator=g, device=DEV).to(dtype)
    lif = lambda: (0.8 + 0.15 * torch.rand(d, generator=g, device=DEV), 1.3 + 0.5 * torch.rand(d, generator=g, device=DEV))
    angle = positions[:, None].to(torch.float32) / 1e6 ** (torch.arange(0, d, 2, device=DEV).to(torch.float32) / d)[None, :]
    angle = torch.cat((angle, angle), dim=-1)
    return dict(tables=tables, lens=torch.tensor([a + b for a, b in zip(new, before)], dtype=torch.int32, device=DEV), slots=slots, k=k, v=v, x=x,
                lif=(lif(), lif(), lif()), rope=(angle.cos().to(dtype), angle.sin().to(dtype)), need=need, new=new, before=before)


def _spike_layer(c: dict, s: dict, i: int, meta: AttentionMetadata) -> torch.Tensor:
    return fused_qkv_attention(s["x"][i], *s["lif"], s["k"][i], s["v"][i], meta, c["heads"], c["kv_heads"], c["dim"], rope=s["rope"])


def _prepare_spike(c: dict, seed: int) -> dict:
    s = _spike_inputs(c, seed)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    if c["kind"] == "spike_prefill":
        starts = [sum(s["new"][:i]) for i in range(len(s["new"]))]
        s["meta"] = AttentionMetadata(slot_mapping=s["slots"], block_size=PAGE, prefill_query_starts=starts, prefill_query_lens=s["new"],
                                      prefill_context_lens=s["before"], prefill_block_tables=[t[:k] for t, k in zip(s["tables"], s["need"])],
                                      status=status)
        return s
    meta = AttentionMetadata(slot_mapping=s["slots"], block_size=PAGE, num_decode_tokens=c["rows"], block_tables=s["tables"], seq_lens=s["lens"],
                             status=status, tables_settled=True)
    step = lambda: [_spike_layer(c, s, i, meta) for i in range(c["layers"])]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    s["graph"] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(s["graph"]):
        s["context"] = step()
    s["meta"] = meta
    return s


def _run_spike(c: dict, s: dict) -> dict:
    if c["kind"] == "spike_prefill":
        return dict(context=[_spike_layer(c, s, 0, s["meta"])], keys=s["k"], values=s["v"])
    s["graph"].replay()
    return dict(context=s["context"], keys=s["k"], values=s["v"])


def _lif_plain(x: torch.Tensor, beta: torch.Tensor, threshold: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """The recurrence is defined in 32-bit operations, each rounded on its own: a spike is a comparison of their result."""
    u = torch.zeros(x.shape[1:], dtype=torch.float32, device=x.device)
    spikes = torch.empty(x.shape, dtype=torch.bool, device=x.device)
    for t in range(x.shape[0]):
        reset = (u - threshold > 0).to(torch.float32) * threshold
        u = beta * u
        u = u + x[t].to(torch.float32)
        u = u - reset
        spikes[t] = u - threshold > 0
    return spikes, u


def _exact_spike(c: dict, seed: int) -> dict:
    s = _spike_inputs(c, seed)
    hq, hkv, d = c["heads"], c["kv_heads"], c["dim"]
    cos, sin = (r[None, :, None, :] for r in s["rope"])
    bits = torch.arange(32, device=DEV)
    unpack = lambda w: ((w[..., None] >> bits) & 1).flatten(-2).to(torch.float64)
    out = []
    for i in range(c.get("layers", 1)):
        q, k, v = s["x"][i].unflatten(-1, (hq + 2 * hkv, d)).split((hq, hkv, hkv), dim=2)
        turn = lambda x: x * cos + torch.cat((-x[..., d // 2:], x[..., : d // 2]), dim=-1) * sin  # rounded to the model dtype as it goes
        q, k, v = (_lif_plain(x, *p)[0].to(torch.float64) for x, p in zip((turn(q), turn(k), v), s["lif"]))
        context = torch.empty(q.shape, dtype=torch.float64, device=DEV)
        at = 0
        for r, (n, before) in enumerate(zip(s["new"], s["before"])):
            pos = torch.arange(before, device=DEV)
            old = s["tables"][r, pos // PAGE].to(torch.int64) * PAGE + pos % PAGE
            whole = lambda pool, now: torch.cat((unpack(pool[i][:, :, old]), now[:, at: at + n].transpose(1, 2)), dim=2)
            keys, values = whole(s["k"], k), whole(s["v"], v)
            hidden = torch.ones(n, before + n, dtype=torch.bool, device=DEV).triu(before + 1)
            for t in range(T):
                for h in range(hkv):
                    mine = slice(h * hq // hkv, (h + 1) * hq // hkv)
                    score = (q[t, at: at + n, mine].transpose(0, 1) @ keys[t, h].T) * d ** -0.5
                    context[t, at: at + n, mine] = (score.masked_fill_(hidden, -math.inf).softmax(-1) @ values[t, h]).transpose(0, 1)
            at += n
        out.append(context.flatten(2))
    return dict(context=out, keys=None, values=None)


def _work_spike(c: dict) -> dict:
    new, before = _spike_sizes(c)
    layers, n, hq, hkv, d = c.get("layers", 1), sum(new), c["heads"], c["kv_heads"], c["dim"]
    size = 4 if c["dtype"] == "fp32" else 2
    bits = T * d // 8
    cached, pairs = sum(before), sum(a * b + a * (a + 1) // 2 for a, b in zip(new, before))
    pages = sum(-(-(a + b) // PAGE) for a, b in zip(new, before))
    nbytes = n * T * d * (2 * hq + 2 * hkv) * size + 2 * hkv * bits * (cached + n) + 4 * pages + n * (8 + 2 * d * size)
    return dict(bytes=layers * nbytes, flops=layers * 4 * T * hq * d * pairs)


# ---- LIF --------------------------------------------------------------------------------------------------------------------

def _prepare_lif(c: dict, seed: int) -> dict:
    g = _gen(seed)
    x = torch.randn((T, c["tokens"], c["width"]), generator=g, device=DEV).to(DTYPES[c["dtype"]])
    return dict(x=x, beta=0.8 + 0.15 * torch.rand(c["width"], generator=g, device=DEV), threshold=1.6 + 0.6 * torch.rand(c["width"], generator=g, device=DEV))


def _run_lif(s: dict) -> dict:
    spikes, membrane = lif_multistep(s["x"], s["beta"], s["threshold"], return_membrane=True)
    return dict(spikes=spikes, membrane=membrane)


# ---- dense designs through the engine ---------------------------------------------------------------------------------------

def _config(design: str, shape: str) -> dict:
    layers, width, heads, kv_heads, d, ff, vocab = {"0.5b": (24, 896, 14, 2, 64, 4864, 151936), "7b4": (4, 3584, 28, 4, 128, 18944, 32768)}[shape]
    common = dict(architecture=design, vocab=vocab, width=width, norm=dict(eps=1e-5))
    if design == "Manirax":
        left = dict(heads=heads, kv_heads=kv_heads, dim=d, vdim=d, scale=d ** -0.5, rot=dict(dims=d, base=1e6))
        right = dict(heads=heads, dim=d, vdim=d, decay=[1 - 2.0 ** -(1 + 8 * i / heads) for i in range(heads)])
        layer = dict(type="parallel", mixer=dict(left=left, right=right, left_scale=1.0, right_scale=1.0), mlp=dict(kind="dense", ff=ff))
        return dict(common, postln_alpha=(2 * layers) ** 0.25, layers=[layer] * layers)
    rot_dim, q_rank, kv_rank = (32, 384, 256) if shape == "0.5b" else (64, 1536, 512)
    out, owner = [], None
    for i in range(layers):
        mlp = dict(kind="moe", router=dict(experts=16, top=2), expert=dict(ff=ff // 4)) if i else dict(kind="dense", ff=ff)
        if i % 2 == 0:
            out.append(dict(type="channel_delta", mixer=dict(heads=heads, kv_heads=heads, dim=d, vdim=d, conv=4), mlp=mlp))
            continue
        mixer = dict(heads=heads, dim=d, rot_dim=rot_dim, vdim=d, q_rank=q_rank, kv_rank=kv_rank, scale=(d + rot_dim) ** -0.5,
                     rot=dict(base=1e6, dims=rot_dim))
        if owner is None:
            owner = i
        else:
            mixer["kv_from"], owner = owner, None
        out.append(dict(type="latent_attention", mixer=mixer, mlp=mlp))
    return dict(common, embedding=dict(scale=width ** 0.5), layers=out)


def _weights(cfg: dict, seed: int) -> dict:
    """Random weights under the checkpoint's names, scaled so that activations stay near one."""
    g = _gen(seed)
    mat = lambda o, i, s=1.0: (torch.randn((o, i), generator=g, device=DEV) * (s * i ** -0.5)).to(torch.bfloat16)
    vec = lambda n, lo=0.6, hi=1.4: (lo + (hi - lo) * torch.rand(n, generator=g, device=DEV)).to(torch.bfloat16)
    width, vocab = cfg["width"], cfg["vocab"]
    manirax = cfg["architecture"] == "Manirax"
    w = {"embed": mat(vocab, width, 1.0 if manirax else width ** 0.5 / cfg["embedding"]["scale"]), "final.norm": vec(width)}
    if not manirax:
        w["head"] = mat(vocab, width)
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        w[p + "norm1"], w[p + "norm2"] = vec(width), vec(width)
        if manirax:
            L, R = m["left"], m["right"]
            w[p + "shift"] = vec(width, 0.0, 0.5)
            a = p + "mix.left."
            w[a + "q"], w[a + "k"], w[a + "v"] = mat(L["heads"] * L["dim"], width), mat(L["kv_heads"] * L["dim"], width), mat(L["kv_heads"] * L["vdim"], width)
            w[a + "pb"], w[a + "o"] = vec(L["heads"], -6.0, -4.0), mat(width, L["heads"] * L["vdim"])
            a = p + "mix.right."
            w.update({a + n: mat(R["heads"] * R["dim"], width) for n in "qkvg"})
            w[a + "norm"], w[a + "o"] = vec(R["heads"] * R["vdim"]), mat(width, R["heads"] * R["vdim"])
            w[p + "mlp.act"] = torch.tensor([0.5, 0.3, 0.2, 0.0], device=DEV, dtype=torch.bfloat16)
        elif layer["type"] == "channel_delta":
            a, H, D, V = p + "mix.", m["heads"], m["dim"], m["vdim"]
            for n, rows in (("q", m["kv_heads"] * D), ("k", m["kv_heads"] * D), ("v", H * V)):
                w[a + n], w[a + n + ".conv"] = mat(rows, width), vec(rows * m["conv"], -0.2, 0.8).view(rows, m["conv"])
            w.update({a + "b": mat(H, width), a + "A_log": vec(H, -1.0, 1.0), a + "dt_bias": vec(H * D, -5.0, 0.0), a + "a1": mat(D, width),
                      a + "a2": mat(H * D, D), a + "g1": mat(D, width), a + "g2": mat(H * V, D), a + "norm": vec(V), a + "o": mat(width, H * V)})
        else:
            a, H, D, R, V, K, Q = p + "mix.", *(m[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
            w.update({a + "dq": mat(Q, width), a + "dq.norm": vec(Q), a + "uq": mat(H * (D + R), Q), a + "uk": mat(H * D, K), a + "uv": mat(H * V, K),
                      a + "sink": vec(H, -1.0, 1.0), a + "g": mat(H * V, width), a + "o": mat(width, H * V)})
            if m.get("kv_from") is None:
                w[a + "dkv"], w[a + "dkv.norm"] = mat(K + R, width), vec(K)
        b = p + "mlp."
        if mlp["kind"] == "dense":
            w[b + "up"], w[b + "down"] = mat(mlp["ff"], width), mat(width, mlp["ff"])
        else:
            E, ff = mlp["router"]["experts"], mlp["expert"]["ff"]
            for e in range(E):
                w[f"{b}e{e}.gate"], w[f"{b}e{e}.up"], w[f"{b}e{e}.down"] = mat(ff, width), mat(ff, width), mat(width, ff)
            w[b + "table"] = torch.rand((vocab, E), generator=g, device=DEV).topk(mlp["router"]["top"]).indices.to(torch.int32)
    return w


def _tokens(c: dict, seed: int) -> torch.Tensor:
    """Token ids ``[sequences, longest]``: prompts, or contexts and the tokens fed after them."""
    longest = c["tokens"] if c["kind"] == "prefill" else c["context"] + c["steps"]
    g = torch.Generator().manual_seed(seed)
    return torch.randint(0, _config(c["design"], c["shape"])["vocab"], (c["prompts"] if c["kind"] == "prefill" else c["rows"], longest), generator=g)


@torch.no_grad()
def _prepare_dense(c: dict, seed: int) -> dict:
    cfg, ids = _config(c["design"], c["shape"]), _tokens(c, seed).tolist()
    model = (ManiraxModel(ManiraxConfig.from_dict(cfg), _weights(cfg, seed), device=DEV) if c["design"] == "Manirax" else
             GotunexModel(GotunexConfig.from_dict(cfg), _weights(cfg, seed), device=DEV))
    seqs, longest = len(ids), len(ids[0])
    engine = new_engine(model, num_blocks=seqs * (-(-longest // PAGE) + 1) + 1, block_size=PAGE, max_num_seqs=seqs, max_model_len=longest + PAGE)
    s = dict(model=model, engine=engine)
    if c["kind"] == "prefill":
        s["prompts"] = [p[:n] for p, n in zip(ids, _lengths(c))]
        s["ends"] = torch.tensor(_lengths(c), device=DEV).cumsum(0) - 1
        return s
    rows = [engine.open_request() for _ in ids]
    group = max(1, 8192 // c["context"])
    for lo in range(0, seqs, group):
        engine.extend([(r, ids[r][: c["context"]]) for r in rows[lo: lo + group]])
    s["snapshot"] = engine.snapshot()
    s["fed"] = [{r: ids[r][c["context"] + k] for r in rows} for k in range(c["steps"])]
    _run_decode(c, s)  # captures the step's graphs, as a server does before it takes requests
    return s


def _run_prefill(c: dict, s: dict) -> dict:
    engine, model = s["engine"], s["model"]
    rows = [engine.open_request() for _ in s["prompts"]]
    hidden = engine.extend(list(zip(rows, s["prompts"])))
    logits = model.compute_logits(hidden, s["ends"])
    for r in rows:
        engine.release(r)
    return dict(hidden=hidden, logits=logits, states=list(engine.cache.recurrent_tensors()))


def _run_decode(c: dict, s: dict) -> dict:
    engine = s["engine"]
    engine.restore(s["snapshot"])
    logits = [engine.feed(tokens) for tokens in s["fed"]]
    return dict(logits=logits, states=list(engine.cache.recurrent_tensors()))


def _rms(x: torch.Tensor, eps: float) -> torch.Tensor:
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _layer_norm(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    return F.layer_norm(x, x.shape[-1:], w, None, eps)


def _rotated(x: torch.Tensor, rot: dict) -> torch.Tensor:
    """``x [B, S, H, >= dims]``: channel i turns with channel i + dims / 2."""
    half = rot["dims"] // 2
    angle = torch.arange(x.shape[1], device=DEV, dtype=torch.float64)[:, None] * rot["base"] ** (-2.0 * torch.arange(half, device=DEV, dtype=torch.float64) / rot["dims"])
    co, si = angle.cos()[:, None], angle.sin()[:, None]
    u, v = x[..., :half], x[..., half: 2 * half]
    return torch.cat((u * co - v * si, v * co + u * si, x[..., 2 * half:]), dim=-1)


def _heads(x: torch.Tensor, h: int) -> torch.Tensor:
    return x.unflatten(-1, (h, -1))


def _manirax_exact(ids: torch.Tensor, w: dict, cfg: dict) -> torch.Tensor:
    """Hidden states ``[B, S, width]`` that the output projection reads, in 64 bits."""
    D = lambda k: w[k].to(torch.float64)
    eps, alpha, S = cfg["norm"]["eps"], cfg["postln_alpha"], ids.shape[1]
    x = D("embed")[ids]
    seen = torch.ones(S, S, dtype=torch.bool, device=DEV).tril()
    gap = (torch.arange(S, device=DEV)[:, None] - torch.arange(S, device=DEV)[None, :]).clamp_min(0).to(torch.float64)
    for i, layer in enumerate(cfg["layers"]):
        p, L, R = f"l{i}.", layer["mixer"]["left"], layer["mixer"]["right"]
        h = x + (F.pad(x, (0, 0, 1, 0))[:, :-1] - x) * D(p + "shift")
        a = p + "mix.left."
        q, k, v = (_heads(h @ D(a + n).T, L[hn]) for n, hn in (("q", "heads"), ("k", "kv_heads"), ("v", "kv_heads")))
        q, k = _rms(_rotated(q, L["rot"]), eps), _rms(_rotated(k, L["rot"]), eps)
        bias, rep = D(a + "pb"), L["heads"] // L["kv_heads"]
        left, b = torch.empty_like(q), p + "mix.right."
        rq, rk, rv = (_heads(F.silu(h @ D(b + n).T), R["heads"]) for n in "qkv")
        right = torch.empty_like(rv)
        for j in range(L["heads"]):
            wt = torch.sigmoid(q[:, :, j] @ k[:, :, j // rep].mT * L["scale"] + bias[j]) * seen
            left[:, :, j] = wt @ v[:, :, j // rep]
        for j in range(R["heads"]):
            right[:, :, j] = ((rq[:, :, j] @ rk[:, :, j].mT) * (seen * torch.pow(torch.tensor(R["decay"][j], device=DEV, dtype=torch.float64), gap))) @ rv[:, :, j]
        right = _rms(right.flatten(2), eps) * D(b + "norm") * torch.sigmoid(h @ D(b + "g").T)
        x = _layer_norm(alpha * x + left.flatten(2) @ D(a + "o").T + right @ D(b + "o").T, D(p + "norm1"), eps)
        z = x @ D(p + "mlp.up").T
        c0, c1, c2, c3 = D(p + "mlp.act")
        x = _layer_norm(alpha * x + (c0 * _rms(z, eps) + c1 * _rms(z * z, eps) + c2 * _rms(z ** 3, eps) + c3) @ D(p + "mlp.down").T, D(p + "norm2"), eps)
    return _layer_norm(x, D("final.norm"), eps)


def _gotunex_exact(ids: torch.Tensor, w: dict, cfg: dict) -> torch.Tensor:
    D = lambda k: w[k].to(torch.float64)
    eps, (B, S) = cfg["norm"]["eps"], ids.shape
    x = D("embed")[ids] * cfg["embedding"]["scale"]
    hidden = torch.ones(S, S, dtype=torch.bool, device=DEV).triu(1)
    cached = {}
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        a, H, V = p + "mix.", m["heads"], m["vdim"]
        n = _rms(x, eps)
        h, h2 = n * D(p + "norm1"), n * D(p + "norm2")
        if layer["type"] == "channel_delta":
            taps = m["conv"]
            conv = lambda n: F.silu(sum(F.pad(h @ D(a + n).T, (0, 0, taps - 1, 0))[:, j: j + S] * D(a + n + ".conv")[:, j] for j in range(taps)))
            unit = lambda y: y * torch.rsqrt(y.square().sum(-1, keepdim=True) + 1e-6)
            rep = H // m["kv_heads"]
            q = unit(_heads(conv("q"), m["kv_heads"])).repeat_interleave(rep, 2) * m["dim"] ** -0.5
            k, v = unit(_heads(conv("k"), m["kv_heads"])).repeat_interleave(rep, 2), _heads(conv("v"), H)
            beta = torch.sigmoid(h @ D(a + "b").T)
            raw = _heads(h @ D(a + "a1").T @ D(a + "a2").T + D(a + "dt_bias"), H)
            decay = torch.exp(-torch.exp(D(a + "A_log"))[:, None] * F.softplus(raw))
            state, o = torch.zeros((B, H, m["dim"], V), dtype=torch.float64, device=DEV), torch.empty_like(v)
            for t in range(S):
                state = state * decay[:, t, :, :, None]
                u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ state).squeeze(2))
                state.addcmul_(k[:, t, :, :, None], u[:, :, None, :])
                o[:, t] = (q[:, t, :, None, :] @ state).squeeze(2)
            y = (_rms(o, eps) * D(a + "norm") * torch.sigmoid(_heads(h @ D(a + "g1").T @ D(a + "g2").T, H))).flatten(2)
        else:
            K, R = m["kv_rank"], m["rot_dim"]
            if m.get("kv_from") is None:
                both = h @ D(a + "dkv").T
                cached[i] = _rms(both[..., :K], eps) * D(a + "dkv.norm"), _rotated(both[..., None, K:], m["rot"])[:, :, 0]
            latent, kr = cached[m.get("kv_from", i)]
            q = _heads(_rms(h @ D(a + "dq").T, eps) * D(a + "dq.norm") @ D(a + "uq").T, H)
            qr = _rotated(q[..., m["dim"]:], m["rot"])
            keys, values = _heads(latent @ D(a + "uk").T, H), _heads(latent @ D(a + "uv").T, H)
            o = torch.empty_like(values)
            for j in range(H):
                score = ((q[:, :, j, : m["dim"]] @ keys[:, :, j].mT + qr[:, :, j] @ kr.mT) * m["scale"]).masked_fill_(hidden, -math.inf)
                sink = D(a + "sink")[j].expand(B, S, 1)
                o[:, :, j] = torch.cat((score, sink), dim=-1).softmax(-1)[..., :-1] @ values[:, :, j]
            y = o.flatten(2) * torch.sigmoid(h @ D(a + "g").T)
        y, b = y @ D(a + "o").T, p + "mlp."
        if mlp["kind"] == "dense":
            y += F.gelu(h2 @ D(b + "up").T, approximate="tanh") @ D(b + "down").T
        else:
            chosen, flat, rows = w[b + "table"][ids.flatten()], y.view(-1, y.shape[-1]), h2.flatten(0, 1)
            for e in range(mlp["router"]["experts"]):
                at = (chosen == e).any(1).nonzero()[:, 0]
                z = rows[at]
                flat.index_add_(0, at, F.silu(z @ D(f"{b}e{e}.gate").T) * (z @ D(f"{b}e{e}.up").T) @ D(f"{b}e{e}.down").T / mlp["router"]["top"])
        x = x + y
    return _rms(x, eps) * D("final.norm")


def _exact_dense(c: dict, seed: int) -> dict:
    cfg, ids = _config(c["design"], c["shape"]), _tokens(c, seed).to(DEV)
    w = _weights(cfg, seed)
    forward = _manirax_exact if c["design"] == "Manirax" else _gotunex_exact
    head = w["embed" if c["design"] == "Manirax" else "head"].to(torch.float64)
    S, layers = ids.shape[1], len(cfg["layers"])
    group = max(1, min(len(ids), (4 << 30) // (8 * S * max(S * 3, 16 * cfg["width"]))))
    hidden = torch.cat([forward(ids[lo: lo + group], w, cfg) for lo in range(0, len(ids), group)])
    states = [None] * (layers * 2 if c["design"] == "Manirax" else -(-layers // 2) * 2)
    if c["kind"] == "decode":
        return dict(logits=[hidden[:, c["context"] + k] @ head.T for k in range(c["steps"])], states=states)
    kept = [h[:n] for h, n in zip(hidden, _lengths(c))]
    return dict(hidden=torch.cat(kept), logits=torch.stack([h[-1] for h in kept]) @ head.T, states=states)


def _work_dense(c: dict) -> dict:
    """A pass reads every weight it needs once per step (of sparse experts at most all), and the state and cache it works on."""
    cfg = _config(c["design"], c["shape"])
    if c["kind"] == "prefill":
        new, before, steps = _lengths(c), [0] * c["prompts"], 1
    else:
        new, before, steps = [1] * c["rows"], [c["context"]] * c["rows"], c["steps"]
    n, seqs, width = sum(new), len(new), cfg["width"]
    pairs, keys = sum(a * b + a * (a + 1) // 2 for a, b in zip(new, before)), sum(a + b for a, b in zip(new, before))
    params = nbytes = flops = 0
    reads_state = 2 if c["kind"] == "decode" else 1
    for layer in cfg["layers"]:
        m, mlp = layer["mixer"], layer["mlp"]
        if layer["type"] == "parallel":
            L, R = m["left"], m["right"]
            mats = width * (2 * L["heads"] + 2 * L["kv_heads"]) * L["dim"] + 5 * width * R["heads"] * R["dim"]
            flops += 4 * L["heads"] * L["dim"] * pairs + 4 * R["heads"] * R["dim"] * R["vdim"] * n
            nbytes += 2 * 2 * L["kv_heads"] * L["dim"] * keys + reads_state * 4 * seqs * (R["heads"] * R["dim"] * R["vdim"] + width)
        elif layer["type"] == "channel_delta":
            H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            mats = width * (2 * G * D + 2 * H * V + H + 2 * D) + D * H * (D + V)
            flops += 8 * H * D * V * n
            nbytes += reads_state * 4 * seqs * (H * D * V + m["conv"] * (2 * G * D + H * V))
        else:
            H, D, R, V, K, Q = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank", "q_rank"))
            mats = width * (Q + 2 * H * V) + H * (D + R) * Q + H * (D + V) * K + (width * (K + R) if m.get("kv_from") is None else 0)
            flops += 2 * H * (D + R + V) * pairs
            nbytes += 2 * (K + R) * keys
        if mlp["kind"] == "dense":
            mats += 2 * width * mlp["ff"]
            used = mats
        else:
            per, top, E = 3 * width * mlp["expert"]["ff"], mlp["router"]["top"], mlp["router"]["experts"]
            used, mats = mats + per * top, mats + per * E * (1 - (1 - top / E) ** n)
        flops += 2 * used * n
        params += mats
    logits = seqs * cfg["vocab"]
    flops += 2 * logits * width
    nbytes += 2 * (params + cfg["vocab"] * width) + 4 * logits + 2 * n * width
    return dict(bytes=steps * nbytes, flops=steps * flops)


# ---- what a timer asks for --------------------------------------------------------------------------------------------------

def prepare(case: dict, seed: int) -> dict:
    make = _prepare_lif if case["kind"] == "lif" else _prepare_spike if case["kind"].startswith("spike") else _prepare_dense
    return dict(make(case, seed), case=case)


@torch.no_grad()
def run(state: dict):
    c = state["case"]
    if c["kind"] == "lif":
        return _run_lif(state)
    if c["kind"].startswith("spike"):
        return _run_spike(c, state)
    return _run_prefill(c, state) if c["kind"] == "prefill" else _run_decode(c, state)


@torch.no_grad()
def exact(case: dict, seed: int):
    if case["kind"] == "lif":
        s = _prepare_lif(case, seed)
        spikes, membrane = _lif_plain(s["x"], s["beta"], s["threshold"])
        return dict(spikes=spikes.to(s["x"].dtype), membrane=membrane)
    return _exact_spike(case, seed) if case["kind"].startswith("spike") else _exact_dense(case, seed)


def work(case: dict) -> dict:
    if case["kind"] == "lif":
        size = 4 if case["dtype"] == "fp32" else 2
        cells = case["tokens"] * case["width"]
        return dict(bytes=cells * (2 * T * size + 4), flops=4 * T * cells)
    return _work_spike(case) if case["kind"].startswith("spike") else _work_dense(case)


def tolerance(case: dict):
    if case["kind"] == "lif":
        return "exact"  # every operation of the recurrence is rounded on its own
    if case["kind"].startswith("spike"):
        # one rounding to the output's type, and 16-bit weights of the keys where the output has 16 bits (bf16: 2e-3 from the 64-bit result)
        return {"rel": {"bf16": 8e-3, "fp16": 4e-3, "fp32": 1e-5}[case["dtype"]], "max": {"bf16": 6e-2, "fp16": 3e-2, "fp32": 1e-4}[case["dtype"]]}
    return {"rel": 3e-2, "max": 0.3}  # bf16 operands through all layers: 1e-2 from the 64-bit result
