"""What the speed of this framework is measured on: decode steps and prompts of three of its model families, as a serving program
runs them on one GPU.

  dense     the grouped-query decoder (``models/dense_gqa.py``), in the sizes of the throughput benchmarks
  falinex   the decoder of retention, lightning and windowed attention layers over an f32 residual (``models/falinex.py``): the
            family that is opened from a checkpoint, with packed steps and recurrent states; same sizes
  mla_moe   the 92B-class latent-attention + routed-expert decoder of the headline benchmark (``models/mla_moe.py``), with 4 of its
            46 equal layers, so that several sets of weights fit one GPU

A pass is one of

  decode    one step of ``rows`` sequences, each with a context of its own (between a quarter of ``context`` and all of it). One
            sequence goes through ``DecodeEngine.step``; more through what the batching engine calls for so many rows: the packed or
            batched executor's ``forward_rows``, or the decoder's captured launch group up to eight rows
  prompt    ``rows`` prompt tokens of one sequence, from the first position: ``DecodeEngine.prefill``, or for falinex
            the packed executor's ``forward_rows`` with ``others`` decode rows of running sequences in the same step

Weights are N(0, 0.02), gains 1 + N(0, 0.02), caches and states hold values of the spread that a run leaves in them. The matrices that
write to a residual without a norm of their own are smaller by sqrt(2 layers), as models are initialised, and embeddings are large beside
what one layer adds (N(0, 1) dense, N(0, 0.2) mla_moe): where every layer is as large as all before it, a single rounding to bf16 grows from
layer to layer. Routers are N(0, 0.05): scores as uneven as trained routers give them, so that a choice between two nearly equal experts
is one between experts of small weight."""
from __future__ import annotations

import math

import torch

from ironpangu_b200.models import dense_gqa, falinex, mla_moe
from ironpangu_b200.models.dense_prefill import DensePrefill
from ironpangu_b200.models.mla_moe_prefill import MlaMoePrefill
from ironpangu_b200.parallel.fabric import Fabric
from ironpangu_b200.runtime.engine import DecodeEngine

BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
STD = 0.02
PAGE = 16
# width, layers, heads, kv heads, head size, feed-forward, vocabulary, window (falinex)
SIZES = {
    "small": (1024, 12, 8, 4, 128, 4096, 32000, 512),
    "2b": (2048, 24, 16, 4, 128, 6144, 151936, 1024),
    "8b": (4096, 16, 32, 8, 128, 16384, 128000, 1024),
}
MLA_LAYERS = 4


def listed():
    return [
        # a small model answering one user: nothing but latency
        dict(name="dense small 1 row", family="dense", size="small", kind="decode", rows=1, context=129),
        # the 2B model, one user with a conversation behind them
        dict(name="dense 2b 1 row", family="dense", size="2b", kind="decode", rows=1, context=2000),
        # a few users at once
        dict(name="dense 2b 8 rows", family="dense", size="2b", kind="decode", rows=8, context=3000),
        # a full server
        dict(name="dense 2b 64 rows", family="dense", size="2b", kind="decode", rows=64, context=4096),
        # an ordinary prompt, of no round length
        dict(name="dense 2b prompt 509", family="dense", size="2b", kind="prompt", rows=509, context=509),
        # a long document
        dict(name="dense 2b prompt 4096", family="dense", size="2b", kind="prompt", rows=4096, context=4096),
        dict(name="falinex 2b 1 row", family="falinex", size="2b", kind="decode", rows=1, context=1500),
        # a server between quiet and full
        dict(name="falinex 2b 27 rows", family="falinex", size="2b", kind="decode", rows=27, context=3000),
        # continuous batching: a prompt's portion beside the decode rows of running sequences
        dict(name="falinex 2b prompt 1500 beside 5", family="falinex", size="2b", kind="prompt", rows=1500, others=5, context=1600),
        # the headline benchmark's step and its prompt
        dict(name="mla_moe 1 row", family="mla_moe", kind="decode", rows=1, context=512, experts="bf16"),
        # the serving configuration: a group of sequences over fp8 experts
        dict(name="mla_moe fp8 experts 8 rows", family="mla_moe", kind="decode", rows=8, context=1024, experts="fp8"),
        dict(name="mla_moe prompt 512", family="mla_moe", kind="prompt", rows=512, context=512, experts="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _seconds(case):
    w = work(case)
    return max(w["bytes"] / 6e12, w["flops"] / 1.2e15)


def draw(rng):
    most = max(_seconds(c) for c in listed())
    while True:
        family = rng.choice(("dense", "dense", "falinex", "mla_moe"))
        kind = rng.choice(("decode", "decode", "prompt"))
        case = dict(family=family, kind=kind)
        if family != "mla_moe":
            case["size"] = rng.choice(("small", "2b", "2b", "8b"))
        if kind == "decode":
            case["rows"] = rng.choice((1, _log(rng, 2, 8 if family == "mla_moe" else 64)))
            case["context"] = _log(rng, 16, 2048 if family == "mla_moe" else 4096)
        else:
            case["rows"] = _log(rng, 16, 512 if family == "mla_moe" else 2048 if family == "falinex" else 4096)
            case["context"] = case["rows"]
            if family == "falinex":
                case["others"] = rng.choice((0, _log(rng, 1, 16)))
                case["context"] = case["rows"] + rng.randrange(1, 200)
        if family == "mla_moe":
            case["experts"] = rng.choice(("bf16", "fp8")) if kind == "decode" and case["rows"] > 1 else "bf16"
        if _seconds(case) <= most:
            return case


# ---------------------------------------------------------------------------------------------------------------------------
# inputs: everything from the seed
# ---------------------------------------------------------------------------------------------------------------------------
def _config(case):
    if case["family"] == "mla_moe":
        c = mla_moe.MlaMoeConfig.flagship()
        c.layers = MLA_LAYERS
        return c
    width, layers, heads, kv, hd, ff, vocab, window = SIZES[case["size"]]
    if case["family"] == "dense":
        return dense_gqa.DenseConfig(layers=layers, hidden=width, heads=heads, kv_heads=kv, head_dim=hd, ffn=ff, vocab=vocab)
    return falinex.FalinexConfig.text2b(layers=layers, width=width, heads=heads, kv_heads=kv, dim=hd, ff=ff, vocab=vocab, window=window)


def _shapes(case, c):
    """Tensor names of the checkpoint or weight dictionary -> shapes."""
    if case["family"] == "dense":
        s = {"embed": (c.vocab, c.hidden), "final_norm": (c.hidden,), "lm_head": (c.vocab, c.hidden)}
        for l in range(c.layers):
            p = f"layers.{l}."
            s.update({p + "attn_norm": (c.hidden,), p + "qkv": ((c.heads + 2 * c.kv_heads) * c.head_dim, c.hidden), p + "o_proj": (c.hidden, c.heads * c.head_dim),
                      p + "ffn_norm": (c.hidden,), p + "gate_up": (2 * c.ffn, c.hidden), p + "down": (c.hidden, c.ffn)})
        return s
    if case["family"] == "mla_moe":
        s = {"embed": (c.vocab, c.hidden), "final_norm": (c.hidden,), "lm_head": (c.vocab, c.hidden)}
        for l in range(c.layers):
            p = f"layers.{l}."
            s.update({p + "attn_norm": (c.hidden,), p + "qkv_a": (c.q_lora + c.kv_lora + c.rope, c.hidden), p + "q_a_norm": (c.q_lora,), p + "kv_a_norm": (c.kv_lora,),
                      p + "q_b": (c.heads * c.qk_dim, c.q_lora), p + "kv_b": (c.heads, c.nope + c.vdim, c.kv_lora), p + "o_proj": (c.hidden, c.heads * c.vdim),
                      p + "ffn_norm": (c.hidden,), p + "router": (c.experts, c.hidden), p + "gate_up": (c.experts, 2 * c.expert_ffn, c.hidden),
                      p + "down": (c.experts, c.hidden, c.expert_ffn), p + "shared_gate_up": (2 * c.shared_ffn, c.hidden), p + "shared_down": (c.hidden, c.shared_ffn)})
        return s
    s = {"embed": (c.vocab, c.width), "final.norm": (c.width,), "head": (c.vocab, c.width)}
    for i, l in enumerate(c.layers):
        p, m = f"l{i}.", l.mixer
        groups = m.heads if m.kind != "attention" else m.kv_heads
        hv = m.heads * m.vdim
        s.update({p + "norm1": (c.width,), p + "mix.q": (m.heads * m.dim, c.width), p + "mix.k": (groups * m.dim, c.width), p + "mix.v": (groups * m.vdim, c.width),
                  p + "mix.g": (hv, c.width), p + "mix.o": (c.width, hv), p + "norm2": (c.width,), p + "mlp.up": (l.ff, c.width), p + "mlp.down": (c.width, l.ff)})
        if m.kind == "lightning":
            s[p + "mix.norm"] = (hv,)
        if m.kind == "attention":
            s.update({p + "mix.q.norm": (m.dim,), p + "mix.k.norm": (m.dim,), p + "mix.sink": (m.heads,)})
    return s


def _weights(case, c, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = {}
    spread = {"embed": {"dense": 1.0, "falinex": 0.1, "mla_moe": 0.2}[case["family"]], "sink": 1.0, "router": 0.05}
    if case["family"] != "falinex":
        depth = c.layers if case["family"] == "dense" else mla_moe.MlaMoeConfig.flagship().layers
        spread.update({n: STD / math.sqrt(2 * depth) for n in ("o_proj", "down", "shared_down")})
    for name, shape in _shapes(case, c).items():
        t = torch.empty(shape, dtype=F32 if name.endswith("router") else BF16, device="cuda")
        t.normal_(0.0, spread.get(name.split(".")[-1], STD), generator=g)
        out[name] = t.add_(1.0) if "norm" in name else t
    return out


def _running(case):
    """Sequences that decode in the pass."""
    return case["rows"] if case["kind"] == "decode" else case.get("others", 0)


def _inputs(case, c, seed):
    """Token ids (host), contexts of the sequences that decode, and what their caches and states hold."""
    g = torch.Generator().manual_seed(seed + 1)
    n, most = _running(case), case["context"]
    tokens = torch.randint(0, c.vocab, (case["rows"] + (n if case["kind"] == "prompt" else 0),), generator=g).tolist()
    contexts = [most] if n == 1 and case["kind"] == "decode" else torch.randint(max(1, most // 4), most + 1, (max(1, n),), generator=g).tolist()[:n]
    return tokens, contexts


def _held(c, layer, what, contexts, seed):
    """``[sequences, longest context, ...]`` of layer ``layer``: the cached rows by position (bf16), or ``[sequences, heads, vdim, dim]`` the states (f32)."""
    g = torch.Generator(device="cuda").manual_seed(seed * 131 + 7 * layer + ord(what[0]))
    n, ctx = len(contexts), max(contexts or [0])
    if what == "latent":
        t = torch.empty(n, ctx, c.kv_lora + c.rope, dtype=BF16, device="cuda")
    elif what == "state":
        m = c.layers[layer].mixer
        return torch.empty(n, m.heads, m.vdim, m.dim, dtype=F32, device="cuda").normal_(0.0, 2.0, generator=g)
    elif isinstance(c, dense_gqa.DenseConfig):
        t = torch.empty(n, ctx, c.kv_heads, c.head_dim, dtype=BF16, device="cuda")
    else:
        m = c.layers[layer].mixer
        t = torch.empty(n, ctx, m.kv_heads, m.dim if what == "key" else m.vdim, dtype=BF16, device="cuda")
    return t.normal_(0.0, 1.0, generator=g)


def _capacity(case):
    return (case["context"] + 1 + PAGE - 1) // PAGE * PAGE + PAGE


def _fill(cache, table, held, contexts):
    """Writes ``held`` (by position) into the pages of the sequences."""
    for s, ctx in enumerate(contexts):
        at = torch.arange(ctx, device="cuda")
        rows = table[s].long()[at // PAGE] * PAGE + at % PAGE
        cache.view(-1, *cache.shape[2:])[rows] = held[s, :ctx].view(ctx, *cache.shape[2:])


# ---------------------------------------------------------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c = _config(case)
    tokens, contexts = _inputs(case, c, seed)
    n, rows, cap = len(contexts), case["rows"], _capacity(case)
    one, prompt = case["kind"] == "decode" and rows == 1, case["kind"] == "prompt"
    s = dict(family=case["family"], kind=case["kind"], rows=rows, tokens=tokens, contexts=contexts)
    fabric = Fabric(0, 1)
    W = _weights(case, c, seed)
    if case["family"] == "dense":
        dec = dense_gqa.DenseDecoder(c, W, fabric, max_tokens=8, max_context=cap, num_slots=max(1, n), keep_logits=True)
        many = DensePrefill(dec, max_rows=min(2048, rows)) if not one else None
        for l in range(c.layers) if contexts else ():
            _fill(dec.k_cache[l], dec.page_table, _held(c, l, "key", contexts, seed), contexts)
            _fill(dec.v_cache[l], dec.page_table, _held(c, l, "value", contexts, seed), contexts)
        s["caches"] = {"k": dec.k_cache, "v": dec.v_cache}
    elif case["family"] == "mla_moe":
        dec = mla_moe.MlaMoeDecoder(c, W, fabric, max_tokens=8, max_context=cap, num_slots=max(1, n), keep_logits=True, expert_fp8=case["experts"] == "fp8")
        many = MlaMoePrefill(dec, max_rows=rows) if prompt else None
        for l in range(c.layers) if contexts else ():
            _fill(dec.caches[l], dec.page_table, _held(c, l, "latent", contexts, seed), contexts)
        s["caches"] = {"latent": dec.caches}
    else:
        dec = falinex.FalinexDecoder(c, W, fabric, max_tokens=8, max_context=cap, num_slots=n + 1 if prompt else n, keep_logits=True)
        many = falinex.FalinexRows(dec, max_rows=rows + n if prompt else rows) if not one else None
        if one:
            s["engine"] = DecodeEngine(dec)             # takes its sequence's pages
        else:
            for r in range(dec.num_slots):
                dec.state_manager.admit(r, cap)
            dec.state_manager.flush()
        for l, L in enumerate(dec.layers):
            if "state" in L:
                if contexts:
                    L["state"][:n].copy_(_held(c, l, "state", contexts, seed))
            elif contexts:
                _fill(L["k_cache"], dec.page_table, _held(c, l, "key", contexts, seed), contexts)
                _fill(L["v_cache"], dec.page_table, _held(c, l, "value", contexts, seed), contexts)
        s["caches"] = {"k": [L["k_cache"] for L in dec.layers if "state" not in L], "v": [L["v_cache"] for L in dec.layers if "state" not in L],
                       "state": [L["state"] for L in dec.layers if "state" in L]}
    s.update(dec=dec, many=many)
    dev = lambda v, dt=torch.int32: torch.tensor(v, dtype=dt, device="cuda")
    if one or (prompt and case["family"] != "falinex"):
        s["engine"] = s.get("engine") or DecodeEngine(dec, prefill=many if prompt else None)
    elif prompt:                                        # the prompt in the last sequence slot, then a row per running sequence
        slots, positions = [n] * rows + list(range(n)), list(range(rows)) + contexts
        s.update(slot_list=slots, position_list=positions, step=(dev(tokens), dev(positions), dev(slots)), select=dev([rows - 1] + list(range(rows, rows + n)), torch.int64))
    else:
        s.update(slot_list=list(range(n)), position_list=contexts, step=(dev(tokens), dev(contexts), dev(list(range(n)))), select=dev(list(range(n)), torch.int64))
        if case["family"] == "mla_moe":
            for at, v in zip((dec.tokens, dec.positions, dec.slots), s["step"]):
                at[:rows].copy_(v)
            s["graph"] = dec.capture(rows)
    return s


def run(s):
    """The logits and the updated caches and states; the token is where the logits are largest, often by less than a rounding."""
    dec = s["dec"]
    if "engine" in s:
        e = s["engine"]
        if s["kind"] == "prompt":
            e.reset()
            e.prefill(s["tokens"])
        else:
            e.pos = s["contexts"][0]
            e.step(s["tokens"][0])
        return {"logits": dec.logits[0], "state": s["caches"]}
    if "graph" in s:
        n = s["rows"]
        for at, v in zip((dec.tokens, dec.positions, dec.slots), s["step"]):
            at[:n].copy_(v)
        s["graph"].replay()
        return {"logits": dec.logits[:n], "state": s["caches"]}
    if s["family"] == "falinex":
        plan = s["many"].plan(s["slot_list"], s["position_list"])
        return {"logits": s["many"].forward_rows(*s["step"], s["select"], plan, plan.control.to("cuda")), "state": s["caches"]}
    return {"logits": s["many"].forward_rows(*s["step"], s["select"]), "state": s["caches"]}


# ---------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------------
def work(case):
    c = _config(case)
    n, prompt = _running(case), case["kind"] == "prompt"
    rows = case["rows"] + (n if prompt else 0)
    # the sequences' contexts are spread evenly between a quarter of the longest and the longest
    contexts = [case["context"]] if n == 1 and not prompt else [case["context"] * (0.25 + 0.75 * (i + 0.5) / max(1, n)) for i in range(n)]
    logit_rows = n + (1 if prompt else 0)
    size, flops = 0.0, 0.0

    def linear(params, r=rows):
        nonlocal size, flops
        size += 2.0 * params
        flops += 2.0 * params * r

    def attend(window, key_bytes, flops_per_pair):
        """Keys read by the decode rows, pairs of all rows, rows written."""
        nonlocal size, flops
        seen = [min(x + 1, window) if window else x + 1 for x in contexts]
        pairs = sum(seen)
        if prompt:
            m = case["rows"]
            pairs += m * (m + 1) / 2 if not window or m <= window else window * (window + 1) / 2 + (m - window) * window
        size += sum(seen) * key_bytes + rows * key_bytes
        flops += pairs * flops_per_pair

    if case["family"] == "dense":
        for _ in range(c.layers):
            linear(c.hidden * (2 * c.heads + 2 * c.kv_heads) * c.head_dim + 3 * c.hidden * c.ffn)
            attend(0, 4 * c.kv_heads * c.head_dim, 4 * c.heads * c.head_dim)
        width = c.hidden
    elif case["family"] == "falinex":
        for l in c.layers:
            m = l.mixer
            groups = m.heads if m.kind != "attention" else m.kv_heads
            linear(c.width * (m.heads * m.dim + groups * (m.dim + m.vdim) + 2 * m.heads * m.vdim) + 2 * c.width * l.ff)
            if m.kind == "attention":
                attend(m.window, 2 * m.kv_heads * (m.dim + m.vdim), 2 * m.heads * (m.dim + m.vdim))
            else:
                size += 4.0 * m.heads * m.dim * m.vdim * (2 * n + (1 if prompt else 0))
                flops += 4.0 * rows * m.heads * m.dim * m.vdim
        width = c.width
    else:
        es = 1 + 4 / 128 if case["experts"] == "fp8" else 2
        for _ in range(c.layers):
            linear(c.hidden * (c.q_lora + c.kv_lora + c.rope) + c.q_lora * c.heads * c.qk_dim + c.heads * (c.nope + c.vdim) * c.kv_lora + c.hidden * c.heads * c.vdim)
            size += 4.0 * c.experts * c.hidden
            flops += 2.0 * rows * c.experts * c.hidden
            chosen = c.experts * (1 - (1 - c.topk / c.experts) ** rows) + c.shared_ffn / c.expert_ffn
            size += es * chosen * 3 * c.hidden * c.expert_ffn
            flops += 2.0 * rows * 3 * c.hidden * (c.topk * c.expert_ffn + c.shared_ffn)
            attend(c.window, 2 * (c.kv_lora + c.rope), 2 * c.heads * (c.qk_dim + c.vdim if prompt else 2 * c.kv_lora + c.rope))
        width = c.hidden
    linear(c.vocab * width, logit_rows)
    size += 2.0 * rows * width + 4.0 * logit_rows * c.vocab
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """bf16 operands and, but for falinex, a bf16 residual over all layers: two orders of the f32 sums, which turn the roundings to bf16 behind
    them, end 0.011 apart in the logits of 24 layers (and each 0.012 from the sums in 64 bits)."""
    return {"rel": 0.03, "max": 0.5}


# ---------------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------------
def _rms(x, eps, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _turn(x, positions, dims, base, interleaved=False):
    """Rotation of the first ``dims`` columns of x ``[rows, heads, d]``."""
    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    a = torch.as_tensor(positions, dtype=F64, device=x.device)[:, None, None] * base ** (-2.0 * i / dims)
    cos, sin = torch.cos(a), torch.sin(a)
    out = x.clone()
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if interleaved else (x[..., :dims // 2], x[..., dims // 2:dims])
    p, q = u * cos - v * sin, v * cos + u * sin
    if interleaved:
        out[..., 0:dims:2], out[..., 1:dims:2] = p, q
    else:
        out[..., :dims // 2], out[..., dims // 2:dims] = p, q
    return out


def _seen(q, k, v, scale, first_pos, window=0, sink=None):
    """q ``[m, H, d]`` at positions first_pos + i over all keys k ``[n, G, d]``, v ``[n, G, e]`` of its sequence from position 0."""
    r = q.shape[1] // k.shape[1]
    out = torch.empty(q.shape[0], q.shape[1], v.shape[-1], dtype=F64, device=q.device)
    j = torch.arange(k.shape[0], device=q.device)[None]
    for i0 in range(0, q.shape[0], 512):
        qi = q[i0:i0 + 512]
        i = first_pos + i0 + torch.arange(qi.shape[0], device=q.device)[:, None]
        hide = j > i
        if window:
            hide |= i - j >= window
        for h in range(q.shape[1]):
            s = (qi[:, h] @ k[:, h // r].T * scale).masked_fill(hide, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
            a = torch.softmax(s, -1)
            out[i0:i0 + 512, h] = (a[:, :-1] if sink is not None else a) @ v[:, h // r]
    return out


def _attend(case, contexts, held, q, k, v, scale, window=0, sink=None):
    """Attention of the pass's rows: the prompt's over itself, then every decode row over what its sequence holds (``held``: keys and
    values by sequence, in 64 bits) and itself."""
    m = case["rows"] if case["kind"] == "prompt" else 0
    out = [_seen(q[:m], k[:m], v[:m], scale, 0, window, sink)] if m else []
    for s, ctx in enumerate(contexts):
        hk, hv = held(s, ctx)
        r = m + s
        out.append(_seen(q[r:r + 1], torch.cat([hk, k[r:r + 1]]), torch.cat([hv, v[r:r + 1]]), scale, ctx, window, sink))
    return torch.cat(out)


def _paged(case, contexts, held, rows):
    """Caches as the pages hold them after the pass, slot after slot: what was there, and the pass's rows by position."""
    pages = _capacity(case) // PAGE
    out = torch.zeros(max(1, len(contexts)), pages * PAGE, *rows.shape[1:], dtype=F64, device="cuda")
    if case["kind"] == "prompt":
        out[0, :case["rows"]] = rows
    for s, ctx in enumerate(contexts):
        out[s, :ctx] = held[s, :ctx].double().view(ctx, *rows.shape[1:])
        out[s, ctx] = rows[s]
    return out.view(-1, PAGE, *rows.shape[1:])


def exact(case, seed):
    c = _config(case)
    W = _weights(case, c, seed)
    tokens, contexts = _inputs(case, c, seed)
    positions = (list(range(case["rows"])) if case["kind"] == "prompt" else []) + contexts
    w = lambda name: W[name].double()
    n_logits = (1 if case["kind"] == "prompt" else 0) + len(contexts)
    x = W["embed"][torch.tensor(tokens, device="cuda")].double()
    how = {"dense": _exact_dense, "falinex": _exact_falinex, "mla_moe": _exact_mla}[case["family"]]
    x, state = how(case, c, w, seed, x, contexts, positions)
    if case["family"] == "falinex":
        logits = _rms(x[-n_logits:], c.eps, w("final.norm")) @ w("head").T
    else:
        logits = _rms(x[-n_logits:], c.eps, w("final_norm")) @ w("lm_head").T
    alone = case["family"] != "falinex" and case["kind"] == "prompt" or case["kind"] == "decode" and case["rows"] == 1
    return {"logits": logits[0] if alone else logits, "state": state}


def _exact_dense(case, c, w, seed, x, contexts, positions):
    hd, hq, hk, T = c.head_dim, c.heads, c.kv_heads, x.shape[0]
    state = {"k": [], "v": []}
    for l in range(c.layers):
        p = f"layers.{l}."
        qkv = _rms(x, c.eps, w(p + "attn_norm")) @ w(p + "qkv").T
        q = _turn(qkv[:, :hq * hd].reshape(T, hq, hd), positions, hd, c.theta)
        k = _turn(qkv[:, hq * hd:(hq + hk) * hd].reshape(T, hk, hd), positions, hd, c.theta)
        v = qkv[:, (hq + hk) * hd:].reshape(T, hk, hd)
        K, V = (_held(c, l, n, contexts, seed) for n in ("key", "value"))
        o = _attend(case, contexts, lambda s, ctx: (K[s, :ctx].double(), V[s, :ctx].double()), q, k, v, hd ** -0.5)
        state["k"].append(_paged(case, contexts, K, k))
        state["v"].append(_paged(case, contexts, V, v))
        x = x + o.reshape(T, hq * hd) @ w(p + "o_proj").T
        gu = _rms(x, c.eps, w(p + "ffn_norm")) @ w(p + "gate_up").T
        x = x + (torch.nn.functional.silu(gu[:, :c.ffn]) * gu[:, c.ffn:]) @ w(p + "down").T
    return x, state


def _decayed(m, q, k, v, decay, S):
    """Rows of one sequence: o_t = S_t^T q_t with S_t = decay S_(t-1) + k_t v_t^T, as blocks of 256 rows; S ``[H, d, e]`` ahead of them."""
    out = []
    for i0 in range(0, q.shape[0], 256):
        a, b, e = q[i0:i0 + 256], k[i0:i0 + 256], v[i0:i0 + 256]
        t = torch.arange(a.shape[0], dtype=F64, device=q.device)
        gap = t[:, None] - t[None]
        fall = torch.where(gap >= 0, decay[:, None, None] ** gap.clamp(min=0), torch.zeros((), dtype=F64, device=q.device))
        o = torch.einsum("hts,she->the", torch.einsum("thd,shd->hts", a, b) * fall, e)
        o = o + torch.einsum("thd,hde->the", a, S) * (decay[None, :] ** (t[:, None] + 1))[:, :, None]
        n = a.shape[0]
        S = decay[:, None, None] ** n * S + torch.einsum("thd,the->hde", b * (decay[None, :] ** (n - 1 - t)[:, None])[:, :, None], e)
        out.append(o)
    return torch.cat(out), S


def _exact_falinex(case, c, w, seed, x, contexts, positions):
    silu, T, n = torch.nn.functional.silu, x.shape[0], len(contexts)
    head = case["rows"] if case["kind"] == "prompt" else 0
    state = {"k": [], "v": [], "state": []}
    for l, L in enumerate(c.layers):
        p, m = f"l{l}.", L.mixer
        q, k, v, g = (x @ w(p + "mix." + name).T for name in "qkvg")
        groups = m.heads if m.kind != "attention" else m.kv_heads
        q, k, v = q.view(T, m.heads, m.dim), k.view(T, groups, m.dim), v.view(T, groups, m.vdim)
        if m.kind == "attention":
            q = _turn(_rms(q, c.eps, w(p + "mix.q.norm")), positions, m.rot_dims, m.rot_base, True)
            k = _turn(_rms(k, c.eps, w(p + "mix.k.norm")), positions, m.rot_dims, m.rot_base, True)
            K, V = (_held(c, l, name, contexts, seed) for name in ("key", "value"))
            o = _attend(case, contexts, lambda s, ctx: (K[s, :ctx].double(), V[s, :ctx].double()), q, k, v, m.scale, m.window, w(p + "mix.sink"))
            y = o.reshape(T, -1) * torch.sigmoid(g)
            state["k"].append(None)        # which pages hold them is the pool's choice
            state["v"].append(None)
        else:
            if m.kind == "retention":
                q, k = _turn(q, positions, m.rot_dims, m.rot_base), _turn(k, positions, m.rot_dims, m.rot_base) * m.dim ** -0.5
            else:
                q, k, v = silu(q), silu(k), silu(v)
            decay = torch.tensor(m.decay, dtype=F64, device="cuda")
            S = _held(c, l, "state", contexts, seed).double().transpose(2, 3)
            out, after = [], [None] * n
            if head:
                o, last = _decayed(m, q[:head], k[:head], v[:head], decay, torch.zeros(m.heads, m.dim, m.vdim, dtype=F64, device="cuda"))
                out.append(o)
                after.append(last)
            for s in range(n):
                o, after[s] = _decayed(m, q[head + s:head + s + 1], k[head + s:head + s + 1], v[head + s:head + s + 1], decay, S[s])
                out.append(o)
            state["state"].append(torch.stack(after).transpose(2, 3))
            o = torch.cat(out)
            y = _rms(o, c.eps).reshape(T, -1) * silu(g) if m.kind == "retention" else _rms(o.reshape(T, -1), c.eps, w(p + "mix.norm")) * torch.sigmoid(g)
        x = x + _rms(y @ w(p + "mix.o").T, c.eps, w(p + "norm1"))
        u = x @ w(p + "mlp.up").T
        u = 0.5 * u * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (u + 0.044715 * u ** 3)))
        x = x + _rms(u @ w(p + "mlp.down").T, c.eps, w(p + "norm2"))
    # the rows that are asked for: the prompt's last, then the decode rows
    return (torch.cat([x[head - 1:head], x[head:]]) if head else x), state


def _narrow(t):
    """A matrix as block-scaled fp8 holds it: e4m3 with an f32 scale (largest / 448) per 128 columns of a row."""
    b = t.float().unflatten(-1, (-1, 128))
    scale = b.abs().amax(-1, keepdim=True) / 448.0
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    return ((b / scale).to(torch.float8_e4m3fn).double() * scale.double()).flatten(-2)


def _exact_mla(case, c, w, seed, x, contexts, positions):
    T, H, state = x.shape[0], c.heads, {"latent": []}
    wide = (lambda t: _narrow(t.to(BF16))) if case["experts"] == "fp8" else (lambda t: t)
    for l in range(c.layers):
        p = f"layers.{l}."
        a = _rms(x, c.eps, w(p + "attn_norm")) @ w(p + "qkv_a").T
        q = (_rms(a[:, :c.q_lora], c.eps, w(p + "q_a_norm")) @ w(p + "q_b").T).view(T, H, c.qk_dim)
        lat = _rms(a[:, c.q_lora:c.q_lora + c.kv_lora], c.eps, w(p + "kv_a_norm"))
        pe = _turn(a[:, None, c.q_lora + c.kv_lora:], positions, c.rope, c.theta)[:, 0]
        q = torch.cat([q[..., :c.nope], _turn(q[..., c.nope:], positions, c.rope, c.theta)], -1)
        kvb = w(p + "kv_b")
        lift = lambda t, e: (torch.cat([torch.einsum("nc,hdc->nhd", t, kvb[:, :c.nope]), e[:, None].expand(-1, H, -1)], -1), torch.einsum("nc,hvc->nhv", t, kvb[:, c.nope:]))
        k, v = lift(lat, pe)
        K = _held(c, l, "latent", contexts, seed)
        o = _attend(case, contexts, lambda s, ctx: lift(K[s, :ctx, :c.kv_lora].double(), K[s, :ctx, c.kv_lora:].double()), q, k, v, c.scale, c.window)
        state["latent"].append(_paged(case, contexts, K, torch.cat([lat, pe], -1)))
        x = x + o.reshape(T, -1) @ w(p + "o_proj").T
        h = _rms(x, c.eps, w(p + "ffn_norm"))
        top = torch.softmax(h @ w(p + "router").T, -1).topk(c.topk, -1)
        weight = top.values / top.values.sum(-1, keepdim=True)
        unit = lambda t, gu, down: (torch.nn.functional.silu(t @ gu[:gu.shape[0] // 2].T) * (t @ gu[gu.shape[0] // 2:].T)) @ down.T
        y = unit(h, wide(w(p + "shared_gate_up")), wide(w(p + "shared_down")))
        gate_up, down = w(p + "gate_up").to(BF16), w(p + "down").to(BF16)
        for e in range(c.experts):
            row, place = (top.indices == e).nonzero(as_tuple=True)
            if row.numel():
                y.index_add_(0, row, weight[row, place][:, None] * unit(h[row], wide(gate_up[e]).double(), wide(down[e]).double()))
        x = x + y
    head = case["rows"] if case["kind"] == "prompt" else 0
    return x[head - 1:head] if head else x, state
