"""What a user of the library has it do, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" names one of the entry points a program calls:

  reply      Engine.step over a Qwen3 decoder: a batch of prompts in one step, then single tokens, logits out
  attention  the attention mixer of the Qwen3 shapes, prompts of unequal lengths or one token against a cache
  mlp        the gated feed-forward, bfloat16 or float32
  delta      the gated delta rule with a decay per key channel, prompts or one token against a state
  window     attention under a sliding window with kept first keys and a sink, float32 softmax weights
  latent     latent attention with a sink, prompts
  experts    routed experts with a shared one
  wkv        time mixing with a decay per key channel and token, prompts

Layer sizes are those of the shapes that bench.py runs (widths 1,024, 2,560 and 4,096). The parts are built through the
registries of abacus_b200.parts, as abacus_b200.models.Model builds them, and own a cache where they need one.
"""
import math

import torch

from abacus_b200.cache import SequenceCache
from abacus_b200.config import Qwen3Config, get_architecture
from abacus_b200.config.specs import (AttentionSpec, DeltaRuleSpec, ExpertSpec, GatedMLPSpec, LatentAttentionSpec,
                                      RotarySpec, RoutedMLPSpec, WkvSpec)
from abacus_b200.engine import Engine
from abacus_b200.engine.batch import Sequence, StepBatch
from abacus_b200.models import Model
from abacus_b200.parts import FEED_FORWARDS, MIXERS, BuildContext, Workspace

EPS = 1e-6
PAGE = 64
# width -> heads of the attention layers, inner size of the feed-forward, heads of the recurrent layers
HEADS = {1024: (16, 8), 2560: (32, 8), 4096: (32, 8)}
INNER = {1024: 3072, 2560: 9728, 4096: 12288}


def _lengths(case):
    return [int(n) for n in case["lengths"].split(",")]


def _text(lengths):
    return ",".join(str(n) for n in lengths)


def listed():
    return [
        # one user's short question to the 0.6B shape and the first tokens of the answer: launches and latency count
        dict(name="reply_one", kind="reply", width=1024, layers=28, lengths="200", steps=12),
        # a batch of unequal questions answered together
        dict(name="reply_batch", kind="reply", width=1024, layers=28, steps=8,
             lengths="64,97,128,160,211,256,301,345,384,407,450,512,577,640,703,768"),
        # an attention layer of the 4B shape over unequal prompts
        dict(name="attention_prompts", kind="attention", width=2560, lengths="64,301,777,1024,1531,2048", decode=False,
             dtype="bfloat16"),
        # an attention layer of the 8B shape, one token each for 32 users with contexts of 128 to 4,096
        dict(name="attention_decode", kind="attention", width=4096, decode=True, dtype="bfloat16",
             lengths=_text([128 + (3968 * i) // 31 for i in range(32)])),
        # the feed-forward of the 4B shape over a step's prompts
        dict(name="mlp_prompts", kind="mlp", width=2560, rows=3967, dtype="bfloat16"),
        # the feed-forward of the 0.6B shape on the 32-bit path
        dict(name="mlp_float32", kind="mlp", width=1024, rows=500, dtype="float32"),
        # a delta-rule layer at width 1,024 over one long prompt
        dict(name="delta_prompt", kind="delta", width=1024, heads=16, kv_heads=8, dim=128, lengths="1999", decode=False),
        # the same at width 2,560, one token each for 64 users
        dict(name="delta_decode", kind="delta", width=2560, heads=32, kv_heads=8, dim=128, decode=True, lengths=_text([1] * 64)),
        # windowed attention with a sink at width 2,560 over unequal prompts
        dict(name="window_prompts", kind="window", width=2560, dim=128, window=1024, keep=4, lengths="345,1500,2048"),
        # latent attention at width 2,560 over two prompts
        dict(name="latent_prompts", kind="latent", width=2560, heads=32, dim=128, rot=64, rank=192, lengths="1111,2048"),
        # routed experts at width 2,560 over a step's prompts
        dict(name="experts_prompts", kind="experts", width=2560, rows=3001, experts=16, top=2, inner=2432),
        # time mixing at width 2,560 over unequal prompts
        dict(name="wkv_prompts", kind="wkv", width=2560, heads=40, dim=64, lengths="500,1023,2048"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_lengths(rng, most, longest=2048, shortest=16):
    """Unequal prompts of `shortest` to `longest` tokens, together at most `most`."""
    lengths, left = [], most
    for _ in range(rng.randint(1, 8)):
        n = min(_log_int(rng, shortest, longest), left)
        if n < shortest:
            break
        lengths.append(n)
        left -= n
    return _text(lengths)


def draw(rng):
    kind = rng.choice(["reply", "attention", "attention", "mlp", "mlp", "delta", "delta", "window", "latent", "experts", "wkv"])
    width = rng.choice([1024, 2560])
    if kind == "reply":
        return dict(kind=kind, width=1024, layers=28, lengths=_draw_lengths(rng, 4000, 1024), steps=rng.randint(2, 12))
    if kind == "attention":
        width = rng.choice([1024, 2560, 4096])
        if rng.random() < 0.4:
            n = rng.randint(8, 48)
            return dict(kind=kind, width=width, decode=True, dtype="bfloat16", lengths=_text([_log_int(rng, 64, 4096) for _ in range(n)]))
        if rng.random() < 0.2:
            return dict(kind=kind, width=1024, lengths=_draw_lengths(rng, 400, 256), decode=False, dtype="float32")
        return dict(kind=kind, width=width, lengths=_draw_lengths(rng, 6000), decode=False, dtype="bfloat16")
    if kind == "mlp":
        if rng.random() < 0.4:
            return dict(kind=kind, width=1024, rows=_log_int(rng, 33, 1500), dtype="float32")
        return dict(kind=kind, width=rng.choice([1024, 2560, 4096]), rows=_log_int(rng, 128, 6000), dtype="bfloat16")
    if kind == "delta":
        heads, dim = rng.choice([8, 16, 32]), rng.choice([64, 128])
        kv_heads = rng.choice([8, heads])
        if rng.random() < 0.4:
            return dict(kind=kind, width=width, heads=heads, kv_heads=kv_heads, dim=dim, decode=True, lengths=_text([1] * rng.randint(8, 96)))
        return dict(kind=kind, width=width, heads=heads, kv_heads=kv_heads, dim=dim, decode=False, lengths=_draw_lengths(rng, 6000))
    if kind == "window":
        return dict(kind=kind, width=width, dim=rng.choice([64, 128]), window=rng.choice([256, 512, 1000, 1024]), keep=rng.choice([0, 4, 64]),
                    lengths=_draw_lengths(rng, 5000))
    if kind == "latent":
        heads = rng.choice([16, 32])
        return dict(kind=kind, width=width, heads=heads, dim=128, rot=64, rank=rng.choice([192, 256]), lengths=_draw_lengths(rng, 4000))
    if kind == "experts":
        return dict(kind=kind, width=width, rows=_log_int(rng, 128, 4000), experts=rng.choice([8, 16]), top=rng.choice([2, 4]),
                    inner=768 if width == 1024 else 2432)
    return dict(kind=kind, width=width, heads=width // 64, dim=64, lengths=_draw_lengths(rng, 5000))


# ------------------------------------------------------------------ what a program has in hand before the call
class _Random:
    """Seeded values on the GPU; one stream per case and seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.gen, device="cuda") * std + mean).to(dtype)

    def matrix(self, *shape, dtype=torch.bfloat16, std=0.02):
        return self.normal(*shape, std=std, dtype=dtype)

    def ints(self, high, n):
        return torch.randint(0, high, (n,), generator=self.gen, device="cuda")


VOCAB = 151936


def _qwen_config(case):
    heads, kv = HEADS[case["width"]]
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=case["width"], intermediate_size=INNER[case["width"]],
                num_hidden_layers=case["layers"], num_attention_heads=heads, num_key_value_heads=kv, head_dim=128, vocab_size=VOCAB,
                max_position_embeddings=40960, rope_theta=1000000.0, rms_norm_eps=EPS, tie_word_embeddings=True)


def _qwen_weights(case, seed):
    """The decoder's tensors by their names in a checkpoint."""
    r, d, inner = _Random(seed), case["width"], INNER[case["width"]]
    heads, kv = HEADS[d]
    w = {"model.embed_tokens.weight": r.matrix(VOCAB, d), "model.norm.weight": r.normal(d, std=0.1, mean=1.0, dtype=torch.bfloat16)}
    for l in range(case["layers"]):
        p = f"model.layers.{l}."
        for n, size in (("input_layernorm", d), ("post_attention_layernorm", d), ("self_attn.q_norm", 128), ("self_attn.k_norm", 128)):
            w[p + n + ".weight"] = r.normal(size, std=0.1, mean=1.0, dtype=torch.bfloat16)
        for n, shape in (("self_attn.q_proj", (heads * 128, d)), ("self_attn.k_proj", (kv * 128, d)), ("self_attn.v_proj", (kv * 128, d)),
                         ("self_attn.o_proj", (d, heads * 128)), ("mlp.gate_proj", (inner, d)), ("mlp.up_proj", (inner, d)),
                         ("mlp.down_proj", (d, inner))):
            w[p + n + ".weight"] = r.matrix(*shape)
    return w


def _qwen_tokens(case, seed):
    """(the prompts, per step one token a sequence) as a program has them: lists of ids."""
    r, lengths = _Random(seed + 1000003), _lengths(case)
    prompts = [r.ints(VOCAB, n).tolist() for n in lengths]
    return prompts, [r.ints(VOCAB, len(lengths)).tolist() for _ in range(case["steps"])]


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _spec(case):
    kind, d = case["kind"], case["width"]
    if kind == "attention":
        heads, kv = HEADS[d]
        return AttentionSpec(hidden=d, n_heads=heads, n_kv_heads=kv, head_dim=128, scale=128 ** -0.5, qk_norm_eps=EPS,
                             position=RotarySpec(theta=1000000.0, rotary_dim=128))
    if kind == "mlp":
        return GatedMLPSpec(d, INNER[d], "silu")
    if kind == "delta":
        return DeltaRuleSpec(hidden=d, n_heads=case["heads"], n_kv_heads=case["kv_heads"], key_dim=case["dim"], value_dim=case["dim"],
                             conv_taps=4, decay_rank=64, gate_rank=64, norm_eps=EPS)
    if kind == "window":
        heads, kv = HEADS[d]
        return AttentionSpec(hidden=d, n_heads=heads, n_kv_heads=kv, head_dim=case["dim"], scale=case["dim"] ** -0.5, qk_norm_eps=EPS,
                             position=RotarySpec(theta=1000000.0, rotary_dim=case["dim"] // 2), window=case["window"],
                             v_head_dim=case["dim"], keep_first=case["keep"], sink=True, exact_weights=True)
    if kind == "latent":
        return LatentAttentionSpec(hidden=d, n_heads=case["heads"], head_dim=case["dim"], rot_dim=case["rot"], v_head_dim=case["dim"],
                                   rank=case["rank"], scale=(case["dim"] + case["rot"]) ** -0.5, norm_eps=EPS, sink=True,
                                   position=RotarySpec(theta=1000000.0, rotary_dim=case["rot"], pairing="interleaved", exact_angles=True))
    if kind == "experts":
        return RoutedMLPSpec(hidden=d, experts=case["experts"], top=case["top"], expert=ExpertSpec(case["inner"]),
                             shared=ExpertSpec(case["inner"]), score="sigmoid", weight_on="input")
    return WkvSpec(hidden=d, n_heads=case["heads"], key_dim=case["dim"], decay_rank=64, norm_eps=EPS)


def _params(case, shapes, seed):
    """The part's tensors by slot: matrices N(0, 0.02), the others as such layers hold them."""
    r, dt, params = _Random(seed), _dtype(case), {}
    for slot, shape in shapes:
        if slot.startswith("conv_"):
            params[slot] = r.normal(*shape, std=0.3, mean=0.3)
        elif slot in ("decay_log", "decay_bias", "w0", "bonus"):
            params[slot] = r.normal(*shape, std=0.5)
        elif slot == "sink":
            params[slot] = r.normal(*shape)
        elif slot.startswith("mu_"):
            params[slot] = r.normal(*shape, std=0.25, mean=0.5)
        elif len(shape) == 1:
            params[slot] = r.normal(*shape, std=0.1, mean=1.0)
        else:
            params[slot] = r.matrix(*shape, dtype=dt)
    return params


def _shapes(case):
    """The slots of the part and their shapes, in a fixed order."""
    kind, d = case["kind"], case["width"]
    if kind in ("attention", "window"):
        (heads, kv), dim = HEADS[d], case.get("dim", 128)
        shapes = [("wq", (heads * dim, d)), ("wk", (kv * dim, d)), ("wv", (kv * dim, d)), ("wo", (d, heads * dim)), ("q_norm", (dim,)),
                  ("k_norm", (dim,))]
        return shapes + ([("sink", (heads,))] if kind == "window" else [])
    if kind == "mlp":
        return [("gate", (INNER[d], d)), ("up", (INNER[d], d)), ("down", (d, INNER[d]))]
    if kind == "delta":
        qk, v, heads = case["kv_heads"] * case["dim"], case["heads"] * case["dim"], case["heads"]
        return [("wq", (qk, d)), ("wk", (qk, d)), ("wv", (v, d)), ("conv_q", (qk, 4)), ("conv_k", (qk, 4)), ("conv_v", (v, 4)),
                ("wb", (heads, d)), ("decay_in", (64, d)), ("decay_out", (v, 64)), ("decay_log", (heads,)), ("decay_bias", (v,)),
                ("gate_in", (64, d)), ("gate_out", (v, 64)), ("out_norm", (case["dim"],)), ("wo", (d, v))]
    if kind == "latent":
        h, dim, rot, rank = case["heads"], case["dim"], case["rot"], case["rank"]
        return [("wq", (h * (dim + rot), d)), ("wuk", (h * dim, rank)), ("wuv", (h * dim, rank)), ("wo", (d, h * dim)),
                ("wdown", (rank + rot, d)), ("down_norm", (rank,)), ("sink", (h,))]
    if kind == "experts":
        shapes = [("router", (case["experts"], d))]
        for e in range(case["experts"]):
            shapes += [(f"up{e}", (case["inner"], d)), (f"down{e}", (d, case["inner"]))]
        return shapes + [("shared_up", (case["inner"], d)), ("shared_down", (d, case["inner"]))]
    size = case["heads"] * case["dim"]
    return ([(f"mu_{b}", (d,)) for b in "rkvgw"] + [(f"w{b}", (size, d)) for b in "rkvg"]
            + [("w1", (64, d)), ("w2", (size, 64)), ("w0", (size,)), ("bonus", (case["heads"], case["dim"])), ("out_norm", (size,)),
               ("wo", (d, size))])


def _rows(case):
    if case.get("decode"):
        return len(_lengths(case))
    return case["rows"] if "rows" in case else sum(_lengths(case))


def _inputs(case, seed):
    """The normed activations that enter the part."""
    return _Random(seed + 500009).normal(_rows(case), case["width"], dtype=_dtype(case))


def _held(case, seed):
    """What the sequences hold before a decode step, sequence by sequence: (keys, values) [tokens before, kv heads, 128], or the
    delta rule's (state [heads, value, key], last rows of the convolution [taps - 1, channels])."""
    r, held = _Random(seed + 900001), []
    if case["kind"] == "attention":
        _, kv = HEADS[case["width"]]
        for n in _lengths(case):
            held.append((r.normal(n - 1, kv, 128, dtype=torch.bfloat16), r.normal(n - 1, kv, 128, dtype=torch.bfloat16)))
    else:
        channels = (2 * case["kv_heads"] + case["heads"]) * case["dim"]
        for _ in _lengths(case):
            held.append((r.normal(case["heads"], case["dim"], case["dim"], std=0.1), r.normal(3, channels, dtype=torch.bfloat16).float()))
    return held


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    device = torch.device("cuda", torch.cuda.current_device())
    if case["kind"] == "reply":
        config = Qwen3Config.from_dict(_qwen_config(case))
        arch, spec = get_architecture(config.architecture), config.to_spec()
        model = Model(spec, arch.layout(spec), _qwen_weights(case, seed), torch.bfloat16, device)
        lengths = _lengths(case)
        context = max(lengths) + case["steps"] + 1
        room = sum(-(-(n + case["steps"] + 1) // PAGE) * PAGE for n in lengths)
        s.engine = Engine(model, max_tokens=max(room, context + PAGE), max_slots=len(lengths), max_context=context)
        s.prompts, s.tokens = _qwen_tokens(case, seed)
        return s
    s.ws = Workspace(device)
    ctx = BuildContext(device=device, dtype=_dtype(case))
    feed_forward = case["kind"] in ("mlp", "experts")
    s.part = (FEED_FORWARDS if feed_forward else MIXERS).build(_spec(case))
    s.part.bind(_params(case, _shapes(case), seed), ctx)
    s.x = _inputs(case, seed)
    n = s.x.shape[0]
    s.out = torch.empty((n, case["width"]), dtype=torch.float32, device=device)
    plans = getattr(s.part, "step_plans", lambda: [])()
    if feed_forward:
        s.batch = StepBatch(n, 1, 1, device).fill([Sequence(0, [0] * n, 0, [])], exact=True)
        return s
    lengths = _lengths(case)
    room = sum(-(-(m + 1) // PAGE) * PAGE for m in lengths)
    longest = max(lengths) + 1
    s.cache = SequenceCache([s.part.cache_need()], [None], max(room, longest + PAGE), ctx.dtype, device, max_slots=len(lengths),
                            max_context=longest)
    if hasattr(s.part, "prepare"):
        s.part.prepare(longest, device)
    s.batch = StepBatch(n, len(lengths), 1, device, plans=plans)
    s.lengths = lengths
    if case.get("decode"):  # the sequences are open and hold what earlier steps left
        s.seqs, view = [], s.cache.views[0]
        for m, held in zip(lengths, _held(case, seed)):
            slot = s.cache.open_slot()
            s.cache.reserve(slot, m)
            s.seqs.append(Sequence(slot, [0], m - 1, []))
            if view.kv is not None:
                pages = view.kv.page_table[slot, :-(-m // PAGE)].long()
                for pool, rows in ((view.kv.k, held[0]), (view.kv.v, held[1])):
                    full = torch.zeros((len(pages) * PAGE,) + tuple(rows.shape[1:]), dtype=rows.dtype, device=device)
                    full[:m - 1] = rows
                    pool[pages] = full.view(len(pages), PAGE, *rows.shape[1:]).transpose(1, 2)
            else:
                view.states["delta"][slot] = held[0]
                view.states["conv_tail"][slot] = held[1]
        if case["kind"] == "delta":  # (past their first tokens, so that the convolution's last rows count)
            s.seqs = [Sequence(q.slot, [0], 100, []) for q in s.seqs]
    return s


def run(s):
    case = s.case
    if case["kind"] == "reply":
        engine = s.engine
        slots = [engine.open() for _ in s.prompts]
        logits = [engine.step([(slot, p, [len(p) - 1]) for slot, p in zip(slots, s.prompts)]).clone()]
        for tokens in s.tokens:
            logits.append(engine.step([(slot, [t], [0]) for slot, t in zip(slots, tokens)]).clone())
        for slot in slots:
            engine.close(slot)
        return logits
    if case["kind"] in ("mlp", "experts"):
        return s.part.forward(s.x, s.out, s.batch, s.ws)
    view = s.cache.views[0]
    if case.get("decode"):
        s.batch.fill(s.seqs, exact=True)
        s.part.forward(s.x, s.out, s.batch, view, s.ws)
        return {"out": s.out, **(view.states or {})}
    slots = [s.cache.open_slot() for _ in s.lengths]
    s.cache.reserve_all(list(zip(slots, s.lengths)))
    s.batch.fill([Sequence(slot, [0] * n, 0, []) for slot, n in zip(slots, s.lengths)], exact=True)
    s.part.forward(s.x, s.out, s.batch, view, s.ws)
    for slot in slots:
        s.cache.close_slot(slot)
    return {"out": s.out, **(view.states or {})}


# ------------------------------------------------------------------ what a pass cannot do without
def _causal_pairs(n, window=None, keep=0):
    """(query, key) pairs of n tokens: the last `window` keys and the first `keep`."""
    if window is None or n <= window:
        return n * (n + 1) // 2
    kept = sum(min(keep, max(0, i - window + 1)) for i in range(n)) if keep else 0
    return window * (window + 1) // 2 + (n - window) * window + kept


def work(case):
    kind, d = case["kind"], case["width"]
    size = 4 if case.get("dtype") == "float32" else 2
    if kind == "reply":
        (heads, kv), lengths, steps = HEADS[d], _lengths(case), case["steps"]
        layer = d * (heads + 2 * kv) * 128 + heads * 128 * d + 3 * d * INNER[d]
        weights = 2 * (case["layers"] * layer + VOCAB * d)
        row = 2 * 2 * kv * 128 * case["layers"]  # a token's keys and values
        nbytes = (steps + 1) * (weights + 4 * len(lengths) * VOCAB)
        nbytes += sum(row * n + sum(row * (n + t + 1) for t in range(steps)) for n in lengths)
        tokens = sum(lengths) + steps * len(lengths)
        flops = 2 * tokens * case["layers"] * layer + 2 * (steps + 1) * len(lengths) * VOCAB * d
        flops += sum(4 * 128 * heads * case["layers"] * _causal_pairs(n + steps) for n in lengths)
        return {"bytes": nbytes, "flops": flops}
    n = _rows(case)
    weights = sum(math.prod(shape) for slot, shape in _shapes(case))
    nbytes, flops = size * (weights + n * d) + 4 * n * d, 2 * n * sum(math.prod(shape) for slot, shape in _shapes(case) if slot[0] in "wgudr")
    if kind == "mlp":
        return {"bytes": nbytes, "flops": 2 * n * weights}
    if kind == "experts":
        return {"bytes": nbytes, "flops": 2 * n * (case["experts"] * d + (case["top"] + 1) * 2 * d * case["inner"])}
    lengths = _lengths(case)
    if kind in ("attention", "window"):
        (heads, kv), dim = HEADS[d], case.get("dim", 128)
        if case.get("decode"):
            pairs, kept = sum(lengths), sum(lengths)
        else:
            pairs, kept = sum(_causal_pairs(m, case.get("window"), case.get("keep", 0)) for m in lengths), n
        return {"bytes": nbytes + 2 * size * kv * dim * kept, "flops": flops + 4 * dim * heads * pairs}
    if kind == "latent":
        h, dim, rot = case["heads"], case["dim"], case["rot"]
        pairs = sum(_causal_pairs(m) for m in lengths)
        return {"bytes": nbytes + 2 * n * (case["rank"] + rot), "flops": flops + 2 * (2 * dim + rot) * h * pairs}
    state = case["heads"] * case["dim"] ** 2  # delta rule, wkv: a state per sequence, walked token by token
    per_token = 7 * state if kind == "delta" else 5 * state
    moved = 4 * state * len(lengths) * (2 if case.get("decode") else 1)
    return {"bytes": nbytes + moved, "flops": flops + n * per_token}


def tolerance(case):
    """Largest relative errors of another correct implementation at the same precision: about four times what a pass is away
    from 64 bits (bfloat16: the roundings of activations between products, and in a whole decoder those of 28 layers)."""
    if case.get("dtype") == "float32":
        return {"rel": 6e-6}
    return {"rel": {"reply": 0.028, "attention": 0.016, "mlp": 0.012, "delta": 0.018, "window": 0.015, "latent": 0.015, "experts": 0.013,
                    "wkv": 0.024}[case["kind"]]}


# ------------------------------------------------------------------ the same in 64 bits
def _f64(params):
    return {n: t.double() for n, t in params.items()}


def _rms(x, w, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, positions, theta, dims, interleaved=False):
    """Pairs of the first `dims` elements of x [tokens, heads, size] turned by their position's angles."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    angle = positions.double()[:, None] * (theta ** (-2.0 * i / dims))[None]
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    turned = x.clone()
    if interleaved:
        a, b = x[..., 0:dims:2], x[..., 1:dims:2]
        turned[..., 0:dims:2], turned[..., 1:dims:2] = a * cos - b * sin, a * sin + b * cos
    else:
        a, b = x[..., :dims // 2], x[..., dims // 2:dims]
        turned[..., :dims // 2], turned[..., dims // 2:dims] = a * cos - b * sin, a * sin + b * cos
    return turned


def _attend(q, k, v, scale, first=0, window=None, keep=0, sink=None):
    """q [n, heads, d] at positions first .. against k, v [m, kv heads, ..] at 0 .. m - 1."""
    n, heads, m, group = q.shape[0], q.shape[1], k.shape[0], q.shape[1] // k.shape[1]
    i = torch.arange(first, first + n, device=q.device)[:, None]
    j = torch.arange(m, device=q.device)[None]
    seen = j <= i
    if window is not None:
        seen = seen & ((i - j < window) | (j < keep))
    out = []
    for h in range(heads):  # a head at a time: the maps of one head fit easily
        z = (q[:, h] @ k[:, h // group].T * scale).masked_fill(~seen, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[h].expand(n, 1)], dim=1)
        out.append(torch.softmax(z, dim=1)[:, :m] @ v[:, h // group])
    return torch.stack(out, dim=1).reshape(n, -1)


def _exact_reply(case, seed):
    w, (prompts, tokens) = _qwen_weights(case, seed), _qwen_tokens(case, seed)
    d, (heads, kv), steps = case["width"], HEADS[case["width"]], case["steps"]
    table = w["model.embed_tokens.weight"]
    lengths = [len(p) + steps for p in prompts]
    ids = torch.tensor([t for i, p in enumerate(prompts) for t in p + [step[i] for step in tokens]], device="cuda")
    x = table[ids].double()
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    for l in range(case["layers"]):
        get = lambda n: w[f"model.layers.{l}.{n}.weight"].double()  # noqa: E731
        xn = _rms(x, get("input_layernorm"))
        q = _rms((xn @ get("self_attn.q_proj").T).view(-1, heads, 128), get("self_attn.q_norm"))
        k = _rms((xn @ get("self_attn.k_proj").T).view(-1, kv, 128), get("self_attn.k_norm"))
        v = (xn @ get("self_attn.v_proj").T).view(-1, kv, 128)
        q, k = (_rotate(t, positions, 1e6, 128) for t in (q, k))
        parts = zip(*(t.split(lengths) for t in (q, k, v)))
        x = x + torch.cat([_attend(*part, 128 ** -0.5) for part in parts]) @ get("self_attn.o_proj").T
        xn = _rms(x, get("post_attention_layernorm"))
        x = x + (torch.nn.functional.silu(xn @ get("mlp.gate_proj").T) * (xn @ get("mlp.up_proj").T)) @ get("mlp.down_proj").T
    start = [sum(lengths[:i]) for i in range(len(lengths))]
    rows = torch.tensor([[s + len(p) - 1 + t for s, p in zip(start, prompts)] for t in range(steps + 1)], device="cuda")
    final, table = _rms(x, w["model.norm.weight"].double()), table.double()
    return [final[r] @ table.T for r in rows]


def _exact_attention(case, seed):
    p, x, lengths = _f64(_params(case, _shapes(case), seed)), _inputs(case, seed).double(), _lengths(case)
    (heads, kv), dim, window = HEADS[case["width"]], case.get("dim", 128), case.get("window")
    rotary = 128 if case["kind"] == "attention" else dim // 2
    decode = bool(case.get("decode"))
    positions = torch.tensor([n - 1 for n in lengths], device="cuda") if decode else torch.cat([torch.arange(n, device="cuda") for n in lengths])
    q = _rotate(_rms((x @ p["wq"].T).view(-1, heads, dim), p["q_norm"]), positions, 1e6, rotary)
    k = _rotate(_rms((x @ p["wk"].T).view(-1, kv, dim), p["k_norm"]), positions, 1e6, rotary)
    v = (x @ p["wv"].T).view(-1, kv, dim)
    scale, outs, at = dim ** -0.5, [], 0
    held = _held(case, seed) if decode else None
    for i, n in enumerate(lengths):
        if decode:
            held_k, held_v = held[i]
            outs.append(_attend(q[i:i + 1], torch.cat([held_k.double(), k[i:i + 1]]), torch.cat([held_v.double(), v[i:i + 1]]), scale, n - 1))
        else:
            outs.append(_attend(q[at:at + n], k[at:at + n], v[at:at + n], scale, 0, window, case.get("keep", 0), p.get("sink")))
            at += n
    return {"out": torch.cat(outs) @ p["wo"].T}


def _exact_mlp(case, seed):
    p, x = _f64(_params(case, _shapes(case), seed)), _inputs(case, seed).double()
    return (torch.nn.functional.silu(x @ p["gate"].T) * (x @ p["up"].T)) @ p["down"].T


def _exact_experts(case, seed):
    p, x = _f64(_params(case, _shapes(case), seed)), _inputs(case, seed).double()
    scores, chosen = torch.sigmoid(x @ p["router"].T).topk(case["top"], dim=1)
    ffn = lambda h, up, down: torch.relu(h @ up.T).square() @ down.T  # noqa: E731
    out = ffn(x, p["shared_up"], p["shared_down"])
    for e in range(case["experts"]):
        row, k = (chosen == e).nonzero(as_tuple=True)
        out[row] += ffn(x[row] * scores[row, k, None], p[f"up{e}"], p[f"down{e}"])
    return out


def _padded(rows, lengths):
    """Rows of sequences one after another -> [longest, sequences, ...], zeros behind a sequence's end."""
    longest = max(lengths)
    out = rows.new_zeros((longest, len(lengths)) + tuple(rows.shape[1:]))
    for i, part in enumerate(rows.split(lengths)):
        out[:len(part), i] = part
    return out


def _unpadded(rows, lengths):
    return torch.cat([rows[:n, i] for i, n in enumerate(lengths)])


def _exact_delta(case, seed):
    p, x = _f64(_params(case, _shapes(case), seed)), _inputs(case, seed).double()
    heads, kv, dim, decode = case["heads"], case["kv_heads"], case["dim"], bool(case.get("decode"))
    lengths = _lengths(case)
    held = _held(case, seed) if decode else None
    rows = x @ torch.cat([p["wq"], p["wk"], p["wv"]]).T
    taps = torch.cat([p["conv_q"], p["conv_k"], p["conv_v"]])
    mixed, tails = [], []
    for i, part in enumerate(rows.split(lengths)):
        tail = held[i][1].double() if decode else part.new_zeros(3, part.shape[1])
        line = torch.cat([tail, part])
        tails.append(line[-3:])
        mixed.append(torch.nn.functional.silu(sum(line[j:j + len(part)] * taps[:, j] for j in range(4))))
    q, k, v = torch.cat(mixed).split([kv * dim, kv * dim, heads * dim], dim=1)
    unit = lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = (unit(q.view(-1, kv, dim)) * dim ** -0.5).repeat_interleave(heads // kv, dim=1)
    k = unit(k.view(-1, kv, dim)).repeat_interleave(heads // kv, dim=1)
    b = torch.sigmoid(x @ p["wb"].T)
    inner = torch.nn.functional.softplus((x @ p["decay_in"].T) @ p["decay_out"].T + p["decay_bias"]).view(-1, heads, dim)
    g = torch.exp(-torch.exp(p["decay_log"])[:, None] * inner)
    q, k, v, b, g = (_padded(t, lengths) for t in (q, k, v.view(-1, heads, dim), b, g))
    state = torch.stack([h[0].double() for h in held]) if decode else x.new_zeros(len(lengths), heads, dim, dim)  # [.., value, key]
    outs, ends = [], [None] * len(lengths)
    for t in range(max(lengths)):
        state = state * g[t][:, :, None, :]
        e = b[t][..., None] * (v[t] - torch.einsum("shvk,shk->shv", state, k[t]))
        state = state + e[..., None] * k[t][:, :, None, :]
        outs.append(torch.einsum("shvk,shk->shv", state, q[t]))
        for i, n in enumerate(lengths):
            if n == t + 1:
                ends[i] = state[i]
    o = _unpadded(torch.stack(outs), lengths)
    gate = torch.sigmoid((x @ p["gate_in"].T) @ p["gate_out"].T).view(-1, heads, dim)
    out = (_rms(o, p["out_norm"]) * gate).reshape(-1, heads * dim) @ p["wo"].T
    return {"out": out, "delta": torch.stack(ends), "conv_tail": torch.stack(tails)}


def _exact_latent(case, seed):
    p, x, lengths = _f64(_params(case, _shapes(case), seed)), _inputs(case, seed).double(), _lengths(case)
    heads, dim, rot, rank = case["heads"], case["dim"], case["rot"], case["rank"]
    positions = torch.cat([torch.arange(n, device="cuda") for n in lengths])
    q = (x @ p["wq"].T).view(-1, heads, dim + rot)
    q = torch.cat([q[..., :dim], _rotate(q[..., dim:], positions, 1e6, rot, True)], dim=-1)
    down = x @ p["wdown"].T
    c = _rms(down[:, :rank], p["down_norm"])
    shared = _rotate(down[:, None, rank:], positions, 1e6, rot, True).expand(-1, heads, -1)
    k = torch.cat([(c @ p["wuk"].T).view(-1, heads, dim), shared], dim=-1)
    v = (c @ p["wuv"].T).view(-1, heads, dim)
    parts = zip(*(t.split(lengths) for t in (q, k, v)))
    return {"out": torch.cat([_attend(*part, (dim + rot) ** -0.5, sink=p["sink"]) for part in parts]) @ p["wo"].T}


def _exact_wkv(case, seed):
    p, x, lengths = _f64(_params(case, _shapes(case), seed)), _inputs(case, seed).double(), _lengths(case)
    heads, dim = case["heads"], case["dim"]
    before = torch.cat([torch.cat([part.new_zeros(1, part.shape[1]), part[:-1]]) for part in x.split(lengths)])
    blend = {b: x + (before - x) * p[f"mu_{b}"] for b in "rkvgw"}
    r, k, v = ((blend[b] @ p[f"w{b}"].T).view(-1, heads, dim) for b in "rkv")
    gate = torch.nn.functional.silu(blend["g"] @ p["wg"].T)
    decay = torch.exp(-torch.exp(torch.tanh(blend["w"] @ p["w1"].T) @ p["w2"].T + p["w0"])).view(-1, heads, dim)
    r, k, v, decay = (_padded(t, lengths) for t in (r, k, v, decay))
    state, outs, ends = x.new_zeros(len(lengths), heads, dim, dim), [], [None] * len(lengths)  # [.., key, value]
    for t in range(max(lengths)):
        new = k[t][..., None] * v[t][:, :, None, :]
        outs.append(torch.einsum("shkv,shk->shv", state + p["bonus"][None, :, :, None] * new, r[t]))
        state = decay[t][..., None] * state + new
        for i, n in enumerate(lengths):
            if n == t + 1:
                ends[i] = state[i]
    o = _rms(_unpadded(torch.stack(outs), lengths), 1.0).reshape(-1, heads * dim) * p["out_norm"] * gate
    return {"out": o @ p["wo"].T, "wkv_state": torch.stack(ends), "wkv_last": torch.stack([part[-1] for part in x.split(lengths)])}


def exact(case, seed):
    kind = case["kind"]
    fn = {"reply": _exact_reply, "attention": _exact_attention, "window": _exact_attention, "mlp": _exact_mlp, "delta": _exact_delta,
          "latent": _exact_latent, "experts": _exact_experts, "wkv": _exact_wkv}[kind]
    return fn(case, seed)
