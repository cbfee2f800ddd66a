"""What a serving program has this engine do, as cases that can be timed and checked.

A case is a dict of plain values.  ``prepare`` makes what such a program holds before the call (weights, the request's
cache, the step's metadata, a captured graph for a decode step), ``run`` is one pass through the engine's public entry
points (``LoadedModel.step.run`` for whole steps, ``forward`` of a part for single layers), ``exact`` is the same result in
64 bits by plain torch.  Sizes are those of ``bench.py``: Llama 3.2 1B, and the layer sizes at which the further designs
are compared (width 2,048 / 3,072 / 4,096).  A step of the engine carries up to a few thousand prompt tokens (its token
budget is 2,048 by default) or one token of each of up to 64 requests.
"""
import json
import math
import os
import tempfile

import torch

import atoma_infer_b200  # noqa: F401
from atoma_infer_b200.cache.manager import CacheManager
from atoma_infer_b200.cache.spec import CacheGroup, LayerCache
from atoma_infer_b200.config.registry import part_class
from atoma_infer_b200.engine import StepEntry
from atoma_infer_b200.engine.runtime import load_model, make_runtime
from atoma_infer_b200.engine.step import StepFunction
from atoma_infer_b200.parts.model import DecoderModel, ModelSpec

PAGE = 16
PAST = 100  # tokens that the requests of a recurrent layer's decode case have behind them
DEV = "cuda:0"
# width: (feed-forward, heads, key/value heads, head size)
SIZES = {2048: (8192, 32, 8, 64), 3072: (8192, 24, 8, 128), 4096: (14336, 32, 8, 128)}


def listed():
    return [
        # A whole decode step of the headline model: 8 requests with 2,048 tokens cached, through the captured graph.
        {"name": "decode-step", "kind": "decode_step", "layers": 16, "vocab": 128256, "requests": 8, "context": 2048},
        # A whole prompt step of the same model: three prompts that together fill the token budget, logits of their last rows.
        {"name": "prompt-step", "kind": "prompt_step", "layers": 16, "vocab": 128256, "lengths": "1391,402,255"},
        # Attention layer, prompt: one long prompt at the 8B sizes (heads of 128), all keys.
        {"name": "attention-prompt", "kind": "attention", "dtype": "bfloat16", "width": 4096, "lengths": "4096"},
        # Attention layer, decode: a full batch of 64 requests whose contexts differ.
        {"name": "attention-decode", "kind": "attention", "dtype": "bfloat16", "width": 2048, "requests": 64, "least": 150, "most": 4001},
        # Feed-forward layer in 32 bits: the trace replay's number format, a prompt of odd length.
        {"name": "feed-forward-f32", "kind": "feed_forward", "dtype": "float32", "width": 2048, "lengths": "333"},
        # State-space layer (Tutezen), prompt: a step's whole token budget of one request.
        {"name": "state-space-prompt", "kind": "state_space", "dtype": "bfloat16", "width": 2048, "lengths": "2048"},
        # The same layer, decode: a few requests, where launches and latency count.
        {"name": "state-space-decode", "kind": "state_space", "dtype": "bfloat16", "width": 2048, "requests": 4},
        # Gated linear attention (Bumolix), prompts of several requests side by side, odd lengths.
        {"name": "gated-linear-prompt", "kind": "gated_linear", "dtype": "bfloat16", "width": 2048, "lengths": "1203,640,205"},
        # Selective scan (Bumolix), a step's whole token budget of one request.
        {"name": "selective-scan-prompt", "kind": "selective_scan", "dtype": "bfloat16", "width": 2048, "lengths": "2048"},
        # Matrix memory with exponential gates (Kavotar), two prompts, the wider layer.
        {"name": "matrix-memory-prompt", "kind": "matrix_memory", "dtype": "bfloat16", "width": 3072, "lengths": "1500,548"},
        # Latent attention (Tutezen) inside its window with learned sinks and gate, a long prompt.
        {"name": "latent-prompt", "kind": "latent", "dtype": "bfloat16", "width": 2048, "lengths": "4096"},
        # Routed experts (Tutezen), a prompt step's rows: two of sixteen experts and the shared one.
        {"name": "experts-prompt", "kind": "experts", "dtype": "bfloat16", "width": 2048, "lengths": "2048"},
    ]


def draw(rng):
    """Sizes are spread over the logarithm; lengths are odd as often as not."""
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def lengths(least, most, parts=4):
        n = rng.choice(range(1, parts + 1))
        total = log(max(least, 16 * n), most)
        cuts = sorted(rng.sample(range(1, total), n - 1))
        return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))

    kind = rng.choice(["decode_step", "prompt_step", "attention", "attention", "feed_forward", "state_space", "state_space", "gated_linear",
                       "selective_scan", "matrix_memory", "latent", "experts"])
    if kind == "decode_step":
        return {"kind": kind, "layers": rng.choice([2, 4, 8]), "vocab": 32768, "requests": log(1, 64), "context": log(100, 3000)}
    if kind == "prompt_step":
        return {"kind": kind, "layers": rng.choice([2, 4, 8]), "vocab": 32768, "lengths": lengths(64, 2048)}
    case = {"kind": kind, "dtype": "bfloat16", "width": rng.choice([2048, 3072, 4096] if kind != "experts" else [2048, 3072])}
    decode = rng.random() < 0.3
    if kind == "feed_forward":
        case["dtype"] = rng.choice(["float32", "bfloat16"])
        case["lengths"] = lengths(17, 700 if case["dtype"] == "float32" else 2048)
        if case["dtype"] == "float32":
            case["width"] = 2048
    elif kind == "attention" and decode:
        most = log(300, 4000)
        case.update(requests=log(1, 64), least=max(1, most // rng.choice([1, 4, 20])), most=most)
    elif kind == "state_space" and decode:
        case["requests"] = log(1, 64)
    else:
        case["lengths"] = lengths(130, 4096 if kind in ("attention", "latent") else 3000)
    return case


# ----------------------------------------------------------------------------- inputs, from the seed alone
class Draw:
    """Numbers on the GPU from one seed, in the order in which they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        t = torch.empty(shape, dtype=torch.float32, device=DEV)
        return t.normal_(mean, std, generator=self.g).to(dtype)

    def uniform(self, a, b, *shape, dtype=torch.float32):
        return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(a, b, generator=self.g).to(dtype)

    def ints(self, n, high):
        return torch.randint(0, high, (n,), generator=self.g, device=DEV).tolist()


def lengths_of(case):
    return [int(n) for n in str(case["lengths"]).split(",")] if "lengths" in case else [1] * int(case["requests"])


def contexts_of(case):
    """Tokens a request of a decode case has cached: evenly spread from ``least`` to ``most``."""
    n, a, b = int(case["requests"]), int(case["least"]), int(case["most"])
    return [a + (b - a) * i // max(n - 1, 1) for i in range(n)]


def dtype_of(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def part_of(case):
    """(part family, part kind, its parameters, its tensors by name: shape and how they are drawn)."""
    H = int(case["width"])
    F, nq, nkv, d = SIZES[H]
    w = ("normal", 0.02)
    if case["kind"] == "attention":
        params = {"hidden": H, "num_heads": nq, "num_kv_heads": nkv, "head_dim": d, "scale": d ** -0.5, "window": None,
                  "position": {"kind": "rope", "head_dim": d, "theta": 500000.0, "scaling": None}}
        return "mixer", "attention", params, {".q_proj.weight": ((nq * d, H), w), ".k_proj.weight": ((nkv * d, H), w),
                                              ".v_proj.weight": ((nkv * d, H), w), ".o_proj.weight": ((H, nq * d), w)}
    if case["kind"] == "feed_forward":
        return "feed_forward", "swiglu", {"hidden": H, "intermediate": F}, {
            ".gate_proj.weight": ((F, H), w), ".up_proj.weight": ((F, H), w), ".down_proj.weight": ((H, F), w)}
    if case["kind"] == "state_space":
        heads, P, N, G, taps = 2 * H // 64, 64, 128, 8, 4
        inner, ch = heads * P, heads * P + 2 * G * N
        params = {"hidden": H, "heads": heads, "head_dim": P, "state": N, "groups": G, "taps": taps, "norm_groups": 8, "eps": 1e-5}
        return "mixer", "mamba2", params, {
            ".in": ((inner + ch + heads, H), w), ".conv": ((ch, taps), ("normal", 0.3)), ".conv.b": ((ch,), ("normal", 0.1)),
            # step sizes of a hundredth to a few tenths, decay rates of 1 to 16: memories of a few to hundreds of tokens
            ".dt_bias": ((heads,), ("uniform", -4.6, -1.0)), ".A_log": ((heads,), ("uniform", 0.0, 2.77)),
            ".D": ((heads,), ("ones", 0.1)), ".norm": ((inner,), ("ones", 0.1)), ".o": ((H, inner), w)}
    if case["kind"] == "gated_linear":
        heads, N, P, rank = H // 256, 128, 256, 16
        params = {"hidden": H, "heads": heads, "dim": N, "vdim": P, "tau": 8.0, "rank": rank, "eps": 1e-5}
        return "mixer", "gated_linear_attention", params, {
            ".q": ((heads * N, H), w), ".k": ((heads * N, H), w), ".v": ((heads * P, H), w), ".g": ((heads * P, H), w),
            ".o": ((H, heads * P), w), ".norm": ((P,), ("ones", 0.1)), ".a1": ((rank, H), w), ".a2": ((heads * N, rank), ("normal", 0.25)),
            ".a2.b": ((heads * N,), ("normal", 1.0, 1.0))}
    if case["kind"] == "selective_scan":
        inner, N, rank, taps = 2 * H, 16, H // 16, 4
        params = {"hidden": H, "inner": inner, "state": N, "dt_rank": rank, "taps": taps}
        return "mixer", "selective_scan", params, {
            ".in": ((2 * inner, H), w), ".conv": ((inner, taps), ("normal", 0.3)), ".conv.b": ((inner,), ("normal", 0.1)),
            ".x": ((rank + 2 * N, inner), w), ".dt": ((inner, rank), ("normal", rank ** -0.5)),
            ".dt.b": ((inner,), ("uniform", -4.6, -1.0)), ".A_log": ((inner, N), ("uniform", 0.0, 2.77)), ".D": ((inner,), ("ones", 0.1)),
            ".o": ((H, inner), w)}
    if case["kind"] == "matrix_memory":
        heads, N, P = H // 256, 128, 256
        params = {"hidden": H, "heads": heads, "dim": N, "vdim": P, "gate_cap": 15.0, "eps": 1e-5}
        return "mixer", "matrix_memory", params, {
            ".q": ((heads * N, H), w), ".k": ((heads * N, H), w), ".v": ((heads * P, H), w), ".g": ((heads * P, H), w),
            ".o": ((H, heads * P), w), ".norm": ((heads * P,), ("ones", 0.1)), ".i": ((heads, H), w), ".f": ((heads, H), w),
            # forget gates near one, so that a memory spans tens to hundreds of tokens
            ".i.b": ((heads,), ("normal", 0.1)), ".f.b": ((heads,), ("uniform", 3.0, 6.0))}
    if case["kind"] == "latent":
        heads, rot, kv, qr = 16, 32, 224, H // 4
        params = {"hidden": H, "heads": heads, "dim": d, "rot_dim": rot, "v_head_dim": d, "q_rank": qr, "kv_rank": kv,
                  "scale": (d + rot) ** -0.5, "window": 1024, "rotary_dims": rot, "theta": 500000.0, "eps": 1e-5, "sink": True, "gate": True}
        return "mixer", "latent_attention", params, {
            ".dq": ((qr, H), w), ".dq.norm": ((qr,), ("ones", 0.1)), ".uq": ((heads * (d + rot), qr), ("normal", qr ** -0.5)),
            ".dkv": ((kv + rot, H), w), ".dkv.norm": ((kv,), ("ones", 0.1)), ".uk": ((heads * d, kv), ("normal", kv ** -0.5)),
            ".uv": ((heads * d, kv), ("normal", kv ** -0.5)), ".o": ((H, heads * d), w), ".sink": ((heads,), ("normal", 1.0)),
            ".g": ((heads * d, H), w)}
    if case["kind"] == "experts":
        E, top, f = 16, 2, F // 4
        params = {"hidden": H, "experts": E, "top": top, "intermediate": f, "shared_intermediate": f}
        tensors = {".router": ((E, H), w)}
        for stem in [f".e{j}" for j in range(E)] + [".shared"]:
            tensors.update({stem + ".gate": ((f, H), w), stem + ".up": ((f, H), w), stem + ".down": ((H, f), w)})
        return "feed_forward", "routed_experts", params, tensors
    raise ValueError(case["kind"])


def layer_inputs(case, seed):
    """A layer's tensors by name and its input rows (rows of a norm: mean square 1), in the case's type."""
    dr, dt = Draw(seed), dtype_of(case)
    tensors = {}
    for name, (shape, how) in part_of(case)[3].items():
        if how[0] == "normal":
            tensors[name] = dr.normal(*shape, std=how[1], mean=how[2] if len(how) > 2 else 0.0, dtype=dt)
        elif how[0] == "ones":
            tensors[name] = dr.normal(*shape, std=how[1], mean=1.0, dtype=dt)
        else:
            tensors[name] = dr.uniform(how[1], how[2], *shape, dtype=dt)
    x = dr.normal(sum(lengths_of(case)), int(case["width"]), dtype=dt)
    return dr, tensors, x


def cached_pages(case, dr):
    """Keys and values of a decode case as whole pages, one tensor [pages, 2, key heads, page, head size] per request."""
    _, _, nkv, d = SIZES[int(case["width"])]
    return [dr.normal(-(-c // PAGE), 2, nkv, PAGE, d, dtype=dtype_of(case)) for c in contexts_of(case)]


def kept_state(case, dr, floats):
    """The per-request state of a decode case, as a scan of normed rows leaves it (numbers of about a half)."""
    return dr.normal(int(case["requests"]), floats, std=0.5)


# ----------------------------------------------------------------------------- single layers
class Layer:
    """A part bound to its tensors, the step's metadata and the request's cache, as the engine holds them."""

    def __init__(self, case, seed):
        family, kind, params, _ = part_of(case)
        dr, tensors, self.x = layer_inputs(case, seed)
        self.family, self.decode = family, "lengths" not in case
        self.rt = make_runtime(case["dtype"], DEV)
        self.part = part_class(family, kind)(params, "p")
        self.part.bind({"p" + n: t for n, t in tensors.items()}, self.rt)
        self.rt.ops.set_weight_order(self.part.streamed_weights())
        lens = lengths_of(case)
        past = contexts_of(case) if "least" in case else [PAST if self.decode else 0] * len(lens)
        need = self.part.cache_need() if family == "mixer" else None
        groups = [CacheGroup(need)] if need is not None else []
        for g in groups:
            g.layers.append(0)
            g.num_pages = 1 + sum(-(-(c + n) // PAGE) for c, n in zip(past, lens))
        model = DecoderModel(ModelSpec(hidden_size=int(case["width"]), vocab_size=16, layers=[],
                                       final_norm={"kind": "rmsnorm", "size": int(case["width"]), "eps": 1e-5}))
        self.manager = CacheManager(PAGE, groups, len(lens))
        self.step = StepFunction(model, None, self.manager, self.rt)
        for r, c in enumerate(past):
            if c:
                self.step.prepare([StepEntry(r, [0] * c)])
                self.manager.advance(r, c)
        host, lay, infos, _ = self.step.prepare([StepEntry(r, [0] * n) for r, n in enumerate(lens)])
        self.meta = host.to(DEV)
        self.ctx = self.step.context(self.meta, lay, infos)
        self.slots = [i.state_slot for i in infos]
        pages = state = None
        if groups:
            pages = torch.zeros((groups[0].num_pages, 2, need.num_kv_heads, PAGE, need.head_dim), dtype=self.rt.dtype, device=DEV)
            if "least" in case:
                for r, kv in enumerate(cached_pages(case, dr)):
                    pages[torch.tensor(self.manager.table(r)[:kv.shape[0]], device=DEV)] = kv
        nbytes = self.part.state_bytes() if family == "mixer" else 0
        if nbytes:
            if self.slots != list(range(len(lens))):
                raise RuntimeError("requests are expected in the order of their state slots")
            state = kept_state(case, dr, nbytes // 4) if self.decode else torch.zeros((len(lens), nbytes // 4), device=DEV)
            state = state.view(torch.uint8)
        self.state = state
        self.cache = LayerCache(group=0 if groups else -1, pages=pages, num_pages=groups[0].num_pages if groups else 0, page_size=PAGE,
                                writes=bool(groups), state=state)
        self.graph = None
        if self.decode:  # the engine runs decode steps as captured graphs
            keep = state.clone() if state is not None else None
            self.forward()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                self.y = self.forward()
            if keep is not None:
                state.copy_(keep)
            self.graph = graph

    def forward(self):
        self.ctx.shared.clear()
        y = self.part.forward(self.x, self.ctx, self.cache) if self.family == "mixer" else self.part.forward(self.x, self.ctx)
        self.rt.ops.join_side_work()
        return y

    def run(self):
        if self.graph is not None:
            self.graph.replay()
            y = self.y
        else:
            if self.state is not None:  # new requests start from a zero state
                for s in self.slots:
                    self.state[s].zero_()
            y = self.forward()
        return (y,) if self.state is None else (y, self.state.view(torch.float32))


# ----------------------------------------------------------------------------- whole steps of the headline model
def model_config(case):
    F, nq, nkv, d = SIZES[2048]
    return {"architectures": ["LlamaForCausalLM"], "hidden_size": 2048, "intermediate_size": F, "vocab_size": int(case["vocab"]),
            "num_hidden_layers": int(case["layers"]), "num_attention_heads": nq, "num_key_value_heads": nkv, "head_dim": d,
            "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "max_position_embeddings": 131072, "tie_word_embeddings": True}


def model_tensors(case, dr):
    cfg, t = model_config(case), {}
    H, F, nq, nkv, d = 2048, cfg["intermediate_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    bf = torch.bfloat16
    t["model.embed_tokens.weight"] = dr.normal(cfg["vocab_size"], H, std=0.02, dtype=bf)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (nq * d, H)), ("self_attn.k_proj", (nkv * d, H)), ("self_attn.v_proj", (nkv * d, H)),
                            ("self_attn.o_proj", (H, nq * d)), ("mlp.gate_proj", (F, H)), ("mlp.up_proj", (F, H)), ("mlp.down_proj", (H, F))):
            t[p + name + ".weight"] = dr.normal(*shape, std=0.02, dtype=bf)
        for name in ("input_layernorm", "post_attention_layernorm"):
            t[p + name + ".weight"] = dr.normal(H, std=0.1, mean=1.0, dtype=bf)
    t["model.norm.weight"] = dr.normal(H, std=0.1, mean=1.0, dtype=bf)
    return t


def step_tokens(case, dr):
    """Prompt tokens per request, and for a decode case the tokens of the steps before the first pass and of every pass."""
    V = int(case["vocab"])
    if case["kind"] == "prompt_step":
        return [dr.ints(n, V) for n in lengths_of(case)], None
    n = int(case["requests"])
    return [dr.ints(int(case["context"]), V) for _ in range(n)], dr.ints(n, V)


class Model:
    def __init__(self, case, seed):
        dr = Draw(seed)
        tensors = model_tensors(case, dr)
        self.prompts, self.next = step_tokens(case, dr)
        room = 0 if self.next is None else 4000  # a decode case's requests grow by a token a pass
        pages = sum(-(-(len(p) + 2 + room) // PAGE) for p in self.prompts) + 8
        with tempfile.TemporaryDirectory() as tmp:
            with open(os.path.join(tmp, "config.json"), "w") as f:
                json.dump(model_config(case), f)
            self.lm = load_model(tmp, dtype="bfloat16", page_size=PAGE, num_pages=pages, max_seqs=len(self.prompts), cuda_graphs=True,
                                 random_weights_seed=0)
        self.lm.model.bind(tensors, self.lm.rt)
        self.calls = 0
        if self.next is not None:
            for r, p in enumerate(self.prompts):
                self.lm.step.run([StepEntry(r, p)])
            for _ in range(2):  # the first step of a batch size runs kernel by kernel, the second is captured
                self.run()

    def run(self):
        if self.next is None:
            ids = [self.calls * len(self.prompts) + i for i in range(len(self.prompts))]
            self.calls += 1
            out = self.lm.step.run([StepEntry(r, p, [len(p) - 1]) for r, p in zip(ids, self.prompts)])
            for r in ids:
                self.lm.step.finish(r)
            return (out,)
        return (self.lm.step.run([StepEntry(r, [t], [0]) for r, t in enumerate(self.next)]),)


def prepare(case, seed):
    return Model(case, seed) if case["kind"] in ("decode_step", "prompt_step") else Layer(case, seed)


def run(state):
    return state.run()


# ----------------------------------------------------------------------------- what a pass cannot do without
def pairs_of(lens, past, window=0):
    """(query, key) pairs of causal attention over what the requests have cached and bring."""
    total = 0
    for n, c in zip(lens, past):
        if window:
            total += sum(min(c + i + 1, window) for i in range(n))
        else:
            total += n * c + n * (n + 1) // 2
    return total


def work(case):
    if case["kind"] in ("decode_step", "prompt_step"):
        F, nq, nkv, d = SIZES[2048]
        H, V, L = 2048, int(case["vocab"]), int(case["layers"])
        per_layer = H * (nq + 2 * nkv) * d + nq * d * H + 3 * H * F
        decode = case["kind"] == "decode_step"
        lens = [1] * int(case["requests"]) if decode else lengths_of(case)
        past = [int(case["context"]) + 2] * len(lens) if decode else [0] * len(lens)
        T, rows = sum(lens), len(lens)
        kv = 2 * nkv * d * 2 * L
        return {"bytes": 2 * (L * per_layer + V * H) + T * H * 2 + kv * (sum(past) + T) + rows * V * 4,
                "flops": 2 * T * L * per_layer + 2 * rows * V * H + 4 * d * nq * L * pairs_of(lens, past)}
    H, lens = int(case["width"]), lengths_of(case)
    F, nq, nkv, d = SIZES[H]
    T, e = sum(lens), 4 if case["dtype"] == "float32" else 2
    _, _, params, tensors = part_of(case)
    params_n = sum(math.prod(shape) for shape, _ in tensors.values())
    matrices = sum(math.prod(shape) for shape, _ in tensors.values() if len(shape) == 2 and min(shape) > 4)
    b, f = e * params_n + 2 * e * T * H, 2 * T * matrices
    if case["kind"] == "attention":
        past = contexts_of(case) if "least" in case else [0] * len(lens)
        b += 2 * nkv * d * e * (sum(past) + T)
        f += 4 * d * nq * pairs_of(lens, past)
    elif case["kind"] == "latent":
        b += 2 * (params["kv_rank"] + params["rot_dim"]) * e * T
        # scores and values in the latent's size, as the layer defines them per head: dim + rot_dim and v_head_dim
        f += 2 * (2 * d + params["rot_dim"]) * params["heads"] * pairs_of(lens, [0] * len(lens), params["window"])
    elif case["kind"] == "experts":
        E, top, f1 = params["experts"], params["top"], params["intermediate"]
        used = min(E, top * T)
        b = e * (E * H + (used + 1) * 3 * f1 * H) + 2 * e * T * H
        f = 2 * T * (E * H + (top + 1) * 3 * f1 * H)
    elif case["kind"] == "state_space":
        N, P, heads = params["state"], params["head_dim"], params["heads"]
        b += 2 * 4 * len(lens) * heads * N * P
        f += 2 * 2 * T * heads * N * P + 2 * T * params["taps"] * (heads * P + 2 * params["groups"] * N)
    elif case["kind"] in ("gated_linear", "matrix_memory"):
        N, P, heads = params["dim"], params["vdim"], params["heads"]
        b += 4 * len(lens) * heads * N * P
        f += 2 * 2 * T * heads * N * P
    elif case["kind"] == "selective_scan":
        b += 4 * len(lens) * params["inner"] * params["state"]
        f += 2 * 2 * T * params["inner"] * params["state"] + 2 * T * params["taps"] * params["inner"]
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case["kind"] in ("decode_step", "prompt_step"):
        # 16 layers of bfloat16 rows: a change of one rounding travels through all that follow
        return {"rel": 5e-2}
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 1.5e-2}


# ----------------------------------------------------------------------------- the same in 64 bits, by plain torch
def rms(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def sigmoid(v):
    return 1 / (1 + torch.exp(-v))


def silu(v):
    return v * sigmoid(v)


def softplus(v):
    return torch.where(v > 30, v, torch.log1p(torch.exp(v.clamp(max=30))))


def rotate_halves(v, positions, theta):
    """Dimension i turns with i + size / 2; v [tokens, heads, size]."""
    d = v.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, dtype=torch.float64, device=v.device) / d)
    ang = positions.double()[:, None, None] * inv
    a, b = v[..., :d // 2], v[..., d // 2:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def rotate_pairs(v, positions, theta):
    """Dimension 2i turns with 2i + 1."""
    d = v.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, dtype=torch.float64, device=v.device) / d)
    ang = positions.double().view(-1, *([1] * (v.dim() - 1))) * inv
    a, b = v[..., 0::2], v[..., 1::2]
    return torch.stack([a * ang.cos() - b * ang.sin(), a * ang.sin() + b * ang.cos()], -1).flatten(-2)


def softmax_attention(q, k, v, scale, start, window=0, sink=None, block=512):
    """q [n, heads, d] of positions start .., k and v [start + n, heads, d]; queries a block at a time."""
    out = []
    j = torch.arange(k.shape[0], device=q.device)
    for a in range(0, q.shape[0], block):
        i = start + torch.arange(a, min(a + block, q.shape[0]), device=q.device)
        s = torch.einsum("ihd,jhd->hij", q[a:a + block], k) * scale
        hidden = j[None, :] > i[:, None]
        if window:
            hidden |= j[None, :] <= i[:, None] - window
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], -1)
        p = torch.softmax(s, -1)[..., :k.shape[0]]
        out.append(torch.einsum("hij,jhd->ihd", p, v))
    return torch.cat(out)


def exact_attention(case, t, x, lens, past, kv):
    H = int(case["width"])
    _, nq, nkv, d = SIZES[H]
    out, at = [], 0
    for r, (n, c) in enumerate(zip(lens, past)):
        rows, at = x[at:at + n], at + n
        pos = torch.arange(c, c + n, device=x.device)
        q = rotate_halves((rows @ t[".q_proj.weight"].T).view(n, nq, d), pos, 500000.0)
        k = rotate_halves((rows @ t[".k_proj.weight"].T).view(n, nkv, d), pos, 500000.0)
        v = (rows @ t[".v_proj.weight"].T).view(n, nkv, d)
        if c:
            old = kv[r].double().permute(1, 0, 3, 2, 4).reshape(2, -1, nkv, d)[:, :c]
            k, v = torch.cat([old[0], k]), torch.cat([old[1], v])
        o = softmax_attention(q, k.repeat_interleave(nq // nkv, 1), v.repeat_interleave(nq // nkv, 1), d ** -0.5, c)
        out.append(o.reshape(n, nq * d) @ t[".o_proj.weight"].T)
    return torch.cat(out)


def convolved(u, w, b, ring, taps):
    """A causal convolution over time on every channel; ring: the rows of positions -(taps - 1) .. -1."""
    full = torch.cat([ring, u])
    return silu(b + sum(w[:, j] * full[j:j + u.shape[0]] for j in range(taps))), full[-(taps - 1):]


def ring_places(rows, end, taps):
    """The last rows as the state keeps them: the row of position p at place p mod (taps - 1)."""
    out = torch.zeros_like(rows)
    for k in range(taps - 1):
        out[(end - (taps - 1) + k) % (taps - 1)] = rows[k]
    return out


def exact_state_space(case, p, t, x, lens, state):
    heads, P, N, G, taps = p["heads"], p["head_dim"], p["state"], p["groups"], p["taps"]
    inner, ch = heads * P, heads * P + 2 * G * N
    proj = x @ t[".in"].T
    ring_floats = -(-(taps - 1) * ch // 4) * 4
    ys, states, at = [], [], 0
    for r, n in enumerate(lens):
        rows, at = proj[at:at + n], at + n
        z, u, dt = rows[:, :inner], rows[:, inner:inner + ch], softplus(rows[:, inner + ch:] + t[".dt_bias"])
        past = 0 if state is None else PAST
        if state is None:
            places, S = torch.zeros(taps - 1, ch, dtype=u.dtype, device=u.device), torch.zeros(heads, N, P, dtype=u.dtype, device=u.device)
        else:
            places = state[r, :(taps - 1) * ch].view(taps - 1, ch).double().clone()
            S = state[r, ring_floats:].view(heads, N, P).double().clone()
        ring = torch.stack([places[(past - (taps - 1) + k) % (taps - 1)] for k in range(taps - 1)])
        xbc, last = convolved(u, t[".conv"], t[".conv.b"], ring, taps)
        xs = xbc[:, :inner].view(n, heads, P)
        B = xbc[:, inner:inner + G * N].view(n, G, N).repeat_interleave(heads // G, 1)
        C = xbc[:, inner + G * N:].view(n, G, N).repeat_interleave(heads // G, 1)
        decay = torch.exp(-torch.exp(t[".A_log"]) * dt)
        y = torch.empty(n, heads, P, dtype=u.dtype, device=u.device)
        dx = dt[..., None] * xs
        for i in range(n):
            S = decay[i][:, None, None] * S + B[i][:, :, None] * dx[i][:, None, :]
            y[i] = torch.einsum("hnp,hn->hp", S, C[i])
        y = (y + t[".D"][:, None] * xs).reshape(n, inner) * silu(z)
        y = rms(y.view(n, p["norm_groups"], -1), p["eps"]).reshape(n, inner) * t[".norm"]
        ys.append(y @ t[".o"].T)
        kept = torch.zeros(ring_floats + heads * N * P, dtype=u.dtype, device=u.device)
        kept[:(taps - 1) * ch] = ring_places(last, past + n, taps).reshape(-1)
        kept[ring_floats:] = S.reshape(-1)
        states.append(kept)
    return torch.cat(ys), torch.stack(states)


def exact_gated_linear(p, t, x, lens):
    heads, N, P = p["heads"], p["dim"], p["vdim"]
    ys, states, at = [], [], 0
    for n in lens:
        rows, at = x[at:at + n], at + n
        q = (rows @ t[".q"].T).view(n, heads, N) * N ** -0.5
        k, v = (rows @ t[".k"].T).view(n, heads, N), (rows @ t[".v"].T).view(n, heads, P)
        z = ((rows @ t[".a1"].T) @ t[".a2"].T + t[".a2.b"]).view(n, heads, N)
        a = torch.exp(-softplus(-z) / p["tau"])
        S = torch.zeros(heads, N, P, dtype=x.dtype, device=x.device)
        o = torch.empty(n, heads, P, dtype=x.dtype, device=x.device)
        for i in range(n):
            S = a[i][:, :, None] * S + k[i][:, :, None] * v[i][:, None, :]
            o[i] = torch.einsum("hnp,hn->hp", S, q[i])
        o = (rms(o, p["eps"]) * t[".norm"]).reshape(n, heads * P) * silu(rows @ t[".g"].T)
        ys.append(o @ t[".o"].T)
        states.append(S.reshape(-1))
    return torch.cat(ys), torch.stack(states)


def exact_matrix_memory(p, t, x, lens):
    heads, N, P, cap = p["heads"], p["dim"], p["vdim"], p["gate_cap"]
    ys, states, at = [], [], 0
    for n in lens:
        rows, at = x[at:at + n], at + n
        q = (rows @ t[".q"].T).view(n, heads, N) * N ** -0.5
        k, v = (rows @ t[".k"].T).view(n, heads, N), (rows @ t[".v"].T).view(n, heads, P)
        i_g = cap * torch.tanh((rows @ t[".i"].T + t[".i.b"]) / cap)
        f_g = -softplus(-cap * torch.tanh((rows @ t[".f"].T + t[".f.b"]) / cap))
        S, nn = torch.zeros(heads, N, P, dtype=x.dtype, device=x.device), torch.zeros(heads, N, dtype=x.dtype, device=x.device)
        m = torch.zeros(heads, dtype=x.dtype, device=x.device)
        o = torch.empty(n, heads, P, dtype=x.dtype, device=x.device)
        for i in range(n):
            m_new = torch.maximum(f_g[i] + m, i_g[i])
            a, b = torch.exp(f_g[i] + m - m_new), torch.exp(i_g[i] - m_new)
            m = m_new
            S = a[:, None, None] * S + (b[:, None] * k[i])[:, :, None] * v[i][:, None, :]
            nn = a[:, None] * nn + b[:, None] * k[i]
            nq = (nn * q[i]).sum(-1).abs()
            o[i] = torch.einsum("hnp,hn->hp", S, q[i]) / (torch.maximum(nq, torch.exp(-m)) + 1e-6)[:, None]
        y = rms(o, p["eps"]).reshape(n, heads * P) * t[".norm"] * sigmoid(rows @ t[".g"].T)
        ys.append(y @ t[".o"].T)
        up = lambda v: torch.nn.functional.pad(v.reshape(-1), (0, -v.numel() % 4))  # noqa: E731
        states.append(torch.cat([up(S), up(nn), up(m)]))
    return torch.cat(ys), torch.stack(states)


def exact_selective_scan(p, t, x, lens):
    inner, N, rank, taps = p["inner"], p["state"], p["dt_rank"], p["taps"]
    proj, A = x @ t[".in"].T, -torch.exp(t[".A_log"])
    ring_floats = -(-(taps - 1) * inner // 4) * 4
    ys, states, at = [], [], 0
    for n in lens:
        rows, at = proj[at:at + n], at + n
        u, last = convolved(rows[:, :inner], t[".conv"], t[".conv.b"], torch.zeros(taps - 1, inner, dtype=x.dtype, device=x.device), taps)
        low = u @ t[".x"].T
        dt = softplus(low[:, :rank] @ t[".dt"].T + t[".dt.b"])
        B, C = low[:, rank:rank + N], low[:, rank + N:]
        S = torch.zeros(inner, N, dtype=x.dtype, device=x.device)
        y = torch.empty(n, inner, dtype=x.dtype, device=x.device)
        for i in range(n):
            S = torch.exp(dt[i][:, None] * A) * S + (dt[i] * u[i])[:, None] * B[i]
            y[i] = S @ C[i]
        y = (y + t[".D"] * u) * silu(rows[:, inner:])
        ys.append(y @ t[".o"].T)
        kept = torch.zeros(ring_floats + inner * N, dtype=x.dtype, device=x.device)
        kept[:(taps - 1) * inner] = ring_places(last, n, taps).reshape(-1)
        kept[ring_floats:] = S.reshape(-1)
        states.append(kept)
    return torch.cat(ys), torch.stack(states)


def exact_latent(p, t, x, lens):
    Hh, d, rot, dv, kv, eps = p["heads"], p["dim"], p["rot_dim"], p["v_head_dim"], p["kv_rank"], p["eps"]
    out, at = [], 0
    for n in lens:
        rows, at = x[at:at + n], at + n
        pos = torch.arange(n, device=x.device)
        q = (rms(rows @ t[".dq"].T, eps) * t[".dq.norm"] @ t[".uq"].T).view(n, Hh, d + rot)
        low = rows @ t[".dkv"].T
        c = rms(low[:, :kv], eps) * t[".dkv.norm"]
        k_rot = rotate_pairs(low[:, kv:], pos, p["theta"])
        q_rot = rotate_pairs(q[..., d:], pos, p["theta"])
        k = torch.cat([(c @ t[".uk"].T).view(n, Hh, d), k_rot[:, None].expand(n, Hh, rot)], -1)
        v = (c @ t[".uv"].T).view(n, Hh, dv)
        o = softmax_attention(torch.cat([q[..., :d], q_rot], -1), k, v, p["scale"], 0, p["window"], t[".sink"])
        out.append((o.reshape(n, Hh * dv) * sigmoid(rows @ t[".g"].T)) @ t[".o"].T)
    return torch.cat(out)


def exact_experts(p, t, x):
    one = lambda h, stem: (silu(h @ t[stem + ".gate"].T) * (h @ t[stem + ".up"].T)) @ t[stem + ".down"].T  # noqa: E731
    s = torch.softmax(x @ t[".router"].T, -1)
    w, ids = s.topk(p["top"], -1)
    w = w / (w.sum(-1, keepdim=True) + 1e-20)
    y = one(x, ".shared")
    for j in range(p["experts"]):
        rows, which = (ids == j).nonzero(as_tuple=True)
        if rows.numel():
            y[rows] += w[rows, which][:, None] * one(x[rows], f".e{j}")
    return y


def exact_model(case, seed):
    dr = Draw(seed)
    tensors = model_tensors(case, dr)
    prompts, nxt = step_tokens(case, dr)
    if nxt is not None and len(prompts) * len(prompts[0]) * int(case["layers"]) > 8 * 2100 * 16:
        return None  # (minutes in 64 bits)
    cfg = model_config(case)
    nq, nkv, d, H = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], 2048
    seqs = [p if nxt is None else p + [nxt[r]] * 3 for r, p in enumerate(prompts)]
    lens = [len(s) for s in seqs]
    w = lambda name: tensors[name].double()  # noqa: E731
    h = tensors["model.embed_tokens.weight"][torch.tensor([x for s in seqs for x in s], device=DEV)].double()
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        a = rms(h, 1e-5) * w(p + "input_layernorm.weight")
        q = rotate_halves((a @ w(p + "self_attn.q_proj.weight").T).view(-1, nq, d), pos, 500000.0)
        k = rotate_halves((a @ w(p + "self_attn.k_proj.weight").T).view(-1, nkv, d), pos, 500000.0)
        v = (a @ w(p + "self_attn.v_proj.weight").T).view(-1, nkv, d)
        o, at = [], 0
        for n in lens:
            part = slice(at, at + n)
            o.append(softmax_attention(q[part], k[part].repeat_interleave(nq // nkv, 1), v[part].repeat_interleave(nq // nkv, 1), d ** -0.5, 0))
            at += n
        h = h + torch.cat(o).reshape(-1, nq * d) @ w(p + "self_attn.o_proj.weight").T
        a = rms(h, 1e-5) * w(p + "post_attention_layernorm.weight")
        h = h + (silu(a @ w(p + "mlp.gate_proj.weight").T) * (a @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
    last = torch.tensor(lens, device=DEV).cumsum(0) - 1
    return (rms(h[last], 1e-5) * w("model.norm.weight")) @ w("model.embed_tokens.weight").T


def exact(case, seed):
    if case["kind"] in ("decode_step", "prompt_step"):
        y = exact_model(case, seed)
        return None if y is None else (y,)
    dr, tensors, x = layer_inputs(case, seed)
    t, x, lens, p = {k: v.double() for k, v in tensors.items()}, x.double(), lengths_of(case), part_of(case)[2]
    if case["kind"] == "attention":
        past = contexts_of(case) if "least" in case else [0] * len(lens)
        return (exact_attention(case, t, x, lens, past, cached_pages(case, dr) if "least" in case else None),)
    if case["kind"] == "feed_forward":
        return ((silu(x @ t[".gate_proj.weight"].T) * (x @ t[".up_proj.weight"].T)) @ t[".down_proj.weight"].T,)
    if case["kind"] == "state_space":
        state = None
        if "lengths" not in case:
            ch = p["heads"] * p["head_dim"] + 2 * p["groups"] * p["state"]
            ring_floats = -(-(p["taps"] - 1) * ch // 4) * 4
            state = kept_state(case, dr, ring_floats + p["heads"] * p["state"] * p["head_dim"])
        return exact_state_space(case, p, t, x, lens, state)
    if case["kind"] == "gated_linear":
        return exact_gated_linear(p, t, x, lens)
    if case["kind"] == "selective_scan":
        return exact_selective_scan(p, t, x, lens)
    if case["kind"] == "matrix_memory":
        return exact_matrix_memory(p, t, x, lens)
    if case["kind"] == "latent":
        return (exact_latent(p, t, x, lens),)
    return (exact_experts(p, t, x),)
