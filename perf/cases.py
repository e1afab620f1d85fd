"""The work whose speed this framework is judged by.

Each case is one pass through a public entry point: a layer (``Block.forward``), a sublayer
(``Mixer.forward`` / ``FeedForward.forward``), the vocabulary head with sampling
(``CudaOps.linear`` and ``CudaOps.sample``), or a whole model (``Runner.step``).  Layers and
sublayers are captured in a CUDA graph once, as the engine captures its steps, and a pass replays
it.  Sizes are those of the model presets (GPT-2 small to XL, ``pedorax-1k``/``-2k``,
``mafuzen-1k``/``-2k``) and of ``bench.py``.

Kinds:

``block``      pre-norm GPT-2 layers over the paged cache: LayerNorm, QKV, append, attention,
               projection, LayerNorm, feed-forward.  ``decode`` single tokens behind ``context``
               cached ones, ``portions`` prompt portions of ``portion`` tokens behind ``prefix``.
``head``       logits of ``rows`` hidden rows over the vocabulary, then one token a row (greedy,
               with a temperature, with a temperature and top-k in turn).
``experts``    routed feed-forward: router, choice within groups, experts, weighted sum.
``latent``     attention over a shared latent with a sink per head.
``delta``      gated delta rule with a decay per key channel.
``retention``  linear attention with a fixed decay per head and rotary positions.
``replay``     a model over given token ids: all prompts as one step, then ``new`` decode steps.

With ``ragged`` lengths spread between half and one and a half times the stated one.
"""

from __future__ import annotations

import math

import torch

from hetero_serve_b200 import architectures  # noqa: F401  (registers the architectures)
from hetero_serve_b200.architectures.gpt2 import GPT2Config, build_spec
from hetero_serve_b200.engine import Runner, StepEntry
from hetero_serve_b200.engine.step import CacheView
from hetero_serve_b200.kernels.ops import CudaOps
from hetero_serve_b200.parts import LayerSpec, Model, PartSpec, PreNormBlock, build_part

PAGE = 16
POSITIONS = 1024                # of the GPT-2 family
EPS = 1e-5
VOCAB = 50257
GPT2_SIZES = {768: 12, 1024: 16, 1280: 20, 1600: 25}       # width -> heads of 64
# width -> sizes of the routed, latent and recurrent sublayers of the measurement presets
EXPERTS = {1024: dict(ff=512, experts=32, top=4, groups=4, keep=2),
           2048: dict(ff=1024, experts=64, top=6, groups=8, keep=4)}
LATENT = {1024: dict(heads=8, dim=128, rot=64, vdim=128, rank=256),
          2048: dict(heads=16, dim=128, rot=64, vdim=128, rank=512)}
DELTA = {1024: dict(heads=8, dim=128, vdim=128, taps=4, low=64),
         2048: dict(heads=16, dim=128, vdim=128, taps=4, low=64)}
RETENTION = {1024: dict(heads=8, dim=128, vdim=128), 2048: dict(heads=16, dim=128, vdim=128)}
LIMIT = 7.0                     # clamp of the experts' activations


def _tokens(kind, name, width, dtype="bfloat16", layers=1, decode=0, context=0, portions=0,
            portion=0, prefix=0, ragged=False):
    return dict(kind=kind, name=name, width=width, dtype=dtype, layers=layers, decode=decode,
                context=context, portions=portions, portion=portion, prefix=prefix, ragged=ragged)


def listed():
    return [
        # one user typing at the smallest model: launches and latency
        _tokens("block", "decode_b1_small", 768, layers=4, decode=1, context=300),
        # a full decode batch late in its requests: the cache is most of the bytes
        _tokens("block", "decode_b64_medium", 1024, layers=2, decode=64, context=700, ragged=True),
        # two whole prompts, the prefill step of the benchmark
        _tokens("block", "prefill_2x1024_medium", 1024, portions=2, portion=1024),
        # continuous batching: cut prompts behind a reused prefix beside decoding requests
        _tokens("block", "mixed_ragged_large", 1280, decode=24, context=500, portions=5,
                portion=211, prefix=300, ragged=True),
        # the 32-bit path: a replayed prompt and a decode batch
        _tokens("block", "prefill_f32_medium", 1024, dtype="float32", portions=2, portion=512),
        _tokens("block", "decode_b8_f32_medium", 1024, dtype="float32", layers=2, decode=8,
                context=700, ragged=True),
        # the end of a decode step of a batch that samples
        dict(kind="head", name="head_sampling_b32", rows=32, width=1024, dtype="bfloat16"),
        # prompts through routed experts
        dict(kind="experts", name="experts_2048", tokens=2048, width=1024, dtype="bfloat16"),
        # prompts through the latent, delta-rule and retention mixers
        _tokens("latent", "latent_prefill_2x1024", 1024, portions=2, portion=1024),
        _tokens("delta", "delta_prefill_2x1024", 1024, portions=2, portion=1024),
        _tokens("retention", "retention_prefill_2x1024", 1024, portions=2, portion=1024),
        # a whole model through the engine's step function
        dict(kind="replay", name="replay_small_b8", layers=12, requests=8, prompt=200, new=16),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block"] * 9 + ["head", "experts", "experts", "latent", "latent", "delta",
                                       "delta", "retention", "retention", "replay"])
    if kind == "replay":
        return dict(kind=kind, layers=12, requests=rng.randint(1, 8), prompt=_spread(rng, 16, 200),
                    new=rng.randint(2, 16))
    if kind == "head":
        return dict(kind=kind, rows=_spread(rng, 1, 64), width=rng.choice(list(GPT2_SIZES)),
                    dtype="bfloat16")
    if kind == "experts":
        return dict(kind=kind, tokens=_spread(rng, 1, 2048), width=rng.choice(list(EXPERTS)),
                    dtype="bfloat16")
    f32 = kind == "block" and rng.random() < 0.3
    width = rng.choice(list(GPT2_SIZES) if kind == "block" else list(LATENT))
    step = rng.choice(["decode", "prefill", "mixed"])
    n_dec = _spread(rng, 1, 16 if f32 else 64) if step != "prefill" else 0
    context = _spread(rng, 16, 680) if n_dec else 0
    portions = rng.randint(1, 6) if step != "decode" else 0
    portion = _spread(rng, 8, (1024 if f32 else 2048) // portions) if portions else 0
    portion = min(portion, POSITIONS)
    prefix = min(_spread(rng, 1, 400), max(0, 680 - portion)) if step == "mixed" else 0
    case = _tokens(kind, "", width, dtype="float32" if f32 else "bfloat16",
                   layers=rng.randint(1, 3) if kind == "block" else 1, decode=n_dec,
                   context=context, portions=portions, portion=portion, prefix=prefix,
                   ragged=rng.random() < 0.7)
    del case["name"]
    return case


# -- the batch of a case ---------------------------------------------------------------------

def _lengths(n, base, ragged, most):
    out = []
    for i in range(n):
        f = 0.5 + ((37 * i + 11) % 64) / 63.0 if ragged else 1.0
        out.append(max(1, min(most, int(base * f))))
    return out


def _entries(case):
    """[(position of the first token, tokens)] of the requests, portions behind single tokens."""
    ragged = case["ragged"]
    out = [(n - 1, 1) for n in _lengths(case["decode"], case["context"], ragged, POSITIONS)]
    news = _lengths(case["portions"], case["portion"], ragged, POSITIONS)
    olds = _lengths(case["portions"], case["prefix"], ragged, POSITIONS) if case["prefix"] \
        else [0] * len(news)
    return out + [(min(p, POSITIONS - n), n) for p, n in zip(olds, news)]


def _dtype(case):
    return torch.bfloat16 if case.get("dtype", "bfloat16") == "bfloat16" else torch.float32


class _Random:
    """Seeded normal tensors on the GPU; matrices come rounded to the compute type."""

    def __init__(self, seed, dtype):
        self.gen = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        self.dtype = dtype

    def vec(self, *shape, std=1.0, mean=0.0):
        return torch.randn(*shape, device="cuda", generator=self.gen) * std + mean

    def mat(self, *shape, std=None):
        std = shape[-1] ** -0.5 if std is None else std
        return (torch.randn(*shape, device="cuda", generator=self.gen) * std).to(self.dtype)


class StepInputs:
    """What layers and sublayers are given while a step runs: the kernels, the batch's tables in
    device memory, the attention work lists and temporary buffers."""

    def __init__(self, entries, dtype, seed, positions):
        self.ops = CudaOps("cuda")
        self.device = self.ops.device
        self.dtype = dtype
        self.status = torch.zeros(1, dtype=torch.int32, device=self.device)
        self.ops.status = self.status
        self.n_requests = len(entries)
        pos, req, start, host = [], [], [], []
        for r, (p, n) in enumerate(entries):
            start.append(len(pos))
            host.append((r, r, p, n))
            pos += range(p, p + n)
            req += [r] * n
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=self.device)  # noqa: E731
        self.n_rows = len(pos)
        self.tok_pos, self.tok_req = i32(pos), i32(req)
        self.req_start, self.req_len = i32(start), i32([n for _, n in entries])
        self.req_slot = i32(list(range(self.n_requests)))
        self.plan = self.ops.make_plan(host, self.n_rows, PAGE)
        pages = [-(-(p + n) // PAGE) for p, n in entries]
        self.num_pages = sum(pages) + 1
        order = torch.randperm(self.num_pages,
                               generator=torch.Generator().manual_seed(int(seed))).tolist()
        width = positions // PAGE
        rows = []
        for k in pages:
            mine, order = order[:k], order[k:]
            rows.append(mine + [-1] * (width - k))
        self.table = i32(rows)
        self._state, self._buffers = None, {}

    def buffer(self, name, shape, dtype):
        key = (name, tuple(shape), dtype)
        if key not in self._buffers:
            self._buffers[key] = torch.zeros(*shape, dtype=dtype, device=self.device)
        return self._buffers[key]

    def state(self):
        return self._state

    def view(self, pool):
        return CacheView(pool=pool, table=self.table, page_size=PAGE, num_pages=self.num_pages,
                         writes=True, group=0)


def _captured(launch):
    """``launch`` run once eagerly, then captured; returns the graph."""
    launch()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        launch()
    return graph


# -- inputs: made from the seed alone, the same for prepare() and exact() ---------------------

def _block_inputs(case, seed):
    g = _Random(seed, _dtype(case))
    E, H = case["width"], GPT2_SIZES[case["width"]]
    entries = _entries(case)
    layers = []
    for _ in range(case["layers"]):
        layers.append({
            "n1.w": g.vec(E, std=0.1, mean=1.0), "n1.b": g.vec(E, std=0.1),
            "qkv.w": g.mat(3 * E, E), "qkv.b": g.vec(3 * E, std=0.1),
            "o.w": g.mat(E, E, std=0.5 * E ** -0.5), "o.b": g.vec(E, std=0.1),
            "n2.w": g.vec(E, std=0.1, mean=1.0), "n2.b": g.vec(E, std=0.1),
            "fc.w": g.mat(4 * E, E), "fc.b": g.vec(4 * E, std=0.1),
            "pr.w": g.mat(E, 4 * E, std=0.5 * (4 * E) ** -0.5), "pr.b": g.vec(E, std=0.1)})
    x = g.vec(sum(n for _, n in entries), E)
    step = StepInputs(entries, _dtype(case), seed, POSITIONS)
    pools = [g.mat(step.num_pages, 2, H, PAGE, 64, std=1.0) for _ in range(case["layers"])]
    return layers, x, pools, step, entries, H


def _head_inputs(case, seed):
    g = _Random(seed, _dtype(case))
    rows, E = case["rows"], case["width"]
    h, w = g.mat(rows, E, std=1.0), g.mat(VOCAB, E, std=2.0 * E ** -0.5)
    i = torch.arange(rows, device="cuda", dtype=torch.int32)
    temperature = torch.where(i % 3 == 0, 0.0, 0.8).float()
    top_k = torch.where(i % 3 == 2, 40, 0).int()
    return h, w, temperature, top_k, (i * 7919 + int(seed)).int(), (i * 0).int(), (i + 100).int()


def _experts_inputs(case, seed):
    g, z = _Random(seed, _dtype(case)), EXPERTS[case["width"]]
    W, F, N = case["width"], z["ff"], z["experts"]
    t = {"gate": g.mat(N, F, W, std=2.0 * W ** -0.5), "up": g.mat(N, F, W, std=2.0 * W ** -0.5),
         "down": g.mat(N, W, F, std=0.5 * F ** -0.5),
         "router": g.mat(N, W, std=2.0 * W ** -0.5).float()}
    return t, g.mat(case["tokens"], W, std=1.0), z


def _latent_inputs(case, seed):
    g, z = _Random(seed, _dtype(case)), LATENT[case["width"]]
    W, H, D, P, V, R = case["width"], z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
    entries = _entries(case)
    t = {"q": g.mat(H * (D + P), W), "dkv": g.mat(R + P, W),
         "norm": g.vec(R, std=0.1, mean=1.0), "uk": g.mat(H * D, R), "uv": g.mat(H * V, R),
         "sink": g.vec(H), "o": g.mat(W, H * V, std=0.5 * (H * V) ** -0.5)}
    h = g.mat(sum(n for _, n in entries), W, std=1.0)
    step = StepInputs(entries, _dtype(case), seed, POSITIONS)
    pool = g.mat(step.num_pages, 1, 1, PAGE, R + P, std=1.0)
    return t, h, pool, step, entries, z


def _delta_inputs(case, seed):
    g, z = _Random(seed, _dtype(case)), DELTA[case["width"]]
    W, H, D, V, taps, low = (case["width"], z["heads"], z["dim"], z["vdim"], z["taps"], z["low"])
    entries = _entries(case)
    t = {"q": g.mat(H * D, W), "k": g.mat(H * D, W), "v": g.mat(H * V, W),
         "q.conv": g.vec(H * D, taps, std=0.5), "k.conv": g.vec(H * D, taps, std=0.5),
         "v.conv": g.vec(H * V, taps, std=0.5), "b": g.mat(H, W),
         "A_log": g.vec(H, std=0.5, mean=-1.0), "norm": g.vec(V, std=0.1, mean=1.0),
         "a1": g.mat(low, W), "a2": g.mat(H * D, low).float(), "dt_bias": g.vec(H * D, std=0.5),
         "g1": g.mat(low, W), "g2": g.mat(H * V, low).float(),
         "o": g.mat(W, H * V, std=0.5 * (H * V) ** -0.5)}
    h = g.mat(sum(n for _, n in entries), W, std=1.0)
    state = g.vec(len(entries), H * D * V + (taps - 1) * H * (2 * D + V), std=0.3)
    for r, (p, _) in enumerate(entries):
        if p == 0:
            state[r] = 0.0                     # a request that starts
    return t, h, state, entries, z


def _retention_inputs(case, seed):
    g, z = _Random(seed, _dtype(case)), RETENTION[case["width"]]
    W, H, D, V = case["width"], z["heads"], z["dim"], z["vdim"]
    entries = _entries(case)
    t = {"q": g.mat(H * D, W), "k": g.mat(H * D, W), "v": g.mat(H * V, W),
         "g": g.mat(H * V, W, std=2.0 * W ** -0.5), "o": g.mat(W, H * V, std=(H * V) ** -0.5)}
    h = g.mat(sum(n for _, n in entries), W, std=1.0)
    state = g.vec(len(entries), H * D * V, std=0.3)
    for r, (p, _) in enumerate(entries):
        if p == 0:
            state[r] = 0.0
    decay = [1.0 - 2.0 ** (-4 - 5 * i / max(1, H - 1)) for i in range(H)]
    return t, h, state, entries, z, decay


def _replay_inputs(case, seed):
    E, L = 768, case["layers"]
    g = _Random(seed, torch.bfloat16)
    w = {"wte.weight": g.mat(VOCAB, E, std=0.05), "wpe.weight": g.mat(POSITIONS, E, std=0.02)}
    for i in range(L):
        p = f"h.{i}."
        for n in ("ln_1", "ln_2"):
            w[p + n + ".weight"], w[p + n + ".bias"] = g.vec(E, std=0.02, mean=1.0), g.vec(E, std=0.02)
        for n, a, b in (("attn.c_attn", E, 3 * E), ("attn.c_proj", E, E), ("mlp.c_fc", E, 4 * E),
                        ("mlp.c_proj", 4 * E, E)):
            w[p + n + ".weight"] = g.mat(a, b, std=0.02)
            w[p + n + ".bias"] = g.vec(b, std=0.01)
    w["ln_f.weight"], w["ln_f.bias"] = g.vec(E, std=0.02, mean=1.0), g.vec(E, std=0.02)
    ids = torch.Generator().manual_seed(int(seed) + 7)
    lens = _lengths(case["requests"], case["prompt"], True, 2048 // case["requests"])
    prompts = [torch.randint(0, VOCAB, (n + case["new"],), generator=ids).tolist() for n in lens]
    return w, prompts, lens


# -- prepare and run --------------------------------------------------------------------------

def _part(family, kind, tensors, **params):
    part = build_part(family, PartSpec(kind, params))
    part.bind(tensors)
    return part


def _prepare_block(case, seed):
    layers, x0, pools, step, _, H = _block_inputs(case, seed)
    E = case["width"]
    norm = lambda n: PartSpec("layernorm", dict(width=E, eps=EPS, weight=n + ".w", bias=n + ".b"))  # noqa: E731
    spec = LayerSpec(
        norm1=norm("n1"), norm2=norm("n2"),
        mixer=PartSpec("causal_attention", dict(
            width=E, n_heads=H, head_dim=64, scale=0.125, qkv_weight="qkv.w", qkv_bias="qkv.b",
            out_weight="o.w", out_bias="o.b", stored_in_out=False)),
        feed_forward=PartSpec("dense", dict(
            width=E, inner=4 * E, activation="gelu_tanh", in_weight="fc.w", in_bias="fc.b",
            out_weight="pr.w", out_bias="pr.b", stored_in_out=False)))
    blocks = []
    for tensors in layers:
        block = PreNormBlock(spec)
        for part in block.parts():
            part.bind({n: tensors[n] for n in part.tensor_requests()})
        blocks.append(block)
    x = torch.empty_like(x0)

    def launch():
        x.copy_(x0)
        for block, pool in zip(blocks, pools):
            block.forward(step, x, step.view(pool))
    return dict(graph=_captured(launch), out=[x, *pools], keep=(step, blocks, x0))


def _prepare_head(case, seed):
    h, w, temperature, top_k, lo, hi, position = _head_inputs(case, seed)
    ops = CudaOps("cuda")
    logits = torch.empty(case["rows"], VOCAB, device="cuda")
    tokens = torch.zeros(case["rows"] + 1, dtype=torch.int32, device="cuda")

    def launch():
        ops.linear(logits, h, w)
        ops.sample(tokens, logits, temperature, top_k, lo, hi, position, status_word=ops.status)
    return dict(graph=_captured(launch), out=[logits, tokens],
                keep=(ops, h, w, temperature, top_k, lo, hi, position))


def _prepare_experts(case, seed):
    t, h, z = _experts_inputs(case, seed)
    tensors = {"router": t["router"]}
    for e in range(z["experts"]):
        for n in ("gate", "up", "down"):
            tensors[f"e{e}.{n}"] = t[n][e]
    part = _part("feed_forward", "routed_experts", tensors, width=case["width"], ff=z["ff"],
                 experts=z["experts"], top=z["top"], groups=z["groups"], keep=z["keep"],
                 limit=LIMIT, router="router", expert_prefix="e")
    step = StepInputs([(0, case["tokens"])], _dtype(case), seed, 2048)
    x = torch.zeros(case["tokens"], case["width"], device="cuda")

    def launch():
        x.zero_()
        part.forward(step, h, x)
    return dict(graph=_captured(launch), out=[x], keep=(step, part, h))


def _prepare_latent(case, seed):
    t, h, pool, step, _, z = _latent_inputs(case, seed)
    D, P = z["dim"], z["rot"]
    part = _part("mixer", "latent_attention", t, width=case["width"], n_heads=z["heads"], dim=D,
                 rot_dim=P, vdim=z["vdim"], kv_rank=z["rank"], scale=(D + P) ** -0.5,
                 rot_base=10000.0, rot_dims=P, eps=1e-6, q_weight="q", latent_weight="dkv",
                 latent_norm="norm", key_up="uk", value_up="uv", sink="sink", out_weight="o")
    x = torch.zeros(h.shape[0], case["width"], device="cuda")

    def launch():
        x.zero_()
        part.forward(step, h, x, step.view(pool))
    return dict(graph=_captured(launch), out=[x, pool], keep=(step, part, h))


def _prepare_recurrent(case, seed):
    if case["kind"] == "delta":
        t, h, state0, entries, z = _delta_inputs(case, seed)
        part = _part("mixer", "channel_delta_rule", t, width=case["width"], n_heads=z["heads"],
                     n_kv_heads=z["heads"], dim=z["dim"], vdim=z["vdim"], taps=z["taps"],
                     eps=1e-6, prefix="")
    else:
        t, h, state0, entries, z, decay = _retention_inputs(case, seed)
        part = _part("mixer", "retention", t, width=case["width"], n_heads=z["heads"],
                     dim=z["dim"], vdim=z["vdim"], decay=decay, eps=1e-6, prefix="",
                     rot_dims=z["dim"])
    step = StepInputs(entries, _dtype(case), seed, POSITIONS)
    step._state = torch.empty_like(state0)
    x = torch.zeros(h.shape[0], case["width"], device="cuda")

    def launch():
        x.zero_()
        step._state.copy_(state0)              # every pass continues the same requests
        part.forward(step, h, x, None)
    return dict(graph=_captured(launch), out=[x, step._state], keep=(step, part, h, state0))


def _prepare_replay(case, seed):
    w, prompts, lens = _replay_inputs(case, seed)
    cfg = GPT2Config.from_dict(dict(n_layer=case["layers"], n_embd=768, n_head=12,
                                    vocab_size=VOCAB, n_positions=POSITIONS))
    model = Model(build_spec(cfg))
    model.bind(w, torch.bfloat16, torch.device("cuda:0"))
    runner = Runner(model, num_pages=case["requests"] * POSITIONS // PAGE, page_size=PAGE,
                    max_requests=case["requests"], dtype=torch.bfloat16, device="cuda:0",
                    cuda_graphs=True)
    return dict(runner=runner, prompts=prompts, lens=lens, new=case["new"])


def prepare(case, seed):
    make = {"block": _prepare_block, "head": _prepare_head, "experts": _prepare_experts,
            "latent": _prepare_latent, "delta": _prepare_recurrent,
            "retention": _prepare_recurrent, "replay": _prepare_replay}
    return make[case["kind"]](case, seed)


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    runner, logits = state["runner"], []
    at = list(state["lens"])
    for i in range(state["new"] + 1):
        entries = []
        for r, (ids, n) in enumerate(zip(state["prompts"], at)):
            part = ids[:n] if i == 0 else ids[n:n + 1]
            entries.append(StepEntry(r, part, [len(part) - 1]))
            at[r] = n + (i > 0)
        logits.append(runner.step(entries, check_status=False).logits.clone())
    for r in range(len(at)):
        runner.close(r)
    return logits


# -- what a pass cannot do without --------------------------------------------------------------

def work(case):
    kind = case["kind"]
    item = 2 if case.get("dtype", "bfloat16") == "bfloat16" else 4
    if kind == "head":
        M, E = case["rows"], case["width"]
        return {"bytes": VOCAB * E * item + M * E * item + 4 * M * VOCAB, "flops": 2 * M * E * VOCAB}
    if kind == "experts":
        z, T, W = EXPERTS[case["width"]], case["tokens"], case["width"]
        pairs = T * z["top"]
        used = min(z["experts"], pairs)
        return {"bytes": used * 3 * z["ff"] * W * item + 4 * z["experts"] * W + T * W * (item + 4),
                "flops": 2 * pairs * 3 * z["ff"] * W + 2 * T * W * z["experts"]}
    if kind == "replay":
        E, L = 768, case["layers"]
        lens = _lengths(case["requests"], case["prompt"], True, 2048 // case["requests"])
        per = 12 * E * E * L
        T, R, new = sum(lens), case["requests"], case["new"]
        weights = 2 * (per + VOCAB * E)
        seen = sum((n + i + 1) for n in lens for i in range(new))
        return {"bytes": (new + 1) * (weights + 4 * R * VOCAB) + 4 * E * L * (seen + 2 * T),
                "flops": 2 * per * (T + R * new) + 2 * R * (new + 1) * E * VOCAB
                + 4 * E * L * (seen + sum(n * (n + 1) // 2 for n in lens))}
    entries, W = _entries(case), case["width"]
    T = sum(n for _, n in entries)
    pairs = sum(n * p + n * (n + 1) // 2 for p, n in entries)      # visible (query, key) pairs
    keys = sum(p + n for p, n in entries)
    if kind == "block":
        L = case["layers"]
        return {"bytes": L * (12 * W * W * item + 2 * W * item * (keys + T)) + 8 * T * W,
                "flops": L * (24 * T * W * W + 4 * W * pairs)}
    if kind == "latent":
        z = LATENT[W]
        H, D, P, V, R = z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
        w = W * (H * (D + P) + R + P) + H * (D + V) * R + W * H * V
        # the cheaper of the two forms: keys and values expanded per head, or the latent itself
        flops = min(2 * pairs * H * (D + P + V) + 2 * keys * H * (D + V) * R,
                    2 * pairs * H * (2 * R + P) + 2 * T * H * (D + V) * R)
        return {"bytes": w * item + (R + P) * item * (keys + T) + T * W * (item + 4),
                "flops": 2 * T * (W * (H * (D + P) + R + P) + W * H * V) + flops}
    if kind == "delta":
        z = DELTA[W]
        H, D, V, low = z["heads"], z["dim"], z["vdim"], z["low"]
        w = W * (H * (2 * D + 2 * V + 1) + 2 * low) + 2 * H * (D + V) * low
        state = len(entries) * (H * D * V + 3 * H * (2 * D + V))
        return {"bytes": w * item + 8 * state + T * W * (item + 4),
                "flops": 2 * T * w + 7 * T * H * D * V}
    z = RETENTION[W]
    H, D, V = z["heads"], z["dim"], z["vdim"]
    w = W * H * (2 * D + 3 * V)
    return {"bytes": w * item + 8 * len(entries) * H * D * V + T * W * (item + 4),
            "flops": 2 * T * w + 5 * T * H * D * V}


def tolerance(case):
    # about four times the distance from exact(): bf16 rows lie between the kernels of a layer
    # (0.8e-3 .. 2.3e-3 a layer, 4e-3 for the latent and for twelve layers), 32-bit sums are
    # 3e-7 .. 1e-6 off
    if case.get("dtype", "bfloat16") == "float32":
        return {"rel": 3e-6}
    return {"block": {"rel": 8e-3}, "head": {"rel": 4e-6, "differ": 0.01},
            "experts": {"rel": 7e-3}, "latent": {"rel": 1.5e-2}, "delta": {"rel": 7e-3},
            "retention": {"rel": 7e-3}, "replay": {"rel": 1.7e-2}}[case["kind"]]


# -- the same in 64 bits, by the formulas --------------------------------------------------------

def _f64(t):
    return t.double()


def _layer_norm(x, w, b):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + EPS) * w + b


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _attend(q, k, v, first, scale):
    """q [n, H, D] at positions first.., k and v [H, keys, D] from position 0 on."""
    s = torch.einsum("nhd,hkd->hnk", q, k) * scale
    at = torch.arange(first, first + q.shape[0], device=q.device)
    s = s.masked_fill(torch.arange(k.shape[1], device=q.device)[None, None] > at[None, :, None],
                      -math.inf)
    return torch.einsum("hnk,hkd->nhd", torch.softmax(s, -1), v)


def _exact_block(case, seed):
    layers, x, pools, step, entries, H = _block_inputs(case, seed)
    x, E = _f64(x), case["width"]
    table, done = step.table.long(), []
    for t, pool in zip(layers, pools):
        t = {n: _f64(v) for n, v in t.items()}
        pool = _f64(pool)
        h = _layer_norm(x, t["n1.w"], t["n1.b"])
        q, k, v = (h @ t["qkv.w"].T + t["qkv.b"]).view(-1, 3, H, 64).unbind(1)
        pos, req = step.tok_pos.long(), step.tok_req.long()
        page = table[req, pos // PAGE]
        pool[page, 0, :, pos % PAGE] = k
        pool[page, 1, :, pos % PAGE] = v
        att, at = torch.empty_like(x), 0
        for r, (p, n) in enumerate(entries):
            keys = p + n
            rows = pool[table[r, :-(-keys // PAGE)]]           # [pages, 2, H, PAGE, 64]
            rows = rows.permute(1, 2, 0, 3, 4).reshape(2, H, -1, 64)[:, :, :keys]
            att[at:at + n] = _attend(q[at:at + n], rows[0], rows[1], p, 0.125).reshape(n, E)
            at += n
        x = x + att @ t["o.w"].T + t["o.b"]
        h = _layer_norm(x, t["n2.w"], t["n2.b"])
        x = x + _gelu(h @ t["fc.w"].T + t["fc.b"]) @ t["pr.w"].T + t["pr.b"]
        done.append(pool)
    return [x, *done]


def _exact_head(case, seed):
    h, w = _head_inputs(case, seed)[:2]
    return [_f64(h) @ _f64(w).T, None]


def _exact_experts(case, seed):
    t, h, z = _experts_inputs(case, seed)
    h, N, G = _f64(h), z["experts"], z["groups"]
    s = torch.sigmoid(h @ _f64(t["router"]).T)
    group = s.view(-1, G, N // G).topk(2, -1).values.sum(-1)
    kept = torch.zeros_like(group).scatter_(1, group.topk(z["keep"], -1).indices, 1.0)
    chosen = s.masked_fill(kept.repeat_interleave(N // G, 1) == 0, -1.0).topk(z["top"], -1).indices
    weight = torch.gather(s, 1, chosen)
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    out = torch.zeros_like(h)
    for e in range(N):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            a = h[rows]
            gate = (a @ _f64(t["gate"][e]).T).clamp(max=LIMIT)
            up = (a @ _f64(t["up"][e]).T).clamp(-LIMIT, LIMIT)
            y = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ _f64(t["down"][e]).T
            out.index_add_(0, rows, y * weight[rows, place, None])
    return [out]


def _frequencies(dims):
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    return (10000.0 ** (-2.0 * i / dims)).float().double()


def _exact_latent(case, seed):
    t, h, pool, step, entries, z = _latent_inputs(case, seed)
    t, h, pool = {n: _f64(v) for n, v in t.items()}, _f64(h), _f64(pool)
    H, D, P, V, R = z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
    pos, req, table = step.tok_pos.long(), step.tok_req.long(), step.table.long()
    angle = pos[:, None].double() * _frequencies(P)

    def turn(u):                                   # neighbours (2i, 2i + 1) turn together
        shape = (-1,) + (1,) * (u.dim() - 2) + (P // 2,)
        c, s = torch.cos(angle).view(shape), torch.sin(angle).view(shape)
        a, b = u[..., 0::2], u[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    q = (h @ t["q"].T).view(-1, H, D + P)
    row = h @ t["dkv"].T
    c = row[:, :R]
    c = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-6) * t["norm"]
    pool[table[req, pos // PAGE], 0, 0, pos % PAGE] = torch.cat([c, turn(row[:, R:])], -1)
    qr, scale, out, at = turn(q[..., D:]), (D + P) ** -0.5, [], 0
    uk, uv = t["uk"].view(H, D, R), t["uv"].view(H, V, R)
    for r, (p, n) in enumerate(entries):
        keys = p + n
        rows = pool[table[r, :-(-keys // PAGE)]].reshape(-1, R + P)[:keys]
        k, v = torch.einsum("hdr,jr->hjd", uk, rows[:, :R]), torch.einsum("hvr,jr->hjv", uv, rows[:, :R])
        s = (torch.einsum("nhd,hjd->hnj", q[at:at + n, :, :D], k)
             + torch.einsum("nhp,jp->hnj", qr[at:at + n], rows[:, R:])) * scale
        seen = torch.arange(keys, device="cuda")[None] <= torch.arange(p, keys, device="cuda")[:, None]
        s = torch.cat([s.masked_fill(~seen, -math.inf),
                       t["sink"].view(H, 1, 1).expand(H, n, 1)], -1)
        out.append(torch.einsum("hnj,hjv->nhv", torch.softmax(s, -1)[..., :-1], v).reshape(n, H * V))
        at += n
    return [torch.cat(out) @ t["o"].T, pool]


def _padded(rows, entries):
    """[requests, longest, ...] from flat rows, and which places hold a token."""
    most = max(n for _, n in entries)
    out, at = rows.new_zeros(len(entries), most, *rows.shape[1:]), 0
    live = torch.zeros(len(entries), most, dtype=torch.bool, device=rows.device)
    for r, (_, n) in enumerate(entries):
        out[r, :n], live[r, :n] = rows[at:at + n], True
        at += n
    return out, live


def _exact_delta(case, seed):
    t, h, state, entries, z = _delta_inputs(case, seed)
    t, h, state = {n: _f64(v) for n, v in t.items()}, _f64(h), _f64(state)
    H, D, V, taps = z["heads"], z["dim"], z["vdim"], z["taps"]
    C, size = H * (2 * D + V), H * D * V
    S = state[:, :size].view(-1, H, D, V).clone()
    history = state[:, size:].view(-1, taps - 1, C)
    fed, live = _padded(h @ torch.cat([t["q"], t["k"], t["v"]]).T, entries)
    seen = torch.cat([history, fed], 1)
    conv = torch.cat([t["q.conv"], t["k.conv"], t["v.conv"]])
    mixed = torch.nn.functional.silu(sum(seen[:, j:j + fed.shape[1]] * conv[:, j] for j in range(taps)))
    unit = lambda u: u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = unit(mixed[..., :H * D].unflatten(-1, (H, D))) * D ** -0.5
    k = unit(mixed[..., H * D:2 * H * D].unflatten(-1, (H, D)))
    v = mixed[..., 2 * H * D:].unflatten(-1, (H, V))
    beta, _ = _padded(torch.sigmoid(h @ t["b"].T), entries)
    rate = torch.nn.functional.softplus((h @ t["a1"].T) @ t["a2"].T + t["dt_bias"]).unflatten(-1, (H, D))
    decay, _ = _padded(torch.exp(-torch.exp(t["A_log"])[:, None] * rate), entries)
    o = torch.zeros_like(v)
    for i in range(fed.shape[1]):
        new = S * decay[:, i, :, :, None]
        u = beta[:, i, :, None] * (v[:, i] - torch.einsum("rhdv,rhd->rhv", new, k[:, i]))
        new = new + k[:, i, :, :, None] * u[:, :, None]
        o[:, i] = torch.einsum("rhdv,rhd->rhv", new, q[:, i])
        S = torch.where(live[:, i, None, None, None], new, S)
    o = o[live]
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * t["norm"]
    o = o.flatten(1) * torch.sigmoid((h @ t["g1"].T) @ t["g2"].T)
    kept = torch.stack([seen[r, n:n + taps - 1] for r, (_, n) in enumerate(entries)])
    return [o @ t["o"].T, torch.cat([S.flatten(1), kept.flatten(1)], 1)]


def _exact_retention(case, seed):
    t, h, state, entries, z, decay = _retention_inputs(case, seed)
    t, h = {n: _f64(v) for n, v in t.items()}, _f64(h)
    H, D, V = z["heads"], z["dim"], z["vdim"]
    S = _f64(state).view(-1, H, D, V)
    pos = torch.cat([torch.arange(p, p + n, device="cuda") for p, n in entries])
    angle = (pos[:, None].double() * _frequencies(D))[:, None]
    c, s = torch.cos(angle), torch.sin(angle)

    def turn(u):                                   # number i turns with i + D / 2
        a, b = u[..., :D // 2], u[..., D // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], -1)
    q, live = _padded(turn((h @ t["q"].T).view(-1, H, D)), entries)
    k, _ = _padded(turn((h @ t["k"].T).view(-1, H, D)) * D ** -0.5, entries)
    v, _ = _padded((h @ t["v"].T).view(-1, H, V), entries)
    keep = torch.tensor(decay, device="cuda").float().double().view(1, H, 1, 1)
    o = torch.zeros_like(v)
    for i in range(q.shape[1]):
        new = S * keep + k[:, i, :, :, None] * v[:, i, :, None]
        o[:, i] = torch.einsum("rhdv,rhd->rhv", new, q[:, i])
        S = torch.where(live[:, i, None, None, None], new, S)
    o = o[live]
    o = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6)).flatten(1)
    return [(o * torch.nn.functional.silu(h @ t["g"].T)) @ t["o"].T, S.flatten(1)]


def _exact_replay(case, seed):
    w, prompts, lens = _replay_inputs(case, seed)
    w = {n: _f64(v) for n, v in w.items()}
    rows = []
    for ids, n in zip(prompts, lens):
        ids = torch.tensor(ids[:n + case["new"]], device="cuda")
        x = w["wte.weight"][ids] + w["wpe.weight"][:len(ids)]
        for i in range(case["layers"]):
            t = {k[len(f"h.{i}."):]: v for k, v in w.items() if k.startswith(f"h.{i}.")}
            lin = lambda a, m: a @ t[m + ".weight"] + t[m + ".bias"]  # noqa: E731
            h = _layer_norm(x, t["ln_1.weight"], t["ln_1.bias"])
            q, k, v = lin(h, "attn.c_attn").view(-1, 3, 12, 64).unbind(1)
            a = _attend(q, k.transpose(0, 1), v.transpose(0, 1), 0, 0.125)
            x = x + lin(a.reshape(len(ids), 768), "attn.c_proj")
            h = _layer_norm(x, t["ln_2.weight"], t["ln_2.bias"])
            x = x + lin(_gelu(lin(h, "mlp.c_fc")), "mlp.c_proj")
        x = _layer_norm(x[n - 1:], w["ln_f.weight"], w["ln_f.bias"])
        rows.append(x @ w["wte.weight"].T)
    return list(torch.stack(rows, 1))


def exact(case, seed):
    make = {"block": _exact_block, "head": _exact_head, "experts": _exact_experts,
            "latent": _exact_latent, "delta": _exact_delta, "retention": _exact_retention,
            "replay": _exact_replay}
    return make[case["kind"]](case, seed)
