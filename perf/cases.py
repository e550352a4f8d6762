"""Workloads that performance work on this package is measured on.

Every case is one piece of the work that a decoder with contextually sparse MLPs has this library
do, called the way such a program calls it:

  layer    SparseLayer.step, token after token (a host that steps layer by layer)
  stack    SparseStack.step, token after token (all sparse MLPs of a model as one graph)
  dropin   the reference's own call sequence: compute_binary_mask, WeightCache, the two getters,
           sparse_mlp_forward
  op       sparse_mlp_forward on weights that were gathered before
  prefill  compute_binary_mask + SkipMLP on whole prompts
  glue     what a decoder layer runs around the MLP at decode time, as one CUDA graph
  model    LlamaSkipModel, decode steps behind a cached prompt

Weights are N(0, 0.02), hidden states follow x_t = 0.9 x_{t-1} + 0.436 n_t, and the streams of a batch
share 70 % of their variance, so consecutive masks overlap, the differential caches have rows to
exchange at every token, and the union of a batch's masks is the one that a batch of related streams
shows.  Thresholds aim at a density per row.
"""
import functools
import math
from statistics import NormalDist

import torch

import sparse_transformers_b200 as stx
from sparse_transformers_b200 import llama_skip as ls

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"fp32": 4, "fp16": 2, "bf16": 2}
WSTD, ALPHA = 0.02, 0.7
# tokens of a decode pass: consecutive masks differ, as in real decoding (a repeated token would leave the caches alone)
TOKENS = 4


# ---------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one layer of a 1B model in 32 bits: the smallest call, nothing but latency around 40 MB of rows
        dict(name="layer-1b-fp32-b1", kind="layer", H=2048, I=8192, r=64, B=1, L=1, dtype="fp32", density=0.20, act="silu", gate=True, rule="naive"),
        # three requests decoded together, 7B ReLU model, top-k rule
        dict(name="layer-7b-fp16-b3-topk", kind="layer", H=4096, I=11008, r=128, B=3, L=1, dtype="fp16", density=0.10, act="relu", gate=True, rule="topk"),
        # an ungated (OPT-like) MLP with the statistical rule, odd number of neurons
        dict(name="layer-nogate-fp16-b1-stat", kind="layer", H=2048, I=8190, r=64, B=1, L=1, dtype="fp16", density=0.15, act="relu", gate=False, rule="statistical_topk"),
        # all MLPs of a 3B model, one stream
        dict(name="stack-3b-fp16-b1", kind="stack", H=3072, I=8192, r=64, B=1, L=28, dtype="fp16", density=0.20, act="silu", gate=True, rule="naive"),
        # a quarter of a 7B model's MLPs, 8 streams
        dict(name="stack-7b-bf16-b8", kind="stack", H=4096, I=14336, r=128, B=8, L=8, dtype="bf16", density=0.15, act="silu", gate=True, rule="naive"),
        # the same with a serving batch of 64 streams
        dict(name="stack-7b-bf16-b64", kind="stack", H=4096, I=14336, r=128, B=64, L=8, dtype="bf16", density=0.15, act="silu", gate=True, rule="naive"),
        # the reference's literal call sequence for one decoded token, getters included
        dict(name="dropin-3b-fp16-b1", kind="dropin", H=3072, I=8192, r=64, B=1, L=1, dtype="fp16", density=0.20, act="silu", gate=True, rule="naive"),
        # a ragged block of prompt rows over an odd number of gathered neurons
        dict(name="op-7b-bf16-777", kind="op", H=4096, I=5501, B=777, L=1, dtype="bf16", act="silu", gate=True),
        # a 300-token prompt, masks of all its tokens united
        dict(name="prefill-3b-fp16-300", kind="prefill", H=3072, I=8192, r=64, B=300, L=1, dtype="fp16", density=0.01, act="silu", gate=True, rule="naive"),
        # four prompts of 2048 tokens: the largest call
        dict(name="prefill-7b-fp16-8192", kind="prefill", H=4096, I=11008, r=128, B=8192, L=1, dtype="fp16", density=0.10, act="relu", gate=True, rule="naive"),
        # norms, attention and output projection of four decoder layers, 4000 tokens of context
        dict(name="glue-3b-fp16-ctx4000", kind="glue", heads=24, kv=8, hd=128, H=3072, ctx=4000, max_len=4096, L=4, dtype="fp16"),
        # a whole decode call, embedding to logits, of four tokens behind a 200-token prompt.  One decoder layer of the 3B shape:
        # with random weights an inactive neuron is not a small one, so a single rounding that moves a neuron across the
        # threshold of a later layer moves the logits by several per cent, and the call could be compared with nothing
        dict(name="model-3b-fp16-1l", kind="model", H=3072, I=8192, r=64, heads=24, kv=8, hd=128, vocab=128256, L=1, prompt=200, max_len=1024, dtype="fp16", density=0.20, act="silu"),
    ]


def _log(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    """One more case of the same ranges; never more work than the largest listed one."""
    kind = rng.choice(["layer", "layer", "stack", "stack", "dropin", "op", "op", "prefill", "glue"])
    dt16 = rng.choice(["fp16", "bf16"])
    if kind == "glue":
        kv = rng.choice([4, 8])
        heads = kv * rng.choice([2, 3, 4])
        hd = rng.choice([64, 128])
        ctx = _log(rng, 16, 8000)
        return dict(kind="glue", heads=heads, kv=kv, hd=hd, H=heads * hd, ctx=ctx, max_len=8192 if ctx > 4000 else 4096, L=4, dtype=dt16)
    H = rng.choice([1024, 2048, 2560, 3072, 4096])
    I = _log(rng, 2048, 14336) if rng.random() < 0.5 else 32 * _log(rng, 64, 448)
    r = rng.choice([32, 64, 128])
    act = rng.choice(["silu", "relu", "gelu_pytorch_tanh"])
    if kind == "op":
        return dict(kind=kind, H=H, I=_log(rng, 512, 11000), B=_log(rng, 1, 4096), L=1, dtype=dt16, act=act, gate=True)
    if kind == "prefill":
        B = _log(rng, 32, 4096)
        return dict(kind=kind, H=H, I=I, r=r, B=B, L=1, dtype=dt16, density=rng.choice([0.005, 0.02, 0.10]), act=act, gate=True, rule="naive")
    if kind == "dropin":
        return dict(kind=kind, H=H, I=I, r=r, B=rng.choice([1, 1, 2, 5, 12]), L=1, dtype=dt16, density=rng.uniform(0.1, 0.25), act=act, gate=True, rule="naive")
    if kind == "layer":
        dtype = rng.choice(["fp32", "fp16", "bf16"])
        gate = rng.random() < 0.8
        B = _log(rng, 1, 8 if dtype == "fp32" or not gate else 96)
        rule = rng.choice(["naive", "naive", "topk", "statistical_topk"])
        return dict(kind=kind, H=H, I=I, r=r, B=B, L=1, dtype=dtype, density=rng.uniform(0.08, 0.25), act=act, gate=gate, rule=rule)
    B = rng.choice([1, 1, _log(rng, 2, 8), _log(rng, 9, 128)])
    return dict(kind=kind, H=H, I=I, r=r, B=B, L=rng.choice([4, 8, 16]) if B == 1 else 4, dtype=dt16, density=rng.uniform(0.1, 0.25), act=act, gate=True, rule="naive")


# ---------------------------------------------------------------------------------- inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + salt) % (1 << 62))


def _rn(g, dtype, *shape, std=1.0):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def _weights(c, seed, l):
    """gate [I,H] (or None), up [I,H], down [H,I], A [r,H], Bm [I,r] of layer l."""
    g, dt = _gen(seed, 10 + l), DTYPES[c["dtype"]]
    gate = _rn(g, dt, c["I"], c["H"], std=WSTD) if c["gate"] else None
    up, down = _rn(g, dt, c["I"], c["H"], std=WSTD), _rn(g, dt, c["H"], c["I"], std=WSTD)
    if "r" not in c:
        return gate, up, down, None, None
    return gate, up, down, _rn(g, dt, c["r"], c["H"], std=WSTD), _rn(g, dt, c["I"], c["r"], std=WSTD)


def _tokens(c, seed, n):
    """n hidden states [B,H] of an AR(1) process; the rows share ALPHA of their variance."""
    g, B, H = _gen(seed, 1), c["B"], c["H"]
    priv, shared = torch.randn(B, H, generator=g, device="cuda"), torch.randn(1, H, generator=g, device="cuda")
    a = ALPHA if B > 1 else 0.0
    got = []
    for _ in range(n):
        got.append((math.sqrt(1 - a) * priv + math.sqrt(a) * shared).to(DTYPES[c["dtype"]]))
        priv = 0.9 * priv + 0.436 * torch.randn(B, H, generator=g, device="cuda")
        shared = 0.9 * shared + 0.436 * torch.randn(1, H, generator=g, device="cuda")
    return got


def _prompt(c, seed):
    return _rn(_gen(seed, 2), DTYPES[c["dtype"]], c["B"], c["H"])


def _param(c):
    """The rule's parameter for the wanted density per row (scores are about N(0, WSTD^4 H r))."""
    z = NormalDist().inv_cdf(1.0 - c["density"])
    if c["rule"] == "topk":
        return float(max(1, int(c["density"] * c["I"])))
    return z if c["rule"] == "statistical_topk" else WSTD ** 2 * math.sqrt(c["H"] * c["r"]) * z


# ---------------------------------------------------------------------------------- prepare / run
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


@torch.no_grad()
def run(state):
    return state["run"](state)


def _sparse_layer(c, seed, l):
    gate, up, down, A, Bm = _weights(c, seed, l)
    return stx.SparseLayer(gate, up, down, A, Bm, act=c["act"], method=c["rule"], param=_param(c), max_batch=c["B"], has_gate=c["gate"])


def _prepare_layer(c, seed):
    xs = _tokens(c, seed, TOKENS)
    layer = _sparse_layer(c, seed, 0)
    layer.step(xs[-1])  # the token before: the cache holds its rows
    return dict(run=_run_layer, layer=layer, xs=xs)


def _run_layer(s):
    return [s["layer"].step(x) for x in s["xs"]]


def _prepare_stack(c, seed):
    xs = _tokens(c, seed, TOKENS)
    layers = [_sparse_layer(c, seed, l) for l in range(c["L"])]
    stack = stx.SparseStack(layers, c["B"])
    out = torch.empty(TOKENS, c["L"], c["B"], c["H"], dtype=DTYPES[c["dtype"]], device="cuda")
    stack.step(xs[-1])
    return dict(run=_run_stack, stack=stack, xs=xs, out=out)


def _run_stack(s):
    for x, o in zip(s["xs"], s["out"]):
        s["stack"].step(x, o)
    return s["out"]


def _mlp(c, seed):
    gate, up, down, A, Bm = _weights(c, seed, 0)
    with torch.device("cuda"):
        lora = stx.FastLoRAProjection(c["H"], c["I"], c["r"])
        mlp = stx.SkipMLP(c["H"], c["I"], 1.0 - c["density"], act_fn=c["act"])
    for lin, w in ((lora.down, A), (lora.up, Bm), (mlp.gate_proj, gate), (mlp.up_proj, up), (mlp.down_proj, down)):
        lin.weight = torch.nn.Parameter(w, requires_grad=False)
    mlp.initialize_weight_cache()
    return lora, mlp


def _prepare_dropin(c, seed):
    xs = _tokens(c, seed, TOKENS)
    lora, mlp = _mlp(c, seed)
    tau = _param(c)
    stx.compute_binary_mask(xs[-1], lora, "naive", threshold=tau, weight_cache=mlp.weight_cache)
    bufs = [torch.zeros(1, 1, dtype=DTYPES[c["dtype"]], device="cuda") for _ in range(2)]
    return dict(run=_run_dropin, lora=lora, mlp=mlp, xs=xs, tau=tau, bufs=bufs, act=c["act"])


def _run_dropin(s):
    masks, outs = [], []
    wc = s["mlp"].weight_cache
    for x in s["xs"]:
        masks.append(stx.compute_binary_mask(x, s["lora"], "naive", threshold=s["tau"], weight_cache=wc))
        y = stx.sparse_mlp_forward(x, wc.get_concat_weight(), wc.get_active_down_weight(), s["bufs"][0], s["bufs"][1], s["act"])
        outs.append(y.clone())
    return dict(masks=masks, outs=outs)


def _prepare_op(c, seed):
    gate, up, down, _, _ = _weights(c, seed, 0)
    dt = DTYPES[c["dtype"]]
    return dict(run=_run_op, x=_prompt(c, seed), concat=torch.cat([gate, up]), down=down.t().contiguous().t(), act=c["act"],
                bufs=[torch.zeros(c["B"], c["H"], dtype=dt, device="cuda"), torch.zeros(c["B"], 2 * c["I"], dtype=dt, device="cuda")])


def _run_op(s):
    # the op leaves act(gate) * up and up in the second buffer, as the reference's does
    return stx.sparse_mlp_forward(s["x"], s["concat"], s["down"], s["bufs"][0], s["bufs"][1], s["act"]), s["bufs"][1]


def _prepare_prefill(c, seed):
    lora, mlp = _mlp(c, seed)
    return dict(run=_run_prefill, lora=lora, mlp=mlp, x=_prompt(c, seed), tau=_param(c))


def _run_prefill(s):
    mask = stx.compute_binary_mask(s["x"], s["lora"], "naive", threshold=s["tau"], weight_cache=s["mlp"].weight_cache)
    return mask, s["mlp"](s["x"], use_sparse=True)


def _glue_inputs(c, seed):
    dt, g = DTYPES[c["dtype"]], _gen(seed, 3)
    n = (c["heads"] + 2 * c["kv"]) * c["hd"]
    lay = []
    for _ in range(c["L"]):
        lay.append(dict(qkv=_rn(g, dt, n), pend=_rn(g, dt, 1, c["H"]), wo=_rn(g, dt, c["H"], c["heads"] * c["hd"], std=WSTD),
                        ln1=1 + _rn(g, dt, c["H"], std=0.1), ln2=1 + _rn(g, dt, c["H"], std=0.1),
                        k=_rn(g, dt, c["kv"], c["max_len"], c["hd"]), v=_rn(g, dt, c["kv"], c["max_len"], c["hd"])))
    cfg = ls.LlamaSkipConfig(head_dim=c["hd"], max_len=c["max_len"])
    return lay, _rn(g, dt, 1, c["H"]), ls.rope_tables(cfg, "cuda")


def _prepare_glue(c, seed):
    lay, h0, (cos, sin) = _glue_inputs(c, seed)
    s = dict(run=_run_glue, lay=lay, h0=h0, pos=torch.full((1,), c["ctx"] - 1, dtype=torch.long, device="cuda"), cos=cos, sin=sin)
    ws = ls.attn_workspace(c["heads"], c["hd"], "cuda")

    def body():
        h, outs = h0.clone(), []
        for L in lay:
            x = ls.add_rmsnorm(h, L["pend"], L["ln1"], 1e-5, torch.empty_like(h))
            o = ls.attn_decode(L["qkv"], cos, sin, s["pos"], L["k"], L["v"], torch.empty(1, c["heads"] * c["hd"], dtype=h.dtype, device="cuda"),
                               c["heads"], c["kv"], c["hd"], ws)
            y = ls.norm_gemv(o, None, None, 0.0, L["wo"])
            outs += [x, o, y, ls.add_rmsnorm(h, y, L["ln2"], 1e-5, torch.empty_like(h))]
        return outs + [h]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        body()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    s["graph"] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(s["graph"]):
        s["outs"] = body()
    s["keep"] = ws
    return s


def _run_glue(s):
    s["graph"].replay()
    return s["outs"]


def _prepare_model(c, seed):
    cfg = ls.LlamaSkipConfig(vocab=c["vocab"], hidden=c["H"], intermediate=c["I"], layers=c["L"], heads=c["heads"], kv_heads=c["kv"],
                             head_dim=c["hd"], predictor_rank=c["r"], density=c["density"], act=c["act"], max_len=c["max_len"],
                             dtype=DTYPES[c["dtype"]])
    m = ls.LlamaSkipModel(cfg, "cuda", seed=seed)
    g = _gen(seed, 4)
    m.prefill(torch.randint(0, c["vocab"], (c["prompt"],), generator=g, device="cuda"))
    ids = torch.randint(0, c["vocab"], (TOKENS, 1), generator=g, device="cuda")
    start = m.pos.clone()
    m.decode_step()
    return dict(run=_run_model, model=m, ids=ids, start=start)


def _run_model(s):
    # scores a given continuation of the cached prompt: the tokens are the caller's, the logits are the result
    m, got = s["model"], []
    m.pos.copy_(s["start"])
    for t in s["ids"]:
        m.token.copy_(t)
        m.decode_step()
        got.append(m.logits.clone())
    return got


# ---------------------------------------------------------------------------------- what a pass cannot do without
@functools.lru_cache(None)
def _union(density, B):
    """Expected share of neurons that at least one of B rows activates (scores of the rows share ALPHA of their variance)."""
    if B == 1:
        return density
    n, z = NormalDist(), NormalDist().inv_cdf(1.0 - density)
    xs = [-6 + 12 * (i + 0.5) / 400 for i in range(400)]
    off = sum(n.pdf(u) * n.cdf((z - math.sqrt(ALPHA) * u) / math.sqrt(1 - ALPHA)) ** B for u in xs) * 12 / 400
    return min(1.0, max(density, 1.0 - off))


#: share of a token's active neurons that the token before did not have (measured: 0.26 for single streams at 20 %)
CHURN = 0.26


def work(case):
    c, s = case, SIZE[case["dtype"]]
    if c["kind"] == "glue":
        kv = 2 * c["ctx"] * c["kv"] * c["hd"] * s
        proj = c["H"] * c["heads"] * c["hd"]
        return {"bytes": c["L"] * (kv + proj * s + 8 * c["H"] * s), "flops": c["L"] * (2 * proj + 4 * c["ctx"] * c["heads"] * c["hd"])}
    H, I, m = c["H"], c["I"], 3 if c.get("gate", True) else 2
    if c["kind"] == "op":
        return {"bytes": s * (m * I * H + 2 * c["B"] * H + (m - 1) * c["B"] * I), "flops": 2 * m * c["B"] * H * I}
    r, B = c["r"], c.get("B", 1)
    if c["kind"] == "prefill":
        K = int(I * (1.0 - (1.0 - c["density"]) ** B))
        return {"bytes": s * (m * K * H + r * (H + I) + 2 * B * H) + I, "flops": 2 * B * (m * H * K + r * (H + I))}
    K = int(_union(c["density"], B) * I)
    # predictor weights and active rows in, rows that the cache did not hold out, rows of x and the result
    token = s * (r * (H + I) + m * K * H + CHURN * m * K * H + 2 * B * H)
    flops = 2 * B * (m * H * K + r * (H + I))
    if c["kind"] == "model":
        qkv = (c["heads"] + 2 * c["kv"]) * c["hd"] * H + c["heads"] * c["hd"] * H
        token += s * (qkv + 2 * (c["prompt"] + 2) * c["kv"] * c["hd"])
        flops += 2 * qkv
        return {"bytes": TOKENS * (c["L"] * token + s * c["vocab"] * H + 4 * c["vocab"]), "flops": TOKENS * (c["L"] * flops + 2 * c["vocab"] * H)}
    return {"bytes": TOKENS * c["L"] * token, "flops": TOKENS * c["L"] * flops}


def tolerance(case):
    """32-bit sums in another order; in 16 bits one rounding of the activations and of the result on either side.  Masks are
    whole values and reproducible bit for bit.  The model's logits differ by 8e-4 when its attention, norms and projections
    round in another order."""
    if case["kind"] == "model":
        return {"rel": 3e-3}
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}


# ---------------------------------------------------------------------------------- the same in 64 bits
def _act64(name, t):
    if name == "relu":
        return torch.relu(t)
    return torch.nn.functional.silu(t) if name == "silu" else torch.nn.functional.gelu(t, approximate="tanh")


def _mask64(c, x, A, Bm):
    """Union of the rows' masks; t and the scores carry the model's roundings, which the rule is defined on."""
    dt = DTYPES[c["dtype"]]
    on = torch.zeros(Bm.shape[0], dtype=torch.bool, device="cuda")
    for xb in x.split(1024):
        t = (xb.double() @ A.double().t()).to(dt)
        sc = (t.double() @ Bm.double().t()).to(dt)
        if c["rule"] == "topk":
            m = torch.zeros_like(sc, dtype=torch.bool).scatter_(1, sc.double().topk(int(_param(c)), dim=1).indices, True)
        elif c["rule"] == "statistical_topk":
            d = sc.double()
            m = d > d.mean(1, keepdim=True) + d.std(1, keepdim=True, unbiased=False) * _param(c)
        else:
            m = sc.double() >= torch.tensor(_param(c), dtype=torch.float32).to(dt).double().item()  # the threshold is of the model's type too
        on |= m.any(0)
    return on


def _mlp64(c, x, gate, up, down):
    x = x.double()
    if gate is None:
        return _act64(c["act"], x @ up.double().t()) @ down.double().t(), None, None
    u = x @ up.double().t()
    a = _act64(c["act"], x @ gate.double().t()) * u
    return a @ down.double().t(), a, u


def _rows(on, gate, up, down):
    return gate[on] if gate is not None else None, up[on], down[:, on]


@torch.no_grad()
def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "model":
        return None
    if kind == "glue":
        return _glue64(c, seed)
    if kind == "op":
        gate, up, down, _, _ = _weights(c, seed, 0)
        y, a, u = _mlp64(c, _prompt(c, seed), gate, up, down)
        return y, torch.cat([a, u], dim=1)
    if kind == "prefill":
        gate, up, down, A, Bm = _weights(c, seed, 0)
        x = _prompt(c, seed)
        on = _mask64(c, x, A, Bm)
        g, u, d = _rows(on, gate, up, down)
        return None, torch.cat([_mlp64(c, xb, g, u, d)[0] for xb in x.split(1024)])
    xs = _tokens(c, seed, TOKENS)
    outs = [[] for _ in xs]
    for l in range(c["L"]):
        gate, up, down, A, Bm = _weights(c, seed, l)
        for i, x in enumerate(xs):
            outs[i].append(_mlp64(c, x, *_rows(_mask64(c, x, A, Bm), gate, up, down))[0])
    if kind == "layer":
        return [o[0] for o in outs]
    if kind == "dropin":
        return dict(masks=None, outs=[o[0] for o in outs])
    return torch.stack([torch.stack(o) for o in outs])


def _glue64(c, seed):
    lay, h0, (cos, sin) = _glue_inputs(c, seed)
    dt, hd, pos = DTYPES[c["dtype"]], c["hd"], c["ctx"] - 1
    h, outs = h0.clone(), []

    def norm(h, w):
        d = h.double()
        return d * torch.rsqrt(d.pow(2).mean() + 1e-5) * w.double()

    def rope(t):
        t = t.double().view(-1, hd)
        rot = torch.cat([-t[:, hd // 2:], t[:, : hd // 2]], dim=1)
        return (t * cos[pos].double() + rot * sin[pos].double()).to(dt)

    for L in lay:
        h = (h.double() + L["pend"].double()).to(dt)
        outs.append(norm(h, L["ln1"]))
        q, k, v = L["qkv"].split([c["heads"] * hd, c["kv"] * hd, c["kv"] * hd])
        q, k = rope(q).double().view(c["kv"], -1, hd), rope(k)
        kc, vc = L["k"][:, : pos + 1].double(), L["v"][:, : pos + 1].double()
        kc[:, pos], vc[:, pos] = k.double(), v.double().view(-1, hd)
        o = torch.softmax(q @ kc.transpose(1, 2) / math.sqrt(hd), dim=-1) @ vc
        outs.append(o.reshape(1, -1))
        y = o.reshape(1, -1).to(dt).double() @ L["wo"].double().t()
        h = (h.double() + y.to(dt).double()).to(dt)
        outs += [y, norm(h, L["ln2"])]
    return outs + [h.double()]
