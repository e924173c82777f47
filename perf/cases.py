"""The work that users of this framework have it do, as cases that can be timed and checked.

Kinds of cases, each driven through the package's public entry points:

  rows       softmax || LayerNorm in fp32 (attention scores of 12 heads beside the layer's norm)
  norm_rope  RMSNorm || RoPE in bf16 (a decoder layer's norm beside the rotation of its queries)
  proj       two dense projections of the same activations (Q || K in tf32 with bias, k || v and gate || up in bf16)
  conv       the two branches of a down-sampling residual block, 3x3 stride 2 || 1x1 stride 2, in tf32
  attention  the causal attention block: QK^T, softmax and PV of groups of heads, software-pipelined
  bert       encoder layers of independent requests through the segment driver, tf32
  llama      the projection half of a decoder layer through the segment driver, bf16
  resnet     stages 2-4 of ResNet-18 through the segment driver, tf32

The first four are registered pairs, one fused launch each; `layers` of them over buffers of their own go out
in one call (a launch, a launch list or a captured graph, as `how` says), which is how a program with that
many layers issues them.  Activations are ~N(0,1), weights and norms as in the package's own workloads.
"""
import math

import torch
import torch.nn.functional as F

import bfuse_project_b200 as bf
from bfuse_project_b200 import segment
from bfuse_project_b200.attention import AttentionBlock

HEADS = 12                       # heads of the softmax case: the rows are heads x tokens
DEV = "cuda"


def listed():
    return [
        # one small call: the norm and the scores of a short prompt, where the launch itself counts
        dict(name="rows_short", kind="rows", tokens=64, keys=256, hidden=768, layers=1, how="launch"),
        # BERT-base at its usual length, all twelve layers
        dict(name="rows_bert", kind="rows", tokens=512, keys=512, hidden=768, layers=12, how="list"),
        # a long odd batch of rows: bound by memory alone
        dict(name="rows_long_odd", kind="rows", tokens=6007, keys=512, hidden=768, layers=1, how="launch"),
        # Llama-3-8B at 512 tokens, eight layers replayed from a graph
        dict(name="norm_rope_llama", kind="norm_rope", tokens=512, heads=32, dim=128, layers=8, how="graph"),
        # BERT-base Q || K projections with bias, twelve layers
        dict(name="proj_qk_tf32", kind="proj", dtype="tf32", tokens=512, k=768, n=768, bias=True, layers=12, how="list"),
        # Llama-3-8B k || v projections of a ragged prompt
        dict(name="proj_kv_ragged", kind="proj", dtype="bf16", tokens=333, k=4096, n=1024, bias=False, layers=8, how="list"),
        # Llama-3-8B gate || up while decoding for 16 sequences: bound by the weights
        dict(name="gate_up_decode", kind="proj", dtype="bf16", tokens=16, k=4096, n=14336, bias=False, layers=1, how="launch"),
        # the same at prefill
        dict(name="gate_up_prefill", kind="proj", dtype="bf16", tokens=2048, k=4096, n=14336, bias=False, layers=1, how="launch"),
        # GPT-2 attention, two groups of heads
        dict(name="attention_causal", kind="attention", heads=12, seq=1024, dim=64, groups=2),
        # the ResNet-18 branch pair at the benchmark's batch
        dict(name="conv_batch256", kind="conv", batch=256, ci=64, hw=56, co=128, layers=1, how="launch"),
        # a BERT-base encoder layer for two requests
        dict(name="bert_layer_x2", kind="bert", replicas=2, seq=512),
        # ResNet-18 stages 2-4 for a serving batch
        dict(name="resnet_stages_b32", kind="resnet", batch=32),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rows", "norm_rope", "proj", "proj", "conv", "attention", "bert", "llama", "resnet"])
    if kind == "rows":
        tokens = _log(rng, 16, 6000)
        layers = rng.randint(1, max(1, min(12, 6000 // tokens)))
        return dict(kind=kind, tokens=tokens, keys=rng.choice([128, 256, 384, 512]), hidden=rng.choice([384, 512, 768, 1024, 1536]),
                    layers=layers, how=rng.choice(["list", "graph"]) if layers > 1 else "launch")
    if kind == "norm_rope":
        tokens = _log(rng, 1, 6000)
        layers = rng.randint(1, max(1, min(8, 6000 // tokens)))
        return dict(kind=kind, tokens=tokens, heads=rng.choice([8, 16, 32]), dim=rng.choice([64, 128]), layers=layers,
                    how=rng.choice(["list", "graph"]) if layers > 1 else "launch")
    if kind == "proj":
        dtype = rng.choice(["tf32", "bf16"])
        k, n = rng.choice([(768, 768), (768, 3072), (3072, 768), (1024, 1024), (512, 2048)] if dtype == "tf32"
                          else [(4096, 1024), (4096, 4096), (4096, 14336), (2048, 2048), (14336, 4096), (2048, 8192)])
        tokens = _log(rng, 1, 2048)
        layers = rng.randint(1, 8) if k * n <= 5_000_000 and tokens <= 700 else 1
        return dict(kind=kind, dtype=dtype, tokens=tokens, k=k, n=n, bias=rng.random() < 0.5, layers=layers,
                    how=rng.choice(["list", "graph"]) if layers > 1 else "launch")
    if kind == "conv":
        ci, hw, co = rng.choice([(64, 56, 128), (128, 28, 256), (256, 14, 512)])
        return dict(kind=kind, batch=_log(rng, 1, 256), ci=ci, hw=hw, co=co, layers=1, how="launch")
    if kind == "attention":
        groups = rng.choice([1, 2, 4])
        return dict(kind=kind, heads=groups * rng.randint(1, 5), seq=rng.choice([128, 256, 384, 512, 768, 1024]), dim=rng.choice([64, 128]), groups=groups)
    if kind == "bert":
        return dict(kind=kind, replicas=rng.randint(1, 4), seq=rng.choice([128, 256, 384, 512]))
    if kind == "llama":
        return dict(kind=kind, seq=_log(rng, 1, 1024))
    return dict(kind=kind, batch=_log(rng, 1, 64))


# --------------------------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, device=DEV, generator=g) * std).to(dtype)


def _gain(g, n, dtype=torch.float32):
    return (torch.rand(n, device=DEV, generator=g) + 0.5).to(dtype)


def _layer_inputs(case, g):
    """The inputs of one registered pair, by name."""
    kind = case["kind"]
    if kind == "rows":
        t, c, h = case["tokens"], case["keys"], case["hidden"]
        return dict(scores=_randn(g, HEADS * t, c), x=_randn(g, t, h), gamma=_gain(g, h), beta=_gain(g, h))
    if kind == "norm_rope":
        t, heads, dim = case["tokens"], case["heads"], case["dim"]
        bf16 = torch.bfloat16
        return dict(x=_randn(g, t, heads * dim, dtype=bf16), w=_gain(g, heads * dim, bf16), q=_randn(g, t, heads, dim, dtype=bf16),
                    inv_freq=(500000.0 ** (-torch.arange(0, dim, 2, device=DEV, dtype=torch.float64) / dim)).float())
    if kind == "proj":
        dt = torch.float32 if case["dtype"] == "tf32" else torch.bfloat16
        t, k, n = case["tokens"], case["k"], case["n"]
        d = dict(a=_randn(g, t, k, dtype=dt), w1=_randn(g, n, k, std=0.02, dtype=dt), w2=_randn(g, n, k, std=0.02, dtype=dt))
        if case["bias"]:
            d.update(b1=_randn(g, n, std=0.1), b2=_randn(g, n, std=0.1))
        return d
    b, ci, hw, co = case["batch"], case["ci"], case["hw"], case["co"]
    return dict(x=_randn(g, b, ci, hw, hw), w3=_randn(g, co, ci, 3, 3, std=math.sqrt(2.0 / (9 * ci))), w1=_randn(g, co, ci, 1, 1, std=math.sqrt(2.0 / ci)))


def _segment_inputs(case, builder, g):
    """Fills the buffers a segment reads and nothing writes; returns them by name."""
    written = set().union(*(o.writes for o in builder.ops))
    given = {}
    for name, t in builder.buf.items():
        if name in written or name == "inv_freq":
            continue
        if name.startswith(("g1", "g2", "wn")):
            t.copy_(1.0 + 0.1 * _randn(g, *t.shape))
        elif name[0] == "b" and t.dim() == 1:
            t.copy_(_randn(g, *t.shape, std=0.1))
        elif t.dim() == 4 and "w_" in name:
            t.copy_(_randn(g, *t.shape, std=math.sqrt(1.0 / t[0].numel())))
        elif name[0] == "w":
            t.copy_(_randn(g, *t.shape, std=1.0 / math.sqrt(t.shape[-1])))
        else:
            t.copy_(_randn(g, *t.shape))
        given[name] = t
    return given


def _build(case, rt, seed):
    kind = case["kind"]
    if kind == "bert":
        b, ops = segment.bert_layer(rt, torch, replicas=case["replicas"], seq=case["seq"], seed=seed)
    elif kind == "llama":
        b, ops = segment.llama_layer_projections(rt, torch, seq=case["seq"], seed=seed)
    else:
        b, ops = segment.resnet18_stages(rt, torch, batch=case["batch"], seed=seed)
    return b, ops


# ------------------------------------------------------------------------------------------ the program

def _register_pair(case, rt, t):
    """Registers the pair of one layer; returns (fusion handle, outputs)."""
    kind, e = case["kind"], torch.empty
    p = lambda *names: [None if n is None else t[n].data_ptr() for n in names]
    if kind == "rows":
        y1, y2 = e(t["scores"].shape, device=DEV), e(t["x"].shape, device=DEV)
        a = rt.describe("softmax", bf.OP_SOFTMAX_F32, t["scores"].shape, p("scores") + [y1.data_ptr()], fparam=(0.125,))
        b = rt.describe("layernorm", bf.OP_LAYERNORM_F32, t["x"].shape, p("x", None, "gamma", "beta") + [y2.data_ptr()], fparam=(1e-5,))
    elif kind == "norm_rope":
        y1, y2 = e(t["x"].shape, device=DEV, dtype=torch.bfloat16), e(t["q"].shape, device=DEV, dtype=torch.bfloat16)
        a = rt.describe("rmsnorm", bf.OP_RMSNORM_BF16, t["x"].shape, p("x", "w") + [y1.data_ptr()], fparam=(1e-5,))
        b = rt.describe("rope", bf.OP_ROPE_BF16, t["q"].shape, p("q", "inv_freq") + [y2.data_ptr()])
    elif kind == "proj":
        op = bf.OP_GEMM_TF32 if case["dtype"] == "tf32" else bf.OP_GEMM_BF16
        m, k, n = case["tokens"], case["k"], case["n"]
        y1, y2 = (e(m, n, device=DEV, dtype=t["a"].dtype) for _ in range(2))
        a, b = (rt.describe("proj%d" % i, op, (1, m, n, k, 0, 0, 0), p("a", "w%d" % i, "b%d" % i if case["bias"] else None) + [y.data_ptr()])
                for i, y in ((1, y1), (2, y2)))
    else:
        n, ci, hw, co = case["batch"], case["ci"], case["hw"], case["co"]
        y1, y2 = (e(n, co, (hw - 1) // 2 + 1, (hw - 1) // 2 + 1, device=DEV) for _ in range(2))
        a = rt.describe("conv3x3_s2", bf.OP_CONV2D_TF32, (n, ci, hw, hw, co, 3, 3, 2, 1, 0, 0, 0), p("x", "w3") + [y1.data_ptr()])
        b = rt.describe("conv1x1_s2", bf.OP_CONV2D_TF32, (n, ci, hw, hw, co, 1, 1, 2, 0, 0, 0, 0), p("x", "w1") + [y2.data_ptr()])
    fusion = rt.register_fusion(rt.register_kernel(a), rt.register_kernel(b), bf.RANGE_SPLIT if kind in ("proj", "conv") else bf.ZIGZAG)
    return fusion, [y1, y2]


def prepare(case, seed):
    rt = bf.Runtime(0)
    g = _gen(seed)
    kind = case["kind"]
    if kind == "attention":
        h, s, d = case["heads"], case["seq"], case["dim"]
        q, k, vt = _randn(g, h, s, d), _randn(g, h, s, d), _randn(g, h, d, s)
        block = AttentionBlock(rt, torch, q, k, vt, groups=case["groups"])
        return dict(rt=rt, block=block, go=lambda: block.run_pipelined(None), out=[block.probs, block.out])
    if kind in ("bert", "llama", "resnet"):
        builder, ops = _build(case, rt, seed)
        _segment_inputs(case, builder, g)
        seg = segment.Segment(rt, ops)
        written = sorted(set().union(*(o.writes for o in ops)))
        return dict(rt=rt, keep=builder, go=seg.run_fused, out={n: builder.buf[n] for n in written})
    keep, fusions, outs = [], [], []
    for _ in range(case["layers"]):
        t = _layer_inputs(case, g)
        f, y = _register_pair(case, rt, t)
        keep.append(t)
        fusions.append(f)
        outs.append(y)
    if case["how"] == "graph":
        graph = rt.graph_create(fusions, bf.MODE_FUSED)
        go = lambda: rt.graph_launch(graph, None)
    elif case["how"] == "list":
        go = lambda: rt.launch_list(fusions, bf.MODE_FUSED, None)
    else:
        go = lambda: rt.launch_fused(fusions[0], None)
    return dict(rt=rt, keep=keep, go=go, out=outs)


def run(state):
    state["go"]()
    return state["out"]


# --------------------------------------------------------------------------------------------- the work

def _conv_work(n, ci, hw, co, k, stride, pad):
    o = (hw + 2 * pad - k) // stride + 1
    return 4 * (n * ci * hw * hw + co * ci * k * k + n * co * o * o), 2.0 * n * co * o * o * ci * k * k


def work(case):
    """Each input read once, each output written once; inputs that several operators share count once."""
    kind = case["kind"]
    if kind == "rows":
        t, c, h, n = case["tokens"], case["keys"], case["hidden"], case["layers"]
        return dict(bytes=n * 4 * (2 * HEADS * t * c + 2 * t * h + 2 * h), flops=n * (8.0 * HEADS * t * c + 8.0 * t * h))
    if kind == "norm_rope":
        t, h, n = case["tokens"], case["heads"] * case["dim"], case["layers"]
        return dict(bytes=n * (2 * (4 * t * h + h) + 2 * case["dim"]), flops=n * 7.0 * t * h)
    if kind == "proj":
        e = 4 if case["dtype"] == "tf32" else 2
        m, k, n, layers = case["tokens"], case["k"], case["n"], case["layers"]
        return dict(bytes=layers * (e * (m * k + 2 * n * k + 2 * m * n) + (8 * n if case["bias"] else 0)), flops=layers * 4.0 * m * n * k)
    if kind == "conv":
        n, ci, hw, co = case["batch"], case["ci"], case["hw"], case["co"]
        b3, f3 = _conv_work(n, ci, hw, co, 3, 2, 1)
        b1, f1 = _conv_work(n, ci, hw, co, 1, 2, 0)
        return dict(bytes=b3 + b1 - 4 * n * ci * hw * hw, flops=f3 + f1)
    if kind == "attention":
        h, s, d = case["heads"], case["seq"], case["dim"]
        return dict(bytes=4 * h * (4 * s * d + s * s), flops=4.0 * h * s * s * d)   # q, k, v, out and the probabilities
    if kind == "bert":
        r, s, h, f = case["replicas"], case["seq"], 768, 3072
        weights = 4 * h * h + 2 * h * f
        return dict(bytes=4.0 * r * (weights + 2 * s * h + 9 * s * h + s * f + 2 * 12 * s * s), flops=r * (2.0 * s * weights + 4.0 * s * s * h))
    if kind == "llama":
        s, h, kv, f = case["seq"], 4096, 1024, 14336
        weights = h * h + 2 * h * kv + 3 * h * f
        return dict(bytes=2.0 * (weights + s * (h + 2 * h + 3 * kv + 2 * h + 2 * f + h)), flops=2.0 * s * weights)
    n, byts, flops, ci, hw = case["batch"], 0, 0.0, 64, 56
    for co in (128, 256, 512):
        for c, w, k, st, pad in ((ci, hw, 3, 2, 1), (ci, hw, 1, 2, 0)) + 3 * ((co, hw // 2, 3, 1, 1),):
            b, fl = _conv_work(n, c, w, co, k, st, pad)
            byts, flops = byts + b, flops + fl
        ci, hw = co, hw // 2
    return dict(bytes=byts, flops=flops)


def tolerance(case):
    """About four times the distance from the 64-bit result that the type gives: 32-bit sums, tf32 operands of
    10 bits of fraction, bf16 outputs; for the chains of tf32 operators, the operators before included."""
    kind = case["kind"]
    if kind == "rows":
        return dict(rel=1e-6, max=1e-4)          # measured 7e-8
    if kind == "norm_rope":
        return dict(rel=7e-3, max=4e-2)          # measured 1.7e-3
    if kind == "proj":                           # measured 7.6e-4 and 1.7e-3
        return dict(rel=3e-3, max=3e-2) if case["dtype"] == "tf32" else dict(rel=7e-3, max=4e-2)
    if kind == "conv":
        return dict(rel=3e-3, max=3e-2)          # measured 7.7e-4
    if kind == "attention":
        return dict(rel=5e-3, max=1e-1)          # measured 1.3e-3
    if kind == "resnet":
        return dict(rel=3e-2, max=3e-1)          # measured 9e-3 after the ninth conv in a row
    return dict(rel=2e-2, max=2e-1)              # measured 4.8e-3


# ------------------------------------------------------------------------------------ the same in 64 bits

def _rope(q, inv_freq):
    # the angle is the product of two 32-bit numbers rounded to 32 bits, as the operator defines it
    ang = (torch.arange(q.shape[0], device=q.device, dtype=torch.float32)[:, None] * inv_freq[None, :]).double()[:, None, :]
    h = q.shape[-1] // 2
    a, b = q[..., :h].double(), q[..., h:].double()
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def _layernorm(x, gamma, beta, eps=1e-5):
    return F.layer_norm(x, x.shape[-1:], gamma.double(), beta.double(), eps)


def _rmsnorm(x, w, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _conv(x, w, stride, pad):
    """conv2d in 64 bits as one matrix product per image chunk."""
    n, o = x.shape[0], (x.shape[2] + 2 * pad - w.shape[2]) // stride + 1
    wm = w.double().reshape(w.shape[0], -1)
    out = torch.empty(n, w.shape[0], o, o, device=x.device, dtype=torch.float64)
    step = max(1, 64_000_000 // (wm.shape[1] * o * o))
    for i in range(0, n, step):
        cols = F.unfold(x[i:i + step].double(), w.shape[2], padding=pad, stride=stride)
        out[i:i + step] = (wm @ cols).reshape(-1, w.shape[0], o, o)
    return out


def _exact_layer(case, t):
    kind = case["kind"]
    if kind == "rows":
        return [torch.softmax(t["scores"].double() * 0.125, -1), _layernorm(t["x"].double(), t["gamma"], t["beta"])]
    if kind == "norm_rope":
        return [_rmsnorm(t["x"].double(), t["w"]), _rope(t["q"], t["inv_freq"])]
    if kind == "proj":
        a = t["a"].double()
        return [a @ t["w%d" % i].double().T + (t["b%d" % i].double() if case["bias"] else 0.0) for i in (1, 2)]
    return [_conv(t["x"], t["w3"], 2, 1), _conv(t["x"], t["w1"], 2, 0)]


def _exact_bert(case, v):
    out, s, hid, heads = {}, case["seq"], 768, 12
    d = hid // heads
    for r in range(case["replicas"]):
        sfx = "" if case["replicas"] == 1 else "_r%d" % r
        w = lambda n: v[n + sfx].double()
        o = {n: w("x") @ w("w" + n).T + w("b" + n) for n in "qkv"}
        # the segment reinterprets its buffers in the layout the next operator wants
        o["scores"] = torch.einsum("hsd,htd->hst", o["q"].reshape(heads, s, d), o["k"].reshape(heads, s, d))
        o["probs"] = torch.softmax(o["scores"] / math.sqrt(d), -1)
        o["ctx"] = torch.einsum("hst,hdt->hsd", o["probs"], o["v"].reshape(heads, d, s)).reshape(s, hid)
        o["attn"] = o["ctx"] @ w("wo").T
        o["h1"] = _layernorm(o["attn"] + w("x"), w("g1"), w("be1"))
        o["f1"] = o["h1"] @ w("w1").T
        o["f2"] = o["f1"] @ w("w2").T
        o["out"] = _layernorm(o["f2"] + o["h1"], w("g2"), w("be2"))
        out.update({n + sfx: t for n, t in o.items()})
    return out


def _exact_llama(case, v, inv_freq):
    s, d = case["seq"], 128
    w = lambda n: v[n].double()
    o = {"xn": _rmsnorm(w("x"), w("wn1"))}
    for n in "qkv":
        o[n] = o["xn"] @ w("w" + n).T
    for n, heads in (("q", 32), ("k", 8)):
        o[n + "_rot"] = _rope(o[n].reshape(s, heads, d), inv_freq).reshape(s, -1)
    o["hn"] = _rmsnorm(o["q_rot"], w("wn2"))
    o["gate"], o["up"] = o["hn"] @ w("wgate").T, o["hn"] @ w("wup").T
    o["down"] = o["gate"] @ w("wdown").T
    return o


def _exact_resnet(v):
    o, x = {}, v["s1"]
    for stage in (2, 3, 4):
        p = "s%d_" % stage
        o[p + "c1"] = _conv(x, v[p + "w_c1"], 2, 1)
        o[p + "sc"] = _conv(x, v[p + "w_sc"], 2, 0)
        x = o[p + "c1"]
        for n in ("c2", "u2c1", "u2c2"):
            x = o[p + n] = _conv(x, v[p + "w_" + n], 1, 1)
    return o


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "attention":
        h, s, d = case["heads"], case["seq"], case["dim"]
        q, k, vt = _randn(g, h, s, d), _randn(g, h, s, d), _randn(g, h, d, s)
        a = torch.einsum("hsd,htd->hst", q.double(), k.double()) / math.sqrt(d)
        a.masked_fill_(torch.ones(s, s, device=DEV, dtype=torch.bool).triu(1), -math.inf)
        p = torch.softmax(a, -1)
        return [p, torch.einsum("hst,hdt->hsd", p, vt.double())]
    if kind in ("bert", "llama", "resnet"):
        builder, _ = _build(case, bf.Runtime(0), seed)     # its buffers' names and shapes; no kernel of it runs here
        v = _segment_inputs(case, builder, g)
        if kind == "bert":
            return _exact_bert(case, v)
        return _exact_llama(case, v, builder.buf["inv_freq"]) if kind == "llama" else _exact_resnet(v)
    return [_exact_layer(case, _layer_inputs(case, g)) for _ in range(case["layers"])]
