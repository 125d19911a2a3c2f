"""The work a server built on this framework does with it, as cases that can be timed: prompts taken in (prefill), tokens generated for one
request or a batch of them (decode), rows of a speculative draft checked (verify), and running requests beside a joining prompt (step).

Three model shapes of the configurations, at their real layer sizes with fewer layers and a smaller vocabulary (in proportion to the depth), so
that several can be built quickly:

  flash     GLM-5.3-Flash: KDA, KDA, KDA and sparse latent attention, hyper-connections of four streams, one dense and three expert layers
            (288 NVFP4 experts, bf16 elsewhere), FP8 cache
  v32       DeepSeek-V3.2: three layers of rotary latent attention with the indexer, one dense and two expert layers (256 experts in groups),
            FP8 weights with 128 x 128 scales, FP8 cache
  gazutar   gazutar-flash: three gated delta-rule layers and one of windowed attention, 64 bf16 experts and 8 identities in groups, bf16 cache

One engine per shape is kept while cases of that shape run, as a server keeps it; a case's state are the sequences that its requests stand in.
Passes leave the state as it was: what a pass appends goes to forks of the state's sequences (a server's cached prefixes), which it frees.
Weights are drawn so that sublayers contribute to the stream as in a trained model, and so that a token's experts stand out of the router's
scores (close calls are rare, loads are uneven); they are values which the storage formats hold exactly.  Prompt tokens are uniform.
"""
from __future__ import annotations

import dataclasses
import math
import weakref
import zlib

import torch

VOCAB, STEPS, CHUNK, PAGE = 16384, 16, 2048, 64
DEV = "cuda"

FLASH = dict(H=4096, layers="kkkm", dense=1, heads=64, q_lora=1536, kv=512, dn=256, dr=0, dv=256, scale=256 ** -0.5, ff=12288, E=288, top=8, eff=2048,
             groups=1, keep=1, routed_scale=2.5, limit=10.0, ih=32, idim=128, itop=2048, pool=4, irot=0, kheads=64, kdim=128, rank=128, eps=1e-5, streams=4)
V32 = dict(H=7168, layers="mmm", dense=1, heads=128, q_lora=1536, kv=512, dn=128, dr=64, dv=128, scale=192 ** -0.5 * (0.1 * math.log(40.0) + 1) ** 2,
           ff=18432, E=256, top=8, eff=2048, groups=8, keep=4, routed_scale=2.5, limit=0.0, ih=64, idim=128, itop=2048, pool=1, irot=64, eps=1e-6, streams=1)
GAZUTAR = dict(H=4096, layers="ddda", dense=0, heads=32, kv_heads=8, dim=128, window=4096, E=64, identity=8, top=8, eff=2048, groups=8, keep=4, kheads=64,
               kdim=128, conv=4, rank=128, eps=1e-5)
SHAPES = {"flash": FLASH, "v32": V32, "gazutar": GAZUTAR}
# sequences and cache pages of the engine: several states of the largest batch, and the forks of one pass
ROOM = {"flash": dict(max_seqs=200, max_batch=32, max_ctx=8704, num_pages=5200), "v32": dict(max_seqs=64, max_batch=8, max_ctx=4608, num_pages=2000),
        "gazutar": dict(max_seqs=130, max_batch=16, max_ctx=4608, num_pages=3000)}


def listed():
    return [
        # a one-line question: what a chat user waits for before the first token; launches and latency
        dict(name="flash prefill 23", model="flash", kind="prefill", tokens=23),
        # one full prompt slice, the unit in which every long prompt is taken in
        dict(name="flash prefill 2048", model="flash", kind="prefill", tokens=2048),
        # a document: several slices, the last one ragged; rows see more keys than the sparse attention selects
        dict(name="flash prefill 5301", model="flash", kind="prefill", tokens=5301),
        # one user's answer at 8k of context: the headline of the benchmark
        dict(name="flash decode 1 at 8176", model="flash", kind="decode", batch=1, ctx=8176, least=8176),
        # a few users at once, at odd lengths of context
        dict(name="flash decode 5 ragged", model="flash", kind="decode", batch=5, ctx=1907, least=301),
        # a full continuous batch
        dict(name="flash decode 32", model="flash", kind="decode", batch=32, ctx=1040, least=620),
        # FP8 weights and rotary latent attention: an ordinary prompt
        dict(name="v32 prefill 777", model="v32", kind="prefill", tokens=777),
        # one user's answer, sparse selection at work
        dict(name="v32 decode 1 at 3001", model="v32", kind="decode", batch=1, ctx=3001, least=3001),
        # a speculative draft of five tokens checked in one pass
        dict(name="v32 verify 6 at 1500", model="v32", kind="verify", rows=6, ctx=1500),
        # bf16 experts, windowed attention, the general delta rule: a prompt
        dict(name="gazutar prefill 1500", model="gazutar", kind="prefill", tokens=1500),
        # a batch of answers
        dict(name="gazutar decode 12", model="gazutar", kind="decode", batch=12, ctx=1203, least=410),
        # running answers beside a joining prompt's slice in one step
        dict(name="gazutar step 7 + 391", model="gazutar", kind="step", batch=7, ctx=800, least=150, tokens=391),
    ]


def draw(rng):
    log = lambda lo, hi: max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    model = rng.choice(["flash", "flash", "v32", "gazutar"])
    top = {"flash": 5300, "v32": 1500, "gazutar": 3000}[model]
    kind = rng.choice({"flash": ["prefill", "decode"], "v32": ["prefill", "decode", "verify"], "gazutar": ["prefill", "decode", "step"]}[model])
    if kind == "prefill":
        return dict(model=model, kind=kind, tokens=log(5, top))
    if kind == "verify":
        return dict(model=model, kind=kind, rows=rng.randint(2, 8), ctx=log(150, 4000))
    batch = log(1, {"flash": 32, "v32": 8, "gazutar": 16}[model])
    ctx = log(150, min({"flash": 8176, "v32": 4000, "gazutar": 4000}[model], 33000 // batch))
    case = dict(model=model, kind=kind, batch=batch, ctx=ctx, least=rng.randint(max(100, ctx // 4), ctx) if batch > 1 else ctx)
    return dict(case, tokens=log(20, 1000)) if kind == "step" else case


# ------------------------------------------------------------------------------------------------ weights
def _specs(model: str) -> dict:
    """{canonical name: (kind, shape, ...)} of a shape's tensors."""
    c, out = SHAPES[model], {}
    H, lin = c["H"], (lambda o, i, s=1.0, kind="lin": (kind, (o, i), s / i ** 0.5))
    dense = "fp8" if model == "v32" else "lin"
    one = lambda n: ("around", (n,), 1.0, 0.1)
    out["embed.weight"], out["head.weight"] = ("embed", (VOCAB, H)), lin(VOCAB, H)
    tot = c["E"] + c.get("identity", 0)
    for i, t in enumerate(c["layers"]):
        p = f"layers.{i}."
        if model == "gazutar":
            for n in ("mix_norm", "ffn_norm"):
                out[p + n + ".weight"], out[p + n + ".bias"] = ("around", (H,), 0.35, 0.05), ("around", (H,), 0.0, 0.03)
        else:
            out[p + "attn_norm.weight"], out[p + "ffn_norm.weight"] = one(H), one(H)
        if c.get("streams", 1) > 1:
            n = c["streams"]
            for q in ("hc_attn.", "hc_ffn."):
                out[p + q + "fn"], out[p + q + "scale"], out[p + q + "base"] = lin(2 * n + n * n, n * H, 0.7, "f32"), one(3), ("around", (2 * n + n * n,), 0.0, 0.5)
        if t in "kd":
            k, C, r = p + "kda.", c["kheads"] * c["kdim"], c["rank"]
            out.update({k + "beta": lin(c["kheads"], H, 1.0), k + "f_a": lin(r, H), k + "g_a": lin(r, H), k + "f_b": lin(C, r), k + "g_b": lin(C, r),
                        k + "o_norm": one(c["kdim"]), k + "o": lin(H, C, 0.6), k + "a_log": ("between", (c["kheads"],), -1.0, 0.5)})
            out[k + "dt_bias"] = ("between", (c["kheads"], c["kdim"]), -5.0, 1.0) if t == "k" else ("between", (C,), -4.0, -1.0)
            for n in "qkv":
                out[k + n], out[k + "conv_" + n] = lin(C, H), ("between", (C, 4), -0.7, 0.7)
        elif t == "m":
            a, h = p + "attn.", c["heads"]
            out.update({a + "q_a": lin(c["q_lora"], H, kind=dense), a + "q_a_norm": one(c["q_lora"]), a + "q_b": lin(h * (c["dn"] + c["dr"]), c["q_lora"], 0.5 if c["dr"] else 1.0, dense),
                        a + "kv_a": lin(c["kv"] + c["dr"], H, kind=dense), a + "kv_a_norm": one(c["kv"]), a + "k_b": ("lin", (h, c["kv"], c["dn"]), c["kv"] ** -0.5),
                        a + "v_b": ("lin", (h, c["dv"], c["kv"]), c["kv"] ** -0.5), a + "o": lin(H, h * c["dv"], 1.0 if c["dr"] else 0.8, dense)})
            x = p + "indexer."
            out.update({x + "wq_b": lin(c["ih"] * c["idim"], c["q_lora"], kind=dense), x + "wk": lin(c["idim"], H, kind=dense), x + "k_norm.weight": one(c["idim"]),
                        x + "k_norm.bias": ("around", (c["idim"],), 0.0, 0.1), x + "weights_proj": lin(c["ih"], H, kind=dense)})
            if c["pool"] > 1:
                out[x + "gate"], out[x + "ape"] = lin(c["idim"], H), ("around", (c["pool"], c["idim"]), 0.0, 0.5)
        else:
            a, q, kv = p + "attn.", c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
            out.update({a + "q": lin(q, H), a + "k": lin(kv, H), a + "v": lin(kv, H), a + "o": lin(H, q), a + "g": lin(q, H), a + "q_norm": ("around", (q,), 1.5, 0.1),
                        a + "k_norm": one(kv), a + "v_mix": ("between", (), 0.3, 0.6)})
        m = p + "moe."
        if i < c["dense"]:
            out.update({p + "mlp.gate": lin(c["ff"], H, kind=dense), p + "mlp.up": lin(c["ff"], H, kind=dense), p + "mlp.down": lin(H, c["ff"], 0.8, dense)})
            continue
        ex = {"flash": "nvfp4", "v32": "fp8", "gazutar": "lin"}[model]
        out[m + "router"], out[m + "router_bias"] = ("router", (tot, H), i), ("around", (tot,), 0.0, 0.002 if model == "gazutar" else 0.01)
        for e in [f"experts.{j}." for j in range(c["E"])] + ([] if model == "gazutar" else ["shared.0."]):
            out[m + e + "gate"], out[m + e + "up"], out[m + e + "down"] = lin(c["eff"], H, kind=ex), lin(c["eff"], H, kind=ex), lin(H, c["eff"], 0.8, ex)
    out["final_norm.weight"] = one(H)
    if model == "gazutar":
        out["final_norm.bias"] = ("around", (H,), 0.0, 0.03)
    return out


class Weights:
    """A shape's tensors by canonical name, made when asked for: fp32 values that the format in which the engine keeps them holds exactly."""

    def __init__(self, model: str):
        self.model, self.c, self.specs = model, SHAPES[model], _specs(model)

    def __contains__(self, name):
        return name in self.specs

    def _gen(self, name):
        return torch.Generator(device=DEV).manual_seed(zlib.crc32(f"{self.model}/{name}".encode()))

    def _directions(self):
        """What in a token's embedding asks for each expert."""
        n = self.c["E"] + self.c.get("identity", 0)
        return torch.randn(n, self.c["H"], generator=self._gen("directions"), device=DEV) / self.c["H"] ** 0.5

    def __getitem__(self, name):
        kind, shape, *a = self.specs[name]
        g = self._gen(name)
        if kind == "between":
            return a[0] + (a[1] - a[0]) * torch.rand(shape, generator=g, device=DEV)
        if kind == "around":
            return a[0] + a[1] * torch.randn(shape, generator=g, device=DEV)
        if kind == "embed":
            # the experts that a token asks for: `top` of them, in `keep` of the groups
            n, per = self.c["E"] + self.c.get("identity", 0), (self.c["E"] + self.c.get("identity", 0)) // self.c["groups"]
            luck = torch.rand(shape[0], n, generator=g, device=DEV)
            if self.c["groups"] > 1:
                grp = torch.rand(shape[0], self.c["groups"], generator=g, device=DEV).topk(self.c["keep"]).indices
                own = luck.view(shape[0], self.c["groups"], per).topk(self.c["top"] // self.c["keep"], dim=2).indices
                ids = (grp[:, :, None] * per + own.gather(1, grp[:, :, None].expand(-1, -1, own.shape[2]))).flatten(1)
            else:
                ids = luck.topk(self.c["top"]).indices
            u = self._directions()
            t = torch.randn(shape, generator=g, device=DEV)
            for k in range(ids.shape[1]):
                t += 11.0 * u[ids[:, k]]
            return t.bfloat16().float()
        if kind == "router":
            # every layer sends the same wish to other experts (whole groups further on)
            n = shape[0]
            return (0.6 if self.model == "gazutar" else 0.33) * self._directions()[(torch.arange(n, device=DEV) + a[0] * (n // self.c["groups"] if self.c["groups"] > 1 else 37)) % n]
        if kind == "nvfp4":
            # 4-bit values times a scale per 16 that E4M3 holds times one power of two; every block and the whole tensor reach the top of their range
            grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0], device=DEV)
            v = grid[torch.randint(0, 16, shape, generator=g, device=DEV)].view(shape[0], shape[1] // 16, 16)
            v[..., 0] = torch.where(v[..., 0] < 0, -6.0, 6.0)
            s = torch.randint(9, 15, (shape[0], shape[1] // 16, 1), generator=g, device=DEV).float() * 32
            s[0, 0] = 448.0
            return (v * s).view(shape) * 2.0 ** round(math.log2(a[0] / 1180.0))
        t = torch.randn(shape, generator=g, device=DEV) * a[0]
        if kind == "fp8":
            s = 2.0 ** math.ceil(math.log2(4.6 * a[0] / 448))
            t.clamp_(-288 * s, 288 * s)
            t[::128, ::128] = 288 * s
            return (t / s).to(torch.float8_e4m3fn).float() * s
        return t if kind == "f32" else t.bfloat16().float()


# ------------------------------------------------------------------------------------------------ the program around a case
_kept = {}


def _engine(model: str):
    """The engine that serves a shape's cases; one at a time is kept."""
    if model not in _kept:
        from layerstorm_b200.models.block_model import BlockModel
        from layerstorm_b200.models.config import get_preset
        from layerstorm_b200.models.device_model import DeviceModel
        from layerstorm_b200.runtime.engine import Engine
        _kept.clear()
        torch.cuda.empty_cache()
        cfg = get_preset({"flash": "glm-5.3-flash", "v32": "deepseek-v3.2", "gazutar": "gazutar-flash"}[model])
        n = len(SHAPES[model]["layers"])
        if cfg.blocks:
            cfg = dataclasses.replace(cfg, vocab=VOCAB, blocks=cfg.blocks[:n], layer_types=[])
            m = BlockModel.from_state_dict(cfg, Weights(model), DEV, page=PAGE)
        else:
            cfg = dataclasses.replace(cfg, vocab=VOCAB, n_layers=n, layer_types=list(cfg.layer_types[:n]), first_k_dense=SHAPES[model]["dense"])
            m = DeviceModel.from_state_dict(cfg, Weights(model), DEV, kv_fmt="fp8", page=PAGE)
        torch.cuda.empty_cache()
        _kept[model] = Engine(m, prefill_chunk=CHUNK, **ROOM[model])
    return _kept[model]


def _lengths(case) -> list:
    """Context of each sequence of the batch: from the longest to the shortest."""
    b = case.get("batch", 1)
    return [case["ctx"] - (case["ctx"] - case.get("least", case["ctx"])) * j // max(1, b - 1) for j in range(b)]


def _tokens(case, seed: int) -> dict:
    """Token ids of the contexts that the sequences stand in and of what a pass feeds."""
    g = torch.Generator().manual_seed(seed)
    ids = lambda *n: torch.randint(0, VOCAB, n, generator=g).tolist()
    if case["kind"] == "prefill":
        return {"contexts": [], "fed": ids(case["tokens"])}
    contexts = [ids(n) for n in _lengths(case)]
    if case["kind"] == "verify":
        return {"contexts": contexts, "fed": ids(case["rows"])}
    return {"contexts": contexts, "fed": ids(STEPS if case["kind"] == "decode" else 1, len(contexts)), "slice": ids(case.get("tokens", 0))}


class State:
    """A case's sequences in the engine; they go when it goes."""

    def __init__(self, case, seed):
        self.kind, self.eng, t = case["kind"], _engine(case["model"]), _tokens(case, seed)
        self.fed, self.slice, self.sids = t["fed"], t.get("slice"), []
        weakref.finalize(self, lambda eng, sids: [eng.free_sequence(s) for s in sids], self.eng, self.sids)
        for c in t["contexts"]:
            self.sids.append(self.eng.create_sequence())
            self.eng.prefill(self.sids[-1], c)


def prepare(case, seed):
    return State(case, seed)


def run(s):
    eng = s.eng
    if s.kind == "prefill":
        sid = eng.create_sequence()
        try:
            return eng.prefill(sid, s.fed, want_logits=True)[1]
        finally:
            eng.free_sequence(sid)
    if s.kind == "verify":
        return eng.forward_rows(s.sids[0], s.fed, commit=False)
    sids = [eng.fork_sequence(p) for p in s.sids]
    try:
        if s.kind == "decode":
            return [eng.decode(sids, toks, return_logits=True)[1] for toks in s.fed]
        from layerstorm_b200.runtime.engine import Portion
        sids.append(eng.create_sequence())
        portions = [Portion(sid, [tok], [0]) for sid, tok in zip(sids, s.fed[0])] + [Portion(sids[-1], s.slice, [len(s.slice) - 1])]
        return torch.cat([logits for _, logits in eng.step(portions, return_logits=True)])
    finally:
        for sid in sids:
            eng.free_sequence(sid)


# ------------------------------------------------------------------------------------------------ what a case cannot do without
def _step_work(c, model, rows, keys, seqs) -> tuple:
    """(bytes, flops) of one step: `rows` new tokens of `seqs` sequences, `keys`: how many cached positions the rows see together."""
    H, wb = c["H"], {"flash": 2.0, "v32": 1.0, "gazutar": 2.0}[model]
    eb = {"flash": 0.5625, "v32": 1.0, "gazutar": 2.0}[model]
    by, fl = 0.0, 0.0
    for i, t in enumerate(c["layers"]):
        if t in "kd":
            C = c["kheads"] * c["kdim"]
            n = H * (4 * C + c["kheads"] + 2 * c["rank"]) + 2 * C * c["rank"]
            state = seqs * C * c["kdim"] * 4
            by, fl = by + n * 2 + 2 * state, fl + 2 * rows * n + 8 * rows * C * c["kdim"]
        elif t == "m":
            h = c["heads"]
            n = H * (c["q_lora"] + c["kv"] + c["dr"] + c["idim"] * (2 if c["pool"] > 1 else 1) + c["ih"]) + c["q_lora"] * (h * (c["dn"] + c["dr"]) + c["ih"] * c["idim"]) + h * c["dv"] * H
            ab = h * c["kv"] * (c["dn"] + c["dv"])
            seen = min(keys / rows, c["itop"])
            by += n * wb + ab * 2 + (min(seqs * keys / rows, seen * rows) * (c["kv"] + 2 * c["dr"]) + keys / rows * seqs * c["idim"] / c["pool"])
            fl += 2 * rows * (n + ab) + 2 * rows * seen * h * (2 * c["kv"] + c["dr"]) + 2 * keys / c["pool"] * c["ih"] * c["idim"]
        else:
            q, kv = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
            n = H * (3 * q + 2 * kv)
            by, fl = by + n * 2 + keys / rows * seqs * 2 * kv * 2, fl + 2 * rows * n + 4 * keys * q
        if i < c["dense"]:
            by, fl = by + 3 * H * c["ff"] * wb, fl + 6 * rows * H * c["ff"]
        else:
            shared = 0 if model == "gazutar" else 1
            hit = c["E"] * (1 - (1 - c["top"] / (c["E"] + c.get("identity", 0))) ** rows) + shared
            by += 3 * H * c["eff"] * eb * hit + c["E"] * H * 4
            fl += 6 * rows * (c["top"] * c["E"] / (c["E"] + c.get("identity", 0)) + shared) * H * c["eff"] + 2 * rows * H * c["E"]
    return by + rows * H * 2, fl


def work(case):
    c, model, kind = SHAPES[case["model"]], case["model"], case["kind"]
    by = fl = 0.0
    if kind == "prefill":
        steps, outs = [(n, sum(range(at + 1, at + n + 1)), 1) for at in range(0, case["tokens"], CHUNK) for n in [min(CHUNK, case["tokens"] - at)]], 1
    elif kind == "verify":
        steps, outs = [(case["rows"], sum(case["ctx"] + j + 1 for j in range(case["rows"])), 1)], case["rows"]
    elif kind == "decode":
        steps, outs = [(case["batch"], sum(_lengths(case)) + case["batch"] * (t + 1), case["batch"]) for t in range(STEPS)], case["batch"] * STEPS
    else:
        n = case["tokens"]
        steps, outs = [(case["batch"] + n, sum(_lengths(case)) + n * (n + 1) // 2, case["batch"] + 1)], case["batch"] + 1
    for rows, keys, seqs in steps:
        b, f = _step_work(c, model, rows, keys, seqs)
        by, fl = by + b, fl + f
    heads = STEPS if kind == "decode" else 1
    return {"bytes": by + heads * VOCAB * c["H"] * 2 + outs * VOCAB * 4, "flops": fl + 2 * outs * VOCAB * c["H"]}


def tolerance(case):
    # bf16 activations through the layers, and for the sparse models an FP8 cache and a selection of keys that close calls turn: about four times
    # what the outputs are off from 64 bits (0.006, 0.01, 0.003)
    return {"rel": {"flash": 0.025, "v32": 0.03, "gazutar": 0.012}[case["model"]], "max": 0.5}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope(x, pos, freq):
    """Adjacent pairs turned by pos * freq; x [T, ..., 2 len(freq)]."""
    a = (pos.double()[:, None] * freq).view(-1, *[1] * (x.dim() - 2), freq.numel())
    e, o = x[..., 0::2], x[..., 1::2]
    return torch.stack((e * a.cos() - o * a.sin(), e * a.sin() + o * a.cos()), -1).flatten(-2)


def _yarn(d):
    """Rotation speeds of DeepSeek-V3.2: base 10000, YaRN factor 40 over 4096 positions between 32 and 1 turns."""
    base = 10000.0 ** (-torch.arange(0, d, 2, dtype=torch.float64, device=DEV) / d)
    at = lambda turns: d * math.log(4096 / (turns * 2 * math.pi)) / (2 * math.log(10000.0))
    lo, hi = max(math.floor(at(32)), 0), min(math.ceil(at(1)), d - 1)
    ramp = ((torch.arange(d // 2, dtype=torch.float64, device=DEV) - lo) / (hi - lo)).clamp(0, 1)
    return base / 40 * ramp + base * (1 - ramp)


def _glu(x, w, p, limit=0.0):
    g, u = x @ w(p + "gate").T, x @ w(p + "up").T
    if limit:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return (g * torch.sigmoid(g) * u) @ w(p + "down").T


def _moe(c, model, w, p, x):
    logits, bias = x @ w(p + "router").T, w(p + "router_bias")
    score = torch.softmax(logits, -1) if model == "gazutar" else torch.sigmoid(logits)
    sel = score + bias
    if c["groups"] > 1:
        g = sel.view(len(x), c["groups"], -1)
        best = g.amax(-1) if model == "gazutar" else g.topk(2, -1).values.sum(-1)
        keep = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(c["keep"], 1).indices, True)
        sel = sel.masked_fill(~keep.repeat_interleave(g.shape[2], 1), -math.inf)
    ids = sel.topk(c["top"], 1).indices
    wt = score.gather(1, ids)
    if model != "gazutar":
        wt = wt / wt.sum(-1, keepdim=True) * c["routed_scale"]
    y = torch.zeros_like(x) if model == "gazutar" else _glu(x, w, p + "shared.0.", c["limit"])
    for e in ids.unique().tolist():
        row, k = (ids == e).nonzero(as_tuple=True)
        xe = x[row]
        y.index_add_(0, row, wt[row, k][:, None] * (xe if e >= c["E"] else _glu(xe, w, p + f"experts.{e}.", c.get("limit", 0.0))))
    return y


def _delta(c, w, p, x, starts, bounded):
    """Gated delta rule over sequences laid end to end; `bounded`: the decay exp(-5 sigmoid(..)), else exp(-exp(a) softplus(..))."""
    h, d, N = c["kheads"], c["kdim"], len(x)
    ends = starts[1:] + [N]

    def conv(n):
        raw, taps = x @ w(p + n).T, w(p + "conv_" + n)
        out = raw * taps[:, 3]
        for s, e in zip(starts, ends):
            for j in range(1, 4):
                out[s + j: e] += raw[s: max(s, e - j)] * taps[:, 3 - j]
        return (out * torch.sigmoid(out)).view(N, h, d)

    q, k, v = conv("q"), conv("k"), conv("v")
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(x @ w(p + "beta").T)
    a = ((x @ w(p + "f_a").T) @ w(p + "f_b").T + w(p + "dt_bias").view(-1)).view(N, h, d)
    rate = w(p + "a_log").exp()[None, :, None]
    decay = torch.exp(-5.0 * torch.sigmoid(rate * a)) if bounded else torch.exp(-rate * torch.nn.functional.softplus(a))
    del a
    core = torch.empty_like(v)
    longest, lens = max(e - s for s, e in zip(starts, ends)), torch.tensor([e - s for s, e in zip(starts, ends)], device=DEV)
    at = torch.tensor(starts, device=DEV)
    S = torch.zeros(len(starts) * h, d, d, dtype=torch.float64, device=DEV)
    for t in range(longest):
        # sequences that have ended go on with their last row; nothing reads what comes of it
        r = at + torch.clamp(lens - 1, max=t)
        f = lambda y: y[r].view(-1, d)
        S.mul_(f(decay)[:, None, :])
        kt = f(k)
        u = (f(v) - torch.bmm(S, kt[:, :, None])[:, :, 0]) * beta[r].view(-1, 1)
        S.baddbmm_(u[:, :, None], kt[:, None, :])
        o = torch.bmm(S, f(q)[:, :, None])[:, :, 0].view(len(starts), h, d)
        live = lens > t
        core[r[live]] = o[live]
    core = _rms(core, w(p + "o_norm"), c["eps"]) * torch.sigmoid((x @ w(p + "g_a").T) @ w(p + "g_b").T).view(N, h, d)
    return core.view(N, h * d) @ w(p + "o").T


def _mla(c, w, p, x, starts, rows):
    """Latent attention of the rows `rows` over their sequences, keys chosen by the indexer."""
    a, ix, h, ends = p + "attn.", p + "indexer.", c["heads"], starts[1:] + [len(x)]
    pos = torch.cat([torch.arange(e - s, device=DEV) for s, e in zip(starts, ends)])
    rot = _yarn(c["dr"]) if c["dr"] else None
    kv = x @ w(a + "kv_a").T
    key = _rms(kv[:, : c["kv"]], w(a + "kv_a_norm"), c["eps"])
    if c["dr"]:
        key = torch.cat([key, _rope(kv[:, c["kv"]:], pos, rot)], 1)
    xr, pr = x[rows], pos[rows]
    qc = _rms(xr @ w(a + "q_a").T, w(a + "q_a_norm"), c["eps"])
    q = (qc @ w(a + "q_b").T).view(len(rows), h, -1)
    ql = torch.einsum("thn,hln->thl", q[..., : c["dn"]], w(a + "k_b"))
    if c["dr"]:
        ql = torch.cat([ql, _rope(q[..., c["dn"]:], pr, rot)], -1)
    ik = torch.nn.functional.layer_norm(x @ w(ix + "wk").T, (c["idim"],), w(ix + "k_norm.weight"), w(ix + "k_norm.bias"), 1e-6)
    iq = (qc @ w(ix + "wq_b").T).view(len(rows), c["ih"], c["idim"])
    if c["irot"]:
        r = c["irot"]
        ik = torch.cat([_rope(ik[:, :r], pos, rot), ik[:, r:]], 1)
        iq = torch.cat([_rope(iq[..., :r], pr, rot), iq[..., r:]], -1)
    iw = xr @ w(ix + "weights_proj").T
    gate = x @ w(ix + "gate").T if c["pool"] > 1 else None
    vb, out = w(a + "v_b"), torch.empty(len(rows), h, c["dv"], dtype=torch.float64, device=DEV)
    P, budget = c["pool"], c["itop"] // c["pool"]
    for s, e in zip(starts, ends):
        mine = ((rows >= s) & (rows < e)).nonzero()[:, 0]
        ent = ik[s:e][: (e - s) // P * P].view(-1, P, c["idim"])
        ent = (torch.softmax(gate[s:e][: len(ent) * P].view(-1, P, c["idim"]) + w(ix + "ape"), 1) * ent).sum(1) if P > 1 else ent[:, 0]
        for b in mine.split(max(1, (1 << 27) // (h * (e - s)))):
            n = (pr[b] + 1) // P                                                     # whole pools that a row sees
            allow = torch.arange(e - s, device=DEV)[None] <= pr[b][:, None]
            if int(n.max()) > budget:
                sc = (torch.relu(torch.einsum("thd,nd->thn", iq[b], ent)) * iw[b][:, :, None]).sum(1)
                sc = sc.masked_fill(torch.arange(len(ent), device=DEV)[None] >= n[:, None], -math.inf)
                pick = torch.zeros_like(sc, dtype=torch.bool).scatter_(1, sc.topk(budget, 1).indices, True) | (n <= budget)[:, None]
                pick = torch.cat([pick.repeat_interleave(P, 1), torch.ones(len(b), e - s - len(ent) * P, dtype=torch.bool, device=DEV)], 1)
                allow &= pick | (torch.arange(e - s, device=DEV)[None] >= n[:, None] * P)
            pr_ = torch.softmax((torch.einsum("thl,sl->ths", ql[b], key[s:e]) * c["scale"]).masked_fill(~allow[:, None], -math.inf), -1)
            out[b] = torch.einsum("thl,hvl->thv", torch.einsum("ths,sl->thl", pr_, key[s:e, : c["kv"]]), vb)
    return out.flatten(1) @ w(a + "o").T


def _attention(c, w, p, x, starts, rows):
    """Windowed attention with a slope per head and a gate."""
    a, ends, G = p + "attn.", starts[1:] + [len(x)], c["heads"] // c["kv_heads"]
    q = _rms(x[rows] @ w(a + "q").T, w(a + "q_norm"), c["eps"]).view(len(rows), c["heads"], -1)
    k = _rms(x @ w(a + "k").T, w(a + "k_norm"), c["eps"]).view(len(x), c["kv_heads"], -1)
    v = (x @ w(a + "v").T).view(len(x), c["kv_heads"], -1)
    slope = 2.0 ** (-8.0 * (torch.arange(c["heads"], dtype=torch.float64, device=DEV) + 1) / c["heads"])
    out = torch.empty_like(q)
    for s, e in zip(starts, ends):
        mine = ((rows >= s) & (rows < e)).nonzero()[:, 0]
        kk, vv = k[s:e].repeat_interleave(G, 1), v[s:e].repeat_interleave(G, 1)
        for b in mine.split(max(1, (1 << 27) // (c["heads"] * (e - s)))):
            dist = (rows[b] - s)[:, None] - torch.arange(e - s, device=DEV)[None]
            sc = torch.einsum("thd,shd->ths", q[b], kk) * c["dim"] ** -0.5 - slope[None, :, None] * dist[:, None]
            out[b] = torch.einsum("ths,shd->thd", torch.softmax(sc.masked_fill(((dist < 0) | (dist >= c["window"]))[:, None], -math.inf), -1), vv)
    return (out.flatten(1) * torch.sigmoid(x[rows] @ w(a + "g").T)) @ w(a + "o").T


class _Streams:
    """Hyper-connections: four copies of the stream, mixed around every sublayer by gates that they set themselves."""

    def __init__(self, c, h):
        self.c, self.res, self.left = c, h[:, None].repeat(1, c["streams"], 1), None

    def enter(self, w, p, norm):
        n = self.c["streams"]
        flat = self.res.flatten(1)
        m = (flat @ w(p + "fn").T) * torch.rsqrt(flat.square().mean(-1, keepdim=True) + self.c["eps"])
        sc, base = w(p + "scale"), w(p + "base")
        pre = torch.sigmoid(m[:, :n] * sc[0] + base[:n]) + 1e-6
        self.post = torch.sigmoid(m[:, n: 2 * n] * sc[1] + base[n: 2 * n]) * 2.0
        k = torch.softmax((m[:, 2 * n:] * sc[2] + base[2 * n:]).view(-1, n, n), -1) + 1e-6
        k = k / (k.sum(-2, keepdim=True) + 1e-6)
        for _ in range(19):
            k = k / (k.sum(-1, keepdim=True) + 1e-6)
            k = k / (k.sum(-2, keepdim=True) + 1e-6)
        self.comb = k
        return _rms((pre[:, :, None] * self.res).sum(1), norm, self.c["eps"])

    def only(self, rows):
        self.res, self.post, self.comb = self.res[rows], self.post[rows], self.comb[rows]

    def leave(self, y):
        self.res = torch.einsum("tij,tih->tjh", self.comb, self.res) + self.post[:, :, None] * y[:, None]


def _forward(model, seqs, want):
    """Logits [rows, vocab] of the rows `want` of sequences laid end to end."""
    c, W = SHAPES[model], Weights(model)
    w = lambda name: W[name].double()
    starts = [0]
    for s in seqs[:-1]:
        starts.append(starts[-1] + len(s))
    x = W["embed.weight"][torch.tensor([t for s in seqs for t in s], device=DEV)].double()
    want, every = torch.tensor(want, device=DEV), torch.arange(len(x), device=DEV)
    hc = _Streams(c, x) if c.get("streams", 1) > 1 else None
    for i, t in enumerate(c["layers"]):
        p, last = f"layers.{i}.", i == len(c["layers"]) - 1
        rows = want if last else every
        if hc:
            h = hc.enter(w, p + "hc_attn.", w(p + "attn_norm.weight"))
        else:
            h = x if model == "gazutar" else _rms(x, w(p + "attn_norm.weight"), c["eps"])
        if t in "kd":
            y = _delta(c, w, p + "kda.", h, starts, t == "k")[rows]
        else:
            y = (_mla if t == "m" else _attention)(c, w, p, h, starts, rows)
        ff = (lambda z: _glu(z, w, p + "mlp.", c.get("limit", 0.0))) if i < c["dense"] else (lambda z: _moe(c, model, w, p + "moe.", z))
        norm = lambda z, n: torch.nn.functional.layer_norm(z, (c["H"],), w(p + n + ".weight"), w(p + n + ".bias"), c["eps"])
        if hc:
            if last:
                hc.only(rows)
            hc.leave(y)
            hc.leave(ff(hc.enter(w, p + "hc_ffn.", w(p + "ffn_norm.weight"))))
        elif model == "gazutar":
            x = x[rows] + norm(y, "mix_norm")
            x = x + norm(ff(x), "ffn_norm")
        else:
            x = x[rows] + y
            x = x + ff(_rms(x, w(p + "ffn_norm.weight"), c["eps"]))
    if hc:
        x = hc.res.mean(1)
    if model == "gazutar":
        x = torch.nn.functional.layer_norm(x, (c["H"],), w("final_norm.weight"), w("final_norm.bias"), c["eps"])
    else:
        x = _rms(x, w("final_norm.weight"), c["eps"])
    return x @ w("head.weight").T


def exact(case, seed):
    t, kind = _tokens(case, seed), case["kind"]
    ctx, fed = t["contexts"], t["fed"]
    if kind == "prefill":
        return _forward(case["model"], [fed], [len(fed) - 1])[0]
    if kind == "verify":
        return _forward(case["model"], [ctx[0] + fed], list(range(len(ctx[0]), len(ctx[0]) + len(fed))))
    seqs = [c + [f[j] for f in fed] for j, c in enumerate(ctx)] + ([t["slice"]] if kind == "step" else [])
    ends, at = [], 0
    for s in seqs:
        at += len(s)
        ends.append(at)
    if kind == "step":
        return _forward(case["model"], seqs, [e - 1 for e in ends])
    out = _forward(case["model"], seqs, [e - STEPS + k for k in range(STEPS) for e in ends])
    return [out[k * len(seqs): (k + 1) * len(seqs)] for k in range(STEPS)]
