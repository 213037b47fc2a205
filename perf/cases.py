"""The work whose time this package is judged by: single layers and two whole calls, each through the entry point a program uses.

A case is a dict of plain values; `kind` names the layer, the rest its sizes.  `prepare` builds what a program holds before the call
(weights, module, state pool, inputs), `run` is one call, `exact` is the same result in 64-bit torch, `work` what the call cannot do
without, `tolerance` how far another correct implementation of the same precision may be off."""
import math

import torch

import lit_llama_b200 as P
from lit_llama_b200 import mixers as X
from lit_llama_b200.int8 import Linear8bitLt
from lit_llama_b200.lugovik import Lugovik, LugovikConfig
from lit_llama_b200.quantization import ColBlockQuantizedLinear
from lit_llama_b200.state import SequenceStatePool

BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
EPS = 1e-6
#: (out, in) of the linears of the 7B and 13B models: attention input and output, feed-forward in and out, head
LINEARS = [(12288, 4096), (4096, 4096), (11008, 4096), (4096, 11008), (32000, 4096), (15360, 5120), (5120, 5120), (13824, 5120), (5120, 13824)]
#: the same for the 8-bit linear, which takes inputs up to 12288 wide
LINEARS8 = [s for s in LINEARS if s[1] <= 12288]
MOST_LINEAR = 4096 * 5120 * 5120          # rows x out x in of the largest linear here


def listed():
    return [
        # one decoded token through an attention output projection of the 7B model: launch latency and 8 MB of weights
        dict(name="int4_one_row", kind="int4", rows=1, out=4096, inp=4096),
        # a batch of eight decoding sequences, 13B feed-forward input
        dict(name="int4_eight_rows", kind="int4", rows=8, out=13824, inp=5120),
        # a chat prompt of ordinary length (ragged) through a 7B feed-forward input
        dict(name="int4_short_prompt", kind="int4", rows=203, out=11008, inp=4096),
        # eight prompts of 512 tokens at once, 13B attention output
        dict(name="int4_long_prompt", kind="int4", rows=4096, out=5120, inp=5120),
        # an ordinary prompt through an LLM.int8() linear of the 7B model
        dict(name="int8_prompt", kind="int8", rows=137, out=11008, inp=4096),
        # a full-context prompt through one 7B attention layer (its two int4 linears included)
        dict(name="llama_attention", kind="attention", batch=1, tokens=2048, heads=32, head_size=128),
        # one token of a whole (8-layer, 7B-wide) int4 LLaMA in the middle of its context
        dict(name="llama_token", kind="token", layers=8, heads=32, head_size=128, batch=1, context=2048, position=1030),
        # a prompt portion through sliding-window attention at width 2048
        dict(name="window_portion", kind="window", tokens=2048, width=2048, heads=16, kv_heads=4, dim=128, window=1024, f32=False),
        # the same layer in the 32-bit mode of trace replay, a ragged portion at width 1024
        dict(name="window_f32", kind="window", tokens=777, width=1024, heads=8, kv_heads=2, dim=128, window=512, f32=True),
        # a prompt portion through latent attention at width 2048
        dict(name="latent_portion", kind="latent", tokens=2048, width=2048, heads=16, dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=512),
        # a prompt portion through the gated delta rule at width 2048
        dict(name="delta_portion", kind="delta", tokens=2048, width=2048, heads=16, dim=128),
        # one engine step of a whole four-layer model (delta rule, two state-space layers, attention beside linear attention, four
        # feed-forwards): a prompt portion of the engine's default length, logits of its last eight tokens
        dict(name="portion_model", kind="model", tokens=512, width=1024, head_size=128, ff=4096, block=1024, vocab=32000, last=8),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["int4", "int4", "int4", "int4", "int8", "attention", "token", "window", "window", "latent", "delta", "model"])
    if kind == "int4":
        out, inp = rng.choice(LINEARS)
        return dict(kind=kind, rows=_log(rng, 1, min(4096, MOST_LINEAR // (out * inp))), out=out, inp=inp)
    if kind == "int8":
        out, inp = rng.choice(LINEARS8)
        return dict(kind=kind, rows=_log(rng, 1, 512), out=out, inp=inp)
    if kind == "attention":
        return dict(kind=kind, batch=1, tokens=_log(rng, 17, 2048), heads=rng.choice([32, 40]), head_size=128)
    if kind == "token":
        return dict(kind=kind, layers=rng.choice([4, 6, 8]), heads=32, head_size=128, batch=rng.choice([1, 1, 1, 4]), context=2048,
                    position=rng.randrange(16, 2047))
    if kind == "window":
        width = rng.choice([1024, 2048])
        f32 = rng.random() < 0.25
        return dict(kind=kind, tokens=_log(rng, 16, 1024 if f32 else 2048), width=width, heads=width // 128, kv_heads=width // 512, dim=128,
                    window=rng.choice([256, 512, 1000, 1024]), f32=f32)
    if kind == "latent":
        big = rng.random() < 0.5
        return dict(kind=kind, tokens=_log(rng, 1, 2048), width=2048 if big else 1024, heads=16 if big else 8, dim=128, rot_dim=64, vdim=128,
                    q_rank=768 if big else 384, kv_rank=512 if big else 256)
    if kind == "delta":
        width = rng.choice([1024, 2048])
        return dict(kind=kind, tokens=_log(rng, 1, 2048), width=width, heads=width // 128, dim=128)
    return dict(kind=kind, tokens=_log(rng, 16, 512), width=1024, head_size=128, ff=4096, block=1024, vocab=32000, last=8)


# ---------------------------------------------------------------------------------------------------- inputs and weights
class _Gen:
    """Random tensors on the GPU from one seed, in the order they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=BF):
        return (torch.randn(*shape, generator=self.g, device="cuda") * std + mean).to(dtype)

    def lin(self, out, inp, dtype=BF):
        return self.normal(out, inp, std=inp ** -0.5, dtype=dtype)

    def ints(self, lo, hi, shape, dtype=torch.int64):
        return torch.randint(lo, hi, shape, generator=self.g, device="cuda", dtype=dtype)


def _packed(g, out, inp):
    """Levels, scales and zero points of a 4-bit linear whose weights have the spread of a trained layer's."""
    qw = g.ints(0, 256, (inp // 2, out), torch.uint8).t()
    scales = (g.normal(out, 1, std=0.1, mean=1.0, dtype=F32) / (4.6 * math.sqrt(inp))).to(BF)
    zeros = (7.5 + g.normal(out, 1, std=0.5, dtype=F32)).to(BF)
    return qw, scales, zeros


def _fill(lin, packed):
    lin.load_state_dict({"quant_weight": packed[0], "scales": packed[1], "zeros": packed[2]})


def _int4(packed):
    prev = torch.get_default_dtype()
    torch.set_default_dtype(BF)
    try:
        with torch.device("cuda"):
            lin = ColBlockQuantizedLinear(packed[0].shape[1] * 2, packed[0].shape[0], bias=False, bits=4, tile_cols=-1)
    finally:
        torch.set_default_dtype(prev)
    _fill(lin, packed)
    return lin


def _dense(packed):
    """The matrix a 4-bit linear stands for, rounded as its get_weight() rounds it."""
    qw, s, z = packed
    lv = torch.stack([qw & 15, qw >> 4], dim=2).reshape(qw.shape[0], -1).to(BF)
    return ((lv - z) * s).to(F64)


def _rope_table(n, hs):
    theta = 1.0 / (10000.0 ** (torch.arange(0, hs, 2, device="cuda", dtype=F32) / hs))
    a = torch.outer(torch.arange(n, device="cuda", dtype=F32), theta)
    return torch.stack([torch.cos(a), torch.sin(a)], dim=-1)


def _window_tensors(c, g):
    dt, W, D, H, G, K = F32 if c["f32"] else BF, {}, c["width"], c["heads"], c["kv_heads"], c["dim"]
    for n, o, i in (("q", H * K, D), ("k", G * K, D), ("v", G * K, D), ("g", H * K, D), ("o", D, H * K)):
        W["a." + n] = g.lin(o, i, dt)
    W["a.q.norm"], W["a.k.norm"] = g.normal(H * K, std=0.1, mean=1.0, dtype=dt), g.normal(G * K, std=0.1, mean=1.0, dtype=dt)
    return W, g.normal(c["tokens"], D, dtype=dt)


def _latent_tensors(c, g):
    W, D, H = {}, c["width"], c["heads"]
    for n, o, i in (("dq", c["q_rank"], D), ("uq", H * (c["dim"] + c["rot_dim"]), c["q_rank"]), ("dkv", c["kv_rank"] + c["rot_dim"], D),
                    ("uk", H * c["dim"], c["kv_rank"]), ("uv", H * c["vdim"], c["kv_rank"]), ("o", D, H * c["vdim"])):
        W["a." + n] = g.lin(o, i)
    W["a.dq.norm"], W["a.dkv.norm"] = g.normal(c["q_rank"], std=0.1, mean=1.0), g.normal(c["kv_rank"], std=0.1, mean=1.0)
    W["a.sink"] = g.normal(H)
    return W, g.normal(c["tokens"], D)


def _delta_weights(W, m, g, D, H, K, rank=64):
    for n in ("q", "k", "v"):
        W[m + n], W[m + n + ".conv"] = g.lin(H * K, D), g.normal(H * K, 4, std=0.5)
    W[m + "b"], W[m + "A_log"], W[m + "norm"] = g.lin(H, D), g.normal(H, std=0.5, mean=-0.5), g.normal(K, std=0.1, mean=1.0)
    W[m + "a1"], W[m + "a2"], W[m + "dt_bias"] = g.lin(rank, D), g.lin(H * K, rank), g.normal(H * K, std=0.5)
    W[m + "g1"], W[m + "g2"], W[m + "o"] = g.lin(rank, D), g.lin(H * K, rank), g.lin(D, H * K)


def _delta_tensors(c, g):
    W = {}
    _delta_weights(W, "a.", g, c["width"], c["heads"], c["dim"])
    return W, g.normal(c["tokens"], c["width"])


ROT = {"base": 1e6, "dims": 128, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}


def _model_config(c):
    D, hs = c["width"], c["head_size"]
    H = D // hs
    ff = {"kind": "dense", "ff": c["ff"]}
    ssm = {"conv": 4, "groups": 1, "heads": 2 * D // 64, "norm_groups": 1, "state": 128, "vdim": 64}
    left = {"heads": H, "kv_heads": max(1, H // 4), "dim": hs, "vdim": hs, "mask": {"size": c["block"]}, "scale": hs ** -0.5, "softcap": 50.0, "rot": ROT}
    right = {"heads": max(1, H // 2), "dim": hs, "vdim": hs, "tau": 16.0}
    return {"architecture": "Lugovik", "vocab": c["vocab"], "width": D, "norm": {"eps": EPS}, "embedding": {"scale": math.sqrt(D)},
            "layers": [{"type": "channel_delta", "mixer": {"conv": 4, "dim": hs, "heads": H, "kv_heads": H, "vdim": hs}, "mlp": ff},
                       {"type": "mamba2", "mixer": ssm, "mlp": ff}, {"type": "mamba2", "mixer": ssm, "mlp": ff},
                       {"type": "parallel", "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}, "mlp": ff}]}


def _model_tensors(c, g):
    cfg, W, D = _model_config(c), {}, c["width"]
    W["embed"], W["head"], W["final.norm"] = g.normal(c["vocab"], D, std=D ** -0.5), g.lin(c["vocab"], D), g.normal(D, std=0.1, mean=1.0)
    for i, layer in enumerate(cfg["layers"]):
        p, m, x = f"l{i}.", f"l{i}.mix.", layer["mixer"]
        for n in ("norm1", "norm2"):
            W[p + n] = g.normal(D, std=0.1, mean=1.0)
        for n in ("norm1b", "norm2b"):
            W[p + n] = g.normal(D, std=0.1, mean=0.5)
        if layer["type"] == "channel_delta":
            _delta_weights(W, m, g, D, x["heads"], x["dim"])
        elif layer["type"] == "mamba2":
            H, V, N = x["heads"], x["vdim"], x["state"]
            ch = H * V + 2 * N
            W[m + "in"], W[m + "conv"], W[m + "conv.b"] = g.lin(2 * H * V + 2 * N + H, D), g.normal(ch, 4, std=0.5), g.normal(ch, std=0.1)
            W[m + "dt_bias"], W[m + "A_log"], W[m + "D"] = g.normal(H, std=0.5), g.normal(H, std=0.5, mean=-0.5), g.normal(H, std=0.1, mean=1.0)
            W[m + "norm"], W[m + "o"] = g.normal(H * V, std=0.1, mean=1.0), g.lin(D, H * V)
        else:
            a, b = x["left"], x["right"]
            H, G, K = a["heads"], a["kv_heads"], a["dim"]
            for n, o, i2 in (("q", H * K, D), ("k", G * K, D), ("v", G * K, D), ("g", H, D), ("o", D, H * K)):
                W[m + "left." + n] = g.lin(o, i2)
            W[m + "left.q.norm"], W[m + "left.k.norm"] = g.normal(K, std=0.1, mean=1.0), g.normal(K, std=0.1, mean=1.0)
            H, K = b["heads"], b["dim"]
            for n, o, i2 in (("q", H * K, D), ("k", H * K, D), ("v", H * K, D), ("g", H * K, D), ("o", D, H * K), ("a1", 64, D), ("a2", H * K, 64)):
                W[m + "right." + n] = g.lin(o, i2)
            W[m + "right.norm"], W[m + "right.a2.b"] = g.normal(K, std=0.1, mean=1.0), g.normal(H * K, std=0.5, mean=2.0)
        W[p + "mlp.gate"], W[p + "mlp.up"], W[p + "mlp.down"] = g.lin(c["ff"], D), g.lin(c["ff"], D), g.lin(D, c["ff"])
    return cfg, W, g.ints(0, c["vocab"], (c["tokens"],)).tolist()


def _int8_tensors(c, g):
    w = g.lin(c["out"], c["inp"])
    x = g.normal(c["rows"], c["inp"])
    loud = g.ints(0, c["inp"], (6,))                      # a few channels carry outliers, as in trained models
    x[:, loud] *= 8.0
    return w, x


def _attention_tensors(c, g):
    C = c["heads"] * c["head_size"]
    return _packed(g, 3 * C, C), _packed(g, C, C), g.normal(c["batch"], c["tokens"], C)


def _token_tensors(c, g):
    C = c["heads"] * c["head_size"]
    ff = int(2 * 4 * C / 3)
    ff = (ff + 255) // 256 * 256
    W = {"wte": g.normal(32000, C), "ln_f": g.normal(C, std=0.1, mean=1.0), "lm_head": _packed(g, 32000, C)}
    for i in range(c["layers"]):
        W[i] = dict(rms_1=g.normal(C, std=0.1, mean=1.0), rms_2=g.normal(C, std=0.1, mean=1.0), c_attn=_packed(g, 3 * C, C), c_proj=_packed(g, C, C),
                    c_fc1=_packed(g, ff, C), c_fc2=_packed(g, ff, C), mlp=_packed(g, C, ff))
    kv = [[g.normal(c["batch"], c["heads"], c["context"], c["head_size"]) for _ in range(2)] for _ in range(c["layers"])]
    return W, kv, g.ints(0, 32000, (c["batch"], 1))


# ---------------------------------------------------------------------------------------------------- one program's state
def _portion(mixer, h, dtype):
    return dict(mixer=mixer, h=h, dtype=dtype, pool=SequenceStatePool(mixer.state_specs(), 1, h.device), meta=torch.zeros(2, dtype=torch.int32, device="cuda"))


def prepare(case, seed):
    c, g = case, _Gen(seed)
    kind = c["kind"]
    if kind == "int4":
        lin = _int4(_packed(g, c["out"], c["inp"]))
        s = dict(kind=kind, module=lin, x=g.normal(c["rows"], c["inp"]))
        lin(s["x"])                                       # the weights are laid out for this many rows at the first call
        return s
    if kind == "int8":
        w, x = _int8_tensors(c, g)
        with torch.device("cuda"):
            lin = Linear8bitLt(c["inp"], c["out"], bias=False)
        lin.load_state_dict({"weight": w})
        lin(x)
        return dict(kind=kind, module=lin, x=x)
    if kind == "attention":
        qkv, proj, x = _attention_tensors(c, g)
        C = c["heads"] * c["head_size"]
        with torch.device("meta"):
            att = P.CausalSelfAttention(P.LLaMAConfig(n_head=c["heads"], n_embd=C, n_layer=1))
        att.c_attn, att.c_proj = _int4(qkv), _int4(proj)
        cache = [torch.zeros(c["batch"], c["heads"], 2048, c["head_size"], dtype=BF, device="cuda") for _ in range(2)]
        s = dict(kind=kind, module=att, x=x, rope=_rope_table(c["tokens"], c["head_size"]), cache=tuple(cache), pos=torch.arange(c["tokens"], device="cuda"))
        run(s)
        return s
    if kind == "token":
        W, kv, idx = _token_tensors(c, g)
        C = c["heads"] * c["head_size"]
        with torch.device("meta"):
            model = P.LLaMA(P.LLaMAConfig(n_head=c["heads"], n_embd=C, n_layer=c["layers"], block_size=c["context"]))
        model.transformer.wte.weight = torch.nn.Parameter(W["wte"], requires_grad=False)
        model.transformer.ln_f.scale = torch.nn.Parameter(W["ln_f"], requires_grad=False)
        model.lm_head = _int4(W["lm_head"])
        for i, blk in enumerate(model.transformer.h):
            w = W[i]
            blk.rms_1.scale, blk.rms_2.scale = (torch.nn.Parameter(w[n], requires_grad=False) for n in ("rms_1", "rms_2"))
            blk.attn.c_attn, blk.attn.c_proj = _int4(w["c_attn"]), _int4(w["c_proj"])
            blk.mlp.c_fc1, blk.mlp.c_fc2, blk.mlp.c_proj = _int4(w["c_fc1"]), _int4(w["c_fc2"]), _int4(w["mlp"])
        model.eval()
        s = dict(kind=kind, module=model, idx=idx, context=c["context"], pos=torch.tensor([c["position"]], device="cuda"))
        for _ in range(4):                                # a decoding loop that is under way
            run(s)
        for (k, v), (k0, v0) in zip(model.kv_caches, kv):
            k.copy_(k0)
            v.copy_(v0)
        return s
    if kind == "window":
        W, h = _window_tensors(c, g)
        m = X.SlidingWindowAttention("a", W, "a.", heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"], vdim=c["dim"], scale=c["dim"] ** -0.5,
                                     window=c["window"], eps=EPS, rot={"base": 10000.0, "dims": c["dim"]})
        return dict(kind=kind, **_portion(m, h, h.dtype))
    if kind == "latent":
        W, h = _latent_tensors(c, g)
        m = X.LatentAttention("a", W, "a.", heads=c["heads"], dim=c["dim"], rot_dim=c["rot_dim"], vdim=c["vdim"], q_rank=c["q_rank"], kv_rank=c["kv_rank"],
                              scale=(c["dim"] + c["rot_dim"]) ** -0.5, eps=EPS, rot={"base": 10000.0, "dims": c["rot_dim"]}, max_positions=4096)
        return dict(kind=kind, **_portion(m, h, h.dtype))
    if kind == "delta":
        W, h = _delta_tensors(c, g)
        m = X.ChannelDeltaMixer("a", W, "a.", heads=c["heads"], kv_heads=c["heads"], dim=c["dim"], vdim=c["dim"], conv=4, eps=EPS)
        return dict(kind=kind, **_portion(m, h, h.dtype))
    if kind == "model":
        cfg, W, tokens = _model_tensors(c, g)
        engine = P.Engine(Lugovik(LugovikConfig.from_dict(cfg), W), n_slots=2)
        n = len(tokens)
        return dict(kind=kind, engine=engine, tokens=tokens, want=list(range(max(0, n - c["last"]), n)))
    raise ValueError(kind)


@torch.no_grad()
def run(s):
    kind = s["kind"]
    if kind in ("int4", "int8"):
        return s["module"](s["x"])
    if kind == "attention":
        y, (k, v) = s["module"](s["x"], s["rope"], None, 2048, s["pos"], s["cache"])
        return y, k, v
    if kind == "token":
        return s["module"](s["idx"], s["context"], s["pos"]), s["module"].kv_caches
    if kind == "model":                                   # a new request's prompt; the request ends with it
        return s["engine"].step([{"id": "r", "tokens": s["tokens"], "want": s["want"]}], end=["r"])[0], dict(s["engine"].pool.tensors)
    pool = s["pool"]                                      # a new sequence's portion through one mixer
    slot = pool.acquire("r")
    ctx = X.StepContext(s["h"].shape[0], s["meta"], pool.tensors, s["dtype"], pos_hint=0, slot_hint=slot)
    y = s["mixer"].forward(s["h"], ctx)
    pool.release("r")
    return y, dict(pool.tensors)


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def _linear_work(rows, out, inp, wbits):
    return out * inp * wbits / 8 + 2 * rows * (inp + out), 2 * rows * out * inp


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("int4", "int8"):
        b, f = _linear_work(c["rows"], c["out"], c["inp"], 4 if kind == "int4" else 8)
        return {"bytes": b, "flops": f}
    if kind == "attention":
        T, C, B = c["tokens"], c["heads"] * c["head_size"], c["batch"]
        b1, f1 = _linear_work(B * T, 3 * C, C, 4)
        b2, f2 = _linear_work(B * T, C, C, 4)
        return {"bytes": b1 + b2 + 4 * B * T * C, "flops": f1 + f2 + 4 * C * B * (T * (T + 1) // 2)}
    if kind == "token":
        C, B = c["heads"] * c["head_size"], c["batch"]
        ff = (int(8 * C / 3) + 255) // 256 * 256
        params = c["layers"] * (4 * C * C + 3 * C * ff) + 32000 * C
        return {"bytes": params / 2 + c["layers"] * 4 * C * B * (c["position"] + 2) + 2 * B * 32000, "flops": 2 * B * params + 4 * c["layers"] * C * B * c["position"]}
    T, D = c["tokens"], c["width"]
    if kind == "window":
        H, G, K, e = c["heads"], c["kv_heads"], c["dim"], 4 if c["f32"] else 2
        n = 3 * H * K + 2 * G * K
        seen = sum(min(t + 1, c["window"]) for t in range(T))
        return {"bytes": e * (D * n + 2 * T * D + 2 * min(T, c["window"]) * G * K), "flops": 2 * T * D * n + 4 * H * K * seen}
    if kind == "latent":
        H = c["heads"]
        n = D * (c["q_rank"] + c["kv_rank"] + c["rot_dim"] + H * c["vdim"]) + H * (c["dim"] + c["rot_dim"]) * c["q_rank"] + H * (c["dim"] + c["vdim"]) * c["kv_rank"]
        return {"bytes": 2 * (n + 2 * T * D + T * (c["kv_rank"] + c["rot_dim"])), "flops": 2 * T * n + 2 * H * (c["dim"] + c["rot_dim"] + c["vdim"]) * (T * (T + 1) // 2)}
    if kind == "delta":
        H, K = c["heads"], c["dim"]
        n = D * (3 * H * K + H + 128) + 128 * H * K + D * H * K
        return {"bytes": 2 * (n + 2 * T * D) + 4 * H * K * K, "flops": 2 * T * n + 7 * T * H * K * K}
    H, I, F = D // c["head_size"], 2 * D, c["ff"]
    delta = D * (3 * D + H + 128) + 128 * D + D * D
    ssm = D * (2 * I + 256 + I // 64) + I * D
    par = D * (D + 2 * (D // 4) + H) + D * D // 2 * 4 + 64 * (D + D // 2) + D * (D + D // 2)
    n = delta + 2 * ssm + par + 12 * D * F
    state = 7 * D * 128 + 2 * 5 * I * 128 + 5 * (D // 2) * 128 + 2 * D * T
    return {"bytes": 2 * (n + c["vocab"] * D + T * D) + 4 * c["vocab"] * c["last"], "flops": 2 * T * n + T * state + 2 * c["last"] * c["vocab"] * D}


def tolerance(case):
    """About four times the distance to `exact` where the result is rounded once or twice, and what bf16 gives to whole layers."""
    kind = case["kind"]
    if kind in ("int4", "int8"):
        return {"rel": 7e-3}                              # one bf16 rounding of the result: 1.7e-3 seen
    if kind == "window" and case["f32"]:
        return {"rel": 1e-5}
    if kind in ("token", "model"):
        return {"rel": 3e-2}
    return {"rel": 2e-2}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _half_rotate(x, dims, base, scaling=None, interleaved=False):
    """x [T, heads, size]: the first `dims` entries of a head turn by the token's position."""
    i = torch.arange(dims // 2, dtype=F64, device="cuda")
    f, m = base ** (-2.0 * i / dims), 1.0
    if scaling:
        def d(t):
            return dims * math.log(scaling["original"] / (2 * math.pi * t)) / (2 * math.log(base))

        lo, hi = max(math.floor(d(scaling["fast"])), 0), min(math.ceil(d(scaling["slow"])), dims - 1)
        r = torch.clamp((i - lo) / max(hi - lo, 0.001), 0, 1)
        f, m = f / scaling["factor"] * r + f * (1 - r), 0.1 * math.log(scaling["factor"]) + 1.0
    f = f.to(F32).to(F64)                                 # the table of frequencies is kept in 32 bits
    a = torch.outer(torch.arange(x.shape[0], dtype=F64, device="cuda"), f)[:, None]
    co, si = torch.cos(a) * m, torch.sin(a) * m
    y = x.clone()
    if interleaved:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        y[..., 0:dims:2], y[..., 1:dims:2] = u * co - v * si, v * co + u * si
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        y[..., :dims // 2], y[..., dims // 2:dims] = u * co - v * si, v * co + u * si
    return y


def _softmax_sum(q, k, v, scale, seen, sink=None, cap=None):
    """q [T, H, K], k [S, H, K], v [S, H, V], seen [T, S]; `sink` [H]: one more term exp(sink) in the denominator."""
    s = torch.einsum("thk,shk->hts", q, k) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    s = s.masked_fill(~seen[None], -math.inf)
    if sink is not None:
        s = torch.cat([s, sink[:, None, None].expand(-1, s.shape[1], 1)], dim=2)
    w = torch.softmax(s, dim=-1)[..., :k.shape[0]]
    return torch.einsum("hts,shv->thv", w, v)


def _causal(T):
    i = torch.arange(T, device="cuda")
    return i[:, None] >= i[None, :]


def _conv_silu(x, w, b=None):
    T, taps = x.shape[0], w.shape[1]
    xp = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(xp[j:j + T] * w[:, j] for j in range(taps))
    return torch.nn.functional.silu(y if b is None else y + b)


def _delta_mix(h, W, p, H, K):
    T = h.shape[0]
    proj = {n: h @ W[p + n].t() for n in ("q", "k", "v")}
    q, k, v = (_conv_silu(proj[n], W[p + n + ".conv"]).view(T, H, K) for n in ("q", "k", "v"))
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q = q * K ** -0.5
    beta = torch.sigmoid(h @ W[p + "b"].t())
    a = (h @ W[p + "a1"].t()) @ W[p + "a2"].t() + W[p + "dt_bias"]
    dec = torch.exp(-torch.exp(W[p + "A_log"])[None, :, None] * torch.nn.functional.softplus(a).view(T, H, K))
    S = torch.zeros(H, K, K, dtype=F64, device="cuda")                    # [head, value, key]
    out = torch.empty(T, H, K, dtype=F64, device="cuda")
    for t in range(T):
        S = S * dec[t][:, None, :]
        u = beta[t][:, None] * (v[t] - torch.bmm(S, k[t][:, :, None])[:, :, 0])
        S = torch.baddbmm(S, u[:, :, None], k[t][:, None, :])
        out[t] = torch.bmm(S, q[t][:, :, None])[:, :, 0]
    gate = torch.sigmoid((h @ W[p + "g1"].t()) @ W[p + "g2"].t())
    y = (_rms(out, W[p + "norm"]).reshape(T, H * K) * gate) @ W[p + "o"].t()
    return y, S, torch.cat([proj["q"], proj["k"], proj["v"]], dim=1)


def _decayed(q, k, v, a):
    """S <- a S + v k^T, o = S q.  q, k [T, H, K], v [T, H, V], a [T, H, K] or [T, H, 1]."""
    T, H, K = q.shape
    S, out = torch.zeros(H, v.shape[2], K, dtype=F64, device="cuda"), torch.empty(T, H, v.shape[2], dtype=F64, device="cuda")
    for t in range(T):
        S = torch.baddbmm(S * a[t][:, None, :], v[t][:, :, None], k[t][:, None, :])
        out[t] = torch.bmm(S, q[t][:, :, None])[:, :, 0]
    return out


def _model_exact(c, cfg, W, tokens):
    T, D, hs = c["tokens"], c["width"], c["head_size"]
    x = W["embed"][torch.tensor(tokens, device="cuda")] * math.sqrt(D)
    for i, layer in enumerate(cfg["layers"]):
        p, m, s = f"l{i}.", f"l{i}.mix.", layer["mixer"]
        h = _rms(x, W[p + "norm1"])
        if layer["type"] == "channel_delta":
            y = _delta_mix(h, W, m, s["heads"], s["dim"])[0]
        elif layer["type"] == "mamba2":
            H, V, N = s["heads"], s["vdim"], s["state"]
            I = H * V
            u = h @ W[m + "in"].t()
            z, xbc, dt = u[:, :I], _conv_silu(u[:, I:2 * I + 2 * N], W[m + "conv"], W[m + "conv.b"]), u[:, 2 * I + 2 * N:]
            dt = torch.nn.functional.softplus(dt + W[m + "dt_bias"])
            xs, B, Cm = xbc[:, :I].view(T, H, V), xbc[:, I:I + N], xbc[:, I + N:]
            o = _decayed(Cm[:, None].expand(T, H, N), B[:, None].expand(T, H, N), dt[:, :, None] * xs, torch.exp(-torch.exp(W[m + "A_log"]) * dt)[:, :, None])
            o = (o + W[m + "D"][:, None] * xs).reshape(T, I) * torch.nn.functional.silu(z)
            y = (_rms(o) * W[m + "norm"]) @ W[m + "o"].t()
        else:
            a, b = s["left"], s["right"]
            H, G = a["heads"], a["kv_heads"]
            q, k = (_rms((h @ W[m + "left." + n].t()).view(T, -1, hs), W[m + "left." + n + ".norm"]) for n in ("q", "k"))
            q, k = (_half_rotate(t, ROT["dims"], ROT["base"], ROT["scaling"]) for t in (q, k))
            v = (h @ W[m + "left.v"].t()).view(T, G, hs)
            blk = torch.arange(T, device="cuda") // c["block"]
            o = _softmax_sum(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), a["scale"], _causal(T) & (blk[:, None] == blk[None]),
                             torch.zeros(H, dtype=F64, device="cuda"), a["softcap"])
            y = (o * torch.sigmoid(h @ W[m + "left.g"].t())[:, :, None]).reshape(T, H * hs) @ W[m + "left.o"].t()
            H = b["heads"]
            q, k, v = ((h @ W[m + "right." + n].t()).view(T, H, hs) for n in ("q", "k", "v"))
            al = torch.sigmoid((h @ W[m + "right.a1"].t()) @ W[m + "right.a2"].t() + W[m + "right.a2.b"]) ** (1.0 / b["tau"])
            o = _rms(_decayed(q * hs ** -0.5, k, v, al.view(T, H, hs)), W[m + "right.norm"]).reshape(T, H * hs)
            y = y + (o * torch.nn.functional.silu(h @ W[m + "right.g"].t())) @ W[m + "right.o"].t()
        x = x + _rms(y, W[p + "norm1b"])
        h = _rms(x, W[p + "norm2"])
        y = (torch.nn.functional.gelu(h @ W[p + "mlp.gate"].t(), approximate="tanh") * (h @ W[p + "mlp.up"].t())) @ W[p + "mlp.down"].t()
        x = x + _rms(y, W[p + "norm2b"])
    return _rms(x[max(0, T - c["last"]):], W["final.norm"]) @ W["head"].t()


def _rope_pairs(x, table):
    """x [..., hs] against table [..., hs/2, 2]: neighbouring entries turn."""
    u, v, co, si = x[..., 0::2], x[..., 1::2], table[..., 0], table[..., 1]
    return torch.stack([u * co - v * si, v * co + u * si], dim=-1).flatten(-2)


@torch.no_grad()
def exact(case, seed):
    c, g = case, _Gen(seed)
    kind = c["kind"]
    if kind == "int4":
        w = _dense(_packed(g, c["out"], c["inp"]))
        return g.normal(c["rows"], c["inp"]).to(F64) @ w.t()
    if kind == "int8":
        w, x = _int8_tensors(c, g)
        wh, a = w.half().to(F64), x.half().to(F64)
        scb = wh.abs().amax(1)
        cb = torch.round(w.half().float() * (127.0 / w.half().float().abs().amax(1).clamp_min(1e-30))[:, None]).clamp(-127, 127).to(F64)
        out = (a.abs() >= 6.0).any(0)
        sca = (a * ~out).abs().amax(1)
        ca = torch.round((a * ~out) * (127.0 / sca)[:, None]).clamp(-127, 127)
        return (ca @ cb.t()) * sca[:, None] * scb / 127.0 ** 2 + (a * out) @ (cb * (scb / 127.0)[:, None]).t()
    if kind == "attention":
        qkv, proj, x = _attention_tensors(c, g)
        B, T, H, hs = c["batch"], c["tokens"], c["heads"], c["head_size"]
        q, k, v = (x.to(F64) @ _dense(qkv).t()).view(B, T, 3, H, hs).unbind(2)
        table = _rope_table(T, hs).to(F64)[None, :, None]
        q, k = _rope_pairs(q, table), _rope_pairs(k, table)
        y = torch.stack([_softmax_sum(q[b], k[b], v[b], hs ** -0.5, _causal(T)) for b in range(B)]).reshape(B, T, H * hs) @ _dense(proj).t()
        full = [torch.nn.functional.pad(t.transpose(1, 2), (0, 0, 0, 2048 - T)) for t in (k, v)]
        return y, full[0], full[1]
    if kind == "token":
        W, kv, idx = _token_tensors(c, g)
        B, H, hs, p = c["batch"], c["heads"], c["head_size"], c["position"]

        def norm(x, w):
            return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.to(F64)

        x = W["wte"][idx[:, 0]].to(F64)
        table = _rope_table(p + 1, hs).to(F64)[p]
        for i in range(c["layers"]):
            w = W[i]
            q, k, v = (norm(x, w["rms_1"]) @ _dense(w["c_attn"]).t()).view(B, 3, H, hs).unbind(1)
            q, k = _rope_pairs(q, table), _rope_pairs(k, table)
            ks, vs = (torch.cat([t[:, :, :p].to(F64), n[:, :, None]], dim=2) for t, n in zip(kv[i], (k, v)))
            a = torch.softmax(torch.einsum("bhd,bhsd->bhs", q, ks) * hs ** -0.5, dim=-1)
            x = x + torch.einsum("bhs,bhsd->bhd", a, vs).reshape(B, H * hs) @ _dense(w["c_proj"]).t()
            n = norm(x, w["rms_2"])
            x = x + (torch.nn.functional.silu(n @ _dense(w["c_fc1"]).t()) * (n @ _dense(w["c_fc2"]).t())) @ _dense(w["mlp"]).t()
        return (norm(x, W["ln_f"]) @ _dense(W["lm_head"]).t())[:, None], None
    if kind == "model":
        cfg, W, tokens = _model_tensors(c, g)
        return _model_exact(c, cfg, {n: t.to(F64) for n, t in W.items()}, tokens), None
    W, h = {"window": _window_tensors, "latent": _latent_tensors, "delta": _delta_tensors}[kind](c, g)
    W, h, T, H = {n: t.to(F64) for n, t in W.items()}, h.to(F64), c["tokens"], c["heads"]
    if kind == "delta":
        y, S, proj = _delta_mix(h, W, "a.", H, c["dim"])
        conv = torch.nn.functional.pad(proj, (0, 0, 3, 0))[-3:]
        return y, {"a.S": S[None], "a.conv": conv[None]}
    if kind == "window":
        G, K = c["kv_heads"], c["dim"]
        q, k = (_rms(h @ W["a." + n].t(), W["a." + n + ".norm"]).view(T, -1, K) for n in ("q", "k"))
        q, k = (_half_rotate(t, K, 10000.0) for t in (q, k))
        v = (h @ W["a.v"].t()).view(T, G, K)
        i = torch.arange(T, device="cuda")
        o = _softmax_sum(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), K ** -0.5, _causal(T) & (i[:, None] - i[None] < c["window"]))
        y = (o.reshape(T, H * K) * torch.sigmoid(h @ W["a.g"].t())) @ W["a.o"].t()
        ring = {}
        for n, t in (("a.k", k), ("a.v", v)):
            r = torch.zeros(1, c["window"], G, K, dtype=F64, device="cuda")
            last = i[max(0, T - c["window"]):]
            r[0, last % c["window"]] = t[last]
            ring[n] = r
        return y, ring
    cq = _rms(h @ W["a.dq"].t(), W["a.dq.norm"])
    q = (cq @ W["a.uq"].t()).view(T, H, c["dim"] + c["rot_dim"])
    ckv = h @ W["a.dkv"].t()
    lat = _rms(ckv[:, :c["kv_rank"]], W["a.dkv.norm"])
    kr = _half_rotate(ckv[:, None, c["kv_rank"]:], c["rot_dim"], 10000.0, interleaved=True)
    qr = _half_rotate(q[..., c["dim"]:], c["rot_dim"], 10000.0, interleaved=True)
    key = torch.cat([(lat @ W["a.uk"].t()).view(T, H, c["dim"]), kr.expand(T, H, c["rot_dim"])], dim=2)
    o = _softmax_sum(torch.cat([q[..., :c["dim"]], qr], dim=2), key, (lat @ W["a.uv"].t()).view(T, H, c["vdim"]), (c["dim"] + c["rot_dim"]) ** -0.5,
                     _causal(T), W["a.sink"])
    cache = torch.zeros(1, 4096, c["kv_rank"] + c["rot_dim"], dtype=F64, device="cuda")
    cache[0, :T] = torch.cat([lat, kr[:, 0]], dim=1)
    return o.reshape(T, H * c["vdim"]) @ W["a.o"].t(), {"a.kv": cache}
