"""What users of this framework have it do, as cases that can be timed and compared.

Kinds of work, each through the public entry points:

* "gemv", "gemm"      one int4 projection of a single token / of a batch of tokens (a host that keeps its own decode loop);
* "deltanet"          consecutive Gated DeltaNet steps with the state held by the caller;
* "attention"         one decode step of grouped-query attention over a long bf16 cache;
* "prompt", "decode"  a model that is kept open: tokens that follow a kept prefix, as one prompt pass or token by token through the
                      captured step.  Models: the int4 hybrid at the widths of the 27B model, Nufalorn at width 4096, Vobunex at width 2048,
                      all with one or two periods of their layers (a deeper model repeats them) and a vocabulary of 32768.

Weights are random and belong to the configuration (a program loads them once); tokens, vectors and states come from the case's seed.
"""
import ctypes
import json
import math
import struct
import tempfile
import zlib
from pathlib import Path

import torch

import lithos_b200 as lb
from lithos_b200 import model as M

VOCAB, MAX_CTX = 32768, 4352


# ---- the models --------------------------------------------------------------------------------------------------
def nufalorn_config():
    """one period: attention in blocks of 2048 positions, HGRN2, GLA, GLA"""
    W, F, H, D = 4096, 12288, 32, 128
    mlp = {"ff": F, "kind": "dense"}
    att = {"heads": H, "kv_heads": 8, "dim": D, "vdim": D, "scale": D ** -0.5, "mask": {"size": 2048}, "rot": {"base": 500000.0, "dims": D}}
    rec = {"heads": H, "dim": D, "vdim": D}
    layers = [{"type": "attention", "mixer": att, "mlp": mlp}, {"type": "hgrn2", "mixer": rec, "mlp": mlp}] + \
             [{"type": "gla", "mixer": dict(rec, tau=16.0), "mlp": mlp} for _ in range(2)]
    return {"architecture": "Nufalorn", "layers": layers, "logit_softcap": 30.0, "norm": {"eps": 1e-6}, "residual_mult": 0.5, "vocab": VOCAB, "width": W}


def vobunex_config():
    """one period: Mamba-2 + dense, Mamba-2 + experts, latent attention + experts, Mamba-2 + dense"""
    W, H = 2048, 16
    rot = {"base": 10000.0, "dims": 64, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    att = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 1024, "kv_rank": 512, "scale": 192 ** -0.5, "rot": rot}
    ssm = {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    moe = {"kind": "moe", "expert": {"ff": 1408, "limit": 7.0}, "router": {"experts": 64, "top": 6}}
    dense = {"kind": "dense", "ff": 8192}
    kinds = [("mamba2", ssm, dense), ("mamba2", ssm, moe), ("latent_attention", att, moe), ("mamba2", ssm, dense)]
    return {"architecture": "Vobunex", "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in kinds], "width": W, "vocab": VOCAB,
            "norm": {"eps": 1e-5}, "embedding": {"bigram": {"buckets": 65521, "mul_prev": 1031, "mul_cur": 7}}}


def hybrid_config():
    """two periods of three DeltaNet layers and one attention layer at the 27B model's widths"""
    c = M.qwen35_27b(max_ctx=MAX_CTX, n_layers=8)
    c.vocab = VOCAB
    return c


def _gen(name):
    return torch.Generator("cuda").manual_seed(zlib.crc32(name.encode()))


def _normal(name, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return (mean + std * torch.randn(shape, generator=_gen(name), device="cuda")).to(dtype)


def _uniform(name, shape, lo, hi, dtype=torch.bfloat16):
    return (lo + (hi - lo) * torch.rand(shape, generator=_gen(name), device="cuda")).to(dtype)


def _int4(name, K, N):
    """a matrix in the GPTQ format: uniform nibbles, zero-points near the middle, outputs of about the inputs' size"""
    g = _gen(name)
    q = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, device="cuda", dtype=torch.int32)
    s = ((0.7 + 0.6 * torch.rand((K // 128, N), generator=g, device="cuda")) / (4.6 * math.sqrt(K))).to(torch.float16)
    z = torch.randint(7, 10, (K // 128, N // 8, 8), generator=g, device="cuda", dtype=torch.int64)
    z = (z << torch.arange(0, 32, 4, device="cuda")).sum(-1)
    return q, s, torch.where(z >= 2 ** 31, z - 2 ** 32, z).to(torch.int32)


def _dense(q, s, z):
    """the same matrix in 64 bits, [K, N]"""
    sh = torch.arange(0, 32, 4, device=q.device)
    w = ((q[:, None, :] >> sh[None, :, None]) & 15).reshape(-1, q.shape[1]).double()
    zero = ((z[:, :, None] >> sh) & 15).reshape(z.shape[0], -1).double()
    return ((w.view(z.shape[0], 128, -1) - zero[:, None]) * s.double()[:, None]).reshape(w.shape)


def hybrid_tensor(c, layer, name):
    """one tensor of a layer, by name; (qweight, scales, qzeros) for the int4 matrices"""
    H, I, V, n = c.hidden, c.inter, c.dn_v_heads * 128, f"hybrid.{layer}.{name}"
    int4 = {"DN_QKV": (H, c.conv_channels), "DN_Z": (H, V), "DN_OUT": (V, H), "FA_Q": (H, 2 * c.fa_q_heads * 256), "FA_K": (H, c.fa_kv_heads * 256),
            "FA_V": (H, c.fa_kv_heads * 256), "FA_O": (c.fa_q_heads * 256, H), "GATE": (H, I), "UP": (H, I), "DOWN": (I, H)}
    if name in int4:
        return _int4(n, *int4[name])
    if name in ("DN_PROJ_A", "DN_PROJ_B"):
        return _normal(n, (c.dn_v_heads, H), 0.02)
    if name == "DN_A_LOG":
        return _uniform(n, (c.dn_v_heads,), 0.0, 2.7, torch.float32)
    if name == "DN_NORM":
        return _normal(n, (128,), 0.02, 1.0, torch.float32)
    return {"DN_DT_BIAS": lambda: _normal(n, (c.dn_v_heads,), 0.1), "DN_CONV1D": lambda: _normal(n, (4, c.conv_channels), 0.3),
            "FA_Q_NORM": lambda: _normal(n, (256,), 0.02, 1.0), "FA_K_NORM": lambda: _normal(n, (256,), 0.02, 1.0),
            "INPUT_NORM": lambda: _normal(n, (H,), 0.02), "POST_NORM": lambda: _normal(n, (H,), 0.02)}[name]()


HYBRID_DN = ("DN_QKV", "DN_Z", "DN_OUT", "DN_PROJ_A", "DN_PROJ_B", "DN_A_LOG", "DN_DT_BIAS", "DN_CONV1D", "DN_NORM")
HYBRID_FA = ("FA_Q", "FA_K", "FA_V", "FA_O", "FA_Q_NORM", "FA_K_NORM")
HYBRID_MLP = ("GATE", "UP", "DOWN", "INPUT_NORM", "POST_NORM")


def hybrid_globals(c):
    return [_normal("hybrid.embed", (c.vocab, c.hidden), 1.0), _normal("hybrid.head", (c.vocab, c.hidden), 0.02), _normal("hybrid.norm", (c.hidden,), 0.02)]


def list_shapes(cfg):
    """{name: (shape, kind, ...)} of a layer-list model's tensors"""
    W, out = cfg["width"], {}

    def mat(n, rows, cols, gain=1.0):
        out[n] = ((rows, cols), "normal", gain / math.sqrt(cols), 0.0)

    def vec(n, size, mean, std):
        out[n] = ((size,), "normal", std, mean)

    def norm(n):
        if cfg["architecture"] == "Vobunex":
            vec(n, W, 1.0, 0.1)
            vec(n + ".b", W, 0.0, 0.1)
        else:
            vec(n, W, 0.0, 0.1)

    out["embed"] = ((cfg["vocab"], W), "normal", 1.0, 0.0)
    mat("head", cfg["vocab"], W)
    norm("final.norm")
    if cfg["architecture"] == "Vobunex":
        out["bigram"] = ((cfg["embedding"]["bigram"]["buckets"] + 1, W), "normal", 0.7, 0.0)
    for i, layer in enumerate(cfg["layers"]):
        m, p, t = layer["mixer"], f"l{i}.mix.", layer["type"]
        H, V = m["heads"], m["vdim"]
        norm(f"l{i}.norm1")
        if t == "latent_attention":
            mat(p + "dq", m["q_rank"], W)
            vec(p + "dq.norm", m["q_rank"], 1.0, 0.2)
            mat(p + "uq", H * (m["dim"] + m["rot_dim"]), m["q_rank"], 1.5)
            mat(p + "dkv", m["kv_rank"] + m["rot_dim"], W)
            vec(p + "dkv.norm", m["kv_rank"], 1.0, 0.2)
            mat(p + "uk", H * m["dim"], m["kv_rank"], 1.5)
            mat(p + "uv", H * V, m["kv_rank"])
            vec(p + "sink", H, 0.5, 1.5)
        elif t == "mamba2":
            C = H * V + 2 * m["groups"] * m["state"]
            mat(p + "in", H * V + C + H, W)
            out[p + "conv"] = ((C, m["conv"]), "normal", 0.6, 0.0)
            vec(p + "conv.b", C, 0.0, 0.2)
            out[p + "dt_bias"] = ((H,), "uniform", -5.0, 0.0)
            out[p + "A_log"] = ((H,), "uniform", -1.5, 2.0)
            vec(p + "D", H, 1.0, 0.3)
            vec(p + "norm", H * V, 1.0, 0.2)
        else:
            mat(p + "q", H * m["dim"], W, 1.5)
            if t == "attention":
                mat(p + "k", m["kv_heads"] * m["dim"], W, 1.5)
                mat(p + "v", m["kv_heads"] * V, W)
            elif t == "hgrn2":
                mat(p + "f", H * m["dim"], W)
                out[p + "f.b"] = ((H * m["dim"],), "uniform", -1.0, 7.0)
                out[p + "lower"] = ((H * m["dim"],), "uniform", 0.0, 0.9)
                mat(p + "v", H * V, W)
                vec(p + "norm", V, 1.0, 0.2)
            else:
                mat(p + "k", H * m["dim"], W)
                mat(p + "v", H * V, W)
                mat(p + "g", H * V, W)
                mat(p + "a1", 16, W)
                mat(p + "a2", H * m["dim"], 16)
                out[p + "a2.b"] = ((H * m["dim"],), "uniform", -2.0, 4.0)
                vec(p + "norm", V, 1.0, 0.2)
        mat(p + "o", W, H * V)
        f, p = layer["mlp"], f"l{i}.mlp."
        norm(f"l{i}.norm2")
        if f["kind"] == "moe":
            for e in range(f["router"]["experts"]):
                mat(f"{p}e{e}.gate", f["expert"]["ff"], W, 1.5)
                mat(f"{p}e{e}.up", f["expert"]["ff"], W)
                mat(f"{p}e{e}.down", W, f["expert"]["ff"])
            out[p + "table"] = ((cfg["vocab"], f["router"]["top"]), "table", f["router"]["experts"])
        else:
            if cfg["architecture"] == "Nufalorn":
                mat(p + "gate", f["ff"], W)
            mat(p + "up", f["ff"], W)
            mat(p + "down", W, f["ff"])
    return out


def list_tensor(cfg, name, spec):
    shape, kind, *a = spec
    n = f"{cfg['architecture']}.{name}"
    if kind == "normal":
        return _normal(n, shape, a[0], a[1])
    if kind == "uniform":
        return _uniform(n, shape, a[0], a[1])
    return torch.rand((shape[0], a[0]), generator=_gen(n), device="cuda").topk(shape[1], dim=1).indices.to(torch.int32)


def write_model(path, cfg):
    """a model directory: config.json and model.safetensors"""
    (path / "config.json").write_text(json.dumps(cfg))
    shapes, head, at = list_shapes(cfg), {}, 0
    for name, spec in shapes.items():
        table = spec[1] == "table"
        size = math.prod(spec[0]) * (4 if table else 2)
        head[name] = {"dtype": "I32" if table else "BF16", "shape": list(spec[0]), "data_offsets": [at, at + size]}
        at += size
    text = json.dumps(head).encode()
    text += b" " * (-len(text) % 8)
    with open(path / "model.safetensors", "wb") as f:
        f.write(struct.pack("<Q", len(text)) + text)
        for name, spec in shapes.items():
            t = list_tensor(cfg, name, spec)
            (t if t.dtype == torch.int32 else t.view(torch.int16)).cpu().numpy().tofile(f)


CONFIGS = {"nufalorn": nufalorn_config, "vobunex": vobunex_config, "hybrid": hybrid_config}
STATE_LAYER = {"hybrid": 6, "nufalorn": 3, "vobunex": 3}  # the last recurrent layer


class Buffer:
    """device memory of a tensor, as the library's calls take it"""

    def __init__(self, t):
        self.t, self.ptr = t, t.data_ptr()


class _View:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


class Server:
    """an open model and the prefix of its live sequence"""

    def __init__(self, name, dtype):
        self.name, self.prefix, self.ctx = name, None, context()
        if name == "hybrid":
            c = hybrid_config()
            self.model = M.Model(self.ctx, c)
            for layer in range(c.n_layers):
                slots = [None] * M.WS_SLOTS
                for n in (HYBRID_FA if c.is_fa(layer) else HYBRID_DN) + HYBRID_MLP:
                    t = hybrid_tensor(c, layer, n)
                    for k, x in enumerate(t if isinstance(t, tuple) else (t,)):
                        slots[M.WS[n] + k] = (x.view(torch.int16) if x.dtype == torch.bfloat16 else x).cpu().numpy()
                self.model.load_layer(layer, slots)
            self.model.load_globals([g.view(torch.int16).cpu().numpy() for g in hybrid_globals(c)])
        else:
            with tempfile.TemporaryDirectory() as d:
                write_model(Path(d), CONFIGS[name]())
                self.model = M.Model.open(self.ctx, d, MAX_CTX, dtype)
        self.model.capture()
        p, n = self.model.state_ptr(STATE_LAYER[name], 0)
        self.state = torch.as_tensor(_View(p, (n // 4,), "<f4"), device="cuda")
        p = ctypes.c_uint64(0)
        self.ctx._check(lb.lib().lb_model_logits_ptr(self.model.h, ctypes.byref(p)))
        self.logits = torch.as_tensor(_View(p.value, (VOCAB,), "<f4"), device="cuda")

    def keep(self, n):
        """the kept prefix: the first n tokens of this model's fixed conversation"""
        if self.prefix != n:
            self.model.reset_state()
            if n:
                self.model.prefill(prefix_tokens(n))
            self.model.checkpoint()
            self.prefix = n

    def __del__(self):
        if getattr(self, "model", None):
            self.model.close()


_kept = {}


def context():
    if "ctx" not in _kept:
        torch.cuda.init()
        _kept["ctx"] = lb.Context(0)
    return _kept["ctx"]


def server(name, dtype):
    """the one model that is open"""
    if _kept.get("key") != (name, dtype):
        _kept.pop("server", None)
        _kept["server"], _kept["key"] = Server(name, dtype), (name, dtype)
    return _kept["server"]


def prefix_tokens(n):
    return torch.randint(0, VOCAB, (MAX_CTX,), generator=torch.Generator().manual_seed(1)).tolist()[:n]


def case_tokens(case, seed):
    return torch.randint(0, VOCAB, (case["tokens"],), generator=torch.Generator().manual_seed(1000 + seed)).tolist()


# ---- the cases ---------------------------------------------------------------------------------------------------
def listed():
    return [
        # one projection of a decode step (gate/up of the 27B model) on weights packed at load: the smallest call, latency counts
        {"name": "gemv_5120x17408", "kind": "gemv", "K": 5120, "N": 17408, "packed": True},
        # a projection for a handful of sequences decoded together
        {"name": "gemm_17408x5120_b12", "kind": "gemm", "K": 17408, "N": 5120, "B": 12},
        # a projection of a ragged prompt chunk
        {"name": "gemm_5120x17408_b150", "kind": "gemm", "K": 5120, "N": 17408, "B": 150},
        # a stretch of DeltaNet steps of the 27B model with the state in the caller's buffer
        {"name": "deltanet_256", "kind": "deltanet", "HV": 48, "HK": 16, "steps": 256, "f32": False},
        # decode attention of the 27B model at an ordinary and at a very long context
        {"name": "attention_4k", "kind": "attention", "HQ": 24, "HKV": 4, "pos": 4096, "f32": False},
        {"name": "attention_100k", "kind": "attention", "HQ": 24, "HKV": 4, "pos": 100000, "f32": False},
        # a long prompt, a short follow-up turn and plain decoding of the int4 hybrid
        {"name": "hybrid_prompt_4096", "kind": "prompt", "model": "hybrid", "dtype": "bfloat16", "prefix": 0, "tokens": 4096},
        {"name": "hybrid_turn_75", "kind": "prompt", "model": "hybrid", "dtype": "bfloat16", "prefix": 2000, "tokens": 75},
        {"name": "hybrid_decode", "kind": "decode", "model": "hybrid", "dtype": "bfloat16", "prefix": 2000, "tokens": 16},
        # prompts of the layer-list models, ragged; decoding of the one with the most launches a step
        {"name": "nufalorn_prompt_3000", "kind": "prompt", "model": "nufalorn", "dtype": "bfloat16", "prefix": 0, "tokens": 3000},
        {"name": "vobunex_prompt_4001", "kind": "prompt", "model": "vobunex", "dtype": "bfloat16", "prefix": 0, "tokens": 4001},
        {"name": "vobunex_decode", "kind": "decode", "model": "vobunex", "dtype": "bfloat16", "prefix": 1000, "tokens": 16},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["gemv", "gemm", "gemm", "deltanet", "attention", "attention", "prompt", "prompt", "prompt", "decode", "decode"])
    if kind in ("gemv", "gemm"):
        K, N = 128 * _log(rng, 8, 136), 32 * _log(rng, 32, 544)
        if kind == "gemv":
            return {"kind": kind, "K": K, "N": N, "packed": rng.random() < 0.7}
        return {"kind": kind, "K": K, "N": N, "B": _log(rng, 2, 256)}
    if kind == "deltanet":
        HK = rng.choice([8, 16])
        return {"kind": kind, "HV": HK * rng.choice([2, 3]), "HK": HK, "steps": _log(rng, 1, 512), "f32": rng.random() < 0.5}
    if kind == "attention":
        HKV = rng.choice([2, 4])
        return {"kind": kind, "HQ": HKV * rng.choice([4, 6]), "HKV": HKV, "pos": _log(rng, 100, 100000), "f32": rng.random() < 0.5}
    name = rng.choice(["hybrid", "nufalorn", "vobunex"])
    f32 = name != "hybrid" and rng.random() < 0.2  # the 32-bit format serves as a check: short calls
    prefix = rng.choice([0, _log(rng, 16, 2000)]) if kind == "prompt" else _log(rng, 16, 4000)
    return {"kind": kind, "model": name, "dtype": "float32" if f32 else "bfloat16", "prefix": prefix,
            "tokens": (_log(rng, 2, 256) if f32 else _log(rng, 2, 4096 - prefix)) if kind == "prompt" else _log(rng, 1, 64)}


# ---- one pass ----------------------------------------------------------------------------------------------------
def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return (std * torch.randn(shape, generator=g, device="cuda")).to(dtype)


def inputs(case, seed):
    """the tensors of a call that is not a model's"""
    g = torch.Generator("cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        K, N, B = case["K"], case["N"], case.get("B", 1)
        q, s, z = _int4(f"seed{seed}", K, N)
        return {"q": q, "s": s, "z": z, "x": _randn(g, B, K, dtype=torch.float16), "y": torch.empty((B, N), device="cuda", dtype=torch.float32)}
    if kind == "deltanet":
        HV, HK, T, dt = case["HV"], case["HK"], case["steps"], torch.float32 if case["f32"] else torch.bfloat16
        unit = lambda t: t / t.norm(dim=-1, keepdim=True)  # noqa: E731
        a, b = _randn(g, T, HV), _randn(g, T, HV)
        a_log = 2.7 * torch.rand(HV, generator=g, device="cuda")
        return {"state": _randn(g, HV, 128, 128, std=0.02), "q": (unit(_randn(g, T, HK, 128)) * 128 ** -0.5).to(dt), "k": unit(_randn(g, T, HK, 128)).to(dt),
                "v": _randn(g, T, HV, 128, dtype=dt), "g": torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(a - 3)), "beta": torch.sigmoid(b),
                "out": torch.empty((T, HV, 128), device="cuda")}
    HQ, HKV, L, dt = case["HQ"], case["HKV"], case["pos"] + 1, torch.float32 if case["f32"] else torch.bfloat16
    cache = lambda: _randn(g, L, HKV, 256, dtype=torch.bfloat16)  # noqa: E731
    return {"q": _randn(g, HQ, 256, dtype=dt), "k": _randn(g, HKV, 256, dtype=dt), "v": _randn(g, HKV, 256, dtype=dt), "gate": _randn(g, HQ, 256, dtype=dt),
            "qn": (1 + _randn(g, 256, std=0.02)).to(torch.bfloat16), "kn": (1 + _randn(g, 256, std=0.02)).to(torch.bfloat16),
            "kc": cache(), "vc": cache(), "out": torch.empty((HQ, 256), device="cuda")}


def prepare(case, seed):
    if "model" in case:
        s = server(case["model"], case["dtype"])
        s.keep(case["prefix"])
        return {"case": case, "server": s, "tokens": case_tokens(case, seed)}
    ctx, t = context(), inputs(case, seed)
    b = {n: Buffer(x) for n, x in t.items()}
    state = {"case": case, "ctx": ctx, "b": b}
    torch.cuda.synchronize()
    if case.get("packed") and ctx.gemv_chain_supports(case["K"], case["N"]):
        state["packed"] = ctx.gemv_pack(b["q"], b["s"], b["z"], case["K"], case["N"])
        state["free"] = _Free(state["packed"])
    ctx.sync()
    return state


class _Free:
    """frees a library buffer with the state that holds it"""

    def __init__(self, buffer):
        self.buffer = buffer

    def __del__(self):
        self.buffer.free()


def run(state):
    c = state["case"]
    if c["kind"] in ("prompt", "decode"):
        s, toks, at = state["server"], state["tokens"], c["prefix"]
        m = s.model
        if at:
            m.rollback()
        else:
            m.reset_state()
        if c["kind"] == "prompt":
            m.prefill(toks, at)
        else:
            for i, t in enumerate(toks):
                m.set_input(t, at + i)
                m.replay(1)
            m.read_next()
        return {"logits": s.logits, "state": s.state}
    ctx, b = state["ctx"], state["b"]
    if c["kind"] == "gemv":
        ctx.gemv_int4(b["q"], b["s"], b["z"], b["x"], b["y"], c["K"], c["N"], lb.GEMV_Y_F32)
        return b["y"].t
    if c["kind"] == "gemm":
        ctx.gemm_int4(b["q"], b["s"], b["z"], b["x"], b["y"], c["K"], c["N"], c["B"], lb.GEMV_Y_F32)
        return b["y"].t
    if c["kind"] == "deltanet":
        ctx.deltanet_step(b["state"], b["q"], b["k"], b["v"], None, b["g"], b["beta"], b["out"], c["HV"], c["HK"], c["steps"], c["f32"])
        return {"out": b["out"].t, "state": b["state"].t}
    ctx.attention_decode(b["q"], b["k"], b["v"], b["gate"], b["qn"], b["kn"], b["kc"], b["vc"], b["out"], c["pos"], c["HQ"], c["HKV"], c["f32"])
    return {"out": b["out"].t, "key": b["kc"].t[c["pos"]], "value": b["vc"].t[c["pos"]]}


def work(case):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        K, N, B = case["K"], case["N"], case.get("B", 1)
        return {"bytes": K * N // 2 + K // 128 * N * 2 + K // 128 * N // 2 + B * K * 2 + B * N * 4, "flops": 2 * B * K * N}
    if kind == "deltanet":
        HV, HK, T = case["HV"], case["HK"], case["steps"]
        return {"bytes": 2 * HV * 65536 + T * ((2 * HK + HV) * 128 * (4 if case["f32"] else 2) + HV * (512 + 8)), "flops": 6 * T * HV * 128 * 128}
    if kind == "attention":
        return {"bytes": (case["pos"] + 1) * case["HKV"] * 1024, "flops": 4 * (case["pos"] + 1) * case["HQ"] * 256}
    P, n = case["prefix"], case["tokens"]
    size, macs, att, state = model_work(case["model"])  # weight bytes, multiplications a token, (heads, K and V widths, row bytes, block), state bytes
    if kind == "decode":
        seen = sum(att[3] * (((P + i) % att[4] if att[4] else P + i) + 1) for i in range(n))
        return {"bytes": n * (size + 2 * state) + seen, "flops": 2 * n * macs}
    pairs = sum(((P + i) % att[4] if att[4] else P + i) + 1 for i in range(n))
    return {"bytes": size + 2 * state, "flops": 2 * n * macs + 2 * pairs * att[0] * (att[1] + att[2])}


def model_work(name):
    """per decoded token: weight bytes and multiplications; attention (heads in all layers, key width, value width, cache bytes a position, block); states"""
    if name == "hybrid":
        c = hybrid_config()
        W, F, V = c.hidden, c.inter, c.dn_v_heads * 128
        macs = 6 * (W * (c.conv_channels + V) + V * W) + 2 * (W * (2 * c.fa_q_heads + 2 * c.fa_kv_heads) * 256 + c.fa_q_heads * 256 * W) + 8 * 3 * W * F
        return macs * 133 // 256 + 2 * VOCAB * W, macs, (2 * c.fa_q_heads, 256, 256, 2 * c.fa_kv_heads * 1024, 0), 6 * c.dn_v_heads * 65536
    cfg = CONFIGS[name]()
    macs, state = 0, 0
    for n, (shape, *_r) in list_shapes(cfg).items():
        if len(shape) == 2 and n.startswith("l") and not n.endswith(("table", "conv")):
            macs += math.prod(shape) * (1 if ".mlp.e" not in n else 6 / 64)
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] in ("hgrn2", "gla"):
            state += m["heads"] * m["dim"] * m["vdim"] * 4
        elif layer["type"] == "mamba2":
            state += m["heads"] * m["state"] * m["vdim"] * 4
    att = (32, 128, 128, 8 * 512, 2048) if name == "nufalorn" else (16, 192, 128, 576 * 2, 0)
    return 2 * (macs + VOCAB * cfg["width"]), macs, att, state


def tolerance(case):
    """about four times the distance from 64 bits that was measured for each kind"""
    kind = case["kind"]
    if kind in ("gemv", "deltanet") or case.get("dtype") == "float32":
        return {"rel": 1e-5}  # 32-bit sums
    if kind == "gemm":
        return {"rel": 1e-5 if case["B"] <= 32 else 1e-3}  # from 33 tokens on the weights are rounded to fp16
    if kind == "attention":
        return {"rel": 1e-4, "max": 5e-3}  # the appended rows are bf16: one may round the other way
    return {"hybrid": {"rel": 1e-3}, "nufalorn": {"rel": 1.5e-2, "max": 0.2}, "vobunex": {"rel": 2e-2, "max": 0.2}}[case["model"]]


# ---- the same in 64 bits -----------------------------------------------------------------------------------------
def exact(case, seed):
    torch.backends.cuda.matmul.allow_tf32 = False
    kind = case["kind"]
    if kind in ("prompt", "decode"):
        toks = prefix_tokens(case["prefix"]) + case_tokens(case, seed)
        x, state = (hybrid_exact if case["model"] == "hybrid" else list_exact)(case["model"], torch.tensor(toks, device="cuda"))
        return {"logits": x, "state": state.reshape(-1)}
    t = inputs(case, seed)
    if kind in ("gemv", "gemm"):
        return t["x"].double() @ _dense(t["q"], t["s"], t["z"])
    if kind == "deltanet":
        rep = case["HV"] // case["HK"]
        q, k = (t[n].double().repeat_interleave(rep, 1) for n in ("q", "k"))
        out, S = delta_rule(q, k, t["v"].double(), t["g"].double(), t["beta"].double(), t["state"].double())
        return {"out": out, "state": S}
    d = {n: x.double() for n, x in t.items() if n not in ("kc", "vc", "out")}
    HQ, HKV, pos = case["HQ"], case["HKV"], case["pos"]
    at = torch.tensor([pos], device="cuda")
    turn = lambda x: rotate(x[None], at, 64, 1e7)[0]  # noqa: E731
    q, k = turn(rms(d["q"]) * d["qn"]), turn(rms(d["k"]) * d["kn"])
    kc, vc = t["kc"].clone(), t["vc"].clone()
    kc[pos], vc[pos] = k.to(torch.bfloat16), d["v"].to(torch.bfloat16)
    out = torch.empty((HQ, 256), dtype=torch.float64, device="cuda")
    for h in range(HQ):
        g = h * HKV // HQ
        w = torch.softmax(kc[:, g].double() @ q[h] / 16, 0)
        out[h] = w @ vc[:, g].double()
    return {"out": out * torch.sigmoid(d["gate"]), "key": None, "value": None}


def rms(x, eps=1e-6):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def rotate(x, pos, dims, base, sign=1.0, freq=None, mul=1.0):
    """neighbouring pairs of the first `dims` features turn with the position; x [T, heads, D]"""
    if freq is None:
        freq = base ** (-torch.arange(0, dims, 2, device=x.device, dtype=torch.float64) / dims)
    ang = sign * pos.double()[:, None] * freq
    c, s = (mul * ang.cos())[:, None], (mul * ang.sin())[:, None]
    y = x.clone()
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    y[..., 0:dims:2] = u * c - v * s
    y[..., 1:dims:2] = v * c + u * s
    return y


def delta_rule(q, k, v, g, beta, S):
    """recall from the old state, read-out from the new one; [T, heads, ...]"""
    out = torch.empty_like(v)
    for t in range(len(q)):
        d = beta[t][:, None] * (v[t] - torch.einsum("hi,hij->hj", k[t], S))
        S = g[t][:, None, None] * S + k[t][:, :, None] * d[:, None, :]
        out[t] = torch.einsum("hij,hi->hj", S, q[t])
    return out, S


def attend(q, k, v, scale, block=0, sink=None):
    """causal, in blocks of positions; q [T, H, D], k, v [T, G, ...]"""
    T, H = q.shape[:2]
    i = torch.arange(T, device=q.device)
    mask = i[None] <= i[:, None]
    if block:
        mask &= (i[None] // block) == (i[:, None] // block)
    out = torch.empty((T, H, v.shape[-1]), dtype=torch.float64, device=q.device)
    for h in range(H):
        g = h * k.shape[1] // H
        s = (q[:, h] @ k[:, g].T * scale).masked_fill_(~mask, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :T] @ v[:, g]
    return out


def hybrid_exact(_name, toks):
    c = hybrid_config()
    embed, head, final = hybrid_globals(c)
    x, T, silu = embed[toks].double(), len(toks), torch.nn.functional.silu
    pos, last = torch.arange(T, device="cuda"), None
    for layer in range(c.n_layers):
        w = lambda n: hybrid_tensor(c, layer, n)  # noqa: B023,E731
        mul = lambda y, n: y @ _dense(*w(n))  # noqa: B023,E731
        h = rms(x) * (1 + w("INPUT_NORM").double())
        if c.is_fa(layer):
            qg = mul(h, "FA_Q").view(T, c.fa_q_heads, 512)
            q = rotate(rms(qg[..., :256]) * w("FA_Q_NORM").double(), pos, 64, 1e7)
            k = rotate(rms(mul(h, "FA_K").view(T, c.fa_kv_heads, 256)) * w("FA_K_NORM").double(), pos, 64, 1e7)
            o = attend(q, k, mul(h, "FA_V").view(T, c.fa_kv_heads, 256), 1 / 16) * torch.sigmoid(qg[..., 256:])
            x = x + mul(o.reshape(T, -1), "FA_O")
        else:
            u, taps = mul(h, "DN_QKV"), w("DN_CONV1D").double()
            u = silu(sum(torch.cat([u.new_zeros((j, u.shape[1])), u])[:T] * taps[j] for j in range(4)))
            qk, n = c.dn_k_heads * 128, c.dn_v_heads
            unit = lambda y: (y / y.norm(dim=-1, keepdim=True)).repeat_interleave(n // c.dn_k_heads, 1)  # noqa: B023,E731
            q, k = unit(u[:, :qk].view(T, -1, 128)) * 128 ** -0.5, unit(u[:, qk:2 * qk].view(T, -1, 128))
            a, b = h @ w("DN_PROJ_A").double().T, h @ w("DN_PROJ_B").double().T
            g = torch.exp(-torch.exp(w("DN_A_LOG").double()) * torch.nn.functional.softplus(a + w("DN_DT_BIAS").double()))
            o, last = delta_rule(q, k, u[:, 2 * qk:].view(T, n, 128), g, torch.sigmoid(b), u.new_zeros((n, 128, 128)))
            o = rms(o) * w("DN_NORM").double() * silu(mul(h, "DN_Z").view(T, n, 128))
            x = x + mul(o.reshape(T, -1), "DN_OUT")
        h = rms(x) * (1 + w("POST_NORM").double())
        x = x + mul(silu(mul(h, "GATE")) * mul(h, "UP"), "DOWN")
    return (rms(x[-1]) * (1 + final.double())) @ head.double().T, last


def yarn(dims, base, s):
    f = base ** (-torch.arange(0, dims, 2, device="cuda", dtype=torch.float64) / dims)
    turning = lambda t: dims * math.log(s["original"] / (2 * math.pi * t)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(turning(s["fast"])), 0), min(math.ceil(turning(s["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0, 1).double()
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1


def list_exact(name, toks):
    cfg = CONFIGS[name]()
    shapes, eps, T, silu = list_shapes(cfg), cfg["norm"]["eps"], len(toks), torch.nn.functional.silu
    w = lambda n: list_tensor(cfg, n, shapes[n]).double()  # noqa: E731
    pos, last, serial = torch.arange(T, device="cuda"), None, name == "vobunex"

    def norm(x, n):
        if not serial:
            return rms(x, eps) * (1 + w(n))
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w(n), w(n + ".b"), eps)

    x = w("embed")[toks]
    if serial:
        b = cfg["embedding"]["bigram"]
        rows = torch.full((T,), b["buckets"], device="cuda")
        rows[1:] = (toks[:-1] * b["mul_prev"] + toks[1:] * b["mul_cur"]) % b["buckets"]
        x = x + w("bigram")[rows]
    for i, layer in enumerate(cfg["layers"]):
        m, p, f = layer["mixer"], f"l{i}.mix.", layer["mlp"]
        H, V = m["heads"], m["vdim"]
        h = norm(x, f"l{i}.norm1")
        mul = lambda n: h @ w(p + n).T  # noqa: B023,E731
        if layer["type"] == "attention":
            G, base = m["kv_heads"], m["rot"]["base"]
            q, k = rotate(mul("q").view(T, H, -1), pos, m["rot"]["dims"], base), rotate(mul("k").view(T, G, -1), pos, m["rot"]["dims"], base)
            v = rotate(rms(mul("v").view(T, G, V), eps), pos, V, base)
            s0 = torch.zeros(H, dtype=torch.float64, device="cuda")
            y = rotate(attend(q, k, v, m["scale"], m["mask"]["size"], s0), pos, V, base, -1.0).reshape(T, -1)
        elif layer["type"] == "latent_attention":
            freq, gain = yarn(m["rot_dim"], m["rot"]["base"], m["rot"]["scaling"])
            D, R, z = m["dim"], m["kv_rank"], mul("dkv")
            lat = rms(z[:, :R], eps) * w(p + "dkv.norm")
            kr = rotate(z[:, None, R:], pos, m["rot_dim"], 0, freq=freq, mul=gain)
            q = ((rms(mul("dq"), eps) * w(p + "dq.norm")) @ w(p + "uq").T).view(T, H, -1)
            q = torch.cat([q[..., :D], rotate(q[..., D:], pos, m["rot_dim"], 0, freq=freq, mul=gain)], -1)
            k = torch.cat([(lat @ w(p + "uk").T).view(T, H, D), kr.expand(T, H, -1)], -1)
            y = attend(q, k, (lat @ w(p + "uv").T).view(T, H, V), m["scale"], 0, w(p + "sink")).reshape(T, -1)
        elif layer["type"] == "mamba2":
            inner, G, N, u = H * V, m["groups"], m["state"], mul("in")
            z, u, dt = u[:, :inner], u[:, inner:2 * inner + 2 * G * N], u[:, 2 * inner + 2 * G * N:]
            taps = w(p + "conv")
            u = silu(sum(torch.cat([u.new_zeros((3 - j, u.shape[1])), u])[:T] * taps[:, j] for j in range(4)) + w(p + "conv.b"))
            B, C = (u[:, inner + j * G * N:inner + (j + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for j in (0, 1))
            xs, dt = u[:, :inner].view(T, H, V), torch.nn.functional.softplus(dt + w(p + "dt_bias"))
            a, S, y = torch.exp(-torch.exp(w(p + "A_log")) * dt), u.new_zeros((H, N, V)), torch.empty_like(xs)
            for t in range(T):
                S = a[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * xs[t][:, None, :]
                y[t] = torch.einsum("hnv,hn->hv", S, C[t])
            last = S
            y = ((y + w(p + "D")[:, None] * xs).reshape(T, inner) * silu(z)).view(T, m["norm_groups"], -1)
            y = rms(y, eps).reshape(T, inner) * w(p + "norm")
        else:
            if layer["type"] == "hgrn2":
                q, low = silu(mul("q")), w(p + "lower")
                a = low + (1 - low) * torch.sigmoid(mul("f") + w(p + "f.b"))
                k = 1 - a
            else:
                q, k = mul("q") * m["dim"] ** -0.5, mul("k")
                a = torch.sigmoid(mul("a1") @ w(p + "a2").T + w(p + "a2.b")) ** (1 / m["tau"])
            q, k, a, v = (t.view(T, H, -1) for t in (q, k, a, mul("v")))
            S, o = x.new_zeros((H, m["dim"], V)), torch.empty_like(v)
            for t in range(T):
                S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hd,hdv->hv", q[t], S)
            last = S
            y = (rms(o, eps) * w(p + "norm")).reshape(T, -1)
            if layer["type"] == "gla":
                y = y * silu(mul("g"))
        y = y @ w(p + "o").T
        p = f"l{i}.mlp."
        if not serial:
            h = norm(x, f"l{i}.norm2")
            x = x + cfg["residual_mult"] * (y + (torch.relu(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T)
            continue
        x = x + y
        h = norm(x, f"l{i}.norm2")
        if f["kind"] == "dense":
            x = x + torch.relu(h @ w(p + "up").T) ** 2 @ w(p + "down").T
            continue
        picks = list_tensor(cfg, p + "table", shapes[p + "table"]).long()[toks]
        y, lim = torch.zeros_like(x), f["expert"]["limit"]
        for e in range(f["router"]["experts"]):
            t = (picks == e).any(1).nonzero()[:, 0]
            gate, up = (h[t] @ w(f"{p}e{e}.gate").T).clamp(max=lim), (h[t] @ w(f"{p}e{e}.up").T).clamp(-lim, lim)
            y[t] += (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ w(f"{p}e{e}.down").T / f["router"]["top"]
        x = x + y
    z = norm(x[-1:], "final.norm")[0] @ w("head").T
    if not serial:
        z = cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])
    return z, last
