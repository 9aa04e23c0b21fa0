"""The work that users of this package have it do, as cases to measure: decode steps of the INT4 models, the
reference-format layer as its consumers call it, the projections alone, and prompts and decode steps of the config.json
models.  ``listed`` are fixed cases, ``draw`` gives others of the same ranges, ``run`` is one pass of a case through the
public entry points and ``exact`` the same outputs evaluated in 64 bits by plain torch."""
import dataclasses
import json
import math
import os
import shutil
import struct
import tempfile

import numpy as np
import torch

from blackwell_b200 import kernels as k
from blackwell_b200 import shapes, synth
from blackwell_b200.decode import DecodeEngine
from blackwell_b200.decode_driver import ModelDriver

SHAPES = {"8b": shapes.QWEN3_8B, "2k": shapes.VIFIVIK_BENCH["2k"][1], "4k": shapes.VIFIVIK_BENCH["4k"][1]}
FORMATS = ("w4a8", "w4a4")
MODELS = {"vifivik": lambda: shapes.vifivik_config(2048, 5632, 32768, 4, 1), "lanedra": lambda: shapes.lanedra_config(2048, 5632, 32768, 4, 1)}


def listed():
    return [
        # one user waiting for an INT4 model's next token (six of its layers): weights once, a chain of dependent launches
        {"name": "int4-step-1", "kind": "int4_step", "shape": "8b", "layers": 6, "batch": 1, "ctx": 2048},
        # a small server batch of the same model
        {"name": "int4-step-8", "kind": "int4_step", "shape": "8b", "layers": 6, "batch": 8, "ctx": 2048},
        # a full server batch: more than 16 sequences take the tcgen05 product
        {"name": "int4-step-64", "kind": "int4_step", "shape": "8b", "layers": 6, "batch": 64, "ctx": 1024},
        # long documents: the cache outweighs the weights
        {"name": "int4-step-4-long", "kind": "int4_step", "shape": "8b", "layers": 6, "batch": 4, "ctx": 16384},
        # a small model a few tokens in, an odd batch and context: launches and latencies
        {"name": "int4-step-3-small", "kind": "int4_step", "shape": "2k", "layers": 6, "batch": 3, "ctx": 101},
        # the five projections of a layer and the head at one sequence, binary16 in: the headline workload
        {"name": "projections-1", "kind": "projections", "shape": "8b", "format": "w4a8", "batch": 1},
        # a layer as consumers of the reference's kernel interface run it: INT4 activations, fp32 scales, fp32 cache
        {"name": "reference-layer-4", "kind": "reference_layer", "shape": "8b", "batch": 4, "ctx": 2048},
        # a long prompt of a config.json model, up to its last logits
        {"name": "prompt-vifivik-4096", "kind": "prompt", "model": "vifivik", "tokens": 4096},
        # a short question: a few dozen rows, everything is latency
        {"name": "prompt-vifivik-37", "kind": "prompt", "model": "vifivik", "tokens": 37},
        # a group of unequal prompts begins together and samples its first ids, as the daemon does
        {"name": "group-lanedra-4", "kind": "group", "model": "lanedra", "batch": 4, "tokens": 1003},
        # decode steps: a server batch, and one sequence
        {"name": "step-vifivik-32", "kind": "model_step", "model": "vifivik", "batch": 32, "ctx": 2048},
        {"name": "step-lanedra-1", "kind": "model_step", "model": "lanedra", "batch": 1, "ctx": 2048},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["int4_step", "int4_step", "projections", "reference_layer", "prompt", "prompt", "group", "model_step", "model_step"])
    case = {"kind": kind}
    if kind in ("int4_step", "projections", "reference_layer"):
        case["shape"] = rng.choice(list(SHAPES))
    else:
        case["model"] = rng.choice(list(MODELS))
    if kind == "int4_step":
        case["layers"] = 6
        case["batch"] = _log(rng, 1, 64)
        case["ctx"] = _log(rng, 17, min(16384, 65536 // case["batch"]))
    elif kind == "projections":
        case["format"] = rng.choice(FORMATS)
        case["batch"] = _log(rng, 1, 64 if case["format"] == "w4a8" else 16)
    elif kind == "reference_layer":
        case["batch"] = _log(rng, 1, 16)
        case["ctx"] = _log(rng, 17, 4096)
    elif kind == "prompt":
        case["tokens"] = _log(rng, 17, 4096)
    elif kind == "group":
        case["batch"] = rng.randint(2, 6)
        case["tokens"] = _log(rng, 17, 6000 // (case["batch"] + 1))
    else:
        case["batch"] = _log(rng, 1, 48)
        case["ctx"] = _log(rng, 17, 2048)
    return case


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# ------------------------------------------------------------------------------------------------ INT4 models
def _int4_shape(case):
    return dataclasses.replace(SHAPES[case["shape"]], layers=case["layers"])


class _Int4Step:
    """A model with its caches filled up to ctx - 1 and the step captured, as a server keeps them."""

    def __init__(self, case, seed):
        self.e = e = DecodeEngine(_int4_shape(case), case["batch"], case["ctx"] + 16, "cuda", seed=seed)
        self.at = case["ctx"] - 1
        e.fill_cache(case["ctx"], seed)
        self.tokens = torch.randint(0, e.s.vocab, (case["batch"],), dtype=torch.int32, device="cuda", generator=_gen(seed))
        self.positions = torch.full_like(self.tokens, self.at)

    def capture(self):
        self.feed()
        self.e.step()   # sizes the library's scratch
        self.feed()
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.e.step()
        return self

    def feed(self):
        self.e.tokens.copy_(self.tokens)
        self.e.pos.copy_(self.positions)

    def run(self):
        self.feed()
        self.graph.replay()
        return {"logits": self.e.logits, "hidden": self.e.x}


class _Projections:
    """The projections of one layer and the head on activations that are at hand: binary16 (w4a8) or INT4 (w4a4)."""

    def __init__(self, case, seed):
        self.M, self.a8 = case["batch"], case["format"] == "w4a8"
        self.mats, x = [], {}
        for i, (_, N, K) in enumerate(SHAPES[case["shape"]].gemv_set()):
            W, sc = synth.int4_weights_device(N, K, seed * 100 + i, scale_dtype=None if self.a8 else torch.float32)
            if K not in x:
                x[K] = self.activations(K, seed * 100 + 50 + i)
            self.mats.append((W, sc, N, K, x[K], torch.empty((self.M, N), device="cuda")))

    def activations(self, K, seed):
        f16 = synth.activations_f16_device(self.M, K, seed)
        if self.a8:
            return f16
        packed = torch.empty((self.M, K // 2), dtype=torch.uint8, device="cuda")
        scale = torch.empty((self.M, K // 16), device="cuda")
        k.quantize_int4_batched(packed, scale, f16.float(), K, self.M)
        return packed, scale

    def run(self):
        for W, sc, N, K, x, y in self.mats:
            if self.a8:
                k.gemv_w4a8_f16in(y, x, W, sc, K, N, self.M)
            else:
                k.gemv_int4_batched(y, x[0], x[1], W, sc, K, N, self.M)
        return [m[5] for m in self.mats]


class _ReferenceLayer:
    """One decoder layer in the reference's formats, by the sequence of calls of its INT4 servers, captured in a graph."""

    def __init__(self, case, seed):
        self.s = s = SHAPES[case["shape"]]
        self.M, self.ctx = M, ctx = case["batch"], case["ctx"]
        H, I, Q, KV = s.hidden, s.inter, s.q_dim, s.kv_dim
        sizes = {"q": (Q, H), "k": (KV, H), "v": (KV, H), "o": (H, Q), "gate": (I, H), "up": (I, H), "down": (H, I)}
        self.W = {n: synth.int4_weights_device(*nk, seed * 100 + i, scale_dtype=torch.float32) for i, (n, nk) in enumerate(sizes.items())}
        g = _gen(seed)
        f32 = lambda *shape: torch.randn(shape, device="cuda", generator=g)
        self.norms = [1.0 + 0.1 * f32(H) for _ in range(2)]
        self.x = f32(M, H)
        self.kc, self.vc = f32(M, s.n_kv_heads, ctx, 128), f32(M, s.n_kv_heads, ctx, 128)
        self.pos = torch.full((1,), ctx - 1, dtype=torch.int32, device="cuda")
        self.n_h = [f32(M, H) for _ in range(5)]
        self.n_q, self.n_k, self.n_v, self.att = f32(M, Q), f32(M, KV), f32(M, KV), f32(M, Q)
        self.n_gate, self.n_up, self.act = f32(M, I), f32(M, I), f32(M, I)
        self.packed = torch.empty((M, max(H, I, Q) // 2), dtype=torch.uint8, device="cuda")
        self.scale = torch.empty((M, max(H, I, Q) // 16), device="cuda")
        self.out = f32(M, H)

    def project(self, y, name):
        W, sc = self.W[name]
        k.gemv_int4_batched(y, self.packed, self.scale, W, sc, W.shape[1] * 2, W.shape[0], self.M)

    def layer(self):
        s, M, H, I, Q, KV = self.s, self.M, self.s.hidden, self.s.inter, self.s.q_dim, self.s.kv_dim
        normed, o, mid, normed2, down = self.n_h
        k.fused_rmsnorm_batched(normed, self.x, self.norms[0], H, s.eps, M)
        k.quantize_int4_batched(self.packed, self.scale, normed, H, M)
        self.project(self.n_q, "q")
        self.project(self.n_k, "k")
        self.project(self.n_v, "v")
        for m in range(M):   # row m of the new keys and values into sequence m's cache
            k.update_kv_cache_device(self.kc[m], self.vc[m], self.n_k[m], self.n_v[m], 0, self.pos, s.n_kv_heads, 128, self.ctx)
        k.attention_decode_batched_gqa_device(self.att, self.n_q, self.kc, self.vc, self.pos, s.n_q_heads, s.n_kv_heads, 128, self.ctx, M,
                                              s.n_kv_heads * self.ctx * 128, 0)
        k.quantize_int4_batched(self.packed, self.scale, self.att, Q, M)
        self.project(o, "o")
        k.vector_add_fp32(mid, self.x, o, M * H)
        k.fused_rmsnorm_batched(normed2, mid, self.norms[1], H, s.eps, M)
        k.quantize_int4_batched(self.packed, self.scale, normed2, H, M)
        self.project(self.n_gate, "gate")
        self.project(self.n_up, "up")
        k.apply_swiglu(self.act, self.n_gate, self.n_up, M * I)
        k.quantize_int4_batched(self.packed, self.scale, self.act, I, M)
        self.project(down, "down")
        k.vector_add_fp32(self.out, mid, down, M * H)

    def capture(self):
        self.layer()
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.layer()
        return self

    def run(self):
        self.graph.replay()
        return {"out": self.out, "attention": self.att, "k": self.n_k, "v": self.n_v}


# ------------------------------------------------------------------------------------------------ config.json models
def _with_model(case, seed, use):
    """use(directory) with a model of random weights in it: a load-time file, gone when the model is loaded."""
    root = tempfile.mkdtemp(dir="/dev/shm" if os.access("/dev/shm", os.W_OK) else None)
    try:
        synth.write_random_model(root, MODELS[case["model"]](), seed=seed)
        return use(root)
    finally:
        shutil.rmtree(root)


def _prompts(case, seed):
    """Token ids by sequence: equal lengths, or unequal ones for a group."""
    rng = np.random.default_rng(seed)
    n, B = case.get("tokens", case.get("ctx")), case.get("batch", 1)
    lengths = [max(2, n * (B - i) // B) for i in range(B)] if case["kind"] == "group" else [n] * B
    return [rng.integers(0, MODELS[case["model"]]()["vocab"], m).tolist() for m in lengths]


class _Driver(ModelDriver):
    def __del__(self):
        if getattr(self, "_h", None):
            self.close()


class _Model:
    def __init__(self, case, seed):
        self.kind = case["kind"]
        self.prompts = _prompts(case, seed)
        longest = max(len(p) for p in self.prompts)
        self.d = _with_model(case, seed, lambda root: _Driver(root, batch=len(self.prompts), max_seq=longest, max_prompt=longest))
        self.logits = self.d.logits()
        self.logits.driver = self.d   # the driver owns the memory
        if self.kind == "model_step":
            self.d.begin(self.prompts)   # the context; the steps below stay at its last position

    def run(self):
        if self.kind == "prompt":
            self.d.release(0)
            return self.d.portion(0, self.prompts[0], [len(self.prompts[0]) - 1])
        if self.kind == "group":
            self.d.begin(self.prompts)
        self.d.step()
        return self.logits


def prepare(case, seed):
    kind = case["kind"]
    if kind == "int4_step":
        return _Int4Step(case, seed).capture()
    if kind == "projections":
        return _Projections(case, seed)
    if kind == "reference_layer":
        return _ReferenceLayer(case, seed).capture()
    return _Model(case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------------ what a pass must do
def work(case):
    kind = case["kind"]
    if kind in ("int4_step", "projections", "reference_layer"):
        s, M = SHAPES[case["shape"]], case["batch"]
        macs = {n: N * K for n, N, K in s.gemv_set()}
        layer = sum(v for n, v in macs.items() if n != "lm_head")
        if kind == "projections":
            x = sum(K * (2 if case["format"] == "w4a8" else 0.75) for K in {K for _, _, K in s.gemv_set()})
            y = sum(4 * N for _, N, _ in s.gemv_set())
            return {"bytes": (layer + macs["lm_head"]) * (0.625 if case["format"] == "w4a8" else 0.75) + M * (x + y),
                    "flops": 2 * M * (layer + macs["lm_head"])}
        pairs = M * case["ctx"] * s.n_kv_heads * 256      # cached numbers that a layer reads
        if kind == "reference_layer":
            return {"bytes": layer * 0.75 + 4 * (pairs + 2 * M * s.hidden), "flops": 2 * M * layer + 2 * pairs * s.n_q_heads / s.n_kv_heads}
        return {"bytes": _step_bytes(case["layers"], layer, macs["lm_head"], pairs, M, s),
                "flops": 2 * M * (case["layers"] * layer + macs["lm_head"]) + case["layers"] * 2 * pairs * s.n_q_heads / s.n_kv_heads}
    cfg = MODELS[case["model"]]()
    lengths = [len(p) for p in _prompts(case, 0)]
    weights, flops, cached = 2 * cfg["vocab"] * cfg["width"], 0, 0
    for L in cfg["layers"]:
        matrix, per_token, per_pair, row, state = _layer_work(cfg["width"], L)
        weights += 2 * matrix
        window = L["mixer"].get("mask", {}).get("size", 1 << 30)
        for n in lengths:
            if kind == "model_step":
                flops += 2 * (matrix + per_token) + 2 * per_pair * min(n, window)
                cached += 2 * state + row * min(n, window)
            else:
                full = max(0, n - window)
                flops += 2 * n * (matrix + per_token) + 2 * per_pair * (full * window + (n - full) * (n - full + 1) // 2)
                cached += state + row * min(n, window)
    flops += 2 * len(lengths) * cfg["vocab"] * cfg["width"]
    return {"bytes": weights + cached + 4 * len(lengths) * cfg["vocab"], "flops": flops}


def _step_bytes(layers, layer, head, pairs, M, s):
    return layers * (layer * 0.625 + pairs * 2) + head * 0.625 + M * (2 * s.hidden + 4 * s.vocab)


def _layer_work(W, L):
    """(weights of the matrices, multiply-adds of a token besides them, of a query-key pair, bytes of a cached row, bytes of
    the recurrent state) of one layer"""
    m, t = L["mixer"], L["type"]
    H, V = m["heads"], m["vdim"]
    ff = 3 * W * L["mlp"]["ff"]
    out = W * H * V
    if t == "mamba2":
        return W * (2 * H * V + 2 * m["groups"] * m["state"] + H) + out + ff, 2 * H * V * m["state"], 0, 0, 4 * H * V * m["state"]
    if t == "retention":
        return W * 2 * H * (m["dim"] + V) + out + ff, 2 * H * V * m["dim"], 0, 0, 4 * H * V * m["dim"]
    if t == "delta":
        return W * (2 * H * (V + 1) + 2 * m["kv_heads"] * m["dim"]) + out + ff, 3 * H * V * m["dim"], 0, 0, 4 * H * V * m["dim"]
    own = "kv_from" not in m
    if t == "attention":
        kv = m["kv_heads"] * (2 * m["dim"] + V)
        return W * (2 * H * m["dim"] + own * kv) + out + ff, 0, 2 * H * (m["dim"] + V), 2 * kv, 0
    R, rot = m["kv_rank"], m["rot_dim"]
    expand = H * (m["dim"] + V) * R
    return W * (H * (m["dim"] + rot + 1) + own * (R + rot)) + expand + out + ff, 0, H * (m["dim"] + rot + V), 2 * (R + rot), 0


def tolerance(case):
    """Against another order of the sums.  Projections: 1e-7 measured, times twenty.  A step rounds its activations to 8 bits in
    every projection, and a tie that falls the other way, with what follows from it, moves the result: 0.010 between two routes of
    six layers (measured; a single reference layer, rounded to 4 bits: 0 to 0.003).  bfloat16 models: 0.007 to 0.011 from 64 bits."""
    kind = case["kind"]
    if kind == "projections":
        return {"rel": 2e-6, "max": 1e-3}
    if kind == "reference_layer":
        return {"rel": 1e-2}
    return {"rel": 3e-2, "max": 0.5}


# ------------------------------------------------------------------------------------------------ 64-bit evaluation
def _blocks(x, levels):
    """x [M][K] with every 16 consecutive values rounded to `levels` steps of their largest magnitude."""
    b = x.double().unflatten(-1, (-1, 16))
    sc = b.abs().amax(-1, keepdim=True) / levels
    sc = torch.where(sc < 1e-10, torch.ones_like(sc), sc)
    q = b / sc
    return ((q.abs() + 0.5).floor() * q.sign() * sc).flatten(-2)


def _dequantized(W, sc):
    q = torch.stack((W & 15, W >> 4), -1).flatten(-2).double() - 8
    return (q.unflatten(-1, (-1, 16)) * sc.double()[..., None]).flatten(-2)


def _product(x, W, sc):
    return torch.cat([x @ _dequantized(W[i:i + 16384], sc[i:i + 16384]).T for i in range(0, W.shape[0], 16384)], -1)


def _unit(x, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt()


def _interleaved(x, positions, dims, base):
    """x [..., T, D]: the pairs (2i, 2i+1) below dims turn by position * base^(-2i/dims)"""
    a = positions.double()[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device, dtype=torch.float64) / dims)
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    turned = torch.stack((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()), -1).flatten(-2)
    return torch.cat((turned, x[..., dims:]), -1)


def _cache_attention(q, kc, vc):
    """q [M][heads][128] over every row of kc, vc [M][kv heads][ctx][128]"""
    g = q.unflatten(1, (kc.shape[1], -1))
    p = torch.einsum("mgqd,mgtd->mgqt", g, kc.double()).mul(128 ** -0.5).softmax(-1)
    return torch.einsum("mgqt,mgtd->mgqd", p, vc.double()).flatten(1)


def _exact_projections(case, seed):
    st = _Projections(case, seed)
    out = []
    for W, sc, _, _, x, _ in st.mats:
        out.append(_product(_blocks(x, 127) if st.a8 else _dequantized(*x), W, sc))
    return out


def _exact_reference_layer(case, seed):
    st = _ReferenceLayer(case, seed)
    s, M, W = st.s, st.M, st.W
    h = _blocks(_unit(st.x.double(), s.eps) * st.norms[0].double(), 7)
    q, kn, v = (_product(h, *W[n]) for n in "qkv")
    kc, vc = st.kc.double(), st.vc.double()
    kc[:, :, -1], vc[:, :, -1] = kn.view(M, -1, 128), v.view(M, -1, 128)
    att = _cache_attention(q.view(M, -1, 128), kc, vc).flatten(1)
    return {"out": None, "attention": att, "k": kn, "v": v}


def _read_tensors(root):
    """name -> float64 tensor of a model.safetensors of bfloat16 tensors"""
    with open(os.path.join(root, "model.safetensors"), "rb") as f:
        header = json.loads(f.read(struct.unpack("<Q", f.read(8))[0]))
        data = f.read()
    raw = torch.frombuffer(bytearray(data), dtype=torch.bfloat16)
    return {n: raw[h["data_offsets"][0] // 2:h["data_offsets"][1] // 2].view(h["shape"]).cuda() for n, h in header.items()}


def _conv(x, taps, bias=None):
    """Causal convolution of every channel; x [B][T][C], taps [C][n], the current token at the last tap"""
    n, T = taps.shape[1], x.shape[1]
    x = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return sum(x[:, j:j + T] * taps[:, j] for j in range(n)) + (0 if bias is None else bias)


def _recurrence(q, kk, v, decay, weight, delta=False):
    """S <- decay_t S (+ the delta rule's correction) + weight_t k_t v_t^T, o_t = S^T q_t; [B][T][heads][...]"""
    S = v.new_zeros(v.shape[0], v.shape[2], kk.shape[-1], v.shape[-1])
    out = torch.empty_like(v)
    for t in range(v.shape[1]):
        S *= decay[:, t, :, None, None]
        new = v[:, t]
        if delta:
            new = new - (kk[:, t, :, None, :] @ S)[..., 0, :]
        S += kk[:, t, :, :, None] * (weight[:, t, :, None] * new)[..., None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :]
    return out


def _mamba2(w, m, eps, x):
    H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    z, xbc, dt = (x @ w("in").T).split((H * V, H * V + 2 * G * N, H), -1)
    xs, B, C = torch.nn.functional.silu(_conv(xbc, w("conv"), w("conv.b"))).split((H * V, G * N, G * N), -1)
    xs = xs.unflatten(-1, (H, V))
    B, C = (y.unflatten(-1, (G, N)).repeat_interleave(H // G, 2) for y in (B, C))
    dt = torch.nn.functional.softplus(dt + w("dt_bias"))
    y = _recurrence(C, B, xs, torch.exp(-w("A_log").exp() * dt), dt) + w("D")[:, None] * xs
    y = y.flatten(2) * torch.nn.functional.silu(z)
    return (_unit(y.unflatten(-1, (m["norm_groups"], -1)), eps).flatten(2) * w("norm")) @ w("o").T


def _retention(w, m, eps, x):
    H, D = m["heads"], m["dim"]
    q, kk, v = ((x @ w(n).T).unflatten(-1, (H, -1)) for n in "qkv")
    decay = torch.tensor(m["decay"], device=x.device, dtype=torch.float64).expand(x.shape[:2] + (H,))
    o = _unit(_recurrence(q, kk * D ** -0.5, v, decay, torch.ones_like(decay)), eps)
    return (o.flatten(2) * torch.nn.functional.silu(x @ w("g").T)) @ w("o").T


def _delta(w, m, eps, x):
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    q, kk, v = (torch.nn.functional.silu(_conv(x @ w(n).T, w(n + ".conv"))) for n in "qkv")
    q, kk = (y.unflatten(-1, (G, D)) for y in (q, kk))
    q, kk = ((y * (y.square().sum(-1, keepdim=True) + 1e-6).rsqrt()).repeat_interleave(H // G, 2) for y in (q, kk))
    decay = torch.exp(-w("A_log").exp() * torch.nn.functional.softplus(x @ w("a").T + w("dt_bias")))
    o = _recurrence(q * D ** -0.5, kk, v.unflatten(-1, (H, -1)), decay, torch.sigmoid(x @ w("b").T), delta=True)
    return ((_unit(o, eps) * w("norm")).flatten(2) * torch.nn.functional.silu(x @ w("g").T)) @ w("o").T


def _latent(w, m, eps, x, cache):
    H, D, R, rot = m["heads"], m["dim"], m["kv_rank"], m["rot"]
    at = torch.arange(x.shape[1], device=x.device)
    if cache is None:
        c, kr = (x @ w("dkv").T).split((R, m["rot_dim"]), -1)
        cache = _unit(c, eps) * w("dkv.norm"), _interleaved(kr, at, rot["dims"], rot["base"])
    c, kr = cache
    q = (x @ w("q").T).unflatten(-1, (H, -1)).transpose(1, 2)
    qr = _interleaved(q[..., D:], at, rot["dims"], rot["base"])
    kk, v = ((c @ w(n).T).unflatten(-1, (H, -1)).transpose(1, 2) for n in ("uk", "uv"))
    hidden = at[:, None] < at
    out = torch.empty_like(v)
    for b in range(x.shape[0]):
        for h in range(H):
            s = (q[b, h, :, :D] @ kk[b, h].T + qr[b, h] @ kr[b].T) * m["scale"]
            s = torch.cat((s.masked_fill_(hidden, -math.inf), w("sink")[h].expand(len(at), 1)), 1).softmax(-1)
            out[b, h] = s[:, :-1] @ v[b, h]
    out = out.transpose(1, 2) * torch.sigmoid(x @ w("g").T)[..., None]
    return out.flatten(2) @ w("o").T, cache


def _turned_halves(y, rot):
    """y [B][T][heads][2][D] with the pairs (i, i + dims / 2) turned by YaRN's angles"""
    dims, sc = rot["dims"], rot["scaling"]
    i = torch.arange(dims // 2, device=y.device, dtype=torch.float64)
    f = rot["base"] ** (-2 * i / dims)
    pair = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))
    lo, hi = max(math.floor(pair(sc["fast"])), 0), min(math.ceil(pair(sc["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    a = torch.arange(y.shape[1], device=y.device).double()[:, None, None, None] * (f / sc["factor"] * ramp + f * (1 - ramp))
    gain = 0.1 * math.log(sc["factor"]) + 1.0
    u, v, rest = y.split((dims // 2, dims // 2, y.shape[-1] - dims), -1)
    return torch.cat(((u * a.cos() - v * a.sin()) * gain, (v * a.cos() + u * a.sin()) * gain, rest), -1)


def _differential(w, m, eps, x, cache):
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    if cache is None:
        cache = _turned_halves((x @ w("k").T).unflatten(-1, (G, 2, D)), m["rot"]), (x @ w("v").T).unflatten(-1, (G, -1))
    kk, v = cache
    q = _turned_halves((x @ w("q").T).unflatten(-1, (H, 2, D)), m["rot"])
    lam = torch.exp(w("lq1") @ w("lk1")) - torch.exp(w("lq2") @ w("lk2")) + m["diff"]
    at = torch.arange(x.shape[1], device=x.device)
    hidden = (at[:, None] < at) | (at[:, None] - at >= m["mask"]["size"])
    out = x.new_empty(x.shape[:2] + (H, m["vdim"]))
    for b in range(x.shape[0]):
        for h in range(H):
            g = h // (H // G)
            a = [((q[b, :, h, i] @ kk[b, :, g, i].T) * m["scale"]).masked_fill_(hidden, -math.inf).softmax(-1) @ v[b, :, g] for i in range(2)]
            out[b, :, h] = a[0] - lam * a[1]
    return (_unit(out, eps) * (1 - m["diff"])).flatten(2) @ w("o").T, cache


def _exact_model(case, seed):
    cfg = MODELS[case["model"]]()
    tensors = _with_model(case, seed, _read_tensors)
    prompts = _prompts(case, seed)
    longest, eps, lanedra = max(map(len, prompts)), cfg["norm"]["eps"], case["model"] == "lanedra"
    ids = torch.tensor([p + [0] * (longest - len(p)) for p in prompts], device="cuda")   # what follows a prompt does not reach it
    at = lambda prefix: lambda name: tensors[prefix + name].double()
    norm = lambda x, w: _unit(x, eps) * (w + 1 if lanedra else w)
    x, cached = tensors["embed"][ids].double() * cfg.get("embedding", {}).get("scale", 1.0), {}
    for i, L in enumerate(cfg["layers"]):
        w, m = at("l%d." % i), L["mixer"]
        mix = at("l%d.mix." % i)
        h = norm(x, w("norm1")) if lanedra else x
        if L["type"] in ("attention", "latent_attention"):
            f = _latent if L["type"] == "latent_attention" else _differential
            y, cached[i] = f(mix, m, eps, h, cached.get(m.get("kv_from")))
        else:
            y = {"mamba2": _mamba2, "retention": _retention, "delta": _delta}[L["type"]](mix, m, eps, h)
        x = x + norm(y, w("norm1b" if lanedra else "norm1"))
        h = norm(x, w("norm2")) if lanedra else x
        y = (torch.nn.functional.silu(h @ w("mlp.gate").T) * (h @ w("mlp.up").T)) @ w("mlp.down").T
        x = x + norm(y, w("norm2b" if lanedra else "norm2"))
    x = x[torch.arange(len(prompts)), [len(p) - 1 for p in prompts]]
    logits = norm(x, at("")("final.norm")) @ at("")("head").T
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def exact(case, seed):
    """None for what depends on activations that were rounded to 4 or 8 bits after a sum: a last bit of the sum that moves one of
    them across a tie moves the result by a whole step of that rounding, so that the 64-bit sums do not say which result is meant."""
    if case["kind"] == "int4_step":
        return None
    with torch.no_grad():
        return {"projections": _exact_projections, "reference_layer": _exact_reference_layer}.get(case["kind"], _exact_model)(case, seed)
