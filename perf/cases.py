"""Workloads of libsmelt_cuda: what a program that uses it spends its time on, from one projection to whole decoders.

Kinds of case, each through the C ABI that ``smelt_b200.capi`` binds:

* ``projection``  one affine u4 matrix times some rows of activations (the typed launchers): what a host that brings its
                  own schedule calls.
* ``decode``      one token per sequence of a plain affine u4 decoder from its captured graph, host tokens in, ids out.
* ``prefill``     a prompt chunk of that decoder, behind a prompt that is already in the cache.
* ``lowbit``      the feed-forward halves of layers with binary or ternary weights.
* ``hybrid``      a new sequence through a decoder with DeltaNet and attention layers: prompt chunks, then decode steps.
* ``pesedra``     the same through a looped decoder with bf16 weights and window + pooled-block attention.
* ``kesedra``     the same through a stack of latent attention, time mixing and expert layers.

Sizes are those of the benchmarks (widths 2048 / 4096 / 5120, the 36-layer model).  Weights are made on the GPU from the
seed, with the distributions of ``smelt_b200.synth``; ``exact`` computes every case again in float64 with plain torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from smelt_b200 import capi

WEIGHTS, LOGITS, KV = 30, 16, 40  # buffer slots
GROUP, EPS, THETA, CHUNK = 64, 1e-6, 1e6, 512
# width -> feed-forward, query heads, key heads, head size
PLAIN = {2048: (6144, 16, 4, 128), 4096: (12288, 32, 8, 128), 5120: (17408, 40, 8, 128)}
# width -> feed-forward, attention heads, query latent, inner size of the decay, expert feed-forward
STACK = {2048: (6144, 16, 768, 64, 768), 4096: (12288, 32, 1536, 64, 1536), 5120: (17408, 40, 1536, 96, 2176)}
WINDOW, POOL, LATENT, ROT, WKV_DIM, EXPERTS, TOP, LIMIT = 1024, 16, 512, 64, 64, 16, 4, 7.0
FEATURES = 6  # elements of a Kesedra stream that no layer changes and that its routers read


# ── what is measured ────────────────────────────────────────────────────────
def listed():
    return [
        # the smallest call there is: one row through one small projection
        {"name": "projection_4096x1024", "kind": "projection", "mode": "matvec", "rows": 4096, "cols": 1024, "batch": 1},
        # the headline benchmark: single-stream decoding of the 36-layer model in the middle of a chat
        {"name": "decode_ctx600", "kind": "decode", "width": 4096, "layers": 36, "vocab": 151936, "batch": 1, "context": 600},
        # the same behind a long document: attention reads as much as the weights
        {"name": "decode_ctx32000", "kind": "decode", "width": 4096, "layers": 36, "vocab": 151936, "batch": 1, "context": 32000},
        # a handful of sequences at once, the batch of the committed fixtures
        {"name": "decode_batch8", "kind": "decode", "width": 4096, "layers": 36, "vocab": 151936, "batch": 8, "context": 1023},
        # a small server: as many sequences as the middle of the range takes
        {"name": "decode_batch32", "kind": "decode", "width": 4096, "layers": 36, "vocab": 151936, "batch": 32, "context": 300},
        # the benchmark's prompt in one chunk
        {"name": "prefill_512", "kind": "prefill", "width": 4096, "layers": 36, "vocab": 151936, "tokens": 512, "start": 0},
        # a short, ragged follow-up turn behind a cached prompt
        {"name": "prefill_77_at_1300", "kind": "prefill", "width": 4096, "layers": 36, "vocab": 151936, "tokens": 77, "start": 1300},
        # single-stream decoding with 1-bit and with ternary weights
        {"name": "lowbit_binary", "kind": "lowbit", "format": 1, "width": 5120, "ff": 17408, "layers": 4, "batch": 1},
        {"name": "lowbit_ternary", "kind": "lowbit", "format": 2, "width": 5120, "ff": 17408, "layers": 4, "batch": 1},
        # a prompt and a short answer on a hybrid decoder
        {"name": "hybrid_turn", "kind": "hybrid", "width": 2048, "layers": 16, "vocab": 32768, "tokens": 300, "steps": 16},
        # a long prompt on the looped bf16 decoder, ragged in its last chunk
        {"name": "pesedra_prompt", "kind": "pesedra", "width": 4096, "precision": "bfloat16", "tokens": 1900, "steps": 0},
        # an answer on the stack, behind a prompt of a few tokens
        {"name": "kesedra_answer", "kind": "kesedra", "width": 4096, "precision": "bfloat16", "tokens": 40, "steps": 24},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["projection"] * 3 + ["decode"] * 4 + ["prefill"] * 2 + ["lowbit"] * 2 + ["hybrid", "pesedra", "pesedra", "kesedra", "kesedra"])
    if kind == "projection":
        return {"kind": kind, "mode": rng.choice(["matvec", "add", "gate_up", "dual"]), "rows": 8 * _log_int(rng, 32, 1536), "cols": 64 * _log_int(rng, 8, 192),
                "batch": _log_int(rng, 1, 512)}
    if kind in ("decode", "prefill"):
        width = rng.choice([2048, 4096, 5120])
        case = {"kind": kind, "width": width, "layers": _log_int(rng, 2, 36 if width < 5120 else 18), "vocab": rng.choice([32768, 151936])}
        if kind == "decode":
            batch = _log_int(rng, 1, 64)
            return {**case, "batch": batch, "context": _log_int(rng, 16, min(32000, 64000 // batch))}
        return {**case, "tokens": _log_int(rng, 2, 512), "start": rng.choice([0, rng.randrange(1, 2000)])}
    if kind == "lowbit":
        return {"kind": kind, "format": rng.choice([1, 2]), "width": 128 * rng.randrange(16, 45), "ff": 128 * rng.randrange(48, 140), "layers": rng.randrange(3, 7),
                "batch": _log_int(rng, 1, 8)}
    if kind == "hybrid":
        return {"kind": kind, "width": rng.choice([1024, 2048]), "layers": 4 * rng.randrange(1, 6), "vocab": 32768, "tokens": _log_int(rng, 2, 700), "steps": rng.randrange(0, 24)}
    case = {"kind": kind, "width": rng.choice([2048, 4096]), "precision": rng.choice(["bfloat16"] * 3 + ["float32"])}
    longest = 512 if case["precision"] == "float32" else 1900 if kind == "pesedra" else 1100
    return {**case, "tokens": _log_int(rng, 2, longest), "steps": rng.randrange(0, 16)}


# ── device memory ───────────────────────────────────────────────────────────
class _Span:
    """A stretch of a context's device memory as torch sees it: a tensor over it keeps the context alive."""

    def __init__(self, ctx, ptr, nbytes):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _slot(ctx, index, dtype, *shape):
    ptr, size = C.c_void_p(), C.c_size_t()
    ctx._check(ctx.lib.smelt_cuda_slot_ptr(ctx.h, index, C.byref(ptr), C.byref(size)))
    n = math.prod(shape) * torch.empty(0, dtype=dtype).element_size() if shape else size.value
    out = torch.as_tensor(_Span(ctx, ptr.value, n), device="cuda").view(dtype)
    return out.view(*shape) if shape else out


def _rng(seed, stream=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) & 0xFFFFFFFF) * 1009 + stream)


class Image:
    """A weights image under construction: offsets first, then the values, made in place."""

    def __init__(self):
        self.size, self.todo = 0, []

    def put(self, dtype, shape, fill):
        """Room for a tensor that ``fill(generator)`` gives; returns its offset."""
        off = -(-self.size // 128) * 128
        self.size = off + math.prod(shape) * torch.empty(0, dtype=dtype).element_size()
        self.todo.append((off, dtype, tuple(shape), fill))
        return off

    def affine(self, rows, cols):
        """An affine u4 matrix: nibbles uniform, scales of a variance-preserving init, biases that centre the nibbles."""
        c = 1.0 / (0.0561 * math.sqrt(cols))
        groups = (rows, cols // GROUP)
        held = {}

        def scales(g):
            held["s"] = ((torch.rand(groups, generator=g, device="cuda") * 0.018 + 0.002) * c).half()
            return held["s"]

        def biases(g):
            return (-7.5 * held.pop("s").float() + (torch.rand(groups, generator=g, device="cuda") * 0.002 - 0.001) * c).half()

        return capi.AffineRef(self.put(torch.uint8, (rows, cols // 2), lambda g: torch.randint(0, 256, (rows, cols // 2), dtype=torch.uint8, device="cuda", generator=g)),
                              self.put(torch.float16, groups, scales), self.put(torch.float16, groups, biases))

    def normal(self, dtype, shape, std, mean=0.0, pad=None):
        """N(mean, std) in the first ``shape`` of a zero-padded ``pad``."""

        def fill(g):
            a = torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(std).add_(mean)
            return a if pad is None else _padded(a, pad)

        return self.put(dtype, pad or shape, fill)

    def make(self, seed):
        """The image on the GPU."""
        out = torch.zeros(-(-self.size // 128) * 128, dtype=torch.uint8, device="cuda")
        g = _rng(seed)
        for off, dtype, shape, fill in self.todo:
            a = fill(g).to(dtype).contiguous()
            out[off:off + a.numel() * a.element_size()] = a.view(torch.uint8).reshape(-1)
        return out


def _padded(a, shape):
    out = torch.zeros(shape, dtype=a.dtype, device=a.device)
    out[tuple(slice(0, n) for n in a.shape)] = a
    return out


def _at(image, off, dtype, *shape):
    return image[off:off + math.prod(shape) * torch.empty(0, dtype=dtype).element_size()].view(dtype).view(*shape)


def _upload(ctx, image):
    ctx.call("alloc_slot", WEIGHTS, C.c_size_t(image.numel()))
    ctx.synchronize()
    _slot(ctx, WEIGHTS, torch.uint8).copy_(image)
    torch.cuda.synchronize()


def _write_table(ctx, build):
    n = C.c_size_t(0)
    build(None, None, C.byref(n))
    table = (capi.DispatchRecord * n.value)()
    ctx._check(build(ctx.h, table, C.byref(n)))
    return table


def _tokens(seed, n, vocab):
    return np.random.default_rng([int(seed) & 0xFFFFFFFF, 5]).integers(0, vocab, n).astype(np.int32)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def _rms(x, eps=EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


# ── one projection ──────────────────────────────────────────────────────────
def _projection_inputs(case, seed):
    """Literal distributions of the kernel benchmarks: scale ~U(0.002, 0.02), bias about -8 scale, activations N(0, 1)."""
    R, K, B, g = case["rows"], case["cols"], case["batch"], _rng(seed)
    out = []
    for _ in range(2 if case["mode"] in ("gate_up", "dual") else 1):
        s = (torch.rand(R, K // GROUP, generator=g, device="cuda") * 0.018 + 0.002).half()
        b = (-8.0 * s.float() + torch.rand(s.shape, generator=g, device="cuda") * 0.002 - 0.001).half()
        out += [torch.randint(0, 256, (R, K // 2), dtype=torch.uint8, device="cuda", generator=g), s, b]
    return out, torch.randn(B, K, generator=g, device="cuda").half(), torch.randn(B, R, generator=g, device="cuda").half()


def _projection_prepare(case, seed):
    w, x, res = _projection_inputs(case, seed)
    ys = [torch.zeros_like(res) for _ in range(2 if case["mode"] == "dual" else 1)]
    name = {"matvec": "affine_matvec", "add": "affine_matvec_add", "gate_up": "affine_gate_up_swiglu", "dual": "affine_dual_matvec"}[case["mode"]]
    tensors = [*w, x, *([res] if case["mode"] == "add" else []), *ys]
    ctx = capi.Context(0)
    return {"ctx": ctx, "name": name, "args": [t.data_ptr() for t in tensors] + [case["rows"], case["cols"], GROUP, case["batch"]], "y": ys, "kept": tensors}


def _projection_run(s):
    s["ctx"].call(s["name"], *s["args"])
    return s["y"]


def _dequant(packed, scales, biases):
    q = torch.stack([packed & 15, packed >> 4], -1).view(packed.shape[0], -1)
    q = q.view(q.shape[0], scales.shape[1], -1).double()
    return (q * scales.double()[..., None] + biases.double()[..., None]).view(packed.shape[0], -1)


def _projection_exact(case, seed):
    w, x, res = _projection_inputs(case, seed)
    ys = [x.double() @ _dequant(*w[i:i + 3]).T for i in range(0, len(w), 3)]
    if case["mode"] == "gate_up":
        ys = [torch.nn.functional.silu(ys[0]) * ys[1]]
    return [ys[0] + res.double()] if case["mode"] == "add" else ys


# ── plain and hybrid affine u4 decoders ─────────────────────────────────────
DELTA_HEADS, DELTA_QK, DELTA_DIM, TAPS = 32, 16, 128, 4


def _plain_image(case):
    """(Image, DecoderDesc, LayerRef array, DeltaRef array, kinds): three DeltaNet layers to one attention layer when hybrid."""
    hybrid = case["kind"] == "hybrid"
    H, L, V = case["width"], case["layers"], case["vocab"]
    I, n_q, n_kv, D = PLAIN.get(H, (3 * H, H // 128, max(1, H // 512), 128))
    qd, kvd, dq, dv = n_q * D, n_kv * D, (2 * DELTA_QK + DELTA_HEADS) * DELTA_DIM, DELTA_HEADS * DELTA_DIM
    img, layers, deltas, kinds = Image(), (capi.LayerRef * L)(), (capi.DeltaRef * L)(), (C.c_uint8 * L)()
    noise = lambda g: ((torch.rand(H, generator=g, device="cuda") * 0.1 - 0.05)).half()  # a norm weight minus one
    for l in range(L):
        ref, d = layers[l], deltas[l]
        kinds[l] = int(hybrid and l % 4 != 3)
        if kinds[l]:
            d.qkv, d.z, d.a, d.b, d.out = img.affine(dq, H), img.affine(dv, H), img.affine(DELTA_HEADS, H), img.affine(DELTA_HEADS, H), img.affine(H, dv)
            d.conv_weight, d.norm_weight = img.normal(torch.float16, (dq, TAPS), 0.5), img.normal(torch.float16, (DELTA_DIM,), 0.1, 1.0)
            d.a_log = img.put(torch.float16, (DELTA_HEADS,), lambda g: torch.rand(DELTA_HEADS, generator=g, device="cuda") * 2.5 - 2.0)
            d.dt_bias = img.put(torch.float16, (DELTA_HEADS,), lambda g: torch.rand(DELTA_HEADS, generator=g, device="cuda") - 0.5)
        else:
            ref.q, ref.k, ref.v, ref.o = img.affine(qd, H), img.affine(kvd, H), img.affine(kvd, H), img.affine(H, qd)
        ref.gate, ref.up, ref.down = img.affine(I, H), img.affine(I, H), img.affine(H, I)
        ref.input_norm, ref.post_norm = img.put(torch.float16, (H,), noise), img.put(torch.float16, (H,), noise)
    desc = capi.DecoderDesc(layers=L, hidden=H, inter=I, n_q=n_q, n_kv=n_kv, head_dim=D, vocab=V, group=GROUP, eps=EPS, rope_theta=THETA,
                            embedding=img.normal(torch.float16, (V, H), 0.02), lm_head=img.normal(torch.float16, (V, H), 0.02),
                            final_norm=img.put(torch.float16, (H,), noise), tp_world=1, tp_rank=0, fuse_residual=3)
    return img, desc, layers, deltas, kinds


def _plain_capacity(case):
    end = case["context"] + 1 if case["kind"] == "decode" else case["tokens"] + case.get("start", 0) + case.get("steps", 0)
    return -(-(end + 16) // 64) * 64  # a user's cache ends a little behind the last position


def _past(case, seed, layer, desc, count, capacity, batch):
    """The cache of one layer as an earlier prompt left it: [batch, heads, capacity, size] with ``count`` positions filled."""
    out = torch.zeros(2, batch, desc.n_kv, capacity, desc.head_dim, dtype=torch.float16, device="cuda")
    out[:, :, :, :count] = torch.randn(2, batch, desc.n_kv, count, desc.head_dim, generator=_rng(seed, 17 + layer), device="cuda", dtype=torch.float16)
    return out


def _edge_layers(L):
    return [0] if L == 1 else [0, L - 1]


def _plain_prepare(case, seed):
    """decode and prefill: weights, cache and a captured graph or a chunk driver."""
    img, desc, layers, _, _ = _plain_image(case)
    B, cap, L = case.get("batch", 1), _plain_capacity(case), case["layers"]
    ctx = capi.Context(0)
    _upload(ctx, img.make(seed))
    table = _write_table(ctx, lambda h, t, n: ctx.lib.smelt_cuda_build_decoder(h, C.byref(desc), layers, cap, B, t, n))
    ctx.synchronize()
    past = case["context"] if case["kind"] == "decode" else case["start"]
    caches = [[_slot(ctx, KV + h * L + l, torch.float16, B, desc.n_kv, cap, desc.head_dim) for h in range(2)] for l in range(L)]
    for l in range(L) if past else ():
        k, v = _past(case, seed, l, desc, past, cap, B)
        caches[l][0].copy_(k)
        caches[l][1].copy_(v)
    torch.cuda.synchronize()
    if case["kind"] == "decode":
        ctx._check(ctx.lib.smelt_cuda_graph_build(ctx.h, table, len(table)))
    ctx.synchronize()
    tokens = _tokens(seed, B if case["kind"] == "decode" else case["tokens"], desc.vocab)
    return {"ctx": ctx, "case": case, "desc": desc, "layers": layers, "table": table, "tokens": tokens, "ids": np.zeros(B, np.int32), "past": past,
            "out": {"logits": _slot(ctx, LOGITS, torch.float16, B, desc.vocab), "caches": [caches[l] for l in _edge_layers(L)]}}


def _plain_run(s):
    ctx = s["ctx"]
    if s["case"]["kind"] == "decode":
        ctx._check(ctx.lib.smelt_cuda_graph_step(ctx.h, _ptr(s["tokens"]), s["past"], _ptr(s["ids"])))
    else:
        ctx._check(ctx.lib.smelt_cuda_prefill(ctx.h, C.byref(s["desc"]), s["layers"], _ptr(s["tokens"]), len(s["tokens"]), s["past"], CHUNK, _ptr(s["ids"])))
    return s["out"]


def _rope(x, positions):
    """x [..., T, D], split halves."""
    h = x.shape[-1] // 2
    a = positions.double()[:, None] * THETA ** (-torch.arange(h, device="cuda").double() / h)
    c, s, u, v = torch.cos(a), torch.sin(a), x[..., :h], x[..., h:]
    return torch.cat([u * c - v * s, u * s + v * c], -1)


def _affine_at(image, ref, rows, cols):
    g = (rows, cols // GROUP)
    return _dequant(_at(image, ref.packed, torch.uint8, rows, cols // 2), _at(image, ref.scales, torch.float16, *g), _at(image, ref.biases, torch.float16, *g))


def _causal(q, k, v, first):
    """q [B, G, r, T, D] at positions first ..; k, v [B, G, S, D]."""
    out = torch.empty_like(q)
    step = max(1, int(2 ** 27 // (q.shape[0] * q.shape[1] * q.shape[2] * k.shape[2])))
    for t in range(0, q.shape[3], step):
        s = torch.einsum("bgrtd,bgsd->bgrts", q[..., t:t + step, :], k) / math.sqrt(q.shape[-1])
        at = first + t + torch.arange(s.shape[3], device="cuda")
        s.masked_fill_(torch.arange(k.shape[2], device="cuda")[None] > at[:, None], -math.inf)
        out[..., t:t + step, :] = torch.einsum("bgrts,bgsd->bgrtd", s.softmax(-1), v)
    return out


def _delta_mixer(image, d, h, H):
    """A DeltaNet block over h [T, H] from a zero state: (output [T, H], taps, recurrent matrices)."""
    T, Hv, Hq, D = len(h), DELTA_HEADS, DELTA_QK, DELTA_DIM
    dq, dv = (2 * Hq + Hv) * D, Hv * D
    x = h @ _affine_at(image, d.qkv, dq, H).T
    z, a, b = h @ _affine_at(image, d.z, dv, H).T, h @ _affine_at(image, d.a, Hv, H).T, h @ _affine_at(image, d.b, Hv, H).T
    past = torch.cat([torch.zeros(TAPS, dq, dtype=torch.float64, device="cuda"), x])
    w = _at(image, d.conv_weight, torch.float16, dq, TAPS).double()
    x = torch.nn.functional.silu(sum(past[1 + i:1 + i + T] * w[:, i] for i in range(TAPS)))
    q, k = _rms(x[:, :Hq * D].view(T, Hq, D)) / D, _rms(x[:, Hq * D:2 * Hq * D].view(T, Hq, D)) / math.sqrt(D)
    q, k, v = q.repeat_interleave(Hv // Hq, 1), k.repeat_interleave(Hv // Hq, 1), x[:, 2 * Hq * D:].view(T, Hv, D)
    beta = torch.sigmoid(b)[..., None]
    decay = torch.exp(-torch.exp(_at(image, d.a_log, torch.float16, Hv).double()) * torch.nn.functional.softplus(a + _at(image, d.dt_bias, torch.float16, Hv).double()))
    S, out = torch.zeros(Hv, D, D, dtype=torch.float64, device="cuda"), torch.empty(T, Hv, D, dtype=torch.float64, device="cuda")
    for t in range(T):  # S [value, key]
        S = S * decay[t][:, None, None]
        delta = (v[t] - torch.einsum("hvk,hk->hv", S, k[t])) * beta[t]
        S = S + delta[:, :, None] * k[t][:, None, :]
        out[t] = torch.einsum("hvk,hk->hv", S, q[t])
    y = _rms(out) * _at(image, d.norm_weight, torch.float16, D).double() * torch.nn.functional.silu(z.view(T, Hv, D))
    return y.reshape(T, dv) @ _affine_at(image, d.out, H, dv).T, past[-TAPS:].T, S


def _plain_exact(case, seed):
    img, desc, layers, deltas, kinds = _plain_image(case)
    image = img.make(seed)
    H, I, D, V, L = desc.hidden, desc.inter, desc.head_dim, desc.vocab, desc.layers
    decode, B = case["kind"] == "decode", case.get("batch", 1)
    T = 1 if decode else case["tokens"] + case.get("steps", 0)
    past, cap = case.get("context", case.get("start", 0)), _plain_capacity(case)
    tokens = torch.from_numpy(_tokens(seed, B if decode else T, V)).cuda().long()
    norm = lambda x, off: _rms(x) * (1.0 + _at(image, off, torch.float16, H).double())
    x = _at(image, desc.embedding, torch.float16, V, H)[tokens].double().view(B, T, H)
    at = past + torch.arange(T, device="cuda")
    caches, states = [], []
    for l in range(L):
        w, h = layers[l], norm(x, layers[l].input_norm)
        if kinds[l]:
            y, taps, S = _delta_mixer(image, deltas[l], h[0], H)
            states.append([taps, S])
            y = y[None]
        else:
            G, r = desc.n_kv, desc.n_q // desc.n_kv
            heads = lambda ref, n: (h.reshape(B * T, H) @ _affine_at(image, ref, n * D, H).T).view(B, T, n, D).transpose(1, 2)
            kv = _past(case, seed, l, desc, past, cap, B)
            q, k, v = _rope(heads(w.q, G * r), at), kv[0].double(), kv[1].double()
            k[:, :, past:past + T], v[:, :, past:past + T] = _rope(heads(w.k, G), at), heads(w.v, G)
            y = _causal(q.reshape(B, G, r, T, D), k[:, :, :past + T], v[:, :, :past + T], past)
            y = y.reshape(B, G * r, T, D).transpose(1, 2).reshape(B, T, G * r * D) @ _affine_at(image, w.o, H, G * r * D).T
            if case["kind"] == "hybrid" or l in _edge_layers(L):
                caches.append([k, v])
            del kv, k, v
        x = x + y
        h = norm(x, w.post_norm)
        x = x + (torch.nn.functional.silu(h @ _affine_at(image, w.gate, I, H).T) * (h @ _affine_at(image, w.up, I, H).T)) @ _affine_at(image, w.down, H, I).T
    last = norm(x[:, -1], desc.final_norm)
    head = _at(image, desc.lm_head, torch.float16, V, H)
    logits = torch.cat([last @ head[i:i + 16384].double().T for i in range(0, V, 16384)], 1)
    out = {"logits": logits, "caches": caches}
    return {**out, "states": states} if case["kind"] == "hybrid" else out


def _hybrid_prepare(case, seed):
    img, desc, layers, deltas, kinds = _plain_image(case)
    cap, L, chunk = _plain_capacity(case), case["layers"], min(CHUNK, case["tokens"])
    dd = capi.DeltaDesc(DELTA_HEADS, DELTA_QK, DELTA_DIM, TAPS)
    ctx = capi.Context(0)
    _upload(ctx, img.make(seed))
    lib, args = ctx.lib, (C.byref(desc), layers, C.byref(dd), deltas, kinds)
    table = _write_table(ctx, lambda h, t, n: lib.smelt_cuda_build_hybrid_decoder(h, *args, cap, t, n))
    prompt = _write_table(ctx, lambda h, t, n: lib.smelt_cuda_build_hybrid_prefill_table(h, *args, chunk, t, n))
    if case["steps"]:
        ctx._check(lib.smelt_cuda_graph_build(ctx.h, table, len(table)))
    ctx.synchronize()
    dq = (2 * DELTA_QK + DELTA_HEADS) * DELTA_DIM
    states = [[_slot(ctx, KV + 2 * L + l, torch.float16, dq, TAPS), _slot(ctx, KV + 3 * L + l, torch.float16, DELTA_HEADS, DELTA_DIM, DELTA_DIM)] for l in range(L) if kinds[l]]
    caches = [[_slot(ctx, KV + h * L + l, torch.float16, 1, desc.n_kv, cap, desc.head_dim) for h in range(2)] for l in range(L) if not kinds[l]]
    return {"ctx": ctx, "case": case, "kept": (img, desc, layers, deltas, kinds, dd), "table": table, "prompt": prompt, "chunk": chunk, "tokens": _tokens(seed, case["tokens"] + case["steps"], desc.vocab),
            "ids": np.zeros(1, np.int32), "clear": [KV + h * L + l for l in range(L) if kinds[l] for h in (2, 3)],
            "out": {"logits": _slot(ctx, LOGITS, torch.float16, 1, desc.vocab), "caches": caches, "states": states}}


def _turn(s, enqueue):
    """A prompt in chunks, its last token's id read back, then decode steps over given tokens."""
    ctx, n, tokens, chunk = s["ctx"], s["case"]["tokens"], s["tokens"], s["chunk"]
    for t0 in range(0, n, chunk):
        enqueue(np.ascontiguousarray(tokens[t0:min(n, t0 + chunk)]), t0, t0 + chunk >= n)
    ctx._check(ctx.lib.smelt_cuda_read_slot(ctx.h, 17, 0, _ptr(s["ids"]), 4))
    for t in range(n, n + s["case"]["steps"]):
        ctx._check(ctx.lib.smelt_cuda_graph_step(ctx.h, _ptr(tokens[t:t + 1]), t, _ptr(s["ids"])))
    return s["out"]


def _hybrid_run(s):
    ctx = s["ctx"]
    for slot in s["clear"]:  # a new sequence: the DeltaNet layers' taps and matrices start at zero
        ctx.call("zero_slot", slot)
    return _turn(s, lambda part, at, last: ctx._check(ctx.lib.smelt_cuda_enqueue_prefill(ctx.h, s["prompt"], len(s["prompt"]), _ptr(part), len(part), at)))


# ── low-bit feed-forward halves ─────────────────────────────────────────────
def _lowbit_inputs(case, seed):
    H, I, g = case["width"], case["ff"], _rng(seed)

    def weights(rows, cols):
        if case["format"] == 1:
            codes = torch.randint(0, 256, (rows, cols // 8), dtype=torch.uint8, device="cuda", generator=g)
        else:
            c = torch.bucketize(torch.rand(rows, cols, generator=g, device="cuda"), torch.tensor([0.335, 0.665], device="cuda")).to(torch.uint8).view(rows, -1, 4)
            codes = c[..., 0] | c[..., 1] << 2 | c[..., 2] << 4 | c[..., 3] << 6
        scales = (torch.rand(rows, cols // 128, generator=g, device="cuda") * 0.025 + 0.005) * (0.8 / (0.0187 * math.sqrt(cols)))
        return [codes.contiguous(), scales.half()]

    layers = [(weights(I, H), weights(I, H), weights(H, I)) for _ in range(case["layers"])]
    return layers, torch.randn(case["batch"], H, generator=g, device="cuda").half()


def _lowbit_prepare(case, seed):
    layers, x = _lowbit_inputs(case, seed)
    B, H, I, f = case["batch"], case["width"], case["ff"], case["format"]
    inner, ys = torch.empty(B, I, dtype=torch.float16, device="cuda"), [torch.empty_like(x) for _ in layers]
    calls = []
    for (gate, up, down), src, dst in zip(layers, [x, *ys], ys):
        p = lambda *ts: [t.data_ptr() for t in ts]
        calls.append(("signed_gate_up_swiglu", [f, *p(*gate, *up, src, inner), I, H, B]))
        calls.append(("signed_matvec_add", [f, *p(*down, inner, src, dst), H, I, B]))
    return {"ctx": capi.Context(0), "calls": calls, "kept": (layers, x, inner), "ys": ys}


def _lowbit_run(s):
    ctx = s["ctx"]
    for name, args in s["calls"]:
        ctx.call(name, *args)
    return s["ys"]


def _lowbit_exact(case, seed):
    layers, x = _lowbit_inputs(case, seed)
    bits = case["format"]

    def dequant(codes, scales):
        c = torch.stack([codes >> s & (1 if bits == 1 else 3) for s in range(0, 8, bits)], -1).view(codes.shape[0], scales.shape[1], 128).double()
        return ((c * 2 - 1 if bits == 1 else c - 1) * scales.double()[..., None]).view(codes.shape[0], -1)

    out, x = [], x.double()
    for gate, up, down in layers:
        x = x + (torch.nn.functional.silu(x @ dequant(*gate).T) * (x @ dequant(*up).T)) @ dequant(*down).T
        out.append(x)
    return out


# ── Pesedra ─────────────────────────────────────────────────────────────────
P_LAYERS, P_LOOP, VOCAB = 5, (1, 4, 2), 32768
CAP, RISING, FALLING = 20.0, math.log1p(math.exp(0.3)), 0.5 + math.log1p(math.exp(-0.2))


def _runs():
    a, b, n = P_LOOP
    return [(l, False) for l in range(a)] + [(l, l == a) for l in range(a, b)] * n + [(l, False) for l in range(b, P_LAYERS)]


def _pesedra_image(case):
    W = case["width"]
    ff, H, G, D = PLAIN[W]
    qkv, img, layers = (H + 2 * G) * D, Image(), (capi.DenseLayer * P_LAYERS)()
    bf = torch.bfloat16
    for i in range(P_LAYERS):
        w = layers[i]
        w.heads, w.kv_heads, w.dim, w.vdim, w.window, w.pool, w.ff = H, G, D, D, WINDOW, POOL, ff
        w.scale, w.softcap, w.norm_gain, w.act_rising, w.act_falling = D ** -0.5, CAP, 0.9 + 0.05 * i, RISING, FALLING
        w.in_proj, w.out_proj = img.normal(bf, (qkv + ff, W), W ** -0.5), img.normal(bf, (W, H * D + ff), 0.5 * (H * D + ff) ** -0.5)
        w.q_norm, w.k_norm = img.normal(bf, (D,), 0.3, 1.0), img.normal(bf, (D,), 0.3, 1.0)
    end = case["tokens"] + case["steps"] + 16
    desc = capi.DenseDesc(layers=P_LAYERS, width=W, vocab=VOCAB, precision={"bfloat16": 0, "float32": 1}[case["precision"]], max_positions=end, loop_start=P_LOOP[0], loop_stop=P_LOOP[1],
                          loop_times=P_LOOP[2], eps=EPS, embedding_scale=1.0, final_gain=1.0, embedding=img.normal(bf, (VOCAB, W), 1.0), positions=img.normal(bf, (end, W), 1.0),
                          loop_in=img.normal(bf, (W, 2 * W), (2 * W) ** -0.5), lm_head=img.normal(bf, (VOCAB, W), W ** -0.5))
    return img, desc, layers


def _dense_prepare(case, seed):
    """pesedra and kesedra: weights, both tables, a graph when there are steps."""
    stack = case["kind"] == "kesedra"
    img, desc, layers = (_kesedra_image if stack else _pesedra_image)(case)
    ctx = capi.Context(0)
    _upload(ctx, img.make(seed))
    lib, cap = ctx.lib, case["tokens"] + case["steps"] + 16
    chunk = min(CHUNK, cap)
    names = ("smelt_cuda_build_stack_decoder", "smelt_cuda_build_stack_prefill_table") if stack else ("smelt_cuda_build_dense_decoder", "smelt_cuda_build_dense_prefill_table")
    table, prompt = (_write_table(ctx, lambda h, t, n, fn=getattr(lib, name): fn(h, C.byref(desc), layers, cap, chunk, t, n)) for name in names)
    if case["steps"]:
        ctx._check(lib.smelt_cuda_graph_build(ctx.h, table, len(table)))
    ctx.synchronize()
    kind = torch.bfloat16 if case["precision"] == "bfloat16" else torch.float32
    n_slots = 2 * len(_runs())
    if stack:
        dtypes = [t for l in layers for t in ([torch.float32] * 2 if l.mixer == capi.MIXER_WKV else [kind] * 2 if l.kv_from < 0 else [])]
    else:
        dtypes = [kind] * n_slots
    return {"ctx": ctx, "case": case, "kept": (img, desc, layers), "table": table, "prompt": prompt, "chunk": chunk, "tokens": _tokens(seed, case["tokens"] + case["steps"], VOCAB),
            "ids": np.zeros(1, np.int32), "out": {"logits": _slot(ctx, LOGITS, torch.float32, 1, VOCAB), "state": [_slot(ctx, KV + i, t) for i, t in enumerate(dtypes)]}}


def _dense_run(s):
    ctx = s["ctx"]

    def enqueue(part, at, last):
        rows = np.array([len(part) - 1] if last else [], np.int32)
        ctx._check(ctx.lib.smelt_cuda_enqueue_prefill_rows(ctx.h, s["prompt"], len(s["prompt"]), _ptr(part), len(part), at, _ptr(rows), len(rows)))

    return _turn(s, enqueue)


def _pesedra_exact(case, seed):
    img, desc, layers = _pesedra_image(case)
    image, W, T, bf = img.make(seed), case["width"], case["tokens"] + case["steps"], torch.bfloat16
    ff, H, G, D = PLAIN[W]
    tokens = torch.from_numpy(_tokens(seed, T, VOCAB)).cuda().long()
    x = x0 = _at(image, desc.embedding, bf, VOCAB, W)[tokens].double() + _at(image, desc.positions, bf, desc.max_positions, W)[:T].double()
    i, j, b = (torch.arange(n, device="cuda") for n in (T, T, T // POOL))
    seen = torch.cat([(j[None] <= i[:, None]) & (j[None] > i[:, None] - WINDOW), b[None] * POOL + POOL - 1 <= i[:, None] - WINDOW], 1)
    for l, begins in _runs():
        w = layers[l]
        if begins:
            x = torch.cat([x, x0], 1) @ _at(image, desc.loop_in, bf, W, 2 * W).double().T
        h = _rms(x) * w.norm_gain
        u = h @ _at(image, w.in_proj, bf, (H + 2 * G) * D + ff, W).double().T
        q, k, v, up = u.split([H * D, G * D, G * D, ff], 1)
        q = _rms(q.view(T, H, D)) * _at(image, w.q_norm, bf, D).double()
        k, v = _rms(k.view(T, G, D)) * _at(image, w.k_norm, bf, D).double(), v.view(T, G, D)
        means = lambda a: torch.cat([a, a[:len(b) * POOL].view(len(b), POOL, G, D).mean(1)])
        k, v, out = means(k), means(v), []
        for g in range(G):
            s = torch.einsum("trd,sd->rts", q[:, g * (H // G):(g + 1) * (H // G)], k[:, g]) * w.scale
            s = (CAP * torch.tanh(s / CAP)).masked_fill(~seen, -math.inf)
            m = s.amax(-1, keepdim=True).clamp(min=0.0)
            e = torch.exp(s - m)
            out.append(torch.einsum("rts,sd->trd", e / (torch.exp(-m) + e.sum(-1, keepdim=True)), v[:, g]))
        neg = up.clamp(max=0.0)
        act = torch.where(up > 0, w.act_rising * up * up, w.act_falling * (torch.expm1(neg) - neg)) + up / 2
        x = x + torch.cat([torch.cat(out, 1).reshape(T, H * D), act], 1) @ _at(image, w.out_proj, bf, W, H * D + ff).double().T
    return {"logits": _rms(x[-1:]) @ _at(image, desc.lm_head, bf, VOCAB, W).double().T, "state": [None] * (2 * len(_runs()))}


# ── Kesedra ─────────────────────────────────────────────────────────────────
def _up(n, k):
    return -(-n // k) * k


def _router_draw(seed):
    """Weights of the features for the 16 experts, and the sign patterns whose choice of four is clear."""
    g = np.random.default_rng([int(seed) & 0xFFFFFFFF, 9])
    signs = np.array([[1.0 if p >> f & 1 else -1.0 for f in range(FEATURES)] for p in range(1 << FEATURES)])
    w = g.standard_normal((EXPERTS, FEATURES)).astype(np.float32)
    w = torch.from_numpy(w).bfloat16().float().numpy()
    z = np.sort(signs @ w.T, 1)[:, ::-1]
    return w, signs[np.argsort(z[:, TOP] - z[:, TOP - 1], kind="stable")[:32]]


def _kesedra_image(case):
    W, img, bf, layers = case["width"], Image(), torch.bfloat16, (capi.StackLayer * 8)()
    ff, H, Q, rank, xf = STACK[W]
    D, n = 128, W
    norm = lambda after=False: img.put(bf, (W,), lambda g: _features(0.3 * torch.randn(W, generator=g, device="cuda"), -1.0 if after else 0.0))
    for i in range(8):
        w = layers[i]
        w.norm1, w.norm1b, w.norm2, w.norm2b, w.kv_from = norm(), norm(True), norm(), norm(True), -1
        if i % 4 < 2:
            w.mixer, w.heads, w.dim, w.rot_dim, w.rot_dims, w.vdim, w.kv_rank, w.q_rank, w.window, w.scale = capi.MIXER_LATENT, H, D, ROT, ROT, D, LATENT, Q, WINDOW, (D + ROT) ** -0.5
            if i % 4:
                w.kv_from = i - 1
            w.in_proj = img.normal(bf, (Q + (0 if i % 4 else LATENT + ROT), W), W ** -0.5)
            w.q_norm, w.kv_norm = img.normal(bf, (Q,), 0.3, 1.0), img.normal(bf, (LATENT,), 0.3, 1.0)
            w.q_proj = img.normal(bf, (H * (D + ROT), Q), Q ** -0.5)
            w.kv_proj, w.out_proj = img.normal(bf, (2 * H * D, LATENT), LATENT ** -0.5), img.normal(bf, (W, H * D), (H * D) ** -0.5)
            w.rot_freq = img.put(torch.float64, (ROT // 2,), lambda g: 10000.0 ** (-torch.arange(ROT // 2, device="cuda").double() * 2 / ROT))
        else:
            w.mixer, w.heads, w.dim, w.rank = capi.MIXER_WKV, W // WKV_DIM, WKV_DIM, rank
            w.in_proj = img.normal(bf, (4 * n + rank, W), W ** -0.5, pad=(4 * n + _up(rank, 64), W))
            w.mu = img.put(bf, (5, W), lambda g: torch.rand(5, W, generator=g, device="cuda"))
            w.w2 = img.normal(bf, (n, rank), rank ** -0.5, pad=(n, _up(rank, 64)))
            w.w0 = img.put(bf, (n,), lambda g: torch.rand(n, generator=g, device="cuda") * 4.5 - 4.0)
            w.bonus, w.head_norm, w.out_proj = img.normal(bf, (n,), 1.0), img.normal(bf, (n,), 0.3, 1.0), img.normal(bf, (W, n), n ** -0.5)
        w.ff_kind = capi.FF_EXPERTS if i % 2 else capi.FF_DENSE
        if i % 2:
            w.experts, w.top, w.limit, w.ff = EXPERTS, TOP, LIMIT, xf
            w.router = img.put(bf, (EXPERTS, W), lambda g: _router(case, g))
            w.router_bias = img.put(bf, (EXPERTS,), lambda g: torch.zeros(EXPERTS, device="cuda"))
            w.up, w.down = img.normal(bf, (EXPERTS, 2 * xf, W), W ** -0.5), img.normal(bf, (EXPERTS, W, xf), xf ** -0.5)
        else:
            w.ff = ff
            w.up, w.up_bias, w.down, w.down_bias = img.normal(bf, (ff, W), W ** -0.5), img.normal(bf, (ff,), 0.5), img.normal(bf, (W, ff), ff ** -0.5), img.normal(bf, (W,), 0.5)
    desc = capi.StackDesc(layers=8, width=W, vocab=VOCAB, precision={"bfloat16": 0, "float32": 1}[case["precision"]], eps=EPS, embedding_scale=1.0,
                          embedding=img.put(bf, (VOCAB, W), lambda g: _embedding(g, W)), lm_head=img.normal(bf, (VOCAB, W), W ** -0.5), final_norm=norm())
    return img, desc, layers


def _features(a, value):
    a[..., :FEATURES] = value
    return a


def _router(case, g):
    """A router that reads the features alone (the rest a little): a choice of experts is never a close one, and differs from token to token."""
    w, _ = _router_draw(int(g.initial_seed()))
    out = torch.randn(EXPERTS, case["width"], generator=g, device="cuda") * (0.02 * case["width"] ** -0.5)
    out[:, :FEATURES] = torch.from_numpy(w).cuda()
    return out


def _embedding(g, width):
    _, signs = _router_draw(int(g.initial_seed()))
    out = torch.randn(VOCAB, width, generator=g, device="cuda")
    pick = torch.randint(0, len(signs), (VOCAB,), generator=g, device="cuda")
    out[:, :FEATURES] = 3.0 * torch.from_numpy(signs).float().cuda()[pick]
    return out


def _kesedra_exact(case, seed):
    img, desc, layers = _kesedra_image(case)
    image, W, T, bf = img.make(seed), case["width"], case["tokens"] + case["steps"], torch.bfloat16
    ff, H, Q, rank, xf = STACK[W]
    D, get = 128, lambda off, *shape: _at(image, off, bf, *shape).double()
    norm = lambda x, off: _rms(x) * (1.0 + get(off, W))
    x = get(desc.embedding, VOCAB, W)[torch.from_numpy(_tokens(seed, T, VOCAB)).cuda().long()]
    i = torch.arange(T, device="cuda")
    seen = (i[None] <= i[:, None]) & (i[None] > i[:, None] - WINDOW)
    angle = i.double()[:, None] * 10000.0 ** (-torch.arange(ROT // 2, device="cuda").double() * 2 / ROT)

    def rotate(a):  # adjacent pairs of the last axis, positions first
        c, s = (f(angle).view(T, *[1] * (a.dim() - 2), ROT // 2) for f in (torch.cos, torch.sin))
        u, v = a[..., 0::2], a[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

    cache = {}
    for l in range(8):
        w, h = layers[l], norm(x, layers[l].norm1)
        if w.mixer == capi.MIXER_LATENT:
            u = h @ get(w.in_proj, Q + (LATENT + ROT if w.kv_from < 0 else 0), W).T
            q = (_rms(u[:, :Q]) * get(w.q_norm, Q) @ get(w.q_proj, H * (D + ROT), Q).T).view(T, H, D + ROT)
            if w.kv_from < 0:
                cache[l] = (_rms(u[:, Q:Q + LATENT]) * get(w.kv_norm, LATENT), rotate(u[:, Q + LATENT:]))
            c, kr = cache[l if w.kv_from < 0 else w.kv_from]
            k, v = (c @ get(w.kv_proj, 2 * H * D, LATENT).T).view(T, 2, H, D).unbind(1)
            s = (torch.einsum("thd,shd->hts", q[..., :D], k) + torch.einsum("thd,sd->hts", rotate(q[..., D:]), kr)) * w.scale
            y = torch.einsum("hts,shd->thd", s.masked_fill(~seen, -math.inf).softmax(-1), v).reshape(T, H * D)
        else:
            n, Hw = W, W // WKV_DIM
            mix = h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * get(w.mu, 5, W)[:, None]
            p = get(w.in_proj, 4 * n + _up(rank, 64), W)
            r, k, v, gate = ((mix[s] @ p[s * n:(s + 1) * n].T).view(T, Hw, WKV_DIM) for s in range(4))
            inner = torch.tanh(mix[4] @ p[4 * n:].T)
            decay = torch.exp(-torch.exp(inner @ get(w.w2, n, _up(rank, 64)).T + get(w.w0, n))).view(T, Hw, WKV_DIM)
            bonus, S, out = get(w.bonus, Hw, WKV_DIM)[..., None], torch.zeros(Hw, WKV_DIM, WKV_DIM, dtype=torch.float64, device="cuda"), []
            for t in range(T):  # S [key, value]
                now = k[t][..., None] * v[t][:, None]
                out.append(torch.einsum("hkv,hk->hv", S + bonus * now, r[t]))
                S = decay[t][..., None] * S + now
            y = (_rms(torch.stack(out)) * get(w.head_norm, Hw, WKV_DIM) * torch.nn.functional.silu(gate)).reshape(T, n)
        x = x + norm(y @ get(w.out_proj, W, y.shape[1]).T, w.norm1b)
        h = norm(x, w.norm2)
        if w.ff_kind == capi.FF_DENSE:
            y = (h @ get(w.up, ff, W).T + get(w.up_bias, ff)).clamp(min=0.0).square() @ get(w.down, W, ff).T + get(w.down_bias, W)
        else:
            z, chosen = (h @ get(w.router, EXPERTS, W).T).topk(TOP, 1)
            weight, y = z.softmax(1), torch.zeros_like(x)
            for e in range(EXPERTS):
                t, slot = (chosen == e).nonzero(as_tuple=True)
                u = (h[t] @ get(w.up + e * 2 * xf * W * 2, 2 * xf, W).T).view(-1, xf, 2)
                g, lin = u[..., 0].clamp(max=LIMIT), u[..., 1].clamp(-LIMIT, LIMIT)
                y.index_add_(0, t, weight[t, slot][:, None] * ((g * torch.sigmoid(1.702 * g) * (lin + 1.0)) @ get(w.down + e * W * xf * 2, W, xf).T))
        x = x + norm(y, w.norm2b)
    slots = sum(2 for l in layers if l.mixer == capi.MIXER_WKV or l.kv_from < 0)
    return {"logits": norm(x[-1:], desc.final_norm) @ get(desc.lm_head, VOCAB, W).T, "state": [None] * slots}


# ── the interface ───────────────────────────────────────────────────────────
_PREPARE = {"projection": _projection_prepare, "decode": _plain_prepare, "prefill": _plain_prepare, "lowbit": _lowbit_prepare, "hybrid": _hybrid_prepare, "pesedra": _dense_prepare,
            "kesedra": _dense_prepare}
_RUN = {"projection": _projection_run, "decode": _plain_run, "prefill": _plain_run, "lowbit": _lowbit_run, "hybrid": _hybrid_run, "pesedra": _dense_run, "kesedra": _dense_run}
_EXACT = {"projection": _projection_exact, "decode": _plain_exact, "prefill": _plain_exact, "lowbit": _lowbit_exact, "hybrid": _plain_exact, "pesedra": _pesedra_exact,
          "kesedra": _kesedra_exact}


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def work(case):
    """Weights, live cache and activations once; multiply-adds of the contractions twice."""
    kind, B = case["kind"], case.get("batch", 1)
    if kind == "projection":
        R, K = case["rows"], case["cols"]
        mats, outs = (2 if case["mode"] in ("gate_up", "dual") else 1), (2 if case["mode"] == "dual" else 1)
        return {"bytes": mats * R * K * 0.5625 + 2 * B * (K + R * (outs + (case["mode"] == "add"))), "flops": 2 * mats * R * K * B}
    if kind == "lowbit":
        n = case["layers"] * 3 * case["width"] * case["ff"]
        return {"bytes": n * (case["format"] / 8 + 2 / 128) + 2 * B * case["width"] * (1 + case["layers"]), "flops": 2 * n * B}
    W = case["width"]
    if kind in ("decode", "prefill", "hybrid"):
        I, n_q, n_kv, D = PLAIN.get(W, (3 * W, W // 128, max(1, W // 512), 128))
        L, V = case["layers"], case["vocab"]
        delta = L * 3 // 4 if kind == "hybrid" else 0
        attn = L - delta
        per = 2 * (n_q + n_kv) * D * W
        dper = ((2 * DELTA_QK + 3 * DELTA_HEADS) * DELTA_DIM + 2 * DELTA_HEADS) * W
        weights = attn * per + delta * dper + L * 3 * I * W
        past = case.get("context", case.get("start", 0))
        prompt, steps = (0, 1) if kind == "decode" else (case["tokens"], case.get("steps", 0))
        rows = B * (prompt + steps)
        seen = B * sum(past + t + 1 for t in range(prompt + steps))
        passes = steps + (-(-prompt // CHUNK))
        heads = steps + (1 if prompt else 0)
        kv = attn * 2 * n_kv * D * 2
        reads = B * (sum(past + prompt + t + 1 for t in range(steps)) + (past + prompt if prompt else 0))
        state = delta * passes * 2 * DELTA_HEADS * DELTA_DIM ** 2 * 2
        return {"bytes": passes * weights * 0.5625 + heads * V * W * 2 + kv * reads + rows * W * 2 + heads * B * V * 2 + state,
                "flops": 2 * rows * weights + 2 * heads * B * V * W + 4 * attn * n_q * D * seen + 6 * delta * rows * DELTA_HEADS * DELTA_DIM ** 2}
    T, steps = case["tokens"], case["steps"]
    passes, rows, es = steps + -(-T // CHUNK), T + steps, 2 if case["precision"] == "bfloat16" else 4
    if kind == "pesedra":
        ff, H, G, D = PLAIN[W]
        n = len(_runs())
        weights = n * ((2 * H + 2 * G) * D + 2 * ff) * W + P_LOOP[2] * 2 * W * W
        keys = [min(t + 1, WINDOW) + max(0, (t + 1 - WINDOW) // POOL) for t in range(rows)]
        return {"bytes": passes * weights * 2 + (steps + 1) * VOCAB * W * 2 + n * 2 * G * D * es * (sum(keys[T:]) + sum(keys[min(T, t0 + CHUNK) - 1] for t0 in range(0, T, CHUNK))),
                "flops": 2 * rows * weights + 2 * (steps + 1) * VOCAB * W + 4 * n * H * D * sum(keys)}
    ff, H, Q, rank, xf = STACK[W]
    D = 128
    latent = 4 * (Q * W + H * (D + ROT) * Q + 2 * H * D * LATENT + W * H * D) + 2 * (LATENT + ROT) * W
    wkv, dense, expert = 4 * (5 * W * W + 2 * rank * W), 4 * 2 * ff * W, 3 * xf * W
    keys = [min(t + 1, WINDOW) for t in range(rows)]
    chunks = [min(CHUNK, T - t0) for t0 in range(0, T, CHUNK)]
    touched = sum(min(EXPERTS, c * TOP) for c in chunks) + steps * TOP
    return {"bytes": 2 * (passes * (latent + wkv + dense + 4 * EXPERTS * W) + 4 * touched * expert + (steps + 1) * VOCAB * W)
            + 4 * (LATENT + ROT) * es * (sum(keys[T:]) + sum(keys[min(T, t0 + CHUNK) - 1] for t0 in range(0, T, CHUNK))) + passes * 4 * 2 * W * WKV_DIM * 4,
            "flops": 2 * rows * (latent + wkv + dense + 4 * TOP * expert) + 2 * (steps + 1) * VOCAB * W + 4 * 2 * H * (2 * D + ROT) * sum(keys) + 4 * 6 * rows * W * WKV_DIM}


def tolerance(case):
    """About four times the distance from ``exact`` that was measured: rounding to fp16 (bf16) at the end of each step,
    carried through the layers."""
    if case.get("precision") == "float32":
        return {"rel": 2e-3}
    return {"rel": {"projection": 1e-3, "decode": 2.5e-2, "prefill": 2.5e-2, "lowbit": 4e-3, "hybrid": 5e-2, "pesedra": 1.5e-2, "kesedra": 4e-2}[case["kind"]]}
