"""The work that users of this framework have it do, as cases that can be timed and checked: single linears over packed
weights, attention over a cache, and whole decoders that read prompts and answer them. All sizes come from the repository's
own configurations and benchmark (Llama-7B shape, the 2B shapes of the Tivazen and Fomalix designs, the linears of the 7B
feed-forward); `draw` gives others of the same ranges.

A linear, an attention and a cache case runs over several weights or caches, as the layers of a decoder do, so that what is
read comes from HBM and not from L2. Weights are normal and packed here with torch; every input follows from the seed."""
from __future__ import annotations

import math

import numpy as np
import torch

from skainet_b200 import device
from skainet_b200.device import Weight

BLOCK = {"Q8_0": (32, 34), "Q4_K": (256, 144), "Q5_K": (256, 176), "Q6_K": (256, 210)}   # elements, bytes
F64 = torch.float64
EPS = 1e-5


def listed():
    llama = {"path": "llama", "layers": 32, "width": 4096, "heads": 32, "kv_heads": 32, "ff": 11008, "vocab": 32000}
    small = {"layers": 24, "width": 2048, "heads": 16, "ff": 5632, "vocab": 32000, "batch": 1, "prompt": 2048, "steps": 0}
    return [
        # one token through the smallest matrices in use: launches and latency count
        {"name": "matvec_q8_0", "path": "linear", "enc": "Q8_0", "rows": 4096, "cols": 4096, "m": 1, "weights": 8},
        # one token through the feed-forward of a 7B model: decoding on one sequence
        {"name": "matvec_q4k", "path": "linear", "enc": "Q4_K", "rows": 11008, "cols": 4096, "m": 1, "weights": 8},
        # 64 sequences in one decode step, or a short prompt
        {"name": "rows64_q4k", "path": "linear", "enc": "Q4_K", "rows": 4096, "cols": 11008, "m": 64, "weights": 4},
        # a prompt's 512 rows
        {"name": "rows512_q4k", "path": "linear", "enc": "Q4_K", "rows": 11008, "cols": 4096, "m": 512, "weights": 2},
        # the down projection of a Q4_K_M file, a ragged handful of rows
        {"name": "rows37_q6k", "path": "linear", "enc": "Q6_K", "rows": 4096, "cols": 11008, "m": 37, "weights": 4},
        # one decode step of 16 sequences over 4096 keys
        {"name": "attn_b16_4096", "path": "attention", "batch": 16, "heads": 32, "kv_heads": 8, "dim": 128, "context": 4096, "caches": 2},
        # the compressed cache, one step over 4096 positions
        {"name": "turboquant_4096", "path": "turboquant", "heads": 8, "kv_heads": 8, "dim": 128, "context": 4096, "bits": 4, "layers": 8},
        # one user's request: a prompt, then an answer token by token
        {"name": "llama_request_b1", **llama, "batch": 1, "prompt": 128, "steps": 32},
        # eight users at once
        {"name": "llama_request_b8", **llama, "batch": 8, "prompt": 64, "steps": 32},
        # a long prompt
        {"name": "llama_prompt_512", **llama, "batch": 1, "prompt": 512, "steps": 0},
        {"name": "tivazen_prompt_2048", "path": "tivazen", "kv_heads": 1, **small},
        {"name": "fomalix_prompt_2048", "path": "fomalix", "kv_heads": 4, **small},
    ]


def _spread(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    path = rng.choice(["linear", "linear", "linear", "attention", "turboquant", "llama", "llama", "tivazen", "fomalix"])
    if path == "linear":
        enc = rng.choice(["Q8_0", "Q4_K", "Q4_K", "Q4_K", "Q5_K", "Q6_K"])
        rows, cols = _spread(rng, 512, 22016), 256 * _spread(rng, 4, 48)
        m = rng.choice([1, 1, _spread(rng, 2, 1024), _spread(rng, 2, 1024)])
        m = max(1, min(m, 512 * 11008 * 4096 // (rows * cols)))
        return {"path": path, "enc": enc, "rows": rows, "cols": cols, "m": m, "weights": max(1, min(8, 200_000_000 // (rows * cols), 2 * 512 * 11008 * 4096 // (rows * cols * m)))}
    if path == "attention":
        kv, batch, dim = rng.choice([1, 2, 4, 8]), _spread(rng, 1, 64), rng.choice([64, 128])
        return {"path": path, "batch": batch, "heads": kv * rng.choice([1, 4, 8]), "kv_heads": kv, "dim": dim,
                "context": max(64, min(_spread(rng, 64, 32768), 2 ** 26 // (batch * kv * dim))), "caches": 2}
    if path == "turboquant":
        kv = rng.choice([2, 4, 8])
        return {"path": path, "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv, "dim": rng.choice([64, 128]), "context": _spread(rng, 64, 4096),
                "bits": rng.choice([2, 3, 4, 4, 8]), "layers": rng.choice([4, 8])}
    if path == "llama":
        width = rng.choice([1024, 2048, 4096])
        heads = width // 128
        batch = rng.choice([1, 1, 2, 4, 8])
        return {"path": path, "layers": rng.randint(2, 12), "width": width, "heads": heads, "kv_heads": heads // rng.choice([1, 2, 4]), "ff": 256 * rng.randint(8, 43),
                "vocab": rng.randint(2000, 32000), "batch": batch, "prompt": _spread(rng, 1, 512 // batch), "steps": rng.choice([0, 8, 32])}
    width = rng.choice([1024, 2048])
    steps = rng.choice([0, 0, 16])
    return {"path": path, "layers": 4 * rng.randint(1, 4), "width": width, "heads": width // 128, "kv_heads": 1 if path == "tivazen" else rng.choice([2, 4]), "ff": 128 * rng.randint(16, 44),
            "vocab": rng.randint(2000, 32000), "batch": 1, "prompt": _spread(rng, 1, 2048), "steps": steps}


# ---- packing: normal matrices in the blocks of GGUF files, on the device ------------------------------------------------------

def _cuda() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed, *what):
    """A generator of its own for each tensor, so that one can be made again without the others."""
    h = seed % (2 ** 31)
    for w in what:
        h = (h * 1000003 + w + 1) % (2 ** 61 - 1)
    return torch.Generator(_cuda()).manual_seed(h)


def _normal(shape, std, seed, *what):
    return torch.randn(shape, device=_cuda(), generator=_generator(seed, *what)) * std


def _halves(v):
    return v.to(torch.float16).contiguous().view(torch.uint8)


def _scaled(w, low, high, d):
    """round(w / d) within [low, high]; 0 where d is 0."""
    return torch.where(d > 0, torch.round(w / torch.where(d > 0, d, torch.ones_like(d))), torch.zeros_like(w)).clamp_(low, high)


def _six_bits(sc, mn):
    """Eight scales and eight minimums of six bits in twelve bytes."""
    lo = torch.cat([sc[..., :4] | ((sc[..., 4:] >> 4) << 6), mn[..., :4] | ((mn[..., 4:] >> 4) << 6)], -1)
    return torch.cat([lo, (sc[..., 4:] & 15) | ((mn[..., 4:] & 15) << 4)], -1)


def _k_codes(w, bits):
    """(d, dmin, scales, minimums, codes) of a matrix in super-blocks of eight times 32."""
    top = 2 ** bits - 1
    low, high = w.amin(-1).clamp_(max=0), w.amax(-1)
    step, off = (high - low) / top, -low
    d, dmin = (v.amax(-1, keepdim=True).div(63).half().float() for v in (step, off))
    sc, mn = _scaled(step, 0, 63, d), _scaled(off, 0, 63, dmin)
    codes = _scaled(w + (dmin * mn)[..., None], 0, top, (d * sc)[..., None])
    return d, dmin, sc.to(torch.uint8), mn.to(torch.uint8), codes.to(torch.uint8)


def _pack(w, enc):
    """The row-major blocks of a float matrix, [rows, bytes] uint8."""
    rows = w.shape[0]
    if enc == "Q8_0":
        b = w.view(rows, -1, 32)
        d = b.abs().amax(-1, keepdim=True).div(127).half().float()
        return torch.cat([_halves(d), _scaled(b, -127, 127, d).to(torch.int8).view(torch.uint8)], -1).view(rows, -1)
    if enc == "Q6_K":
        b = w.view(rows, -1, 16, 16)
        step = b.abs().amax(-1) / 31
        d = step.amax(-1, keepdim=True).div(127).half().float()
        sc = _scaled(step, 0, 127, d)
        q = (_scaled(b, -32, 31, (d * sc)[..., None]) + 32).to(torch.uint8).view(rows, -1, 2, 4, 32)
        ql = torch.stack([(q[..., 0, :] & 15) | ((q[..., 2, :] & 15) << 4), (q[..., 1, :] & 15) | ((q[..., 3, :] & 15) << 4)], -2)
        qh = (q[..., 0, :] >> 4) | ((q[..., 1, :] >> 4) << 2) | ((q[..., 2, :] >> 4) << 4) | ((q[..., 3, :] >> 4) << 6)
        return torch.cat([ql.reshape(rows, -1, 128), qh.reshape(rows, -1, 64), sc.to(torch.uint8), _halves(d)], -1).view(rows, -1)
    d, dmin, sc, mn, q = _k_codes(w.view(rows, -1, 8, 32), 4 if enc == "Q4_K" else 5)
    pairs = q.view(rows, -1, 4, 2, 32)
    qs = ((pairs[..., 0, :] & 15) | ((pairs[..., 1, :] & 15) << 4)).reshape(rows, -1, 128)
    head = torch.cat([_halves(d), _halves(dmin), _six_bits(sc, mn)], -1)
    if enc == "Q4_K":
        return torch.cat([head, qs], -1).view(rows, -1)
    qh = sum(((q[..., j, :] >> 4) << j) for j in range(8)).to(torch.uint8)
    return torch.cat([head, qh, qs], -1).view(rows, -1)


def _unpack(p, enc):
    """The matrix that packed blocks stand for, in 64 bits."""
    rows, (n, nbytes) = p.shape[0], BLOCK[enc]
    b = p.view(rows, -1, nbytes)
    half = lambda at: b[..., at:at + 2].contiguous().view(torch.float16).to(F64)  # noqa: E731
    if enc == "Q8_0":
        return (half(0) * b[..., 2:].contiguous().view(torch.int8).to(F64)).view(rows, -1)
    if enc == "Q6_K":
        ql, qh = b[..., :128].view(rows, -1, 2, 2, 32), b[..., 128:192].view(rows, -1, 2, 32)
        q = torch.stack([(ql[..., 0, :] & 15) | ((qh & 3) << 4), (ql[..., 1, :] & 15) | (((qh >> 2) & 3) << 4), (ql[..., 0, :] >> 4) | (((qh >> 4) & 3) << 4),
                         (ql[..., 1, :] >> 4) | ((qh >> 6) << 4)], -2)
        sc = b[..., 192:208].contiguous().view(torch.int8).to(F64) * half(208)
        return ((q.reshape(rows, -1, 16, 16).to(F64) - 32) * sc[..., None]).view(rows, -1)
    s = b[..., 4:16]
    sc = torch.cat([s[..., :4] & 63, (s[..., 8:] & 15) | ((s[..., :4] >> 6) << 4)], -1).to(F64) * half(0)
    mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1).to(F64) * half(2)
    qs = b[..., -128:].reshape(rows, -1, 4, 32)
    q = torch.stack([qs & 15, qs >> 4], -2).view(rows, -1, 8, 32)
    if enc == "Q5_K":
        q = q | torch.stack([((b[..., 16:48] >> j) & 1) << 4 for j in range(8)], -2)
    return (q.to(F64) * sc[..., None] - mn[..., None]).view(rows, -1)


def _resident(packed, enc, rows, cols):
    torch.cuda.synchronize()
    return Weight.from_device(packed.data_ptr(), packed.numel() * packed.element_size(), enc, rows, cols)


def _rounded(x, enc):
    """The activations that the encoding's kernels multiply: K-quants of four and six bits take one int8 code per value with a
    scale per 256 (part of the format's definition), the others the values themselves."""
    if enc not in ("Q4_K", "Q6_K"):
        return x.to(F64)
    b = x.float().reshape(*x.shape[:-1], -1, 256)
    top = b.abs().amax(-1, keepdim=True)
    q = torch.round(b * torch.where(top > 0, torch.full_like(top, 127.0).div(top), torch.zeros_like(top))).clamp_(-127, 127)
    return (q.to(F64) * (top / 127.0).to(F64)).view(x.shape)


# ---- single linears -----------------------------------------------------------------------------------------------------------

class _Linear:
    @staticmethod
    def matrix(c, seed, i):
        return _pack(_normal((c["rows"], c["cols"]), 0.02, seed, 1, i), c["enc"])

    @staticmethod
    def prepare(c, seed):
        ws = [_resident(_Linear.matrix(c, seed, i), c["enc"], c["rows"], c["cols"]) for i in range(c["weights"])]
        x = _normal((c["m"], c["cols"]), 1.0, seed, 2)
        return {"run": _Linear.run, "w": ws, "x": x, "y": [torch.empty(c["m"], c["rows"], device="cuda") for _ in ws], "m": c["m"]}

    @staticmethod
    def run(s):
        for w, y in zip(s["w"], s["y"]):
            device.matmul(w, s["x"].data_ptr(), s["m"], y.data_ptr())
        return s["y"]

    @staticmethod
    def exact(c, seed):
        x = _rounded(_normal((c["m"], c["cols"]), 1.0, seed, 2), c["enc"])
        return [x @ _unpack(_Linear.matrix(c, seed, i), c["enc"]).T for i in range(c["weights"])]

    @staticmethod
    def work(c):
        n, nbytes = BLOCK[c["enc"]]
        return {"bytes": c["weights"] * (c["rows"] * c["cols"] // n * nbytes + 4 * c["m"] * (c["rows"] + c["cols"])), "flops": 2 * c["weights"] * c["m"] * c["rows"] * c["cols"]}

    @staticmethod
    def tolerance(c):
        return {"rel": 2e-4 if c["enc"] == "Q8_0" else 2e-6}   # four times what is measured; Q8_0: activations carried with 15 bits


# ---- attention over a binary16 cache ------------------------------------------------------------------------------------------

class _Attention:
    @staticmethod
    def inputs(c, seed, i):
        kv = (c["batch"], c["kv_heads"], c["context"], c["dim"])
        return _normal((c["batch"], c["heads"], c["dim"]), 1.0, seed, 1, i), _normal(kv, 1.0, seed, 2, i).half(), _normal(kv, 1.0, seed, 3, i).half()

    @staticmethod
    def lengths(c, seed):
        """Sequences of a batch are of different lengths: from half the context on, the first of them whole."""
        n = np.random.default_rng(seed).integers((c["context"] + 1) // 2, c["context"] + 1, c["batch"]).astype(np.int32)
        n[0] = c["context"]
        return torch.from_numpy(n)

    @staticmethod
    def prepare(c, seed):
        caches = [_Attention.inputs(c, seed, i) for i in range(c["caches"])]
        return {"run": _Attention.run, "c": c, "caches": caches, "n": _Attention.lengths(c, seed).cuda(), "out": [torch.empty_like(q) for q, _, _ in caches]}

    @staticmethod
    def run(s):
        c = s["c"]
        for (q, k, v), o in zip(s["caches"], s["out"]):
            device.attn_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), c["batch"], c["heads"], c["kv_heads"], c["dim"], c["context"], s["n"].data_ptr(),
                               c["context"], c["dim"] ** -0.5)
        return s["out"]

    @staticmethod
    def attend(q, k, v, scale):
        """[heads, dim] over [kv_heads, n, dim]."""
        g = q.shape[0] // k.shape[0]
        k, v = k.repeat_interleave(g, 0), v.repeat_interleave(g, 0)
        return torch.einsum("hn,hnd->hd", torch.softmax(torch.einsum("hd,hnd->hn", q, k) * scale, -1), v)

    @staticmethod
    def exact(c, seed):
        out, lengths = [], _Attention.lengths(c, seed)
        for i in range(c["caches"]):
            q, k, v = _Attention.inputs(c, seed, i)
            out.append(torch.stack([_Attention.attend(q[b].to(F64), k[b, :, :n].to(F64), v[b, :, :n].to(F64), c["dim"] ** -0.5) for b, n in enumerate(lengths.tolist())]))
        return out

    @staticmethod
    def work(c):
        n = 0.75 * c["context"] * c["batch"] * c["caches"]
        return {"bytes": n * c["kv_heads"] * c["dim"] * 4 + 8 * c["caches"] * c["batch"] * c["heads"] * c["dim"], "flops": 4 * n * c["heads"] * c["dim"]}

    @staticmethod
    def tolerance(c):
        return {"rel": 3e-6}   # four times what is measured


# ---- attention over the compressed cache --------------------------------------------------------------------------------------

class _TurboQuant:
    @staticmethod
    def inputs(c, seed, layer):
        shape = (c["context"], c["kv_heads"], c["dim"])
        return _normal(shape, 1.0, seed, 1, layer), _normal(shape, 1.0, seed, 2, layer), _normal((c["heads"], c["dim"]), 1.0, seed, 3, layer)

    @staticmethod
    def prepare(c, seed):
        from skainet_b200.kvstore import DeviceKvCacheStore, TurboQuantConfig
        cfg = TurboQuantConfig.polarOnly(c["bits"])
        store = DeviceKvCacheStore(c["layers"], c["kv_heads"], c["dim"], c["context"], keyConfig=cfg, valueConfig=cfg)
        row = c["kv_heads"] * c["dim"] * 4
        layers = [_TurboQuant.inputs(c, seed, l) for l in range(c["layers"])]
        for p in range(c["context"]):                # a token goes into all layers before the next one
            for l, (k, v, _) in enumerate(layers):
                store.appendTokenDevice(l, k.data_ptr() + p * row, v.data_ptr() + p * row)
        queries = [q for _, _, q in layers]
        torch.cuda.synchronize()
        return {"run": _TurboQuant.run, "c": c, "store": store, "q": queries, "out": [torch.empty_like(q) for q in queries]}

    @staticmethod
    def run(s):
        c = s["c"]
        for l, (q, o) in enumerate(zip(s["q"], s["out"])):
            s["store"].decodeStep(l, q.data_ptr(), o.data_ptr(), c["heads"], 0, c["context"])
        return s["out"]

    @staticmethod
    def signs(c, layer, flip):
        """[context, kv_heads, dim] of 1 and -1: the seeded sign of every element (a polynomial of layer, head and position through
        MurmurHash3's finalizer seeds Marsaglia's xorwow, whose first 64 draws are dropped)."""
        m32 = 0xFFFFFFFF
        pos, head = np.meshgrid(np.arange(c["context"], dtype=np.uint64), np.arange(c["kv_heads"], dtype=np.uint64), indexing="ij")
        h = (((layer * 31 + head) & m32) * 31 + pos) & m32
        h ^= h >> 16
        h = (h * 0x85EBCA6B) & m32
        h ^= h >> 13
        h = (h * 0xC2B2AE35) & m32
        h = (h ^ (h >> 16)) ^ flip
        high = np.where(h >> 31, np.uint64(m32), np.uint64(0))
        x, y, z, w, v, add = h, high, h * 0, h * 0, h ^ m32, ((h << 10) & m32) ^ (high >> 4)
        out = np.empty(h.shape + (c["dim"],))
        for i in range(64 + c["dim"]):
            t = x ^ (x >> 2)
            x, y, z, w = y, z, w, v
            v = (t ^ ((t << 1) & m32)) ^ v ^ ((v << 4) & m32)
            add = (add + 362437) & m32
            if i >= 64:
                out[..., i - 64] = np.where(((v + add) & m32) >> 31, -1.0, 1.0)
        return torch.from_numpy(out).to(_cuda())

    @staticmethod
    def stored(x, signs, bits):
        """What the codec gives back for rows x: rotated, rounded per 32 values in 32 bits, rotated back."""
        def hadamard(v):
            n, h = v.shape[-1], 1
            while h < n:
                a = v.view(*v.shape[:-1], -1, 2, h)
                v = torch.stack([a[..., 0, :] + a[..., 1, :], a[..., 0, :] - a[..., 1, :]], -2).view(v.shape)
                h *= 2
            return v * torch.tensor(1.0 / np.sqrt(np.float32(n)), dtype=v.dtype, device=v.device)
        top = 2 ** (bits - 1) - 1
        g = hadamard(x * signs.float()).view(*x.shape[:-1], -1, 32)
        scale = g.abs().amax(-1, keepdim=True) / top
        return hadamard((torch.round(g * (1.0 / scale)).clamp_(-top, top).to(F64) * scale.to(F64)).view(x.shape)) * signs

    @staticmethod
    def exact(c, seed):
        out = []
        for l in range(c["layers"]):
            k, v, q = _TurboQuant.inputs(c, seed, l)
            k, v = (_TurboQuant.stored(t, _TurboQuant.signs(c, l, flip), c["bits"]).transpose(0, 1) for t, flip in ((k, 0), (v, 0x5A5A5A5A)))
            out.append(_Attention.attend(q.to(F64), k, v, c["dim"] ** -0.5))
        return out

    @staticmethod
    def work(c):
        n = c["layers"] * c["context"] * c["kv_heads"]
        return {"bytes": 2 * n * (c["dim"] * c["bits"] // 8 + c["dim"] // 8) + 8 * c["layers"] * c["heads"] * c["dim"], "flops": 4 * c["layers"] * c["context"] * c["heads"] * c["dim"]}

    @staticmethod
    def tolerance(c):
        return {"rel": 2e-3}   # measured 5e-4: decoded rows are held in binary16


# ---- whole decoders -----------------------------------------------------------------------------------------------------------

def _tokens(c, seed):
    """[batch, prompt + steps] token numbers; an answer's tokens are given, so that no near tie decides what comes next."""
    return np.random.default_rng(seed + 17).integers(0, c["vocab"], (c["batch"], c["prompt"] + c["steps"])).astype(np.int32)


def _answer(s):
    """A request from the start: the prompts, then step by step with the logits of every step; a prompt alone gives the logits
    after its last token."""
    m, c, t = s["model"], s["c"], s["tokens"]
    m.reset()
    if not c["steps"]:
        return [m.forward(t[b, :], [c["prompt"] - 1], b) for b in range(c["batch"])]
    for b in range(c["batch"]):
        m.prefill(t[b, :c["prompt"]], b, want_next=False)
    out = np.empty((c["steps"], c["batch"], c["vocab"]), np.float32)
    picked = np.zeros(c["batch"], np.int32)
    for i in range(c["steps"]):
        m.decode(np.ascontiguousarray(t[:, c["prompt"] + i]), picked)
        out[i] = m.logits(c["batch"])
    return [out]


def _laid_out(c, logits):
    """Logits [batch, positions wanted, vocab] as `_answer` returns them."""
    return [torch.stack(logits, 1)] if c["steps"] else logits


def _rms(x, gain):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain


def _causal_softmax(score, extra=None):
    n = score.shape[-1]
    score = score.masked_fill(torch.ones(n, n, dtype=torch.bool, device=score.device).triu(1), -math.inf)
    if extra is not None:
        return torch.softmax(torch.cat([score, extra.expand(*score.shape[:-1], 1)], -1), -1)[..., :-1]
    return torch.softmax(score, -1)


def _decoder_work(c, per_token, weight_bytes, cache_bytes):
    """per_token: multiply-adds of one token's linears; the head runs for the tokens whose logits are wanted."""
    steps, prompt = c["steps"], c["prompt"]
    tokens = c["batch"] * (prompt + steps)
    passes = (1 if prompt else 0) + steps
    seen = c["batch"] * (prompt + sum(prompt + i + 1 for i in range(steps)))
    pairs = c["batch"] * (prompt + steps) ** 2 // 2
    flops = 2 * (tokens * per_token + c["batch"] * max(1, steps) * c["width"] * c["vocab"]) + 4 * pairs * c["layers"] * c["heads"] * 128
    return {"bytes": passes * weight_bytes + seen * cache_bytes + 4 * c["vocab"] * c["batch"] * max(1, steps), "flops": flops}


class _Llama:
    """Q4_K linears, Q8_0 tables, as the configurations of the benchmark."""
    NAMES = ("q", "k", "v", "o", "gate", "up", "down")

    @staticmethod
    def shape(c, name):
        w, kv = c["width"], c["kv_heads"] * 128
        return {"q": (w, w), "k": (kv, w), "v": (kv, w), "o": (w, w), "gate": (c["ff"], w), "up": (c["ff"], w), "down": (w, c["ff"]), "table": (c["vocab"], w)}[name]

    @staticmethod
    def packed(c, seed, layer, name):
        """Normal weights; what one layer writes into the residual stream is small beside it, as in trained models."""
        std = 0.02 / (3 * math.sqrt(2 * c["layers"])) if name in ("o", "down") else 0.02
        return _pack(_normal(_Llama.shape(c, name), std, seed, layer + 1, _Llama.NAMES.index(name)), "Q4_K")

    @staticmethod
    def table(c, seed, which):
        return _pack(_normal(_Llama.shape(c, "table"), 1.0 if which == 0 else 0.02, seed, 0, which), "Q8_0")

    @staticmethod
    def gain(c, seed, layer, which):
        return 1.0 + _normal((c["width"],), 0.1, seed, 1000 + layer, which)

    @staticmethod
    def prepare(c, seed):
        from skainet_b200.llama import W_ATTN_NORM, W_DOWN, W_EMBED, W_FFN_NORM, W_GATE, W_HEAD, W_K, W_O, W_OUT_NORM, W_Q, W_UP, W_V, Llama, LlamaConfig
        m = Llama(LlamaConfig(c["layers"], c["width"], c["heads"], c["kv_heads"], 128, c["ff"], c["vocab"], rms_eps=EPS, max_seq=max(64, c["prompt"] + c["steps"]), max_batch=c["batch"]))
        for which, at in ((0, W_EMBED), (1, W_HEAD)):
            m.set_weight(0, at, _resident(_Llama.table(c, seed, which), "Q8_0", c["vocab"], c["width"]))
        m.set_norm(0, W_OUT_NORM, _Llama.gain(c, seed, -1, 0).cpu().numpy())
        for l in range(c["layers"]):
            for name, at in zip(_Llama.NAMES, (W_Q, W_K, W_V, W_O, W_GATE, W_UP, W_DOWN)):
                m.set_weight(l, at, _resident(_Llama.packed(c, seed, l, name), "Q4_K", *_Llama.shape(c, name)))
            for which, at in ((0, W_ATTN_NORM), (1, W_FFN_NORM)):
                m.set_norm(l, at, _Llama.gain(c, seed, l, which).cpu().numpy())
        m.finalize()
        return {"run": _answer, "model": m, "c": c, "tokens": _tokens(c, seed)}

    @staticmethod
    def exact(c, seed):
        tokens = torch.from_numpy(_tokens(c, seed)).long().to(_cuda())
        B, n, H, G = c["batch"], tokens.shape[1], c["heads"], c["kv_heads"]
        x = _unpack(_Llama.table(c, seed, 0), "Q8_0")[tokens]
        ang = torch.arange(n, dtype=F64, device=x.device)[:, None] * 1e4 ** (-torch.arange(64, dtype=F64, device=x.device) / 64)
        cos, sin = ang.cos()[:, None], ang.sin()[:, None]

        def turn(v):
            a, b = v[..., 0::2], v[..., 1::2]
            return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).view(v.shape)

        for l in range(c["layers"]):
            lin = lambda name, v: _rounded(v, "Q4_K") @ _unpack(_Llama.packed(c, seed, l, name), "Q4_K").T  # noqa: B023, E731
            h = _rms(x, _Llama.gain(c, seed, l, 0).to(F64))
            q, k, v = (lin(name, h).view(B, n, heads, 128) for name, heads in (("q", H), ("k", G), ("v", G)))
            q, k, v = turn(q), turn(k).half().to(F64), v.half().to(F64)              # the cache is binary16
            k, v = (t.repeat_interleave(H // G, 2) for t in (k, v))
            a = torch.stack([torch.einsum("hij,jhd->ihd", _causal_softmax(torch.einsum("ihd,jhd->hij", q[b], k[b]) * 128 ** -0.5), v[b]) for b in range(B)])
            x = x + lin("o", a.reshape(B, n, H * 128))
            h = _rms(x, _Llama.gain(c, seed, l, 1).to(F64))
            x = x + lin("down", torch.nn.functional.silu(lin("gate", h)) * lin("up", h))
        head = _unpack(_Llama.table(c, seed, 1), "Q8_0")
        x = _rms(x, _Llama.gain(c, seed, -1, 0).to(F64))
        at = slice(c["prompt"], n) if c["steps"] else slice(n - 1, n)
        return _laid_out(c, [x[b, at] @ head.T for b in range(B)])

    @staticmethod
    def work(c):
        params = c["layers"] * sum(math.prod(_Llama.shape(c, n)) for n in _Llama.NAMES)
        return _decoder_work(c, params, params * 144 // 256 + c["vocab"] * c["width"] * 34 // 32, c["layers"] * 2 * c["kv_heads"] * 128 * 2)

    @staticmethod
    def tolerance(c):
        return {"rel": 3e-2, "max": 0.3}   # measured 1e-2: an int8 code that falls the other way is worth 1/127 of its block's largest value, four times per layer


class _Bf16Decoder:
    """What the two BF16 designs share: matrices by name, rounded to bf16."""

    @classmethod
    def matrix(cls, c, seed, layer, name, rows, cols, gain=1.0):
        names = sorted(cls.IDS)
        return _normal((rows, cols), gain / math.sqrt(cols), seed, layer + 1, names.index(name)).bfloat16()

    @classmethod
    def vector(cls, seed, layer, which, shape, mean=0.0, std=1.0):
        return mean + _normal(shape, std, seed, 5000 + layer, which)

    @staticmethod
    def tolerance(c):
        return {"rel": 2.5e-2, "max": 0.3}   # measured 3e-3 to 6e-3


def _put(m, layer, which, t):
    w = _resident(t, "BF16", *t.shape)
    m.set_weight(layer, which, w)
    torch.cuda.synchronize()
    w.free()


class _Tivazen(_Bf16Decoder):
    """Every second layer reads the cache of the one before it. (The routed form is left out: a near tie between two experts
    makes outputs that cannot be compared.)"""
    IDS = ("embed", "head", "q", "dkv", "uk", "uv", "g", "o", "gate", "up", "down")
    RANK, WINDOW = 512, 1024

    @classmethod
    def matrices(cls, c, layer):
        W, H = c["width"], c["heads"]
        shapes = {"q": (H * 192, W, 1.0), "uk": (H * 128, cls.RANK, 1.0), "uv": (H * 128, cls.RANK, 1.0), "g": (H, W, 1.0), "o": (W, H * 128, 1.0), "gate": (c["ff"], W, 1.0),
                  "up": (c["ff"], W, 1.0), "down": (W, c["ff"], 1.0)}
        if layer % 2 == 0:
            shapes["dkv"] = (cls.RANK + 64, W, 1.0)
        return shapes

    @staticmethod
    def norm(layer, which):
        return 0.12 + 0.002 * layer + 0.02 * which

    @classmethod
    def depth(cls, seed, layer):
        return torch.cat([cls.vector(seed, layer, 9, (layer + 1,), 0.0, 0.02), torch.ones(1, device=_cuda())])

    @classmethod
    def prepare(cls, c, seed):
        from skainet_b200 import tivazen as T
        at = {"q": T.W_Q, "dkv": T.W_DKV, "uk": T.W_UK, "uv": T.W_UV, "g": T.W_G, "o": T.W_O, "gate": T.W_GATE, "up": T.W_UP, "down": T.W_DOWN}
        layers = [T.TivazenLayer(c["heads"], 128, 64, 128, cls.RANK, cls.WINDOW, 192 ** -0.5, 1e4, l - 1 if l % 2 else None, T.MLP_DENSE, c["ff"]) for l in range(c["layers"])]
        m = T.Tivazen(T.TivazenConfig(c["width"], c["vocab"], EPS, layers, max_seq=max(64, c["prompt"] + c["steps"]), max_batch=c["batch"]))
        _put(m, 0, T.W_EMBED, cls.matrix(c, seed, -1, "embed", c["vocab"], c["width"], math.sqrt(c["width"])))
        _put(m, 0, T.W_HEAD, cls.matrix(c, seed, -1, "head", c["vocab"], c["width"]))
        m.set_vector(0, T.V_FINAL_NORM, [1.0])
        for l in range(c["layers"]):
            for name, shape in cls.matrices(c, l).items():
                _put(m, l, at[name], cls.matrix(c, seed, l, name, *shape))
            if l % 2 == 0:
                m.set_vector(l, T.V_DKV_NORM, cls.vector(seed, l, 8, (cls.RANK,), 1.0, 0.1).cpu().numpy())
            m.set_vector(l, T.V_NORM1, [cls.norm(l, 0)])
            m.set_vector(l, T.V_NORM2, [cls.norm(l, 1)])
            m.set_vector(l, T.V_DEPTH, cls.depth(seed, l).cpu().numpy())
        m.finalize()
        return {"run": _answer, "model": m, "c": c, "tokens": _tokens(c, seed)}

    @classmethod
    def exact(cls, c, seed):
        tokens = torch.from_numpy(_tokens(c, seed)[0]).long().to(_cuda())
        n, H, R = tokens.numel(), c["heads"], cls.RANK
        ang = torch.arange(n, dtype=F64, device=tokens.device)[:, None] * 1e4 ** (-torch.arange(32, dtype=F64, device=tokens.device) / 32)

        def turn(v):
            cos, sin = (f(ang).view(n, *([1] * (v.dim() - 2)), 32) for f in (torch.cos, torch.sin))
            a, b = v[..., :32], v[..., 32:]
            return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

        i = torch.arange(n, device=tokens.device)
        hidden = (i[None] > i[:, None]) | (i[:, None] - i[None] >= cls.WINDOW)
        x = cls.matrix(c, seed, -1, "embed", c["vocab"], c["width"], math.sqrt(c["width"])).to(F64)[tokens]
        states, kv = [x], None
        for l in range(c["layers"]):
            w = {name: cls.matrix(c, seed, l, name, *shape).to(F64) for name, shape in cls.matrices(c, l).items()}
            if l % 2 == 0:
                y = x @ w["dkv"].T
                kv = _rms(y[:, :R], cls.vector(seed, l, 8, (R,), 1.0, 0.1).to(F64)), turn(y[:, R:])
            q = (x @ w["q"].T).view(n, H, 192)
            k, v = (kv[0] @ w["uk"].T).view(n, H, 128), (kv[0] @ w["uv"].T).view(n, H, 128)
            score = (torch.einsum("ihd,jhd->hij", q[..., :128], k) + torch.einsum("ihd,jd->hij", turn(q[..., 128:]), kv[1])) * 192 ** -0.5
            a = torch.einsum("hij,jhd->ihd", torch.softmax(score.masked_fill_(hidden, -math.inf), -1), v) * torch.sigmoid(x @ w["g"].T)[..., None]
            del score
            x = x + _rms(a.reshape(n, -1) @ w["o"].T, cls.norm(l, 0))
            x = x + _rms((torch.nn.functional.silu(x @ w["gate"].T) * (x @ w["up"].T)) @ w["down"].T, cls.norm(l, 1))
            states.append(x)
            x = sum(a * s for a, s in zip(cls.depth(seed, l).to(F64), states))
        at = slice(c["prompt"], n) if c["steps"] else slice(n - 1, n)
        return _laid_out(c, [_rms(x, 1.0)[at] @ cls.matrix(c, seed, -1, "head", c["vocab"], c["width"]).to(F64).T])

    @classmethod
    def work(cls, c):
        params = sum(r * k for l in range(c["layers"]) for r, k, _ in cls.matrices(c, l).values())
        return _decoder_work(c, params, 2 * (params + c["vocab"] * c["width"]), c["layers"] * (cls.RANK + 64))


class _Fomalix(_Bf16Decoder):
    """Layers in turns of four: two of the delta rule, one Mamba-2, one attention, each with a feed-forward."""
    IDS = ("embed", "head", "q", "k", "v", "b", "a", "g", "in", "o", "gate", "up", "down")
    CHUNK, SCALE = 2048, 12.0

    @staticmethod
    def sizes(c, l):
        """(kind, heads, key/value heads, key size, value size)."""
        H = c["heads"]
        return [("delta", H, H // 2, 128, 128), ("delta", H, H // 2, 128, 128), ("mamba2", 4 * H, 4, 128, 64), ("attention", H, c["kv_heads"], 128, 128)][l % 4]

    @classmethod
    def matrices(cls, c, l):
        kind, H, G, D, V = cls.sizes(c, l)
        W, qk, inner = c["width"], G * D, H * V
        mixer = {"attention": {"q": (H * D, W), "k": (qk, W), "v": (G * V, W)}, "delta": {"q": (qk, W), "k": (qk, W), "v": (inner, W), "b": (H, W), "a": (H, W), "g": (inner, W)},
                 "mamba2": {"in": (2 * inner + 2 * qk + H, W)}}[kind]
        return {**mixer, "o": (W, inner), "gate": (c["ff"], W), "up": (c["ff"], W), "down": (W, c["ff"])}

    @classmethod
    def vectors(cls, c, seed, l):
        """By name; decays run from almost none to strong, the norms that close a sublayer keep it small beside the stream."""
        kind, H, G, D, V = cls.sizes(c, l)
        W, qk, inner = c["width"], G * D, H * V
        at = iter(range(100))
        new = lambda shape, mean=0.0, std=1.0: cls.vector(seed, l, next(at), shape, mean, std)  # noqa: E731
        v = {"norm1": new((W,), 1.0, 0.1), "norm1b": new((W,), 0.5, 0.05), "norm2": new((W,), 1.0, 0.1), "norm2b": new((W,), 0.5, 0.05)}
        if kind == "attention":
            return {**v, "q.b": new((H * D,), 0.0, 0.1), "k.b": new((qk,), 0.0, 0.1), "v.b": new((G * V,), 0.0, 0.1), "sink": new((H,))}
        base = torch.tensor([-6.0, 0.0, -3.0, 1.0], device=_cuda()).repeat((H + 3) // 4)[:H]
        v.update({"A_log": base + new((H,), 0.0, 0.2), "dt_bias": new((H,), -1.0, 0.5)})
        if kind == "delta":
            return {**v, "q.conv": new((qk, 4), 0.0, 0.5), "k.conv": new((qk, 4), 0.0, 0.5), "v.conv": new((inner, 4), 0.0, 0.5), "norm": new((V,), 1.0, 0.1)}
        return {**v, "conv": new((inner + 2 * qk, 4), 0.0, 0.5), "conv.b": new((inner + 2 * qk,), 0.0, 0.3), "D": new((H,)), "norm": new((inner,), 1.0, 0.1)}

    @classmethod
    def prepare(cls, c, seed):
        from skainet_b200 import fomalix as X
        wat = {"q": X.W_Q, "k": X.W_K, "v": X.W_V, "b": X.W_B, "a": X.W_A, "g": X.W_G, "in": X.W_IN, "o": X.W_O, "gate": X.W_GATE, "up": X.W_UP, "down": X.W_DOWN}
        vat = {"norm1": X.V_NORM1, "norm1b": X.V_NORM1B, "norm2": X.V_NORM2, "norm2b": X.V_NORM2B, "q.b": X.V_Q_BIAS, "k.b": X.V_K_BIAS, "v.b": X.V_V_BIAS, "sink": X.V_SINK,
               "q.conv": X.V_Q_CONV, "k.conv": X.V_K_CONV, "v.conv": X.V_V_CONV, "conv": X.V_CONV, "conv.b": X.V_CONV_BIAS, "A_log": X.V_A_LOG, "dt_bias": X.V_DT_BIAS, "D": X.V_D,
               "norm": X.V_MIX_NORM}
        layers = []
        for l in range(c["layers"]):
            kind, H, G, D, V = cls.sizes(c, l)
            more = {"delta": {"type": X.DELTA, "conv": 4}, "mamba2": {"type": X.MAMBA2, "conv": 4, "norm_groups": 1}, "attention": {"type": X.ATTENTION, "chunk": cls.CHUNK, "scale": D ** -0.5 * 4}}[kind]
            layers.append(X.FomalixLayer(heads=H, kv_heads=G, dim=D, vdim=V, ff=c["ff"], **more))
        m = X.Fomalix(X.FomalixConfig(c["width"], c["vocab"], EPS, layers, cls.SCALE, max_seq=max(64, c["prompt"] + c["steps"]), max_batch=c["batch"]))
        _put(m, 0, X.W_EMBED, cls.matrix(c, seed, -1, "embed", c["vocab"], c["width"], math.sqrt(c["width"]) / 4))
        _put(m, 0, X.W_HEAD, cls.matrix(c, seed, -1, "head", c["vocab"], c["width"]))
        m.set_vector(0, X.V_FINAL_NORM, np.ones(c["width"], np.float32))
        for l in range(c["layers"]):
            for name, shape in cls.matrices(c, l).items():
                _put(m, l, wat[name], cls.matrix(c, seed, l, name, *shape))
            for name, v in cls.vectors(c, seed, l).items():
                m.set_vector(l, vat[name], v.cpu().numpy())
        m.finalize()
        return {"run": _answer, "model": m, "c": c, "tokens": _tokens(c, seed)}

    @staticmethod
    def conv(x, taps, bias=0.0):
        T = taps.shape[1]
        xp = torch.cat([torch.zeros(T - 1, x.shape[1], dtype=F64, device=x.device), x])
        return torch.nn.functional.silu(sum(xp[j:j + x.shape[0]] * taps[:, j] for j in range(T)) + bias)

    @staticmethod
    def delta(h, w, v, H, G, D, V):
        n = h.shape[0]
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k, x = (_Fomalix.conv(h @ w[a].T, v[a + ".conv"]) for a in ("q", "k", "v"))
        q, k = (unit(t.view(n, G, D)).repeat_interleave(H // G, 1) for t in (q, k))
        q, x = q * D ** -0.5, x.view(n, H, V)
        decay = torch.exp(-torch.exp(v["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + v["dt_bias"]))
        beta = torch.sigmoid(h @ w["b"].T)
        S, out = torch.zeros(H, D, V, dtype=F64, device=h.device), []
        for t in range(n):
            S = S * decay[t][:, None, None]
            u = beta[t][:, None, None] * (x[t][:, None] - k[t][:, None] @ S)
            S = torch.baddbmm(S, k[t][:, :, None], u)
            out.append(q[t][:, None] @ S)
        o = torch.cat(out, 1).transpose(0, 1)
        return _rms(o, v["norm"]) * torch.nn.functional.silu(h @ w["g"].T).view(n, H, V)

    @staticmethod
    def mamba2(h, w, v, H, G, D, V):
        n, inner = h.shape[0], H * V
        z, xbc, dt = torch.split(h @ w["in"].T, [inner, inner + 2 * G * D, H], 1)
        x, B, C = torch.split(_Fomalix.conv(xbc, v["conv"], v["conv.b"]), [inner, G * D, G * D], 1)
        x = x.view(n, H, V)
        B, C = (t.view(n, G, D).repeat_interleave(H // G, 1) for t in (B, C))
        dt = torch.nn.functional.softplus(dt + v["dt_bias"])
        decay = torch.exp(-torch.exp(v["A_log"]) * dt)
        S, out = torch.zeros(H, D, V, dtype=F64, device=h.device), []
        for t in range(n):
            S = torch.baddbmm(S * decay[t][:, None, None], B[t][:, :, None] * dt[t][:, None, None], x[t][:, None])
            out.append(C[t][:, None] @ S)
        y = torch.cat(out, 1).transpose(0, 1) + v["D"][:, None] * x
        return _rms(y.reshape(n, inner) * torch.nn.functional.silu(z), v["norm"])

    @staticmethod
    def attention(h, w, v, H, G, D, V):
        n = h.shape[0]
        q, k, x = ((h @ w[a].T + v[a + ".b"]).view(n, heads, -1) for a, heads in (("q", H), ("k", G), ("v", G)))
        q, k, x = _rms(q, 1.0), _rms(k, 1.0).repeat_interleave(H // G, 1), x.repeat_interleave(H // G, 1)
        i = torch.arange(n, device=h.device) // _Fomalix.CHUNK
        score = torch.einsum("ihd,jhd->hij", q, k) * (D ** -0.5 * 4)
        score = score.masked_fill(i[:, None] != i[None], -math.inf)
        return torch.einsum("hij,jhd->ihd", _causal_softmax(score, v["sink"].view(H, 1, 1)), x)

    @classmethod
    def exact(cls, c, seed):
        tokens = torch.from_numpy(_tokens(c, seed)[0]).long().to(_cuda())
        n, W = tokens.numel(), c["width"]
        ang = torch.arange(n, dtype=F64, device=tokens.device)[:, None] * 1e4 ** (-2.0 * torch.arange(W // 2, dtype=F64, device=tokens.device) / W)
        x = cls.matrix(c, seed, -1, "embed", c["vocab"], W, math.sqrt(W) / 4).to(F64)[tokens] * cls.SCALE + torch.stack([ang.sin(), ang.cos()], -1).view(n, W)
        for l in range(c["layers"]):
            kind, H, G, D, V = cls.sizes(c, l)
            w = {name: cls.matrix(c, seed, l, name, *shape).to(F64) for name, shape in cls.matrices(c, l).items()}
            v = {name: t.to(F64) for name, t in cls.vectors(c, seed, l).items()}
            o = getattr(cls, kind)(_rms(x, v["norm1"]), w, v, H, G, D, V).reshape(n, -1) @ w["o"].T
            x = x + _rms(o, v["norm1b"])
            h = _rms(x, v["norm2"])
            x = x + _rms((torch.nn.functional.gelu(h @ w["gate"].T, approximate="tanh") * (h @ w["up"].T)) @ w["down"].T, v["norm2b"])
        at = slice(c["prompt"], n) if c["steps"] else slice(n - 1, n)
        return _laid_out(c, [_rms(x, 1.0)[at] @ cls.matrix(c, seed, -1, "head", c["vocab"], W).to(F64).T])

    @classmethod
    def work(cls, c):
        params = sum(r * k for l in range(c["layers"]) for r, k in cls.matrices(c, l).values())
        return _decoder_work(c, params, 2 * (params + c["vocab"] * c["width"]), c["layers"] // 4 * c["kv_heads"] * 256 * 2)


PATHS = {"linear": _Linear, "attention": _Attention, "turboquant": _TurboQuant, "llama": _Llama, "tivazen": _Tivazen, "fomalix": _Fomalix}


def prepare(case, seed):
    return PATHS[case["path"]].prepare(case, seed)


def run(state):
    return state["run"](state)


def work(case):
    return PATHS[case["path"]].work(case)


def tolerance(case):
    return PATHS[case["path"]].tolerance(case)


def exact(case, seed):
    return PATHS[case["path"]].exact(case, seed)
