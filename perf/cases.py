"""The performance cases of this framework: what a model's forward has it do, through its public entry points.

Every case is a sequence of `LaunchKernel` records, made once as a decode loop makes them (`LaunchBatch`, with
`Projector` choosing the projection ids as the reference's `ProjectBatch` does), and submitted per pass with
`LaunchMany` and `Flush` to a backend whose deferred queue is on, the mode the C++ backend starts in.  Weights,
activations and caches are seeded random tensors in the formats' own layouts with zero-mean values of a trained
layer's size; shapes are those of `tessera_b200.workload` (hidden 5120, feed-forward 17408, 24 query heads over 4
kv heads of 256, 48 linear-attention heads of 128) and of the benchmark's routed-expert row (256 experts of 2048 ->
512 -> 2048, eight selected).  Sequences run over several layers with weights of their own, so that a pass streams
them from memory as a forward does instead of finding them in the cache.

Paths (`case["path"]`):
  ffn        rmsnorm, gate and up projections, silu_mul, down projection, add (Q4_K, down Q4_K or Q6_K)
  project    the three projection shapes of a layer in one weight format: MXFP4, FP8, W4A8, bf16, fp32
  moe        router, top-k, gates, the selected experts, the shared expert, of one token
  attention  attention over the key / value cache, in each cache format
  linear     what a linear-attention layer does between its projections (gates, convolution, norms, delta rule)
  token      a whole forward of one token: embedding, layers of both kinds, head; returns the logits
"""
import math

import numpy as np
import torch

from tessera_b200.backend import DEVICE, CreateBackend, KernelLaunch, LaunchBatch
from tessera_b200.project import F4E2M1, Q4K, Q6K, Projector

EPS = 1e-6
THETA, ROPE_DIM, SECTIONS = 1e7, 64, (11, 11, 10)
CONV_WIDTH = 4


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a decoded token's feed-forward blocks: the bulk of what a token streams
        dict(name="ffn_decode", path="ffn", m=1, hidden=5120, ffn=17408, down=Q4K, layers=2),
        # one of eight tensor-parallel ranks' share of it (8 of 68 blocks): small launches, latency counts
        dict(name="ffn_decode_shard", path="ffn", m=1, hidden=5120, ffn=2048, down=Q6K, layers=8),
        # sixteen drafted tokens checked at once (speculative decoding)
        dict(name="ffn_verify", path="ffn", m=16, hidden=5120, ffn=17408, down=Q6K, layers=2),
        # one chunk of a prompt
        dict(name="ffn_prefill", path="ffn", m=512, hidden=5120, ffn=17408, down=Q6K, layers=1),
        # verification over MXFP4 weights, activations kept in full / quantised to FP8 per token
        dict(name="mxfp4_verify", path="project", fmt="mxfp4", m=16, hidden=5120, ffn=17408, layers=2),
        dict(name="w4a8_verify", path="project", fmt="w4a8", m=16, hidden=5120, ffn=17408, layers=2),
        # a few tokens decoded together over FP8 weights
        dict(name="fp8_small_batch", path="project", fmt="fp8", m=4, hidden=5120, ffn=17408, layers=1),
        # a token through mixture-of-experts layers: many small launches
        dict(name="moe_decode", path="moe", hidden=2048, inter=512, experts=256, top_k=8, down=Q4K, layers=4),
        # attention of a decoded token over an FP8 cache, the full-attention layers of a model
        dict(name="attention_decode", path="attention", kv="fp8", m=1, n=4096, heads=24, kv_heads=4, head_dim=256, window=0, layers=16),
        # attention of a prompt's last chunk, and the linear-attention layers' part of a first chunk
        dict(name="attention_prefill", path="attention", kv="fp8", m=512, n=4096, heads=24, kv_heads=4, head_dim=256, window=0, layers=1),
        dict(name="linear_prefill", path="linear", rows=512, k_heads=16, v_heads=48, head=128, layers=1),
        # a whole forward: three linear-attention layers and one full-attention layer, and the head over the vocabulary
        dict(name="token", path="token", hidden=5120, ffn=17408, vocab=151936, heads=24, kv_heads=4, head_dim=256, k_heads=16,
             v_heads=48, head=128, kv="fp8", n=4096, layers=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["ffn", "ffn", "project", "project", "moe", "attention", "attention", "linear", "token"])
    if path == "ffn":
        m, hidden, ffn = _log(rng, 1, 512), 256 * rng.randint(4, 20), 256 * rng.randint(4, 68)
        down = rng.choice([Q4K, Q6K])
        layers = max(1, min(8, int(1.5e8 / (1.7 * hidden * ffn)))) if m <= 64 else 1
        return dict(path=path, m=m, hidden=hidden, ffn=ffn, down=down, layers=layers)
    if path == "project":
        fmt = rng.choice(["mxfp4", "mxfp4", "fp8", "w4a8", "bf16", "f32"])
        m = _log(rng, 1, 16 if fmt == "f32" else 64 if fmt in ("bf16", "w4a8") else 512)
        hidden, ffn = 64 * rng.randint(16, 80), 64 * rng.randint(16, 272)
        return dict(path=path, fmt=fmt, m=m, hidden=hidden, ffn=ffn, layers=rng.randint(1, 2))
    if path == "moe":
        return dict(path=path, hidden=256 * rng.randint(4, 16), inter=256 * rng.randint(1, 4), experts=rng.choice([32, 60, 64, 128, 256]),
                    top_k=rng.randint(2, 8), down=rng.choice([Q4K, Q6K]), layers=rng.randint(1, 4))
    if path == "attention":
        kv, head_dim, kv_heads, group = rng.choice(["f32", "f16", "q8", "q4", "fp8"]), rng.choice([128, 256]), rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 6, 8])
        heads = kv_heads * group
        while heads > 32:
            kv_heads, heads = kv_heads // 2, heads // 2
        m = _log(rng, 1, 512)
        most = int(512 * 4096 * 24 * 256 / (m * heads * head_dim))
        n = _log(rng, max(64, m), max(64, m, min(32768, most)))
        window = rng.choice([0, 0, 0, max(1, n // 3)])
        return dict(path=path, kv=kv, m=m, n=n, heads=heads, kv_heads=kv_heads, head_dim=head_dim, window=window, layers=rng.randint(1, 8) if m == 1 else 1)
    if path == "linear":
        k_heads = rng.choice([4, 8, 16])
        return dict(path=path, rows=_log(rng, 1, 512), k_heads=k_heads, v_heads=k_heads * rng.choice([1, 2, 3]), head=128, layers=1)
    return dict(path=path, hidden=256 * rng.randint(4, 16), ffn=256 * rng.randint(8, 48), vocab=rng.randint(1000, 151936), heads=16, kv_heads=rng.choice([2, 4]),
                head_dim=rng.choice([128, 256]), k_heads=8, v_heads=rng.choice([8, 16, 24]), head=128, kv=rng.choice(["f32", "f16", "q8", "fp8"]),
                n=_log(rng, 64, 4096), layers=4)


# ------------------------------------------------------------------ weights in the formats' layouts

class Random:
    """Seeded tensors on the GPU, one generator for a case."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)

    def bytes(self, *shape):
        return torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=self.g)

    def ints(self, lo, hi, *shape):
        return torch.randint(lo, hi, shape, device="cuda", generator=self.g)

    def uniform(self, lo, hi, *shape):
        return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=self.g)

    def normal(self, *shape):
        return torch.randn(shape, device="cuda", generator=self.g)

    def q4k(self, n, k):
        """n rows of k/256 Q4_K blocks (fp16 d, dmin; 12 bytes of 6-bit scales and mins; 128 nibble bytes), zero-mean
        values of standard deviation about 1/sqrt(k)."""
        nb = n * (k // 256)
        w = self.bytes(nb, 144)
        sc = self.ints(24, 64, nb, 8)
        mn = (sc + self.ints(-4, 5, nb, 8)).clamp_(0, 63)
        d = self.uniform(0.7, 1.3, nb) / (math.sqrt(k) * 4.61 * 44.0)
        w[:, 0:2] = d.half().view(torch.uint8).view(nb, 2)
        w[:, 2:4] = (7.5 * d).half().view(torch.uint8).view(nb, 2)
        w[:, 4:8] = ((sc[:, 0:4] & 63) | ((sc[:, 4:8] >> 4) << 6)).to(torch.uint8)
        w[:, 8:12] = ((mn[:, 0:4] & 63) | ((mn[:, 4:8] >> 4) << 6)).to(torch.uint8)
        w[:, 12:16] = ((sc[:, 4:8] & 15) | ((mn[:, 4:8] & 15) << 4)).to(torch.uint8)
        return w.view(-1)

    def q6k(self, n, k):
        """n rows of k/256 Q6_K blocks (128 low-nibble bytes, 64 high-bit bytes, 16 int8 scales, fp16 d)."""
        nb = n * (k // 256)
        w = self.bytes(nb, 210)
        w[:, 192:208] = self.ints(-64, 64, nb, 16).to(torch.int8).view(torch.uint8)
        d = self.uniform(0.7, 1.3, nb) / (math.sqrt(k) * 684.0)
        w[:, 208:210] = d.half().view(torch.uint8).view(nb, 2)
        return w.view(-1)

    def block(self, fmt, n, k):
        return self.q4k(n, k) if fmt == Q4K else self.q6k(n, k)

    def mxfp4(self, n, k):
        """Packed E2M1 nibbles (uniform codes) followed by one E8M0 byte per 32 values, exponents -8..0."""
        return torch.cat([self.bytes(n * k // 2), self.ints(119, 128, n * k // 32).to(torch.uint8)])

    def fp8(self, n, k):
        """E4M3 bytes and a scale per row of N(0, 0.02) weights."""
        w = self.normal(n, k) * 0.02
        s = w.abs().amax(dim=1) / 448.0
        return (w / s[:, None]).to(torch.float8_e4m3fn).view(torch.uint8).view(-1), s


def _deq_q4k(w, n, k):
    b = w.view(-1, 144)
    d, dmin = (b[:, i:i + 2].contiguous().view(torch.float16).double() for i in (0, 2))
    p = b[:, 4:16].to(torch.int32)
    sc = torch.cat([p[:, 0:4] & 63, (p[:, 8:12] & 15) | ((p[:, 0:4] >> 6) << 4)], 1).double() * d
    mn = torch.cat([p[:, 4:8] & 63, (p[:, 8:12] >> 4) | ((p[:, 4:8] >> 6) << 4)], 1).double() * dmin
    q = b[:, 16:144].view(-1, 4, 1, 32)
    q = torch.cat([q & 15, q >> 4], 2).view(-1, 8, 32)
    return (q.double() * sc[:, :, None] - mn[:, :, None]).view(n, k)


def _deq_q6k(w, n, k):
    b = w.view(-1, 210)
    d = b[:, 208:210].contiguous().view(torch.float16).double()
    s = b[:, 192:208].contiguous().view(torch.int8).double() * d
    ql, qh = b[:, 0:128].view(-1, 2, 2, 32), b[:, 128:192].view(-1, 2, 1, 32)
    low = torch.cat([ql & 15, ql >> 4], 2)
    high = torch.cat([(qh >> i) & 3 for i in (0, 2, 4, 6)], 2)
    q = (low.to(torch.int16) | (high.to(torch.int16) << 4)) - 32
    return (q.view(-1, 16, 16).double() * s[:, :, None]).view(n, k)


def _deq_mxfp4(w, n, k):
    grid = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, -0., -.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device="cuda")
    b = w[:n * k // 2].long()
    v = torch.stack([grid[b & 15], grid[b >> 4]], 1).view(-1, 32)
    return (v * torch.exp2(w[n * k // 2:].double() - 127.0)[:, None]).view(n, k)


def _times(fmt, a, w, n, k):
    """a (rows x k, 64 bits) times the transposed weights, some rows of W at a time."""
    if fmt in ("bf16", "f32"):
        return a @ w.view(n, k).double().t()
    if fmt == "fp8":
        return (a @ w[0].view(torch.float8_e4m3fn).view(n, k).double().t()) * w[1].double()
    out, per = [], max(1, (1 << 26) // k)
    for r in range(0, n, per):
        rows = min(per, n - r)
        if fmt == "mxfp4":
            part = torch.cat([w[r * k // 2:(r + rows) * k // 2], w[n * k // 2 + r * k // 32:n * k // 2 + (r + rows) * k // 32]])
            out.append(a @ _deq_mxfp4(part, rows, k).t())
        else:
            step = k // 256 * (144 if fmt == Q4K else 210)
            out.append(a @ (_deq_q4k if fmt == Q4K else _deq_q6k)(w[r * step:(r + rows) * step], rows, k).t())
    return torch.cat(out, 1)


_WEIGHT_BYTES = {Q4K: 144 / 256, Q6K: 210 / 256, "mxfp4": 17 / 32, "w4a8": 17 / 32, "fp8": 1.0, "bf16": 2.0, "f32": 4.0}
_KV_BYTES = {"f32": 4.0, "f16": 2.0, "q8": 1.0, "q4": 0.5, "fp8": 1.0}


# ------------------------------------------------------------------ device buffers and launch sequences

_BACKEND = None


def _backend():
    global _BACKEND
    if _BACKEND is None:
        _BACKEND = CreateBackend()
        _BACKEND.SetDeviceIndex(torch.cuda.current_device())
        _BACKEND.Init()
        _BACKEND.SetDeferred(1)
    return _BACKEND


class Memory:
    """A buffer of the backend as a torch tensor sees it."""

    _CODES = {torch.float32: "<f4", torch.uint8: "|u1", torch.int32: "<i4", torch.int64: "<i8"}

    def __init__(self, shape, dtype):
        item = torch.empty(0, dtype=dtype).element_size()
        self.buffer = _backend().AllocateBuffer(max(1, math.prod(shape) * item), DEVICE)
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=self._CODES[dtype], data=(self.buffer.Handle(), False), version=3)


class Program:
    """A state: its buffers by name, and the launches of a pass."""

    def __init__(self, tensors):
        self.b, self.batch, self.kernels = _backend(), LaunchBatch(), {}
        self.buffers, self.tensors = {}, {}
        for name, t in tensors.items():
            self.new(name, t.shape, t.dtype)
        self.b.Synchronize()
        for name, t in tensors.items():
            self.tensors[name].copy_(t)
        self.projector = Projector(self)

    # what Projector asks of a backend
    def LoadKernel(self, name):
        if name not in self.kernels:
            self.kernels[name] = self.b.LoadKernel(name)
        return self.kernels[name]

    def AllocateBuffer(self, nbytes):
        return self.b.AllocateBuffer(nbytes)

    def LaunchKernel(self, kernel, launch):
        self.batch.add(kernel, launch)

    def new(self, name, shape, dtype=torch.float32):
        m = Memory(shape, dtype)
        self.buffers[name], self.tensors[name] = m.buffer, torch.as_tensor(m, device="cuda")
        return name

    def do(self, kernel, names, scalars):
        self.batch.add(self.LoadKernel(kernel), KernelLaunch(buffers=[self.buffers[x] for x in names], scalars=[int(s) for s in scalars]))

    def project(self, fmt, a, w, out, m, n, k):
        if fmt in (Q4K, Q6K, "mxfp4"):
            self.projector.ProjectBatch({"mxfp4": F4E2M1}.get(fmt, fmt), self.buffers[a], self.buffers[w], self.buffers[out], m, n, k)
        elif fmt == "fp8":
            self.do("gemm_fp8", [a, w, w + ".scale", out], [m, n, k])
        else:
            self.do("gemm_bf16" if fmt == "bf16" else "gemm_f32", [a, w, out], [m, n, k])


def _bits(x):
    return int(np.float32(x).view(np.uint32))


def prepare(case, seed):
    tensors = _INPUTS[case["path"]](case, Random(seed))
    p = Program({k: v.view(torch.uint8).view(-1) if v.dtype in (torch.float16, torch.bfloat16) else v for k, v in tensors.items()})
    del tensors
    outs = _RECORD[case["path"]](case, p)
    p.b.Flush()
    return p, {name: p.tensors[name] for name in outs}


def run(state):
    program, outs = state
    program.b.LaunchMany(program.batch)
    program.b.Flush()
    return outs


def exact(case, seed):
    return _EXACT[case["path"]](case, _INPUTS[case["path"]](case, Random(seed)))


def tolerance(case):
    return _TOLERANCE[case["path"]](case)


def work(case):
    return _WORK[case["path"]](case)


def _norm64(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w.double()


def _silu64(x):
    return x / (1.0 + torch.exp(-x))


# ------------------------------------------------------------------ ffn

def _ffn_inputs(c, r):
    t = dict(x0=r.normal(c["m"], c["hidden"]))
    for i in range(c["layers"]):
        _ffn_weights(c, r, t, i, c["down"])
    return t


def _ffn_weights(c, r, t, i, down):
    t["norm%d" % i] = 1.0 + 0.1 * r.normal(c["hidden"])
    t["gate%d" % i], t["up%d" % i] = r.q4k(c["ffn"], c["hidden"]), r.q4k(c["ffn"], c["hidden"])
    t["down%d" % i] = r.block(down, c["hidden"], c["ffn"])


def _ffn_layer(p, m, hidden, ffn, down, i, x, out):
    p.do("rmsnorm", [x, "norm%d" % i, "xn"], [m, hidden, _bits(EPS)])
    p.project(Q4K, "xn", "gate%d" % i, "g", m, ffn, hidden)
    p.project(Q4K, "xn", "up%d" % i, "u", m, ffn, hidden)
    p.do("silu_mul", ["g", "u", "act"], [m * ffn])
    p.project(down, "act", "down%d" % i, "proj", m, hidden, ffn)
    p.do("add", [x, "proj", out], [m * hidden])


def _ffn_record(c, p):
    m, hidden, ffn = c["m"], c["hidden"], c["ffn"]
    for name, cols in (("xn", hidden), ("g", ffn), ("u", ffn), ("act", ffn), ("proj", hidden)):
        p.new(name, (m, cols))
    for i in range(c["layers"]):
        p.new("x%d" % (i + 1), (m, hidden))
        _ffn_layer(p, m, hidden, ffn, c["down"], i, "x%d" % i, "x%d" % (i + 1))
    return ["x%d" % (i + 1) for i in range(c["layers"])] + ["act"]


def _ffn64(t, x, i, hidden, ffn, down):
    xn = _norm64(x, t["norm%d" % i])
    act = _silu64(_times(Q4K, xn, t["gate%d" % i], ffn, hidden)) * _times(Q4K, xn, t["up%d" % i], ffn, hidden)
    return x + _times(down, act, t["down%d" % i], hidden, ffn), act


def _ffn_exact(c, t):
    out, x = {}, t["x0"].double()
    for i in range(c["layers"]):
        x, out["act"] = _ffn64(t, x, i, c["hidden"], c["ffn"], c["down"])
        out["x%d" % (i + 1)] = x
    return out


def _ffn_work(c):
    per = c["hidden"] * c["ffn"]
    weights = per * (2 * _WEIGHT_BYTES[Q4K] + _WEIGHT_BYTES[c["down"]]) + 4 * c["hidden"]
    return dict(bytes=c["layers"] * weights + 4 * c["m"] * (c["hidden"] * (1 + c["layers"]) + c["ffn"]), flops=6.0 * c["layers"] * c["m"] * per)


# ------------------------------------------------------------------ project

def _project_shapes(c):
    h, f = c["hidden"], c["ffn"]
    return [(h, h), (f, h), (h, f)]


def _project_inputs(c, r):
    t = dict(x=r.normal(c["m"], c["hidden"]).bfloat16().float(), act=r.normal(c["m"], c["ffn"]).bfloat16().float())
    for i in range(c["layers"]):
        for j, (n, k) in enumerate(_project_shapes(c)):
            w = "w%d_%d" % (i, j)
            if c["fmt"] in ("mxfp4", "w4a8"):
                t[w] = r.mxfp4(n, k)
            elif c["fmt"] == "fp8":
                t[w], t[w + ".scale"] = r.fp8(n, k)
            else:
                t[w] = (r.normal(n, k) * 0.02).to(torch.bfloat16 if c["fmt"] == "bf16" else torch.float32)
    return t


def _project_record(c, p):
    m, outs = c["m"], []
    if c["fmt"] == "w4a8":
        for a, k in (("x", c["hidden"]), ("act", c["ffn"])):
            p.new(a + ".codes", (m, k), torch.uint8)
            p.new(a + ".scale", (m,))
        for i in range(c["layers"]):
            for j, (n, k) in enumerate(_project_shapes(c)):  # the weights' reference scales, made when they are loaded
                w = "w%d_%d" % (i, j)
                p.new(w + ".ref", (n,), torch.uint8)
                p.b.LaunchKernel(p.LoadKernel("mxfp4_row_ref"), KernelLaunch(buffers=[p.buffers[w], p.buffers[w + ".ref"]], scalars=[n, k]))
    for i in range(c["layers"]):
        for j, (n, k) in enumerate(_project_shapes(c)):
            a, w, out = "act" if j == 2 else "x", "w%d_%d" % (i, j), p.new("out%d_%d" % (i, j), (m, n))
            outs.append(out)
            if c["fmt"] == "w4a8":
                p.do("quantize_fp8_pack_rows", [a, a + ".codes", a + ".scale"], [m, k])
                p.do("gemm_mxfp4_wmma", [a + ".codes", w, a + ".scale", w + ".ref", out], [m, n, k, 1, 0])
            else:
                p.project(c["fmt"], a, w, out, m, n, k)
    return outs


def _fp8_rows64(x):
    """Values of x after the per-row FP8 E4M3 quantisation with an absmax scale (a division by a number would be
    a multiplication by its rounded reciprocal, and move the ties of bf16 inputs)."""
    s = x.float().abs().amax(-1, keepdim=True)
    s = s / torch.full_like(s, 448.0)
    return (x.float() / s).clamp(-448, 448).to(torch.float8_e4m3fn).double() * s.double()


def _project_exact(c, t):
    out = {}
    for i in range(c["layers"]):
        for j, (n, k) in enumerate(_project_shapes(c)):
            a, w = t["act" if j == 2 else "x"], "w%d_%d" % (i, j)
            a = _fp8_rows64(a) if c["fmt"] == "w4a8" else a.double()
            fmt = "mxfp4" if c["fmt"] == "w4a8" else c["fmt"]
            out["out%d_%d" % (i, j)] = _times(fmt, a, (t[w], t[w + ".scale"]) if fmt == "fp8" else t[w], n, k)
    return out


def _project_work(c):
    total = sum(n * k for n, k in _project_shapes(c)) * c["layers"]
    rows = sum(n for n, _ in _project_shapes(c)) * c["layers"]
    return dict(bytes=total * _WEIGHT_BYTES[c["fmt"]] + 4 * c["m"] * (c["hidden"] + c["ffn"] + rows), flops=2.0 * c["m"] * total)


# ------------------------------------------------------------------ moe

def _moe_inputs(c, r):
    h, f, e = c["hidden"], c["inter"], c["experts"]
    t = dict(x0=r.normal(1, h))
    for i in range(c["layers"]):
        t["norm%d" % i] = 1.0 + 0.1 * r.normal(h)
        t["router%d" % i] = r.normal(e, h) / math.sqrt(h)
        t["sgate%d" % i] = r.normal(h) / math.sqrt(h)
        t["gate%d" % i], t["up%d" % i], t["down%d" % i] = r.q4k(e * f, h), r.q4k(e * f, h), r.block(c["down"], e * h, f)
        t["sg%d" % i], t["su%d" % i], t["sd%d" % i] = r.q4k(f, h), r.q4k(f, h), r.q4k(h, f)
    return t


def _moe_record(c, p):
    h, f, e, k = c["hidden"], c["inter"], c["experts"], c["top_k"]
    per_gu, per_d = f * (h // 256) * 144, h * (f // 256) * (144 if c["down"] == Q4K else 210)
    for name, cols in (("xn", h), ("logits", e), ("vals", k), ("wts", k), ("sig", 1), ("phi", k * f), ("routed", h), ("g", f), ("u", f), ("act", f), ("shared", h), ("ff", h)):
        p.new(name, (1, cols))
    outs = []
    for i in range(c["layers"]):
        x, out, ids = "x%d" % i, p.new("x%d" % (i + 1), (1, h)), p.new("ids%d" % i, (1, k), torch.int32)
        p.do("rmsnorm", [x, "norm%d" % i, "xn"], [1, h, _bits(EPS)])
        p.do("gemm_f32", ["xn", "router%d" % i, "logits"], [1, e, h])
        p.do("top_k_rows", ["logits", ids, "vals"], [1, e, k, 0])
        p.do("moe_gate", ["vals", "xn", "sgate%d" % i, "wts", "sig"], [k, h])
        p.do("moe_experts_gate_up_q4k", ["xn", "gate%d" % i, "up%d" % i, ids, "phi"], [h, f, k, per_gu, per_gu])
        p.do("moe_experts_down_" + c["down"], ["phi", "down%d" % i, ids, "wts", "routed"], [h, f, k, per_d, 0])
        p.project(Q4K, "xn", "sg%d" % i, "g", 1, f, h)
        p.project(Q4K, "xn", "su%d" % i, "u", 1, f, h)
        p.do("silu_mul", ["g", "u", "act"], [f])
        p.project(Q4K, "act", "sd%d" % i, "shared", 1, h, f)
        p.do("moe_scale_add", ["routed", "shared", "sig", "ff"], [h, 0])
        p.do("add", [x, "ff", out], [h])
        outs += [out, ids]
    return outs


def _moe_exact(c, t):
    h, f, e, k = c["hidden"], c["inter"], c["experts"], c["top_k"]
    out, x, bb = {}, t["x0"].double(), 144 if c["down"] == Q4K else 210
    for i in range(c["layers"]):
        xn = _norm64(x, t["norm%d" % i])
        vals, ids = torch.topk((xn @ t["router%d" % i].double().t())[0], k)
        wts, sig = torch.softmax(vals, 0), torch.sigmoid(xn[0] @ t["sgate%d" % i].double())
        ff = torch.zeros_like(xn)
        for w, id_ in zip(wts, ids.tolist()):
            gu, dn = slice(id_ * f * (h // 256) * 144, (id_ + 1) * f * (h // 256) * 144), slice(id_ * h * (f // 256) * bb, (id_ + 1) * h * (f // 256) * bb)
            phi = _silu64(_times(Q4K, xn, t["gate%d" % i][gu], f, h)) * _times(Q4K, xn, t["up%d" % i][gu], f, h)
            ff = ff + w * _times(c["down"], phi, t["down%d" % i][dn], h, f)
        act = _silu64(_times(Q4K, xn, t["sg%d" % i], f, h)) * _times(Q4K, xn, t["su%d" % i], f, h)
        x = x + ff + sig * _times(Q4K, act, t["sd%d" % i], h, f)
        out["x%d" % (i + 1)], out["ids%d" % i] = x, None
    return out


def _moe_work(c):
    h, f = c["hidden"], c["inter"]
    blocks = c["top_k"] * h * f * (2 * _WEIGHT_BYTES[Q4K] + _WEIGHT_BYTES[c["down"]]) + 3 * h * f * _WEIGHT_BYTES[Q4K]
    return dict(bytes=c["layers"] * (blocks + 4 * h * (c["experts"] + 3)), flops=c["layers"] * 2.0 * (3 * (c["top_k"] + 1) * h * f + c["experts"] * h))


# ------------------------------------------------------------------ attention

def _cache(r, kv, n, cols):
    """n cache rows of cols values in the cache's format, and the scale of each row."""
    if kv == "f32":
        return r.normal(n, cols), None
    if kv == "f16":
        return r.normal(n, cols).half(), None
    s = r.uniform(0.5, 1.5, n)
    if kv == "fp8":
        return (r.normal(n, cols) * 100.0).clamp_(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8), s / 100.0
    if kv == "q8":
        return (r.normal(n, cols) * 30.0).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8), s / 30.0
    return r.bytes(n, cols // 2), s / 4.0


def _cache64(kv, t, s, n, cols):
    if kv in ("f32", "f16"):
        return t.view(n, cols).double()
    if kv == "fp8":
        v = t.view(torch.float8_e4m3fn).view(n, cols).double()
    elif kv == "q8":
        v = t.view(torch.int8).view(n, cols).double()
    else:
        b = t.view(n, cols // 2).to(torch.int32)
        v = torch.stack([b & 15, b >> 4], 2).view(n, cols)
        v = torch.where(v >= 8, v - 16, v).double()
    return v * s.double()[:, None]


def _attention_inputs(c, r):
    t, cols = {}, c["kv_heads"] * c["head_dim"]
    for i in range(c["layers"]):
        t["q%d" % i] = r.normal(c["m"], c["heads"], c["head_dim"])
        for x in "kv":
            t["%s%d" % (x, i)], s = _cache(r, c["kv"], c["n"], cols)
            if s is not None:
                t["%s%d.scale" % (x, i)] = s
    return t


def _attend(p, kv, q, k, v, out, m, n, heads, kv_heads, dim, window):
    if kv in ("f32", "f16"):
        p.do("attention", [q, k, v, out], [m, n, heads, kv_heads, dim, n - m, 0, window, int(kv == "f16"), 1])
    else:
        p.do("attention_" + kv, [q, k, v, k + ".scale", v + ".scale", out], [m, n, heads, kv_heads, dim, n - m, 0, window, ("q8", "q4", "fp8").index(kv)])


def _attention_record(c, p):
    outs = []
    for i in range(c["layers"]):
        outs.append(p.new("out%d" % i, (c["m"], c["heads"], c["head_dim"])))
        _attend(p, c["kv"], "q%d" % i, "k%d" % i, "v%d" % i, outs[-1], c["m"], c["n"], c["heads"], c["kv_heads"], c["head_dim"], c["window"])
    return outs


def _attention64(q, k, v, heads, kv_heads, dim, window):
    """q: rows x heads x dim at the last positions; k, v: keys x (kv_heads * dim)."""
    m, n, group = q.shape[0], k.shape[0], heads // kv_heads
    k, v = k.view(n, kv_heads, dim), v.view(n, kv_heads, dim)
    pos, key = torch.arange(n - m, n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
    hidden = (key > pos) if window == 0 else (key > pos) | (key < pos + 1 - window)
    out = torch.empty_like(q)
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].t() / math.sqrt(dim)).masked_fill_(hidden, -math.inf)
        out[:, h] = torch.softmax(s, 1) @ v[:, h // group]
    return out


def _attention_exact(c, t):
    out, cols = {}, c["kv_heads"] * c["head_dim"]
    for i in range(c["layers"]):
        k, v = (_cache64(c["kv"], t["%s%d" % (x, i)], t.get("%s%d.scale" % (x, i)), c["n"], cols) for x in "kv")
        out["out%d" % i] = _attention64(t["q%d" % i].double(), k, v, c["heads"], c["kv_heads"], c["head_dim"], c["window"])
    return out


def _attention_keys(c):
    """(query, key) pairs that are not masked, and keys that any row reads."""
    m, n, w = c["m"], c["n"], c["window"]
    pairs = sum(min(n - m + i + 1, w or n) for i in range(m))
    return pairs, min(n, (w or n) + m - 1)


def _attention_work(c):
    pairs, keys = _attention_keys(c)
    scale = 8 if c["kv"] in ("q8", "q4", "fp8") else 0
    per = 2 * keys * c["kv_heads"] * c["head_dim"] * _KV_BYTES[c["kv"]] + scale * keys + 8 * c["m"] * c["heads"] * c["head_dim"]
    return dict(bytes=c["layers"] * per, flops=c["layers"] * 4.0 * pairs * c["heads"] * c["head_dim"])


# ------------------------------------------------------------------ linear

def _linear_weights(c, r, t, i):
    conv = (2 * c["k_heads"] + c["v_heads"]) * c["head"]
    t["conv_w%d" % i] = r.normal(conv, CONV_WIDTH) * 0.5
    t["a_log%d" % i], t["dt%d" % i] = -torch.exp(r.normal(c["v_heads"])), r.normal(c["v_heads"])
    t["ssm_norm%d" % i] = 1.0 + 0.1 * r.normal(c["head"])


def _linear_inputs(c, r):
    t, rows, conv = {}, c["rows"], (2 * c["k_heads"] + c["v_heads"]) * c["head"]
    for i in range(c["layers"]):
        _linear_weights(c, r, t, i)
        t["qkv%d" % i], t["z%d" % i] = r.normal(rows, conv), r.normal(rows, c["v_heads"] * c["head"])
        t["alpha_raw%d" % i], t["beta_raw%d" % i] = r.normal(rows, c["v_heads"]), r.normal(rows, c["v_heads"])
    return t


def _linear_buffers(p, rows, kh, vh, d):
    for name, cols in (("alpha", vh), ("beta", vh), ("q", kh * d), ("k", kh * d), ("v", vh * d), ("qe", vh * d), ("ke", vh * d)):
        p.new(name, (rows, cols))


def _linear_layer(p, rows, kh, vh, d, i, qkv, z, alpha_raw, beta_raw, hist, state, core, out):
    conv = (2 * kh + vh) * d
    p.do("ssm_gate", ["a_log%d" % i, "dt%d" % i, alpha_raw, beta_raw, "alpha", "beta"], [vh, rows])
    p.do("conv1d_state", [qkv, "conv_w%d" % i, hist, "q", "k", "v", hist], [conv, CONV_WIDTH, kh * d, 0, rows, 0])
    p.do("l2norm", ["q", "q"], [rows * kh, d, _bits(EPS), _bits(1.0 / math.sqrt(d))])
    p.do("l2norm", ["k", "k"], [rows * kh, d, _bits(EPS), _bits(1.0)])
    p.do("repeat_heads", ["q", "qe"], [vh, d, vh // kh, rows])
    p.do("repeat_heads", ["k", "ke"], [vh, d, vh // kh, rows])
    p.do("delta_step_heads", [state, "ke", "v", "qe", core, "alpha", "beta"], [vh, d, d, rows, 0, 0, 0])
    p.do("rmsnorm_gated", [core, "ssm_norm%d" % i, z, out], [rows * vh, d, _bits(EPS), 0, 0])


def _linear_record(c, p):
    rows, kh, vh, d, outs = c["rows"], c["k_heads"], c["v_heads"], c["head"], []
    _linear_buffers(p, rows, kh, vh, d)
    p.new("core", (rows, vh * d))
    for i in range(c["layers"]):
        hist, state = p.new("hist%d" % i, ((2 * kh + vh) * d, CONV_WIDTH - 1)), p.new("state%d" % i, (vh, d, d))
        out = p.new("out%d" % i, (rows, vh * d))
        # a prompt's first chunk starts from an empty history and state
        p.do("fill", [hist], [0, (2 * kh + vh) * d * (CONV_WIDTH - 1)])
        p.do("fill", [state], [0, vh * d * d])
        _linear_layer(p, rows, kh, vh, d, i, "qkv%d" % i, "z%d" % i, "alpha_raw%d" % i, "beta_raw%d" % i, hist, state, "core", out)
        outs += [out, hist, state]
    return outs


def _linear64(t, i, qkv, z, alpha_raw, beta_raw, hist, state, kh, vh, d):
    """hist: channels x 3, newest first.  Returns (out, hist, state)."""
    rows = qkv.shape[0]
    alpha = torch.exp(t["a_log%d" % i].double() * torch.nn.functional.softplus(alpha_raw + t["dt%d" % i].double(), threshold=700.0))
    beta = torch.sigmoid(beta_raw)
    line = torch.cat([hist.flip(1).t(), qkv])  # oldest first
    conv = _silu64(sum(line[j:j + rows] * t["conv_w%d" % i].double()[:, j] for j in range(CONV_WIDTH)))
    q, k, v = conv[:, :kh * d].reshape(rows, kh, d), conv[:, kh * d:2 * kh * d].reshape(rows, kh, d), conv[:, 2 * kh * d:].reshape(rows, vh, d)
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + EPS) for x in (q / 1.0, k))
    q = (q / math.sqrt(d)).repeat(1, vh // kh, 1)
    k = k.repeat(1, vh // kh, 1)
    core = []
    for r in range(rows):
        a, b, kr = alpha[r][:, None, None], beta[r][:, None, None], k[r][:, :, None]
        read = (state * kr).sum(1, keepdim=True)
        state = a * (state - b * kr * read) + b * v[r][:, None, :] * kr
        core.append((state * q[r][:, :, None]).sum(1))
    core = torch.stack(core)
    out = _norm64(core, t["ssm_norm%d" % i]) * _silu64(z.view(rows, vh, d))
    return out.view(rows, vh * d), line[-(CONV_WIDTH - 1):].flip(0).t(), state


def _linear_exact(c, t):
    out, kh, vh, d = {}, c["k_heads"], c["v_heads"], c["head"]
    for i in range(c["layers"]):
        hist = torch.zeros((2 * kh + vh) * d, CONV_WIDTH - 1, dtype=torch.float64, device="cuda")
        state = torch.zeros(vh, d, d, dtype=torch.float64, device="cuda")
        args = (t[x + str(i)].double() for x in ("qkv", "z", "alpha_raw", "beta_raw"))
        out["out%d" % i], out["hist%d" % i], out["state%d" % i] = _linear64(t, i, *args, hist, state, kh, vh, d)
    return out


def _linear_work(c):
    rows, kh, vh, d = c["rows"], c["k_heads"], c["v_heads"], c["head"]
    conv = (2 * kh + vh) * d
    per = 4 * (rows * (conv + 2 * vh * d + 2 * vh) + conv * (2 * CONV_WIDTH - 1) + vh * d * d)
    return dict(bytes=c["layers"] * per, flops=c["layers"] * rows * (7.0 * vh * d * d + 2.0 * conv * CONV_WIDTH))


# ------------------------------------------------------------------ token

def _token_plan(c):
    """Per layer: whether it is a full-attention layer, and the format of its mixed tensors."""
    return [(i % 4 == 3, Q6K if i % 2 else Q4K) for i in range(c["layers"])]


def _token_inputs(c, r):
    h, qd, kvd = c["hidden"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    vd, conv = c["v_heads"] * c["head"], (2 * c["k_heads"] + c["v_heads"]) * c["head"]
    t = dict(id=r.ints(0, c["vocab"], 1).to(torch.int32), table=r.q4k(c["vocab"], h), pos=torch.full((1, 3), c["n"] - 1, dtype=torch.int64, device="cuda"))
    t["table"].view(-1, 144)[:, 0:4] = t["table"].view(-1, 144)[:, 0:4].contiguous().view(torch.float16).float().mul(math.sqrt(h)).half().view(torch.uint8).view(-1, 4)
    for i, (full, mixed) in enumerate(_token_plan(c)):
        t["anorm%d" % i] = 1.0 + 0.1 * r.normal(h)
        if full:
            t["wq%d" % i], t["wk%d" % i], t["wv%d" % i], t["wo%d" % i] = r.q4k(2 * qd, h), r.q4k(kvd, h), r.block(mixed, kvd, h), r.q4k(h, qd)
            t["qnorm%d" % i], t["knorm%d" % i] = 1.0 + 0.1 * r.normal(c["head_dim"]), 1.0 + 0.1 * r.normal(c["head_dim"])
            for x in "kv":
                t["c%s%d" % (x, i)], s = _cache(r, c["kv"], c["n"], kvd)
                if s is not None:
                    t["c%s%d.scale" % (x, i)] = s
        else:
            _linear_weights(c, r, t, i)
            t["wqkv%d" % i], t["wz%d" % i], t["wo%d" % i] = r.q4k(conv, h), r.q4k(vd, h), r.q4k(h, vd)
            t["walpha%d" % i], t["wbeta%d" % i] = r.q4k(c["v_heads"], h), r.q4k(c["v_heads"], h)
            t["hist%d" % i], t["state%d" % i] = r.normal(conv, CONV_WIDTH - 1), r.normal(c["v_heads"], c["head"], c["head"]) * 0.1
        _ffn_weights(c, r, t, i, mixed)
    t["onorm"], t["head"] = 1.0 + 0.1 * r.normal(h), r.q6k(c["vocab"], h)
    return t


def _token_record(c, p):
    h, heads, kvh, dim, n, kv = c["hidden"], c["heads"], c["kv_heads"], c["head_dim"], c["n"], c["kv"]
    qd, kvd, vd, conv = heads * dim, kvh * dim, c["v_heads"] * c["head"], (2 * c["k_heads"] + c["v_heads"]) * c["head"]
    row = int(kvd * _KV_BYTES[kv])
    for name, cols in (("x", h), ("x1", h), ("xn", h), ("proj", h), ("g", c["ffn"]), ("u", c["ffn"]), ("act", c["ffn"]), ("fused", 2 * qd), ("aq", qd), ("agate", qd),
                       ("ak", kvd), ("av", kvd), ("attn", qd), ("rscale", 1), ("qkv", conv), ("z", vd), ("araw", c["v_heads"]), ("braw", c["v_heads"]), ("core", vd),
                       ("mix", vd), ("logits", c["vocab"])):
        p.new(name, (1, cols))
    p.new("row", (kvd * 4,), torch.uint8)
    _linear_buffers(p, 1, c["k_heads"], c["v_heads"], c["head"])
    p.do("embedding_q4k", ["id", "table", "x"], [1, h, c["vocab"]])
    outs = ["logits"]
    for i, (full, mixed) in enumerate(_token_plan(c)):
        p.do("rmsnorm", ["x", "anorm%d" % i, "xn"], [1, h, _bits(EPS)])
        if full:
            p.project(Q4K, "xn", "wq%d" % i, "fused", 1, 2 * qd, h)
            p.project(Q4K, "xn", "wk%d" % i, "ak", 1, kvd, h)
            p.project(mixed, "xn", "wv%d" % i, "av", 1, kvd, h)
            p.do("qgate_split", ["fused", "aq", "agate"], [heads, dim, 1])
            p.do("rmsnorm", ["aq", "qnorm%d" % i, "aq"], [heads, dim, _bits(EPS)])
            p.do("rmsnorm", ["ak", "knorm%d" % i, "ak"], [kvh, dim, _bits(EPS)])
            p.do("mrope", ["aq", "pos"], [1, heads, dim, ROPE_DIM, _bits(THETA), *SECTIONS])
            p.do("mrope", ["ak", "pos"], [1, kvh, dim, ROPE_DIM, _bits(THETA), *SECTIONS])
            for src, cache in (("ak", "ck%d" % i), ("av", "cv%d" % i)):
                if kv == "f32":
                    p.do("copy_d2d", [src, cache], [0, (n - 1) * row, row])
                    continue
                if kv == "f16":
                    p.do("cast_f32_f16", [src, "row"], [kvd])
                else:
                    p.do("quantize_fp8_pack" if kv == "fp8" else "quantize_" + kv, [src, "row", "rscale"], [1, kvd])
                    p.do("copy_d2d", ["rscale", cache + ".scale"], [0, (n - 1) * 4, 4])
                p.do("copy_d2d", ["row", cache], [0, (n - 1) * row, row])
            _attend(p, kv, "aq", "ck%d" % i, "cv%d" % i, "attn", 1, n, heads, kvh, dim, 0)
            p.do("sigmoid_gate", ["attn", "agate", "attn"], [qd])
            p.project(Q4K, "attn", "wo%d" % i, "proj", 1, h, qd)
        else:
            p.project(Q4K, "xn", "wqkv%d" % i, "qkv", 1, conv, h)
            p.project(Q4K, "xn", "wz%d" % i, "z", 1, vd, h)
            p.project(Q4K, "xn", "wbeta%d" % i, "braw", 1, c["v_heads"], h)
            p.project(Q4K, "xn", "walpha%d" % i, "araw", 1, c["v_heads"], h)
            _linear_layer(p, 1, c["k_heads"], c["v_heads"], c["head"], i, "qkv", "z", "araw", "braw", "hist%d" % i, "state%d" % i, "core", "mix")
            p.project(Q4K, "mix", "wo%d" % i, "proj", 1, h, vd)
            outs.append("state%d" % i)
        p.do("add", ["x", "proj", "x1"], [h])
        _ffn_layer(p, 1, h, c["ffn"], mixed, i, "x1", "x")
    p.do("rmsnorm", ["x", "onorm", "xn"], [1, h, _bits(EPS)])
    p.project(Q6K, "xn", "head", "logits", 1, c["vocab"], h)
    return outs


def _rope64(x, pos):
    """x: heads x dim, one position."""
    half = ROPE_DIM // 2
    angle = pos * THETA ** (-2.0 * torch.arange(half, dtype=torch.float64, device="cuda") / ROPE_DIM)
    a, b = x[:, :half], x[:, half:ROPE_DIM]
    return torch.cat([a * torch.cos(angle) - b * torch.sin(angle), a * torch.sin(angle) + b * torch.cos(angle), x[:, ROPE_DIM:]], 1)


def _stored64(kv, x):
    """A row as the cache holds it."""
    if kv == "f32":
        return x
    if kv == "f16":
        return x.float().half().double()
    if kv == "fp8":
        return _fp8_rows64(x)
    s = x.float().abs().amax(-1, keepdim=True)
    s = s / torch.full_like(s, 127.0)
    return (x.float() / s).round().clamp(-127, 127).double() * s.double()


def _token_exact(c, t):
    h, heads, kvh, dim, n, out = c["hidden"], c["heads"], c["kv_heads"], c["head_dim"], c["n"], {}
    qd, kvd, vd, conv = heads * dim, kvh * dim, c["v_heads"] * c["head"], (2 * c["k_heads"] + c["v_heads"]) * c["head"]
    step = h // 256 * 144
    row = int(t["id"])
    x = _deq_q4k(t["table"][row * step:(row + 1) * step], 1, h)
    for i, (full, mixed) in enumerate(_token_plan(c)):
        xn = _norm64(x, t["anorm%d" % i])
        if full:
            fused = _times(Q4K, xn, t["wq%d" % i], 2 * qd, h).view(heads, 2 * dim)
            k, v = _times(Q4K, xn, t["wk%d" % i], kvd, h).view(kvh, dim), _times(mixed, xn, t["wv%d" % i], kvd, h)
            q, k = _rope64(_norm64(fused[:, :dim], t["qnorm%d" % i]), n - 1), _rope64(_norm64(k, t["knorm%d" % i]), n - 1)
            ck, cv = (_cache64(c["kv"], t["c%s%d" % (y, i)], t.get("c%s%d.scale" % (y, i)), n, kvd).clone() for y in "kv")
            ck[-1], cv[-1] = _stored64(c["kv"], k.reshape(1, kvd))[0], _stored64(c["kv"], v)[0]
            mix = _attention64(q.reshape(1, heads, dim), ck, cv, heads, kvh, dim, 0).view(1, qd) * torch.sigmoid(fused[:, dim:].reshape(1, qd))
            x = x + _times(Q4K, mix, t["wo%d" % i], h, qd)
        else:
            qkv, z = _times(Q4K, xn, t["wqkv%d" % i], conv, h), _times(Q4K, xn, t["wz%d" % i], vd, h)
            a, b = _times(Q4K, xn, t["walpha%d" % i], c["v_heads"], h), _times(Q4K, xn, t["wbeta%d" % i], c["v_heads"], h)
            mix, _, out["state%d" % i] = _linear64(t, i, qkv, z, a, b, t["hist%d" % i].double(), t["state%d" % i].double(), c["k_heads"], c["v_heads"], c["head"])
            x = x + _times(Q4K, mix, t["wo%d" % i], h, vd)
        x, _ = _ffn64(t, x, i, h, c["ffn"], mixed)
    out["logits"] = _times(Q6K, _norm64(x, t["onorm"]), t["head"], c["vocab"], h)
    return out


def _token_work(c):
    h, qd, kvd, vd = c["hidden"], c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c["v_heads"] * c["head"]
    conv = (2 * c["k_heads"] + c["v_heads"]) * c["head"]
    nbytes, weights = c["vocab"] * h * _WEIGHT_BYTES[Q6K] + 4 * c["vocab"], float(c["vocab"] * h)
    for full, mixed in _token_plan(c):
        if full:
            nbytes += (2 * qd + kvd + qd) * h * _WEIGHT_BYTES[Q4K] + kvd * h * _WEIGHT_BYTES[mixed] + 2 * c["n"] * kvd * _KV_BYTES[c["kv"]]
            weights += (3 * qd + 2 * kvd) * h + 2 * c["n"] * qd
        else:
            nbytes += (conv + 2 * vd + 2 * c["v_heads"]) * h * _WEIGHT_BYTES[Q4K] + 8 * vd * c["head"]
            weights += (conv + 2 * vd) * h + 3 * vd * c["head"]
        nbytes += h * c["ffn"] * (2 * _WEIGHT_BYTES[Q4K] + _WEIGHT_BYTES[mixed])
        weights += 3 * h * c["ffn"]
    return dict(bytes=nbytes, flops=2.0 * weights)


_INPUTS = dict(ffn=_ffn_inputs, project=_project_inputs, moe=_moe_inputs, attention=_attention_inputs, linear=_linear_inputs, token=_token_inputs)
_RECORD = dict(ffn=_ffn_record, project=_project_record, moe=_moe_record, attention=_attention_record, linear=_linear_record, token=_token_record)
_EXACT = dict(ffn=_ffn_exact, project=_project_exact, moe=_moe_exact, attention=_attention_exact, linear=_linear_exact, token=_token_exact)
_WORK = dict(ffn=_ffn_work, project=_project_work, moe=_moe_work, attention=_attention_work, linear=_linear_work, token=_token_work)

# Largest differences of a correct implementation at the same precision, about four times the measured distance of the
# paths from `exact`.  Q4_K / Q6_K projections of up to eight rows carry their activations as integer digits (three of
# them up to two rows, two above); larger batches round weights and activations to binary16 (9e-4 measured, 1.7e-3 over several layers), as
# MXFP4 and FP8 do beyond 128 rows; what sums in fp32 shows 1e-7 to 2e-6.
_TOLERANCE = dict(
    ffn=lambda c: dict(rel=5e-3, max=5e-2) if c["m"] > 8 else dict(rel=1e-3, max=1e-2) if c["m"] > 2 else dict(rel=1e-5, max=4e-4),
    project=lambda c: dict(rel=4e-3, max=4e-2) if c["m"] > 128 and c["fmt"] in ("mxfp4", "fp8") else dict(rel=1e-5, max=4e-4),
    moe=lambda c: dict(rel=1e-5, max=4e-4, differ=0.005),
    attention=lambda c: dict(rel=4e-6, max=1e-4),
    linear=lambda c: dict(rel=4e-6, max=4e-4),
    token=lambda c: dict(rel=1e-5 if c["kv"] in ("f32", "f16") else 1e-4, max=4e-3),
)
