"""Attention over the key / value cache on the GPU (ids attention, attention_q8 / _q4 / _fp8, their split
halves and attention_combine) against the CPU oracle, which is bit-equal to the reference's AttentionRef
family (tests/test_oracle_golden.py).  The device adds the keys' contributions in a different order (lanes
split head_dim, warps split the keys, chunks merge at the end), so results agree to fp32 rounding."""
import os

import numpy as np
import pytest
import torch

from tessera_b200 import capi
from tessera_b200.backend import KernelLaunch

pytestmark = pytest.mark.gpu

TAGS = ("f32", "f16", "i8", "i4", "f8")
QUANT_ID = {2: "attention_q8", 3: "attention_q4", 4: "attention_fp8"}
QUANT_KIND = {2: 0, 3: 1, 4: 2}
TOL = 2e-5  # of the largest output magnitude


def run(backend, name, buffers, scalars):
    backend.LaunchKernel(backend.LoadKernel(name), KernelLaunch(buffers=buffers, scalars=scalars))


def near(y, r):
    return float(np.max(np.abs(y - r))) <= TOL * float(np.max(np.abs(r)))


def near_each(y, r, head_dim):
    """`near` for every (row, head) by itself."""
    y, r = y.reshape(-1, head_dim).astype(np.float64), r.reshape(-1, head_dim).astype(np.float64)
    return bool(np.all(np.abs(y - r).max(1) <= TOL * np.abs(r).max(1)))


def device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, q_base, window, causal, row_base=0):
    width = heads * head_dim
    qfull = np.zeros((row_base + m, width), np.float32)
    qfull[row_base:] = q.reshape(m, width)
    out = backend.AllocateBuffer((row_base + m) * width * 4)
    if fmt < 2:
        run(backend, "attention", [backend.upload(qfull), backend.upload(k), backend.upload(v), out],
            [m, n, heads, kv_heads, head_dim, q_base, row_base, window, fmt, 1 if causal else 0])
    else:
        run(backend, QUANT_ID[fmt],
            [backend.upload(qfull), backend.upload(k), backend.upload(v), backend.upload(ks), backend.upload(vs), out],
            [m, n, heads, kv_heads, head_dim, q_base, row_base, window, QUANT_KIND[fmt]])
    return backend.download(out, np.float32, (row_base + m) * width).reshape(row_base + m, width)[row_base:]


def make_cache(g, fmt, n, row):
    """(k, v, k_scale, v_scale) of a seeded cache in the format."""
    ks = (0.004 + 0.01 * g.random(n)).astype(np.float32)
    vs = (0.004 + 0.01 * g.random(n)).astype(np.float32)

    def one():
        if fmt == 0:
            return g.standard_normal((n, row)).astype(np.float32)
        if fmt == 1:
            return g.standard_normal((n, row)).astype(np.float16).view(np.uint8)
        if fmt == 2:
            return g.integers(-127, 128, (n, row)).astype(np.int8).view(np.uint8)
        if fmt == 3:
            nib = g.integers(0, 16, (n, row)).astype(np.uint8)
            return (nib[:, 0::2] | (nib[:, 1::2] << 4)).astype(np.uint8)
        b = g.integers(0, 256, (n, row)).astype(np.uint8)
        b[(b & 0x7F) == 0x7F] = 0x3C
        return b
    return one(), one(), ks, vs


def test_golden_cases_every_format(backend):
    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "attention_golden.npz"))
    m, n, heads, kv_heads, head_dim = (int(x) for x in g["dims"])
    checked = 0
    for fmt, tag in enumerate(TAGS):
        for si, (q_base, window, causal) in enumerate(g["settings"]):
            key = f"out_{tag}_{si}"
            if key not in g:
                continue
            y = device_attention(backend, fmt, g["q"], g["k_" + tag], g["v_" + tag], g["k_scale"], g["v_scale"], m, n, heads,
                                 kv_heads, head_dim, int(q_base), int(window), bool(causal))
            assert near(y, g[key]), key
            checked += 1
    assert checked == 16


@pytest.mark.parametrize("fmt", [0, 1, 2, 3, 4])
def test_decode_row_over_a_long_cache(backend, oracle, fmt):
    """One query row, 24 heads over 4 kv heads of 256, 4096 keys: 64 chunks (fp32, fp16), a cluster of sixteen CTAs (the others)."""
    g = np.random.default_rng(10 + fmt)
    n, heads, kv_heads, head_dim = 4096, 24, 4, 256
    q = g.standard_normal((1, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    y = device_attention(backend, fmt, q, k, v, ks, vs, 1, n, heads, kv_heads, head_dim, n - 1, 0, True)
    r = oracle.attention(fmt, q, k, v, 1, n, heads, kv_heads, head_dim, n - 1, 0, True, ks, vs)
    assert near(y, r)


@pytest.mark.parametrize("fmt,window", [(0, 0), (1, 300), (4, 1000)])
def test_verify_rows_with_row_base_and_window(backend, oracle, fmt, window):
    """Five query rows at the end of a 1500-key cache, written at rows 2..6 of a shared batch buffer."""
    g = np.random.default_rng(20 + fmt)
    m, n, heads, kv_heads, head_dim = 5, 1500, 16, 2, 128
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, n - m, window, True, row_base=2)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, n - m, window, True, ks, vs)
    assert near(y, r)


@pytest.mark.parametrize("fmt", [0, 1, 2, 4])
@pytest.mark.parametrize("q_base,split", [(2047, 16), (5, 16), (2047, 64)])
def test_split_and_combine_ids(backend, oracle, fmt, q_base, split):
    """The caller's chunk count and partial buffers (the reference's single-token path): partials in the reference's
    layout, empty chunks as the null partial (0, -1e30, 0), attention_combine merges them."""
    g = np.random.default_rng(30 + fmt)
    n, heads, kv_heads, head_dim = 2048, 8, 2, 256
    q = g.standard_normal((1, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    parts = heads * split
    pacc, pmax, psum = (backend.AllocateBuffer(parts * c * 4) for c in (head_dim, 1, 1))
    out = backend.AllocateBuffer(heads * head_dim * 4)
    if fmt < 2:
        for name in ("attention_split", "attention_split_gqa"):
            run(backend, name, [backend.upload(q), backend.upload(k), backend.upload(v), pacc, pmax, psum],
                [1, n, heads, kv_heads, head_dim, q_base, 0, fmt, 1, split])
    else:
        run(backend, QUANT_ID[fmt] + "_split",
            [backend.upload(q), backend.upload(k), backend.upload(v), backend.upload(ks), backend.upload(vs), pacc, pmax, psum],
            [1, n, heads, kv_heads, head_dim, q_base, 0, QUANT_KIND[fmt], split])
    run(backend, "attention_combine", [pacc, pmax, psum, out], [1, heads, head_dim, split])
    y = backend.download(out, np.float32, heads * head_dim).reshape(1, -1)
    r = oracle.attention(fmt, q, k, v, 1, n, heads, kv_heads, head_dim, q_base, 0, True, ks, vs)
    assert near(y, r)
    mx = backend.download(pmax, np.float32, parts).reshape(heads, split)
    sm = backend.download(psum, np.float32, parts).reshape(heads, split)
    acc = backend.download(pacc, np.float32, parts * head_dim).reshape(heads, split, head_dim)
    span = q_base + 1
    chunk = (span + split - 1) // split
    for s in range(split):
        if s * chunk >= span:
            assert np.all(mx[:, s] == np.float32(-1e30)) and np.all(sm[:, s] == 0) and np.all(acc[:, s] == 0)
        else:
            assert np.all(mx[:, s] > -1e29) and np.all(sm[:, s] >= 1.0)  # the chunk's own max contributes exp(0)


def test_rejects_what_it_does_not_serve(backend):
    buf = backend.AllocateBuffer(1 << 20)
    cases = [
        ("attention", [buf] * 4, [1, 16, 4, 2, 64, 15, 0, 0, 0, 1], capi.StatusCode.UnsupportedFeature),      # head_dim 64
        ("attention", [buf] * 4, [1, 16, 32, 2, 128, 15, 0, 0, 0, 1], capi.StatusCode.UnsupportedFeature),    # 16 heads per kv head
        ("attention", [buf] * 4, [1, 16, 6, 4, 128, 15, 0, 0, 0, 1], capi.StatusCode.InvalidArgument),        # heads % kv_heads
        ("attention", [buf] * 4, [1, 4096, 8, 8, 256, 15, 0, 0, 0, 1], capi.StatusCode.InvalidArgument),      # cache beyond the buffer
        ("attention_q8", [buf] * 6, [1, 16, 4, 2, 128, 15, 0, 0, 2], capi.StatusCode.InvalidArgument),        # kind of another id
        ("attention_split", [buf] * 6, [1, 16, 4, 2, 128, 15, 0, 0, 1, 65], capi.StatusCode.InvalidArgument),  # more than 64 chunks
        ("attention_combine", [buf] * 4, [1, 4, 128, 0], capi.StatusCode.InvalidArgument),
    ]
    for name, buffers, scalars, code in cases:
        with pytest.raises(capi.StatusError) as e:
            run(backend, name, buffers, scalars)
        assert e.value.code == code, name
    backend.Synchronize()


def bits(x):
    return int(np.float32(x).view(np.uint32))


def test_rope_against_golden_and_oracle(backend, oracle):
    """The angle is formed in double precision on both sides; the device's double sine and cosine may differ from
    the host's in the last bit, which shows as one ulp of an fp32 factor."""
    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "attention_golden.npz"))
    buf = backend.upload(g["rope_io"])
    run(backend, "rope", [buf], [3, 2, 64, 48, 1021, bits(1e6)])
    got = backend.download(buf, np.float32, g["rope_io"].size)
    assert np.all(np.abs(got - g["rope_out"]) <= 3e-7 * (np.abs(g["rope_out"]) + np.abs(g["rope_io"])))
    untouched = np.arange(got.size) % 64 >= 48
    assert np.array_equal(got[untouched], g["rope_io"][untouched])
    rng = np.random.default_rng(41)
    rows, heads, dim, rdim = 5, 24, 256, 64
    io = rng.standard_normal(rows * heads * dim).astype(np.float32)
    buf = backend.upload(io)
    run(backend, "rope", [buf], [rows, heads, dim, rdim, 100000, bits(1e7)])
    want = oracle.rope(io, rows, heads, dim, rdim, 100000, float(np.float32(1e7)))
    assert np.all(np.abs(backend.download(buf, np.float32, io.size) - want) <= 3e-7 * (np.abs(want) + np.abs(io)))


@pytest.mark.parametrize("kind,name", [(0, "quantize_q8"), (1, "quantize_q4")])
def test_cache_writers_are_bit_equal(backend, oracle, kind, name):
    """quantize_q8 / quantize_q4 (the int8 / 4-bit cache rows): golden cases with ties and a zero row, then
    a cache-sized row; the row maximum is exact in any order, so codes and scales are bit-equal."""
    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "attention_golden.npz"))
    tag = "kvq8" if kind == 0 else "kvq4"
    rng = np.random.default_rng(43 + kind)
    big = (rng.standard_normal((7, 1024)) * 3).astype(np.float32)
    for x, want in ((g["kvq_in"], (g[tag + "_codes"], g[tag + "_scale"])), (big, oracle.quantize_rows(kind, big))):
        rows, cols = x.shape
        nbytes = rows * cols if kind == 0 else rows * cols // 2
        codes, scale = backend.AllocateBuffer(nbytes), backend.AllocateBuffer(rows * 4)
        run(backend, name, [backend.upload(x), codes, scale], [rows, cols])
        assert np.array_equal(backend.download(codes, np.uint8, nbytes).reshape(want[0].shape), want[0])
        assert np.array_equal(backend.download(scale, np.float32, rows), want[1])
    buf = backend.AllocateBuffer(4096)
    with pytest.raises(capi.StatusError):
        run(backend, name, [buf, buf, buf], [1, 1020 if kind == 1 else 1022])  # cols not a multiple of 8 / 4
    backend.Synchronize()


def test_written_cache_feeds_attention(backend, oracle):
    """quantize_q8 rows written by the device, read back by attention_q8: the pair the int8 cache path runs."""
    rng = np.random.default_rng(47)
    n, heads, kv_heads, head_dim = 300, 8, 2, 128
    row = kv_heads * head_dim
    kf, vf = (rng.standard_normal((n, row)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((1, heads * head_dim)).astype(np.float32)
    bufs = []
    for x in (kf, vf):
        codes, scale = backend.AllocateBuffer(n * row), backend.AllocateBuffer(n * 4)
        run(backend, "quantize_q8", [backend.upload(x), codes, scale], [n, row])
        bufs += [codes, scale]
    out = backend.AllocateBuffer(heads * head_dim * 4)
    run(backend, "attention_q8", [backend.upload(q), bufs[0], bufs[2], bufs[1], bufs[3], out],
        [1, n, heads, kv_heads, head_dim, n - 1, 0, 0, 0])
    (kc, ks), (vc, vs) = oracle.quantize_rows(0, kf), oracle.quantize_rows(0, vf)
    want = oracle.attention(2, q, kc, vc, 1, n, heads, kv_heads, head_dim, n - 1, 0, True, ks, vs)
    assert near(backend.download(out, np.float32, heads * head_dim).reshape(1, -1), want)


# (m, n, heads, kv_heads, head_dim, q_base, window): the fewest rows the tile takes, a second row tile of four rows, one
# head per kv head on a first chunk, a window that starts inside tiles, query rows past the cache, eight heads per kv
# head over many chunks, five and seven heads per kv head (a row tile ends inside a query row), one chunk
BATCHES = [(4, 2100, 24, 4, 256, 2096, 0), (22, 400, 24, 4, 256, 378, 0), (130, 130, 8, 8, 128, 0, 0), (101, 1500, 16, 2, 128, 1399, 300),
           (57, 160, 24, 4, 256, 120, 0), (129, 700, 4, 4, 128, 500, 130), (16, 2049, 16, 2, 256, 2033, 0), (40, 900, 15, 3, 128, 860, 70),
           (39, 640, 14, 2, 256, 601, 0), (600, 64, 4, 2, 128, 0, 0)]


@pytest.mark.parametrize("fmt", [1, 2, 3, 4])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim,q_base,window", BATCHES)
def test_batches_on_the_tensor_pipe(backend, oracle, fmt, m, n, heads, kv_heads, head_dim, q_base, window):
    """Batches of query rows (two binary16 terms per query element and weight, exact cache elements): fp32 rounding."""
    g = np.random.default_rng(50 + fmt + m)
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32) * np.float32(10.0) ** g.integers(-3, 2, (m, 1)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, q_base, window, True, row_base=1)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, q_base, window, True, ks, vs)
    assert near(y, r)


# (m, n, heads, kv_heads, head_dim, q_base, window): one key, fewer keys than a warp's sixteen, a chunk that ends inside a
# warp's keys, eight rows of the sixteen over two row tiles, a window whose first keys leave chunks empty for the last row,
# sixteen chunks of unequal length, query rows past the cache, five heads per kv head; then the first rows of a long cache,
# where most CTAs of a cluster (counted on all keys) have none and still take part in the merge, in both row widths; sixteen
# CTAs of which the last has no key; batches in several clusters a kv head of eight, four and two CTAs
FEW = [(1, 1, 24, 4, 256, 0, 0), (1, 13, 8, 8, 128, 12, 0), (1, 1000, 8, 1, 128, 900, 0), (3, 333, 16, 2, 256, 330, 0),
       (3, 500, 6, 1, 128, 450, 70), (1, 4097, 24, 4, 256, 4096, 0), (2, 64, 12, 4, 256, 70, 0), (2, 700, 10, 2, 128, 698, 0),
       (1, 4096, 8, 2, 128, 0, 0), (1, 4096, 24, 4, 256, 20, 0), (3, 4096, 16, 2, 128, 5, 0), (2, 3000, 24, 4, 256, 0, 0),
       (1, 129, 8, 2, 128, 128, 0), (9, 150, 24, 4, 256, 141, 0), (70, 90, 16, 4, 128, 20, 0), (200, 70, 16, 4, 128, 0, 33)]


@pytest.mark.parametrize("fmt", [2, 3, 4])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim,q_base,window", FEW)
def test_few_rows_on_the_tensor_pipe(backend, oracle, fmt, m, n, heads, kv_heads, head_dim, q_base, window):
    """A cluster per kv head and sixteen (row, head) pairs (two binary16 terms per query element and weight, exact cache
    elements): fp32 rounding."""
    g = np.random.default_rng(80 + fmt + n)
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32) * np.float32(10.0) ** g.integers(-3, 2, (m, 1)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, q_base, window, True, row_base=1)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, q_base, window, True, ks, vs)
    assert near(y, r)


def test_few_rows_with_nonfinite_values(backend, oracle):
    """Two rows of which only the second sees a key whose scale is infinite and a NaN value."""
    g = np.random.default_rng(90)
    m, n, heads, kv_heads, head_dim = 2, 200, 8, 2, 128
    q = np.abs(g.standard_normal((m, heads * head_dim))).astype(np.float32)
    k, v, ks, vs = make_cache(g, 4, n, kv_heads * head_dim)
    v[n - 1] = 0x7F
    ks[n - 1] = np.inf
    y = device_attention(backend, 4, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, n - 2, 0, True)
    r = oracle.attention(4, q, k, v, m, n, heads, kv_heads, head_dim, n - 2, 0, True, ks, vs).reshape(y.shape)
    assert near(y[:1], r[:1])
    assert np.isnan(y[1:]).all() and np.isnan(r[1:]).all()


def test_batch_without_causal_mask(backend, oracle):
    g = np.random.default_rng(60)
    m, n, heads, kv_heads, head_dim = 320, 333, 8, 2, 128
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, 1, n, kv_heads * head_dim)
    y = device_attention(backend, 1, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, 0, 0, False)
    assert near(y, oracle.attention(1, q, k, v, m, n, heads, kv_heads, head_dim, 0, 0, False, ks, vs))


@pytest.mark.parametrize("fmt", [1, 4])
def test_nonfinite_values_reach_only_the_rows_that_see_them(backend, oracle, fmt):
    """A NaN value in key 250 and an infinite fp16 key 255: rows at positions below see neither."""
    g = np.random.default_rng(70 + fmt)
    m, n, heads, kv_heads, head_dim = 120, 300, 8, 2, 128
    q = np.abs(g.standard_normal((m, heads * head_dim))).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    if fmt == 1:
        v.view(np.float16)[250] = np.nan
        k.view(np.float16)[255, 3] = -np.inf
    else:
        v[250] = 0x7F
    y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, n - m, 0, True)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, n - m, 0, True, ks, vs).reshape(y.shape)
    clean = 250 - (n - m)
    assert near(y[:clean], r[:clean])
    assert np.isnan(y[clean:]).all() and np.isnan(r[clean:]).all()


# (m, n, heads, kv_heads, head_dim) of both kernels: row tiles over few and many chunks and over one, a cluster of one and
# of many CTAs with up to eight and up to sixteen rows
SHAPES = [(22, 400, 24, 4, 256), (40, 4000, 16, 2, 128), (600, 64, 4, 2, 128), (1, 300, 16, 2, 256), (1, 60, 8, 2, 128),
          (3, 1000, 24, 4, 128)]


@pytest.mark.parametrize("fmt", [2, 3, 4])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim", SHAPES)
def test_value_scales_of_unlike_size(backend, oracle, fmt, m, n, heads, kv_heads, head_dim):
    """Value scales over twelve decades, the largest on a key that only the last rows see, and a large one on a key of
    negligible weight: every row is as exact as its own keys allow, whatever the other keys' scales are (the weights of a
    row are split relative to that row's own largest contribution)."""
    g = np.random.default_rng(100 + fmt + n)
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    vs *= (10.0 ** g.uniform(-6, 6, n)).astype(np.float32)
    q_base = max(0, n - m)
    vs[n - max(1, min(m, n) // 2):] *= np.float32(1e9)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, q_base, 0, True, ks, vs)
    y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, q_base, 0, True)
    assert near_each(y, r, head_dim)


@pytest.mark.parametrize("fmt", [2, 3, 4])
@pytest.mark.parametrize("exponent", [112, 103, -118])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim", SHAPES)
def test_value_scales_at_the_ends_of_their_range(backend, oracle, fmt, exponent, m, n, heads, kv_heads, head_dim):
    """Finite value scales near the largest and the smallest fp32 numbers give finite results."""
    g = np.random.default_rng(110 + fmt + n)
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    if fmt == 4:
        v = np.where((v & 0x7F) > 0x40, v & 0xBF, v)      # |v| <= 2, so that the sums stay in range
    q_base = max(0, n - m)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, q_base, 0, True, ks, vs)
    factor = np.float32(2.0 ** (exponent + 7))            # vs is about 2^-7; a power of two changes nothing else
    y = device_attention(backend, fmt, q, k, v, ks, vs * factor, m, n, heads, kv_heads, head_dim, q_base, 0, True)
    assert np.isfinite(y).all()
    assert near_each(y / factor, r, head_dim)


@pytest.mark.parametrize("fmt,scale,value", [(2, "k", np.nan), (2, "v", np.inf), (3, "k", np.nan), (3, "v", -np.inf), (4, "v", np.nan)])
@pytest.mark.parametrize("m,n", [(120, 300), (2, 200)])
def test_nonfinite_scales_reach_only_the_rows_that_see_them(backend, oracle, fmt, scale, value, m, n):
    """A key in the middle of the rows' positions has a scale that is not finite: the rows before it are untouched, the
    others get the oracle's infinities and NaN."""
    g = np.random.default_rng(120 + fmt + m)
    heads, kv_heads, head_dim = 8, 2, 128
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    (ks if scale == "k" else vs)[n - m // 2] = value
    y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, n - m, 0, True)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, n - m, 0, True, ks, vs).reshape(y.shape)
    clean = m - m // 2
    assert near_each(y[:clean], r[:clean], head_dim)
    assert not np.isfinite(y[clean:]).any()
    assert np.array_equal(np.isnan(y), np.isnan(r)) and np.array_equal(np.isposinf(y), np.isposinf(r))


@pytest.mark.parametrize("fmt,bad", [(4, False), (4, True), (3, False), (1, False), (2, True)])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim", SHAPES)
def test_sigmoid_gate_inside_attention(backend, oracle, fmt, bad, m, n, heads, kv_heads, head_dim):
    """attention and the sigmoid_gate of its output, queued side by side, run as one operation: in the tile's own output,
    in the merge of its chunks and in a cluster's merge, also where a value that is not finite is among the keys."""
    g = np.random.default_rng(130 + fmt + m)
    q, gate = (g.standard_normal((m, heads * head_dim)).astype(np.float32) for _ in range(2))
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    if bad and fmt == 4:
        v[n - 1, 3] = 0x7F
    elif bad:
        vs[n - 1] = np.nan
    up, out = backend.upload, backend.AllocateBuffer(m * heads * head_dim * 4)
    bufs, tail = [up(q), up(k), up(v)], [n - m if n >= m else 0, 0, 0]
    if fmt >= 2:
        bufs += [up(ks), up(vs)]
    gb = up(gate)

    def kernels(gated):
        before = backend.LaunchStats()[1]
        run(backend, "attention" if fmt < 2 else QUANT_ID[fmt], bufs + [out],
            [m, n, heads, kv_heads, head_dim] + tail + ([fmt, 1] if fmt < 2 else [QUANT_KIND[fmt]]))
        if gated:
            run(backend, "sigmoid_gate", [out, gb, out], [m * heads * head_dim])
        backend.Synchronize()
        return backend.LaunchStats()[1] - before
    backend.Synchronize()
    backend.SetDeferred(2)
    try:
        alone, merged = kernels(False), kernels(True)
    finally:
        backend.SetDeferred(0)
    assert merged == alone
    y = backend.download(out, np.float32, q.size).reshape(m, -1)
    r = oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, tail[0], 0, True, ks, vs).reshape(m, -1)
    r = oracle.sigmoid_gate(r.reshape(-1), gate.reshape(-1)).reshape(m, -1)
    assert np.array_equal(np.isnan(y), np.isnan(r)) and np.isnan(y).any() == bad
    assert near(np.nan_to_num(y), np.nan_to_num(r))


@pytest.mark.parametrize("fmt", [3, 4])
@pytest.mark.parametrize("over", ["q", "v"])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim", SHAPES)
def test_result_over_an_input(backend, oracle, fmt, over, m, n, heads, kv_heads, head_dim):
    """In place over the queries (a CTA or a cluster reads its own rows first), and over the values (everything is read
    before anything is written)."""
    g = np.random.default_rng(140 + fmt + m)
    q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
    k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
    q_base = n - m if n >= m else 0
    qb, kb = backend.upload(q), backend.upload(k)
    vb = backend.upload(np.concatenate([v.reshape(-1), np.zeros(max(16, q.nbytes - v.nbytes), np.uint8)]))
    out = qb if over == "q" else vb
    run(backend, QUANT_ID[fmt], [qb, kb, vb, backend.upload(ks), backend.upload(vs), out],
        [m, n, heads, kv_heads, head_dim, q_base, 0, 0, QUANT_KIND[fmt]])
    y = backend.download(out, np.float32, q.size).reshape(m, -1)
    assert near(y, oracle.attention(fmt, q, k, v, m, n, heads, kv_heads, head_dim, q_base, 0, True, ks, vs).reshape(m, -1))


def decoded64(fmt, cache, scale, n):
    """A cache in 64 bits."""
    if fmt == 1:
        return cache.view(np.float16).reshape(n, -1).astype(np.float64)
    if fmt == 2:
        x = cache.view(np.int8).astype(np.float64)
    elif fmt == 3:
        x = np.stack([cache & 15, cache >> 4], 2).reshape(n, -1).astype(np.float64)
        x = np.where(x >= 8, x - 16, x)
    else:
        mag, man = (cache >> 3) & 15, (cache & 7).astype(np.float64)
        x = np.where(mag == 0, man / 8 * 2.0 ** -6, (1 + man / 8) * 2.0 ** (mag.astype(np.float64) - 7))
        x = np.where(cache & 0x80, -x, x)
    return x.reshape(n, -1) * scale.astype(np.float64)[:, None]


def attention64(q, k, v, heads, kv_heads, head_dim, q_base):
    m, n = q.shape[0], k.shape[0]
    hidden = np.arange(n)[None] > q_base + np.arange(m)[:, None]
    q, k, v = (x.reshape(-1, h, head_dim).astype(np.float64) for x, h in ((q, heads), (k, kv_heads), (v, kv_heads)))
    out = np.empty_like(q)
    for h in range(heads):
        s = q[:, h] @ k[:, h * kv_heads // heads].T / np.sqrt(head_dim)
        s[hidden] = -np.inf
        w = np.exp(s - s.max(1, keepdims=True))
        out[:, h] = (w / w.sum(1, keepdims=True)) @ v[:, h * kv_heads // heads]
    return out.reshape(m, -1)


@pytest.mark.parametrize("fmt", [1, 2, 3, 4])
@pytest.mark.parametrize("m,n,heads,kv_heads,head_dim,draws", [(96, 2048, 16, 2, 256, 2), (160, 1500, 8, 2, 128, 3), (1, 4096, 24, 4, 256, 12),
                                                               (3, 2000, 16, 2, 128, 12)])
def test_as_close_to_64_bits_as_fp32_sums(backend, fmt, m, n, heads, kv_heads, head_dim, draws):
    """The tensor-pipe kernels against attention_*_split and attention_combine, whose products and sums are fp32 throughout:
    the error (2-norm, over all draws) is no larger, on keys and values of unit size.  2 %: the spread between draws."""
    mine = chunks = 0.0
    for seed in range(draws):
        g = np.random.default_rng(1000 * fmt + seed)
        q = g.standard_normal((m, heads * head_dim)).astype(np.float32)
        k, v, ks, vs = make_cache(g, fmt, n, kv_heads * head_dim)
        if fmt == 4:
            k, v = (torch.from_numpy(np.clip(g.standard_normal(x.shape).astype(np.float32) * 100, -448, 448)).to(torch.float8_e4m3fn).view(torch.uint8).numpy() for x in (k, v))
        ks, vs = (g.uniform(0.5, 1.5, n).astype(np.float32) / np.float32({1: 1, 2: 74, 3: 4.6, 4: 100}[fmt]) for _ in range(2))
        want = attention64(q, decoded64(fmt, k, ks, n), decoded64(fmt, v, vs, n), heads, kv_heads, head_dim, n - m)
        y = device_attention(backend, fmt, q, k, v, ks, vs, m, n, heads, kv_heads, head_dim, n - m, 0, True)
        split = min(64, n // 64)
        bufs = [backend.upload(x) for x in ((q, k, v) if fmt == 1 else (q, k, v, ks, vs))]
        parts = [backend.AllocateBuffer(m * heads * split * c * 4) for c in (head_dim, 1, 1)]
        out = backend.AllocateBuffer(q.nbytes)
        run(backend, "attention_split" if fmt == 1 else QUANT_ID[fmt] + "_split", bufs + parts,
            [m, n, heads, kv_heads, head_dim, n - m, 0] + ([1, 1] if fmt == 1 else [QUANT_KIND[fmt]]) + [split])
        run(backend, "attention_combine", parts + [out], [m, heads, head_dim, split])
        x = backend.download(out, np.float32, q.size).reshape(q.shape)
        mine += float(np.sum((y - want) ** 2) / np.sum(want ** 2))
        chunks += float(np.sum((x - want) ** 2) / np.sum(want ** 2))
    print("error %.3e, fp32 sums %.3e" % ((mine / draws) ** 0.5, (chunks / draws) ** 0.5))
    assert mine <= 1.04 * chunks      # (1.02 ** 2)
