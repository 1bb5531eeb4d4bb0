"""Parity of the CUDA path with the CPU oracle, through the C ABI, on a B200.

Modelled on the reference's generic device suite (gpu/tests.rs): the same
deterministic generator, the same shape lists, the same two error checks —
plus bit-exact checks of the decoders and quantizers, the committed golden
cases, and the stricter "max relative error 1e-3" bar.
"""
import json
import os

import numpy as np
import pytest

from conftest import close, close_batch, max_rel_err

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
KATS = json.load(open(os.path.join(HERE, "golden", "reference_kats.json")))
FORMATS = ("q4_k", "q6_k", "q8_0")

# max |got - want| / max(|want|, rms(want)); the matmul bar
TOL = 1e-3


def kcols(fmt, cols):
    """The reference's shapes with cols made whole blocks of the format."""
    per = 32 if fmt == "q8_0" else 256
    return (cols + per - 1) // per * per


def lcg_weights(oracle, rng, fmt, rows, cols):
    """Rng::q8_0-style (gpu/tests.rs:87-103): a row of LCG floats at a time, quantized."""
    w = rng.floats(rows * cols).reshape(rows, cols)
    return oracle.quantize(fmt, w)


def upload(dev, fmt, rows, cols, blocks):
    from dwim_b200 import Tensor
    return dev.upload(Tensor(fmt, (rows, cols), blocks))


def random_pair(dev, oracle, fmt, rows, cols, rng):
    """A matrix of N(0, 0.02) weights and the same rows in another order, uploaded, and what the oracle decodes
    from their blocks, in double precision: (matrix, its weights, reordered matrix, its weights)."""
    blocks = dev.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)).data.reshape(rows, -1)
    other = np.roll(blocks, 1, axis=0)
    w = oracle.dequantize(fmt, blocks.reshape(-1), rows, cols).reshape(rows, cols).astype(np.float64)
    return (upload(dev, fmt, rows, cols, blocks.reshape(-1)), w, upload(dev, fmt, rows, cols, np.ascontiguousarray(other).reshape(-1)),
            np.roll(w, 1, axis=0))


def silu_times(gate, up):
    return gate / (1 + np.exp(-gate)) * up


# ---- device plumbing (gpu/tests.rs:166-186, 962-975) --------------------------------
def test_write_and_read_round_trip(dev, oracle):
    data = oracle.Lcg(1).floats(100_003)
    assert np.array_equal(dev.read(dev.buffer(data)), data)


def test_alloc_is_zeroed_and_resize_keeps_capacity(dev):
    from dwim_b200 import DeviceError
    buf = dev.alloc(1000)
    assert not dev.read(buf).any()
    dev.write(buf, np.arange(1000, dtype=np.float32))
    dev.resize(buf, 10)
    assert np.array_equal(dev.read(buf), np.arange(10, dtype=np.float32))
    dev.resize(buf, 1000)
    assert np.array_equal(dev.read(buf)[:10], np.arange(10, dtype=np.float32))
    with pytest.raises(DeviceError):
        dev.resize(buf, 1001)
    assert len(dev.read(dev.alloc(0))) == 0


def test_device_reports_itself(dev):
    assert "B200" in dev.name()
    assert dev.memory() > 1 << 30
    assert dev.batch() == 2048


# ---- decoders: bit-exact -----------------------------------------------------------------
@pytest.mark.parametrize("fmt", FORMATS)
def test_dequantize_is_bit_exact(dev, oracle, fmt):
    rng = np.random.default_rng(21)
    for rows, cols in [(1, 256), (37, 1024), (300, 5120)]:
        w = (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)
        blocks = oracle.quantize(fmt, w)
        got = dev.dequantize(upload(dev, fmt, rows, cols, blocks))
        want = oracle.dequantize(fmt, blocks, rows, cols)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("fmt", FORMATS)
def test_dequantize_random_bit_patterns_is_bit_exact(dev, oracle, fmt):
    """Every field at arbitrary values, not only what a quantizer emits."""
    from dwim_b200 import row_bytes
    rng = np.random.default_rng(22)
    rows, cols = 64, 1024
    blocks = rng.integers(0, 256, rows * row_bytes(fmt, cols), dtype=np.uint8)
    # keep the f16 scales finite (inf/nan scales are not weights)
    size = {"q4_k": 144, "q6_k": 210, "q8_0": 34}[fmt]
    b = blocks.reshape(-1, size)
    for off in {"q4_k": (1, 3), "q6_k": (209,), "q8_0": (1,)}[fmt]:
        b[:, off] &= 0x3B          # exponent below 0x1f
    got = dev.dequantize(upload(dev, fmt, rows, cols, blocks))
    want = oracle.dequantize(fmt, blocks, rows, cols)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def test_q6_k_known_answers_on_the_device(dev, oracle):
    # inference/quants.rs:236-275, decoded by the device
    block = np.zeros(210, np.uint8)
    block[37], block[128 + 5], block[192 + 2] = 0b1010, 0b1100, 3
    block[208:210] = np.frombuffer(oracle.to_f16([0.25]).tobytes(), np.uint8)
    out = dev.dequantize(upload(dev, "q6_k", 1, 256, block))[0]
    assert out[37] == 19.5 and all(out[i] == -24.0 for i in range(32, 48) if i != 37)
    assert not out[:32].any() and not out[48:].any()


@pytest.mark.parametrize("fmt", FORMATS)
def test_quantize_is_byte_exact(dev, oracle, fmt):
    rng = np.random.default_rng(23)
    w = (0.02 * rng.standard_normal((96, 2048))).astype(np.float32)
    w[0, :256] = 0.0
    w[1, 7] = 5.0
    w[2, :64] = np.float32(1e-30)
    w[3, 300] = -65536.0
    assert np.array_equal(dev.quantize(fmt, w).data, oracle.quantize(fmt, w))
    lcg = oracle.Lcg(5).floats(64 * 512).reshape(64, 512)
    assert np.array_equal(dev.quantize(fmt, lcg).data, oracle.quantize(fmt, lcg))


# ---- matmul ---------------------------------------------------------------------------
@pytest.mark.parametrize("fmt", FORMATS)
def test_block_matmul_matches_cpu(dev, oracle, fmt):
    """block_matmul_matches_cpu (gpu/tests.rs:219-262): the reference's shapes, its
    generator (weights Rng(80) shape after shape, x = Rng(rows + n)), its checks."""
    rng = oracle.Lcg(80)
    for rows, cols, n in KATS["matmul_shapes"]["shapes"]:
        cols = kcols(fmt, cols)
        blocks = lcg_weights(oracle, rng, fmt, rows, cols)
        x = oracle.Lcg(rows + n).floats(n * cols)
        want = oracle.matmul(fmt, blocks, rows, cols, x)
        out = dev.alloc(n * rows)
        dev.matmul(out, upload(dev, fmt, rows, cols, blocks), dev.buffer(x))
        got = dev.read(out).reshape(n, rows)
        what = f"{fmt} {rows}x{cols} n={n}"
        if n == 1:
            close(got, want, 1e-4)
        close_batch(got, want, what)
        assert max_rel_err(got, want) <= TOL, what


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17])
def test_matmul_token_counts_at_model_width(dev, oracle, fmt, n):
    rng = np.random.default_rng(31 + n)
    rows, cols = 333, 5120
    blocks = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    x = rng.standard_normal((n, cols)).astype(np.float32)
    out = dev.alloc(n * rows)
    dev.matmul(out, upload(dev, fmt, rows, cols, blocks), dev.buffer(x))
    got, want = dev.read(out).reshape(n, rows), oracle.matmul(fmt, blocks, rows, cols, x)
    assert max_rel_err(got, want) <= TOL
    # the small-M kernel keeps products exact: expect fp32-summation noise only
    assert max_rel_err(got, want) <= 2e-5


@pytest.mark.parametrize("fmt", FORMATS)
def test_matmul_bf16_activations(dev, oracle, fmt):
    """Config 2's inputs: rows of N(0,1) scaled to RMS 1, rounded to bf16."""
    rng = np.random.default_rng(41)
    rows, cols = 1000, 5120
    blocks = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    weight = upload(dev, fmt, rows, cols, blocks)
    for n in (1, 7, 16):
        x = rng.standard_normal((n, cols)).astype(np.float32)
        x /= np.sqrt((x * x).mean(1, keepdims=True))
        bits = oracle.to_bf16(x)
        xb = dev.alloc(n * cols)
        dev.write_bf16(xb, bits)
        assert np.array_equal(dev.read(xb), oracle.bf16(bits))
        out = dev.alloc(n * rows)
        dev.matmul(out, weight, xb)
        want = oracle.matmul(fmt, blocks, rows, cols, oracle.bf16(bits))
        assert max_rel_err(dev.read(out).reshape(n, rows), want) <= 2e-5


@pytest.mark.parametrize("fmt", FORMATS)
def test_matmul_golden_cases(dev, fmt):
    """The committed oracle outputs (tests/golden/oracle_cases.npz)."""
    g = np.load(os.path.join(HERE, "golden", "oracle_cases.npz"))
    w, x, blocks = g[f"{fmt}_w"], g[f"{fmt}_x"], g[f"{fmt}_blocks"]
    rows, cols = w.shape
    n = x.shape[0]
    assert np.array_equal(dev.quantize(fmt, w).data, blocks)
    weight = upload(dev, fmt, rows, cols, blocks)
    assert np.array_equal(dev.dequantize(weight).view(np.uint32), g[f"{fmt}_dequant"].view(np.uint32))
    out, scratch = dev.alloc(n * rows), dev.alloc(n * rows)
    dev.matmul(out, weight, dev.buffer(x))
    assert max_rel_err(dev.read(out), g[f"{fmt}_matmul"]) <= 2e-5
    dev.swiglu(out, weight, upload(dev, fmt, rows, cols, g[f"{fmt}_up_blocks"]), dev.buffer(x), scratch)
    assert max_rel_err(dev.read(out), g[f"{fmt}_swiglu"]) <= 1e-4


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("rows,cols", [(2384, 1024), (2400, 5120), (7105, 768), (9500, 1280), (17, 6144), (2369, 6400), (65, 17408), (33, 30464),
                                       (40, 70400), (7105, 5888), (7200, 5120)])
def test_small_m_row_tiles_and_boxes(dev, oracle, fmt, rows, cols):
    """One to four row tiles a CTA (ragged last tiles), whole rows and boxes of odd numbers of units (a last
    box that is part padding, part past the row), planes resident and travelling, up to a row too long for
    more than one row tile; the three epilogues.  Eight tokens round an activation at 2^-23 of its unit's
    largest: 1e-5 of the result's root mean square is sixty times that."""
    rng = np.random.default_rng(rows + cols)
    weight, w, other, w2 = random_pair(dev, oracle, fmt, rows, cols, rng)
    for n in (1, 2, 3, 5, 8):
        x = rng.standard_normal((n, cols)).astype(np.float32)
        res = rng.standard_normal((n, rows)).astype(np.float32)
        xb, out, acc = dev.buffer(x), dev.alloc(n * rows), dev.buffer(res)
        want = x.astype(np.float64) @ w.T
        bar = 1e-5 * np.sqrt((want ** 2).mean())
        dev.matmul(out, weight, xb)
        assert np.abs(dev.read(out).reshape(n, rows) - want).max() <= bar, n
        dev.matmul_add(acc, weight, xb)
        assert np.abs(dev.read(acc).reshape(n, rows) - (want + res)).max() <= bar + 1e-6, n
        dev.swiglu(out, weight, other, xb, dev.alloc(n * rows))
        silu = silu_times(want, x.astype(np.float64) @ w2.T)
        assert np.abs(dev.read(out).reshape(n, rows) - silu).max() <= 4 * bar * max(1.0, np.abs(want).max()), n


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("fmt,rows,cols,n", [("q8_0", 100, 96, 530), ("q8_0", 300, 5120, 64), ("q8_0", 33, 2048, 17), ("q6_k", 2400, 768, 23),
                                             ("q6_k", 40, 6144, 41), ("q8_0", 16, 32, 9), ("q6_k", 48, 12544, 70)])
def test_groups_of_eight_tokens(dev, oracle, fmt, rows, cols, n, bf16):
    """Full groups in one launch (up to 64 of them), the rest in another (by f32 activations of 25 tokens and more, rows of
    whole units: the dense kernel); every token against the oracle's weights in double precision, 1e-5 of the result's
    root mean square as for eight tokens."""
    rng = np.random.default_rng(rows + n)
    weight, w, _, _ = random_pair(dev, oracle, fmt, rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    xb = dev.buffer(x)
    if bf16:
        bits = oracle.to_bf16(x)
        dev.write_bf16(xb, bits)
        x = oracle.bf16(bits).reshape(n, cols)
    want = x.astype(np.float64) @ w.T
    res = rng.standard_normal((n, rows)).astype(np.float32)
    out, acc = dev.alloc(n * rows), dev.buffer(res)
    bar = 1e-5 * np.sqrt((want ** 2).mean())
    dev.matmul(out, weight, xb)
    assert np.abs(dev.read(out).reshape(n, rows) - want).max() <= bar
    dev.matmul_add(acc, weight, xb)
    assert np.abs(dev.read(acc).reshape(n, rows) - (want + res)).max() <= bar + 1e-6


@pytest.mark.parametrize("bf16", [False, True])
def test_groups_under_capture(oracle, bf16):
    """A product of more than eight tokens captured into a CUDA graph after a warm-up at another token count
    (the buffer resized between): no allocation is needed there, and none made later takes away what a captured
    graph reads.  Every token as the eager product gives it.  (By f32 activations the longer ones are the dense
    kernel's.)"""
    import torch
    from dwim_b200 import B200, Tensor
    stream = torch.cuda.Stream()
    d = B200(0, stream=stream.cuda_stream)
    try:
        rng = np.random.default_rng(71)
        rows, cols, most = 96, 2048, 48
        blocks = oracle.quantize("q8_0", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
        weight = d.upload(Tensor("q8_0", (rows, cols), blocks))
        x = rng.standard_normal((most, cols)).astype(np.float32)
        if bf16:
            x = oracle.bf16(oracle.to_bf16(x)).reshape(most, cols)
        want = oracle.matmul("q8_0", blocks, rows, cols, x).reshape(most, rows)
        xb, out = d.buffer(x), d.alloc(most * rows)

        def at(n):
            d.resize(xb, n * cols)
            d.resize(out, n * rows)

        def right(n):
            got = d.read(out).reshape(n, rows)
            d.write(out, np.zeros(n * rows, np.float32))
            return max_rel_err(got, want[:n]) <= 2e-5

        def captured(n):
            at(n)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                d.matmul(out, weight, xb)
            return graph

        if bf16:
            d.touch_bf16(xb)
        at(8)
        d.matmul(out, weight, xb)
        assert right(8)
        graphs = {n: captured(n) for n in (most, 16)}
        at(most)
        d.matmul(out, weight, xb)                       # eager: the planes of all its groups at once, or the operand
        assert right(most)
        graphs[24] = captured(24)
        for n, graph in list(graphs.items()) * 2:
            at(n)
            with torch.cuda.stream(stream):
                graph.replay()
            assert right(n), n
        del graphs
    finally:
        d.close()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n", [40, 9, 16, 32, 130])
def test_q4_k_gemm_scale_extremes(dev, oracle, n, bf16):
    """The tensor-core kernel folds a block's minimums into the same accumulator
    as its quants, scaled by dmin/d: rows whose blocks have d = 0, dmin = 0, either
    sign, or dmin up to 2^40 times d must still match the CPU result."""
    rng = np.random.default_rng(47)
    rows, cols = 256, 1024
    blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)).copy()
    regimes = [(1e-3, 2e-3), (0.0, 0.05), (0.05, 0.0), (0.0, 0.0), (1e-3, 0.1), (1e-4, 6.0), (2.4e-7, 30.0),
               (6e-8, 60000.0), (-1e-3, 2e-3), (1e-3, -2e-3), (3e-5, 1.0), (1.0, 6e-8)]
    v = blocks.reshape(rows, cols // 256, 144)
    for r in range(rows):
        d, dmin = regimes[r % len(regimes)]
        v[r, :, 0:2] = np.frombuffer(np.float16(d).tobytes(), np.uint8)
        v[r, :, 2:4] = np.frombuffer(np.float16(dmin).tobytes(), np.uint8)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    xb = dev.alloc(n * cols)
    if bf16:
        bits = oracle.to_bf16(x)
        dev.write_bf16(xb, bits)
        x = oracle.bf16(bits).reshape(n, cols)
    else:
        dev.write(xb, x)
    out = dev.alloc(n * rows)
    dev.matmul(out, upload(dev, "q4_k", rows, cols, blocks), xb)
    got, want = dev.read(out).reshape(n, rows), oracle.matmul("q4_k", blocks, rows, cols, x).reshape(n, rows)
    for k, (d, dmin) in enumerate(regimes):
        g, w = got[:, k::len(regimes)], want[:, k::len(regimes)]
        if d == 0.0 and dmin == 0.0:
            assert not g.any() and not w.any()
        else:
            assert max_rel_err(g, w) <= 2e-5, f"d={d} dmin={dmin}: {max_rel_err(g, w):.2e}"


def test_shadow_is_rebuilt_after_a_write(dev, oracle):
    """One input buffer reused: across formats (different operand layouts) and
    after being overwritten."""
    rng = np.random.default_rng(43)
    rows, cols = 64, 512
    w = (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)
    xb, out = dev.alloc(2 * cols), dev.alloc(2 * rows)
    for trial in range(2):
        x = rng.standard_normal((2, cols)).astype(np.float32)
        dev.write(xb, x)
        for fmt in FORMATS:
            blocks = oracle.quantize(fmt, w)
            dev.matmul(out, upload(dev, fmt, rows, cols, blocks), xb)
            assert max_rel_err(dev.read(out), oracle.matmul(fmt, blocks, rows, cols, x)) <= 2e-5


# ---- fused operators (gpu/tests.rs:816-871) ---------------------------------------------
@pytest.mark.parametrize("fmt", FORMATS)
def test_swiglu_matches_cpu(dev, oracle, fmt):
    rng = oracle.Lcg(22)
    for rows, cols, n in KATS["fused_shapes"]["shapes"]:
        cols = kcols(fmt, cols)
        gate, up = lcg_weights(oracle, rng, fmt, rows, cols), lcg_weights(oracle, rng, fmt, rows, cols)
        x = rng.floats(n * cols)
        want = oracle.swiglu(fmt, gate, up, rows, cols, x)
        out, scratch = dev.alloc(n * rows), dev.alloc(n * rows)
        dev.swiglu(out, upload(dev, fmt, rows, cols, gate), upload(dev, fmt, rows, cols, up), dev.buffer(x), scratch)
        got = dev.read(out)
        close_batch(got, want, f"{fmt} {rows}x{cols} n={n}")
        assert max_rel_err(got, want) <= TOL


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 9])
def test_swiglu_one_launch_at_model_width(dev, oracle, fmt, n):
    """Up to eight tokens take gate and up in a single launch; nine go the
    two-launch way.  Rows that are not a whole tile, both ways against the CPU."""
    rng = np.random.default_rng(53 + n)
    rows, cols = 1000, 5120
    gate = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    up = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    x = rng.standard_normal((n, cols)).astype(np.float32)
    out, scratch = dev.alloc(n * rows), dev.alloc(n * rows)
    dev.swiglu(out, upload(dev, fmt, rows, cols, gate), upload(dev, fmt, rows, cols, up), dev.buffer(x), scratch)
    want = oracle.swiglu(fmt, gate, up, rows, cols, x)
    assert max_rel_err(dev.read(out), want) <= 2e-5


@pytest.mark.parametrize("fmt", FORMATS)
def test_matmul_add_matches_cpu(dev, oracle, fmt):
    rng = oracle.Lcg(23)
    for rows, cols, n in KATS["fused_shapes"]["shapes"]:
        cols = kcols(fmt, cols)
        blocks = lcg_weights(oracle, rng, fmt, rows, cols)
        inp, x = rng.floats(n * cols), rng.floats(n * rows)
        want = oracle.matmul_add(fmt, blocks, rows, cols, inp, x).ravel()
        out, scratch = dev.buffer(x), dev.alloc(n * rows)
        dev.matmul_add(out, upload(dev, fmt, rows, cols, blocks), dev.buffer(inp), scratch)
        got = dev.read(out)
        # what was added, which is what a batch's error is a part of
        close_batch(got - x, want - x, f"{fmt} {rows}x{cols} n={n}")
        assert max_rel_err(got - x, want - x) <= TOL


# ---- misuse is an error code, never a fault (the trait's panics) ------------------------------
def test_misuse_is_reported(dev, oracle):
    from dwim_b200 import DeviceError, Tensor
    rng = np.random.default_rng(47)
    blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((32, 512))).astype(np.float32))
    w = upload(dev, "q4_k", 32, 512, blocks)
    with pytest.raises(DeviceError):               # x is not rows of cols
        dev.matmul(dev.alloc(32), w, dev.alloc(500))
    with pytest.raises(DeviceError):               # out has the wrong length
        dev.matmul(dev.alloc(33), w, dev.alloc(512))
    with pytest.raises(DeviceError):               # write of the wrong length
        dev.write(dev.alloc(8), np.zeros(9, np.float32))
    with pytest.raises(DeviceError):               # gate and up differ
        w2 = upload(dev, "q4_k", 16, 512, blocks[: 16 * 288])
        dev.swiglu(dev.alloc(32), w, w2, dev.alloc(512), dev.alloc(32))
    L = dev._L
    import ctypes as C
    h = C.c_void_p()
    assert L.dwim_b200_upload(dev._ctx, 12, 32, 512, blocks.ctypes.data, blocks.size - 1, C.byref(h)) == -1   # truncated
    assert L.dwim_b200_upload(dev._ctx, 2, 32, 512, blocks.ctypes.data, blocks.size, C.byref(h)) == -2        # Q4_0: unknown here
    assert L.dwim_b200_upload(dev._ctx, 12, 32, 500, blocks.ctypes.data, blocks.size, C.byref(h)) == -2       # not whole blocks
    assert b"blocks" in L.dwim_b200_last_error(dev._ctx)
    # the device still works afterwards
    out = dev.alloc(32)
    x = rng.standard_normal(512).astype(np.float32)
    dev.matmul(out, w, dev.buffer(x))
    assert max_rel_err(dev.read(out), oracle.matmul("q4_k", blocks, 32, 512, x)) <= 2e-5
    dev.sync()


def test_empty_inputs(dev, oracle):
    blocks = oracle.quantize("q8_0", np.ones((4, 64), np.float32))
    w = upload(dev, "q8_0", 4, 64, blocks)
    dev.matmul(dev.alloc(0), w, dev.alloc(0))       # no tokens
    w0 = upload(dev, "q8_0", 0, 64, np.zeros(0, np.uint8))
    dev.matmul(dev.alloc(0), w0, dev.alloc(64))     # no rows
    dev.sync()


# ---- BASELINE's full sizes: oracle on a row sample + size-independent properties ------------------
def full_size_case(dev, oracle, fmt, rows, cols, n, seed, bf16=False):
    rng = np.random.default_rng(seed)
    w = (0.02 * rng.standard_normal((rows, cols), dtype=np.float32)).astype(np.float32)
    t = dev.quantize(fmt, w)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    weight = dev.upload(t)
    xb = dev.alloc(n * cols)
    if bf16:
        bits = oracle.to_bf16(x)
        x = oracle.bf16(bits).reshape(n, cols)
        dev.write_bf16(xb, bits)
    else:
        dev.write(xb, x)
    out = dev.alloc(n * rows)
    dev.matmul(out, weight, xb)
    got = dev.read(out).reshape(n, rows)
    # (1) the oracle on every row
    want = oracle.matmul(fmt, t.data, rows, cols, x)
    assert max_rel_err(got, want) <= TOL
    # (2) the device quantizer wrote the oracle's bytes (a row sample) and decodes them bit-exactly
    sample = rng.choice(rows, 64, replace=False)
    assert np.array_equal(t.select_rows(sample).data, oracle.quantize(fmt, w[sample]))
    # (3) linearity: W.(2x) = 2 W.x (a power of two scales every term; only
    # f16-subnormal remainders of tiny activations can round differently)
    dev.write(xb, 2.0 * x)
    out2 = dev.alloc(n * rows)
    dev.matmul(out2, weight, xb)
    assert max_rel_err(dev.read(out2).reshape(n, rows), 2.0 * got) <= 1e-6
    # (4) a second run gives the same bits (fixed summation order)
    dev.write(xb, x)
    dev.matmul(out2, weight, xb)
    assert np.array_equal(dev.read(out2).reshape(n, rows), got)
    return got, want


def test_config1_q4_k_gemv_full_size(dev, oracle):
    """Q4_K [17408, 5120] . x[1, 5120], W seed 0, x seed 1."""
    w = (0.02 * np.random.default_rng(0).standard_normal((17408, 5120), dtype=np.float32))
    x = np.random.default_rng(1).standard_normal((1, 5120)).astype(np.float32)
    t = dev.quantize("q4_k", w)
    assert t.data.size == 50_135_040
    weight = dev.upload(t)
    assert np.array_equal(dev.dequantize(weight).view(np.uint32),
                          oracle.dequantize("q4_k", t.data, 17408, 5120).view(np.uint32))
    out = dev.alloc(17408)
    dev.matmul(out, weight, dev.buffer(x))
    got, want = dev.read(out), oracle.matmul("q4_k", t.data, 17408, 5120, x).ravel()
    close(got, want, 1e-4)
    assert max_rel_err(got, want) <= 2e-5
    # against the unquantized product: within quantization noise (a sanity check on the format itself)
    exact = (w.astype(np.float64) @ x[0].astype(np.float64))
    assert np.sqrt(np.mean((got - exact) ** 2)) < 0.12 * np.sqrt(np.mean(exact ** 2))


@pytest.mark.parametrize("fmt,rows,cols,n", [
    ("q4_k", 12288, 5120, 8), ("q8_0", 5120, 5120, 8), ("q4_k", 5120, 17408, 4), ("q6_k", 151936, 5120, 1)])
def test_config3_shapes_full_size(dev, oracle, fmt, rows, cols, n):
    full_size_case(dev, oracle, fmt, rows, cols, n, seed=3)


def test_config2_q4_k_m16_bf16_full_size(dev, oracle):
    full_size_case(dev, oracle, "q4_k", 17408, 5120, 16, seed=2, bf16=True)


# ---- sharding: the device's re-assembly against the host statement of it ---------------------
def test_gather_rows_matches_the_host_assembly(dev):
    from dwim_b200 import shard
    rng = np.random.default_rng(51)
    for rows, world, align, n in [(17408, 8, 16, 3), (5120, 2, 16, 16), (77, 4, 16, 2), (100, 3, 7, 5)]:
        pr = shard.part_rows(rows, world, align)
        parts = rng.standard_normal((world, n, pr)).astype(np.float32)
        out = dev.alloc(n * rows)
        dev.gather_rows(out, dev.buffer(parts), n, rows, world, align)
        assert np.array_equal(dev.read(out).reshape(n, rows), shard.assemble(parts, n, rows, world, align))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 40])
def test_feed_forward_block_on_one_gpu(dev, oracle, n):
    """ShardedFFN with a world of one: swiglu, then the down projection of the
    f32 intermediate, against the CPU's two steps."""
    from dwim_b200 import Tensor, shard
    rng = np.random.default_rng(61 + n)
    hidden, inner = 512, 1024
    mk = lambda r, c: Tensor("q4_k", (r, c), oracle.quantize("q4_k", (0.05 * rng.standard_normal((r, c))).astype(np.float32)))
    gate, up, down = mk(inner, hidden), mk(inner, hidden), mk(hidden, inner)
    x = rng.standard_normal((n, hidden)).astype(np.float32)
    block = shard.ShardedFFN(dev, gate, up, down)
    got = dev.read(block.forward(dev.buffer(x))).reshape(n, hidden)
    h = oracle.swiglu("q4_k", gate.data, up.data, inner, hidden, x)
    want = oracle.matmul("q4_k", down.data, hidden, inner, h).reshape(n, hidden)
    assert max_rel_err(got, want) <= 5e-5


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n", [1, 2, 5, 8])
def test_int8_routine_activation_extremes(dev, oracle, fmt, n):
    """Up to eight tokens go through int8 digit planes with one exponent per 256
    activations: outliers, zeros, a zero unit, tiny and huge magnitudes."""
    rng = np.random.default_rng(71 + n)
    rows, cols = 96, 2048
    blocks = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    weight = upload(dev, fmt, rows, cols, blocks)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    x[:, 7] = 3.0e4                   # an outlier in the first unit
    x[:, 256:512] = 0.0               # a unit of zeros
    x[:, 512:768] *= 1e-30            # tiny
    x[:, 768:1024] *= 1e20            # huge
    x[:, 1024:1280:2] = 0.0           # every other one zero
    x[:, 1300] = -65504.0
    out = dev.alloc(n * rows)
    dev.matmul(out, weight, dev.buffer(x))
    got, want = dev.read(out).reshape(n, rows), oracle.matmul(fmt, blocks, rows, cols, x)
    assert np.isfinite(got).all()
    # three digit planes (three to eight tokens) round an activation at 2^-23 of its unit's largest
    assert max_rel_err(got, want) <= (2e-5 if n <= 2 else 1e-4)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("scale", [1e5, 1e20, 1e-30])
def test_gemm_activation_range(dev, oracle, scale, bf16):
    """Forty tokens through the tensor-core kernel with activations far outside
    f16's range: every token's row is scaled by its own power of two on the way in
    and back on the way out, so nothing is clamped or flushed."""
    rng = np.random.default_rng(79)
    rows, cols, n = 256, 1024, 40
    blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    x = rng.standard_normal((n, cols)).astype(np.float32)
    x[::2] *= np.float32(scale)               # every other token: neighbours keep their own range
    x[1, 7] = 3.0e4
    xb = dev.alloc(n * cols)
    if bf16:
        bits = oracle.to_bf16(x)
        dev.write_bf16(xb, bits)
        x = oracle.bf16(bits).reshape(n, cols)
    else:
        dev.write(xb, x)
    out = dev.alloc(n * rows)
    dev.matmul(out, upload(dev, "q4_k", rows, cols, blocks), xb)
    got, want = dev.read(out).reshape(n, rows), oracle.matmul("q4_k", blocks, rows, cols, x)
    assert np.isfinite(got).all()
    for t in range(n):                         # per token: the tokens' magnitudes differ by up to 10^30
        assert max_rel_err(got[t], want[t]) <= 2e-5, (t, max_rel_err(got[t], want[t]))


@pytest.mark.parametrize("cols", [256, 1024, 3328, 5120, 5376, 6144, 10496, 18432, 18688, 26880])
@pytest.mark.parametrize("n,norm", [(9, False), (9, True), (40, False), (150, True), (300, False)])
def test_gemm_operand_rows_of_every_length(dev, oracle, cols, n, norm):
    """The tensor-core kernels' operand, rows held by one block or a cluster's, in whole chunks of 1024 and 2048 and
    a rest: a norm's row and its product, an infinite and a NaN activation that stay their token's own."""
    rng = np.random.default_rng(cols + n)
    rows = 16
    blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    w = oracle.dequantize("q4_k", blocks, rows, cols).reshape(rows, cols).astype(np.float64)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    x[2, cols - 1] = 50.0
    out, xb = dev.alloc(n * rows), dev.buffer(x)
    x = x.astype(np.float64)
    if norm:
        gain = (1 + 0.1 * rng.standard_normal(cols)).astype(np.float32)
        xn = dev.alloc(n * cols)
        dev.normalize(xn, xb, dev.buffer(gain), n * cols, 1e-6)
        x = x / np.sqrt((x * x).mean(1, keepdims=True) + 1e-6) * gain
        # scale and product rounded to fp32 each, a sum of cols terms: a few 2^-24
        assert max_rel_err(dev.read(xn), x) <= 2e-6
        xb = xn
    elif n == 9:
        bad = x.astype(np.float32)
        bad[4, cols // 2], bad[5, 3] = np.inf, np.nan
        dev.write(xb, bad)
    dev.matmul(out, upload(dev, "q4_k", rows, cols, blocks), xb)
    got, want = dev.read(out).reshape(n, rows), x @ w.T
    assert np.isfinite(got).all()
    good = [t for t in range(n) if norm or n != 9 or t not in (4, 5)]
    # fp32 sums of up to 26880 products, f16 pairs for the activations (2^-22): 1e-5 of the result's magnitude
    assert max_rel_err(got[good], want[good]) <= 1e-5


# ---- the operators either side of the product (the norm before it, the arg-max after it, bf16 matrices) ----
def test_normalize_matches_cpu(dev, oracle):
    """normalize_matches_cpu (gpu/tests.rs:788-812): the reference's shapes and
    generator; then the model's width, where the same launch also writes the next
    product's operand form: the product of the normalized rows must match too."""
    rng = oracle.Lcg(21)
    for dim, rows in KATS["normalize_shapes"]["shapes"]:
        w, x = rng.floats(dim), rng.floats(dim * (rows + 1))
        rng.floats(dim * rows)                 # the reference draws y for its add check here
        out = dev.alloc(dim * rows)
        dev.normalize(out, dev.buffer(x), dev.buffer(w), dim * rows, 1e-6)
        close(dev.read(out), oracle.rmsnorm(x[: dim * rows], w, 1e-6), 1e-5)
    g = np.random.default_rng(83)
    cols, wrows = 5120, 320
    blocks = oracle.quantize("q4_k", (0.02 * g.standard_normal((wrows, cols))).astype(np.float32))
    weight = upload(dev, "q4_k", wrows, cols, blocks)
    for n in (1, 2, 5, 8, 12, 40, 300):
        x = (3.0 * g.standard_normal((n, cols))).astype(np.float32)
        w = (1.0 + 0.1 * g.standard_normal(cols)).astype(np.float32)
        normed, out = dev.alloc(n * cols), dev.alloc(n * wrows)
        dev.normalize(normed, dev.buffer(x), dev.buffer(w), n * cols, 1e-6)
        launches = dev.launches
        dev.matmul(out, weight, normed)
        want_n = oracle.rmsnorm(x, w, 1e-6)
        close(dev.read(normed), want_n, 1e-5)
        # the device's own normalized rows (they differ from the CPU's by summation order) through the oracle
        want = oracle.matmul("q4_k", blocks, wrows, cols, dev.read(normed).reshape(n, cols))
        assert max_rel_err(dev.read(out), want) <= (2e-5 if n <= 2 or n > 8 else 1e-4), n
        assert dev.launches - launches == 1, "the product ran an activation prologue of its own"


@pytest.mark.parametrize("dim", [256, 1024, 1280, 5120, 8192, 8448, 17408])
@pytest.mark.parametrize("n", [1, 5, 8])
def test_normalize_in_place_across_blocks(dev, oracle, dim, n):
    """A row dealt to one to eight blocks, whole rounds and remainders, the output over the input;
    then a product that reads the digit planes of the same launch.  The norm's own error: a few
    roundings of 2^-24 beside those of the sum of squares."""
    rng = np.random.default_rng(dim + n)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    gain = (1 + 0.1 * rng.standard_normal(dim)).astype(np.float32)
    buf = dev.buffer(x)
    dev.normalize(buf, buf, dev.buffer(gain), n * dim, 1e-6)
    x64 = x.astype(np.float64)
    want = x64 / np.sqrt((x64 ** 2).mean(axis=1, keepdims=True) + 1e-6) * gain
    got = dev.read(buf).reshape(n, dim)
    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max()
    blocks = oracle.quantize("q8_0", (0.02 * rng.standard_normal((48, dim))).astype(np.float32))
    out = dev.alloc(n * 48)
    dev.matmul(out, upload(dev, "q8_0", 48, dim, blocks), buf)
    ref = want @ oracle.dequantize("q8_0", blocks, 48, dim).astype(np.float64).reshape(48, dim).T
    assert max_rel_err(dev.read(out).reshape(n, 48), ref.astype(np.float32)) <= 2e-5


def test_bf16_matmul_matches_cpu(dev, oracle):
    """matmul_matches_cpu (gpu/tests.rs:178-196): bf16 weights, the reference's
    shapes, generator and tolerance; and the gate matrices' shape in the model."""
    from dwim_b200 import Tensor
    rng = oracle.Lcg(4)
    shapes = [tuple(s) for s in KATS["bf16_matmul_shapes"]["shapes"]] + [(96, 5120, 1), (96, 5120, 5)]
    for rows, cols, n in shapes:
        wbits = (rng.floats(rows * cols).view(np.uint32) >> 16).astype(np.uint16)   # Rng::bf16, gpu/tests.rs:60-68
        x = rng.floats(n * cols)
        weight = dev.upload(Tensor("bf16", (rows, cols), wbits))
        assert np.array_equal(dev.dequantize(weight), oracle.bf16(wbits).reshape(rows, cols))
        out = dev.alloc(n * rows)
        dev.matmul(out, weight, dev.buffer(x))
        close(dev.read(out), oracle.matmul_bf16(wbits, rows, cols, x), 1e-4)


@pytest.mark.parametrize("rows,cols,n", [(1, 8, 1), (33, 2048, 3), (5, 2056, 8), (96, 5120, 16), (3, 8, 17), (33, 520, 64), (31, 72, 65), (33, 136, 128),
                                         (96, 5120, 129)])
def test_bf16_matmul_edges(dev, oracle, rows, cols, n):
    """Both kernels at the edges of their tiles (rows of 32, tokens of 32, K of 64 dealt to eight
    blocks), with the three epilogues.  fp32 sums of at most 5120 products: 1e-5 of the result's
    root mean square is sixteen times 2^-24 * sqrt(5120)."""
    from dwim_b200 import Tensor
    rng = np.random.default_rng(rows + cols + n)
    bits = oracle.to_bf16(rng.standard_normal((rows, cols)).astype(np.float32))
    w = oracle.bf16(bits).reshape(rows, cols).astype(np.float64)
    weight = dev.upload(Tensor("bf16", (rows, cols), bits.view(np.uint8)))
    x = rng.standard_normal((n, cols)).astype(np.float32)
    res = rng.standard_normal((n, rows)).astype(np.float32)
    want = x.astype(np.float64) @ w.T
    bar = 1e-5 * np.sqrt((want ** 2).mean())
    xb, out, acc = dev.buffer(x), dev.alloc(n * rows), dev.buffer(res)
    dev.matmul(out, weight, xb)
    assert np.abs(dev.read(out).reshape(n, rows) - want).max() <= bar
    dev.matmul_add(acc, weight, xb)
    assert np.abs(dev.read(acc).reshape(n, rows) - (want + res)).max() <= bar + 1e-6
    gated = dev.alloc(n * rows)
    dev.swiglu(gated, weight, weight, xb, dev.alloc(n * rows))
    silu = want / (1 + np.exp(-want)) * want
    assert np.abs(dev.read(gated).reshape(n, rows) - silu).max() <= 4 * bar * max(1.0, np.abs(want).max())


def test_argmax_on_the_device(dev, oracle):
    rng = np.random.default_rng(91)
    vocab = 151936
    for n in (1, 5):
        logits = rng.standard_normal((n, vocab)).astype(np.float32)
        logits[0, 777] = logits[0, 99999] = 9.0     # a tie: the first index wins (inference/qwen35/mod.rs:702-710)
        if n > 1:
            logits[1, :] = -np.inf
            logits[2, 5] = np.nan
            logits[3, 0] = 50.0
        got = dev.argmax(dev.buffer(logits), vocab)
        want = [oracle.argmax(row) for row in logits]
        assert got.tolist() == want


@pytest.mark.parametrize("n,length", [(1, 1), (1, 2048), (3, 2049), (8, 151936), (700, 3000), (1, 700001)])
def test_argmax_blocks(dev, n, length):
    """One block to two per SM and row, fewer where the rows are many; ties (the first index), infinities,
    NaNs (never chosen), rows of NaNs (index 0)."""
    rng = np.random.default_rng(n + length)
    x = rng.integers(-50, 50, (n, length)).astype(np.float32)
    x[rng.random((n, length)) < 0.1] = np.nan
    x[0, length // 2] = np.inf
    if n > 2:
        x[1] = np.nan
        x[2] = -np.inf
    want = np.where(np.isnan(x).all(axis=1), 0, np.argmax(np.where(np.isnan(x), -np.inf, x), axis=1))
    if n > 2:
        want[2] = 0
    for _ in range(2):
        assert np.array_equal(dev.argmax(dev.buffer(x), length), want)


def test_back_to_back_products_see_their_own_inputs(dev, oracle):
    """Small-M kernels start while the kernel ahead still runs: every product of a
    chain must still use the input written just before it, and accumulate in order."""
    rng = np.random.default_rng(83)
    rows, cols = 640, 1024
    tensors = [oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)) for _ in range(2)]
    weights = [upload(dev, "q4_k", rows, cols, t) for t in tensors]
    xb, acc = dev.alloc(cols), dev.alloc(rows)
    xs = rng.standard_normal((12, cols)).astype(np.float32)
    want = np.zeros(rows, np.float32)
    for i, x in enumerate(xs):
        dev.write(xb, x)
        dev.matmul_add(acc, weights[i % 2], xb)        # acc += w . x, twelve times without a sync
        want = oracle.matmul_add("q4_k", tensors[i % 2], rows, cols, x, want).reshape(rows)
    assert max_rel_err(dev.read(acc), want) <= 2e-5


def test_gemm_above_the_batch_size(dev, oracle):
    """More tokens than Device::batch() in one call, ragged against every tile size."""
    rng = np.random.default_rng(89)
    rows, cols, n = 200, 512, 2049
    blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    x = rng.standard_normal((n, cols)).astype(np.float32)
    out = dev.alloc(n * rows)
    dev.matmul(out, upload(dev, "q4_k", rows, cols, blocks), dev.buffer(x))
    assert max_rel_err(dev.read(out), oracle.matmul("q4_k", blocks, rows, cols, x)) <= 2e-5


# ---- the benchmarked GEMM configurations at full size -----------------------------------------
def bf16_rows(oracle, rng, n, cols):
    """Config 2's activations: rows of N(0,1) scaled to RMS 1, rounded to bf16."""
    x = rng.standard_normal((n, cols)).astype(np.float32)
    x /= np.sqrt((x * x).mean(1, keepdims=True))
    bits = oracle.to_bf16(x)
    return bits, oracle.bf16(bits).reshape(n, cols)


def sampled_rows(rows, rng, count=384):
    """First, last and a ragged middle stretch of the 128-row tiles, plus random rows."""
    picks = set(range(min(rows, 130))) | set(range(max(0, rows - 130), rows)) | set(range(rows // 2 - 3, min(rows, rows // 2 + 64)))
    picks |= set(int(r) for r in rng.choice(rows, min(rows, count), replace=False))
    return np.array(sorted(picks))


_full_weights = {}


def full_weight(dev, rows, cols, seed):
    """A full-size Q4_K matrix, quantized on the device once per session."""
    key = (rows, cols, seed)
    if key not in _full_weights:
        w = 0.02 * np.random.default_rng(seed).standard_normal((rows, cols), dtype=np.float32)
        t = dev.quantize("q4_k", w)
        _full_weights.clear()                      # one at a time: 50 MB of blocks, 356 MB of f32 behind them
        _full_weights[key] = (t, dev.upload(t))
    return _full_weights[key]


@pytest.mark.parametrize("rows,cols,n", [
    (17408, 5120, 128), (17408, 5120, 512), (17408, 5120, 2048),       # config 2: gate / up
    (5120, 17408, 128), (5120, 17408, 2048),                            # the transposed down projection
    (17401, 5120, 512)])                                                # a ragged last row tile
def test_config2_gemm_full_size(dev, oracle, rows, cols, n):
    """BASELINE config 2 as the benchmark runs it: Q4_K W x bf16 X through the
    256-column tensor-core kernel, against the oracle on a row sample that covers
    the first, last and middle row tiles and every token; plus run-to-run bit
    equality over the whole output."""
    rng = np.random.default_rng(2000 + n)
    t, weight = full_weight(dev, rows, cols, seed=0 if rows != 17401 else 9)
    bits, x = bf16_rows(oracle, rng, n, cols)
    xb, out = dev.alloc(n * cols), dev.alloc(n * rows)
    dev.write_bf16(xb, bits)
    dev.matmul(out, weight, xb)
    got = dev.read(out).reshape(n, rows)
    assert np.isfinite(got).all()
    sample = sampled_rows(rows, rng)
    want = oracle.matmul("q4_k", t.select_rows(sample).data, sample.size, cols, x)
    err = max_rel_err(got[:, sample], want)
    assert err <= TOL, f"max relative error {err:.2e}"
    assert err <= 2e-5, f"exact products: only summation order may differ, got {err:.2e}"
    close_batch(got[:, sample], want, f"q4_k {rows}x{cols} n={n}")
    dev.matmul(out, weight, xb)
    assert np.array_equal(dev.read(out).reshape(n, rows), got)


@pytest.mark.parametrize("n", [17, 33, 130, 300])
def test_gemm_bf16_token_counts(dev, oracle, n):
    """bf16 activations (one f16 term) in tiles of 32, 64 and 192 or
    256 columns of the tensor-core kernel, ragged against each."""
    rng = np.random.default_rng(3000 + n)
    rows, cols = 1000, 5120
    blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    bits, x = bf16_rows(oracle, rng, n, cols)
    xb, out = dev.alloc(n * cols), dev.alloc(n * rows)
    dev.write_bf16(xb, bits)
    dev.matmul(out, upload(dev, "q4_k", rows, cols, blocks), xb)
    assert max_rel_err(dev.read(out).reshape(n, rows), oracle.matmul("q4_k", blocks, rows, cols, x)) <= 2e-5


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n", [9, 16, 17, 32, 33, 64, 65, 128, 129, 192, 193, 256, 257])
def test_gemm_terms_at_tile_edges(dev, oracle, fmt, n):
    """f32 activations' two terms side by side or in turn, bf16's one, at the edges of the tiles' token counts."""
    rng = np.random.default_rng(n)
    rows, cols = 129, 768
    weight, w, _, _ = random_pair(dev, oracle, fmt, rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    bits = oracle.to_bf16(x)
    out, xb = dev.alloc(n * rows), dev.alloc(n * cols)
    for bf16 in (False, True):
        dev.write_bf16(xb, bits) if bf16 else dev.write(xb, x)
        dev.matmul(out, weight, xb)
        want = (oracle.bf16(bits).reshape(n, cols) if bf16 else x).astype(np.float64) @ w.T
        # sums of 768 products in the tensor cores' fp32, f16 pairs for the activations: a few 2^-20 of the result
        assert max_rel_err(dev.read(out).reshape(n, rows), want) <= 1e-5, bf16


@pytest.mark.parametrize("rows,cols,n,bf16", [(129, 256, 9, False), (1000, 512, 16, True), (77, 768, 17, False), (640, 1024, 32, True),
                                              (1024, 5120, 12, False), (5121, 2304, 31, False), (300, 17408, 16, False), (19000, 512, 20, True)])
def test_q4_k_few_tokens(dev, oracle, rows, cols, n, bf16):
    """9 to 32 tokens: one to 68 units of K dealt to four groups and to a cluster's blocks, ragged rows, every epilogue."""
    rng = np.random.default_rng(rows)
    weight, w, other, w2 = random_pair(dev, oracle, "q4_k", rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    x[1] *= 30.0
    xb = dev.alloc(n * cols)
    if bf16:
        bits = oracle.to_bf16(x)
        dev.write_bf16(xb, bits)
        x = oracle.bf16(bits).reshape(n, cols)
    else:
        dev.write(xb, x)
    x = x.astype(np.float64)
    y, z = x @ w.T, x @ w2.T
    out, scratch, h = dev.alloc(n * rows), dev.alloc(n * rows), rng.standard_normal((n, rows)).astype(np.float32)
    res = dev.buffer(h)
    dev.matmul(out, weight, xb)
    got = dev.read(out).reshape(n, rows)
    dev.matmul_add(res, weight, xb)
    added = dev.read(res).reshape(n, rows)
    dev.swiglu(out, weight, other, xb, scratch)
    gated = dev.read(out).reshape(n, rows)
    # the products' sums to 1e-5 of a token's typical result; silu(g) u by twice that of its factors
    for t in range(n):
        assert max_rel_err(got[t], y[t]) <= 1e-5
        assert max_rel_err(added[t], h[t] + y[t]) <= 2e-5
        assert np.abs(gated[t] - silu_times(y[t], z[t])).max() <= 3e-5 * np.sqrt((y[t] ** 2).mean()) * np.abs(z[t]).max()


@pytest.mark.parametrize("rows,cols,n,bf16", [(1024, 5120, 70, False), (1024, 5120, 131, True), (129, 768, 70, True), (100, 2048, 300, False),
                                              (640, 2304, 600, True), (1024, 17408, 131, False), (5120, 4096, 90, True),
                                              (700, 1280, 161, True), (700, 1280, 192, True), (1500, 1024, 97, False), (2000, 512, 385, True)])
def test_gemm_shares_k_between_blocks(dev, oracle, rows, cols, n, bf16):
    """Few row tiles: two to eight blocks of a cluster share a tile's K (uneven shares, ragged rows and
    tokens), with the three epilogues.  fp32 sums: the oracle in double precision from the decoded
    weights, 2e-5 of the result's root mean square (measured 2e-6)."""
    rng = np.random.default_rng(rows + n)
    weight, w, other, w2 = random_pair(dev, oracle, "q4_k", rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    xb = dev.alloc(n * cols)
    if bf16:
        bits = oracle.to_bf16(x)
        dev.write_bf16(xb, bits)
        x = oracle.bf16(bits).reshape(n, cols)
    else:
        dev.write(xb, x)
    want = x.astype(np.float64) @ w.T
    bar = 2e-5 * np.sqrt((want ** 2).mean())
    out, again = dev.alloc(n * rows), dev.alloc(n * rows)
    dev.matmul(out, weight, xb)
    got = dev.read(out)
    assert np.abs(got.reshape(n, rows) - want).max() <= bar
    dev.matmul(again, weight, xb)
    assert np.array_equal(dev.read(again), got)           # the blocks' sums are added in a fixed order
    res = rng.standard_normal((n, rows)).astype(np.float32)
    acc = dev.buffer(res)
    dev.matmul_add(acc, weight, xb)
    assert np.abs(dev.read(acc).reshape(n, rows) - (want + res)).max() <= bar + 1e-6
    dev.swiglu(out, weight, other, xb, again)
    silu = silu_times(want, x.astype(np.float64) @ w2.T)
    assert np.abs(dev.read(out).reshape(n, rows) - silu).max() <= 4 * bar * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n,cut", [(300, 128), (40, 17), (8, 3)])
def test_chunks_and_shards_agree_with_the_whole(dev, oracle, fmt, n, cut):
    """What the header says of a result's bits: a call gives the same ones every time; the same tokens in
    another batch, or the same rows in another matrix, may be summed in another order and agree within
    1e-5 of the result's root mean square (either is within 5e-6 of it from the exact sum)."""
    rng = np.random.default_rng(n)
    rows, cols, row_cut = 1030, 2304, 517
    blocks = dev.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)).data.reshape(rows, -1)
    x = rng.standard_normal((n, cols)).astype(np.float32)

    def product(r, t):
        part = np.ascontiguousarray(blocks[r]).reshape(-1)
        xs = np.ascontiguousarray(x[t])
        out = dev.alloc(xs.shape[0] * blocks[r].shape[0])
        weight, xb = upload(dev, fmt, blocks[r].shape[0], cols, part), dev.buffer(xs)
        results = []
        for _ in range(2):
            dev.matmul(out, weight, xb)
            results.append(dev.read(out).reshape(xs.shape[0], -1))
        assert np.array_equal(results[0], results[1])
        return results[0]

    whole = product(slice(0, rows), slice(0, n))
    bar = 1e-5 * np.sqrt((whole.astype(np.float64) ** 2).mean())
    chunks = np.concatenate([product(slice(0, rows), slice(0, cut)), product(slice(0, rows), slice(cut, n))], axis=0)
    shards = np.concatenate([product(slice(0, row_cut), slice(0, n)), product(slice(row_cut, rows), slice(0, n))], axis=1)
    assert np.abs(chunks - whole).max() <= bar and np.abs(shards - whole).max() <= bar


@pytest.mark.parametrize("fmt", ["q6_k", "q8_0"])
@pytest.mark.parametrize("n", [80, 40, 150])
def test_dense_kernel_scale_extremes(dev, oracle, fmt, n):
    """Block scales over f16's range within a unit (Q8_0's power of two), sub-scales at both ends (Q6_K's
    13-bit products), zero scales, signed ones: random bit patterns with finite scales, against the decoded
    weights in double precision, per row."""
    from dwim_b200 import Tensor
    rng = np.random.default_rng(5)
    rows, cols = 200, 1024
    size = 34 if fmt == "q8_0" else 210
    blocks = rng.integers(0, 256, (rows, cols // (32 if fmt == "q8_0" else 256), size), dtype=np.uint8)
    exponent = rng.integers(0, 31, blocks.shape[:2])
    exponent[: rows // 2] = rng.integers(12, 18, exponent[: rows // 2].shape)      # half the rows: ordinary scales
    d = ((rng.integers(0, 2, exponent.shape) << 15) | (exponent << 10) | rng.integers(0, 1024, exponent.shape)).astype(np.uint16)
    d[rng.random(d.shape) < 0.05] = 0
    at = 0 if fmt == "q8_0" else 208
    blocks[:, :, at] = d & 0xff
    blocks[:, :, at + 1] = d >> 8
    weight = dev.upload(Tensor(fmt, (rows, cols), blocks.reshape(-1)))
    w = oracle.dequantize(fmt, blocks.reshape(-1), rows, cols).reshape(rows, cols).astype(np.float64)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    out = dev.alloc(n * rows)
    dev.matmul(out, weight, dev.buffer(x))
    got, want = dev.read(out).reshape(n, rows), x.astype(np.float64) @ w.T
    rms = np.sqrt((want ** 2).mean(axis=0))
    assert (np.abs(got - want).max(axis=0) <= 2e-5 * np.maximum(rms, 1e-30)).all()


@pytest.mark.parametrize("fmt", ["q6_k", "q8_0"])
@pytest.mark.parametrize("rows,cols,n", [(129, 256, 65), (96, 2048, 70), (300, 2304, 66), (1024, 5120, 80), (640, 6144, 131), (77, 12288, 70)])
def test_dense_kernel_shares_k_between_blocks(dev, oracle, fmt, rows, cols, n):
    """The dense kernel with one to eight blocks on a tile (uneven shares of K, ragged rows and tokens), with
    the three epilogues.  The tensor cores' additions within a unit are not rounded to nearest: 2e-5 of the
    result's root mean square (the largest difference measured at any K is 4.2e-6 of it)."""
    rng = np.random.default_rng(rows + n)
    weight, w, other, w2 = random_pair(dev, oracle, fmt, rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    xb, out, again = dev.buffer(x), dev.alloc(n * rows), dev.alloc(n * rows)
    want = x.astype(np.float64) @ w.T
    bar = 2e-5 * np.sqrt((want ** 2).mean())
    dev.matmul(out, weight, xb)
    got = dev.read(out)
    assert np.abs(got.reshape(n, rows) - want).max() <= bar
    dev.matmul(again, weight, xb)
    assert np.array_equal(dev.read(again), got)
    res = rng.standard_normal((n, rows)).astype(np.float32)
    acc = dev.buffer(res)
    dev.matmul_add(acc, weight, xb)
    assert np.abs(dev.read(acc).reshape(n, rows) - (want + res)).max() <= bar + 1e-6
    dev.swiglu(out, weight, other, xb, again)
    silu = silu_times(want, x.astype(np.float64) @ w2.T)
    assert np.abs(dev.read(out).reshape(n, rows) - silu).max() <= 4 * bar * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("fmt", ["q6_k", "q8_0"])
@pytest.mark.parametrize("rows,cols,n", [(129, 256, 25), (300, 2304, 64), (2600, 1024, 33), (96, 17408, 30), (64, 12544, 130)])
def test_dense_kernel_drained_every_k_block(dev, oracle, fmt, rows, cols, n):
    """f32 activations of 25 to 64 tokens, and of rows above 12288: as exact as the digit planes that it replaces."""
    rng = np.random.default_rng(cols)
    weight, w, _, _ = random_pair(dev, oracle, fmt, rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    want = x.astype(np.float64) @ w.T
    out, xb, h = dev.alloc(n * rows), dev.buffer(x), rng.standard_normal((n, rows)).astype(np.float32)
    dev.matmul(out, weight, xb)
    got = dev.read(out).reshape(n, rows)
    # three digit planes round an activation at 2^-23 of its unit's largest, three to four times its size: 3e-7 in 2-norm
    assert np.linalg.norm(got - want) <= 3e-7 * np.linalg.norm(want)
    res = dev.buffer(h)
    dev.matmul_add(res, weight, xb)                       # the operand kept from the product before
    assert max_rel_err(dev.read(res).reshape(n, rows), h + want) <= 1e-5
    dev.write(xb, x[::-1])                                # and made anew after a write
    dev.matmul(out, weight, xb)
    assert np.array_equal(dev.read(out).reshape(n, rows), got[::-1])


@pytest.mark.parametrize("fmt", ["q6_k", "q8_0"])
def test_dense_kernel_of_few_tokens_under_capture(oracle, fmt):
    """The operand is not the shadow's: captured after a product that left one, a graph makes its own at every replay,
    and a shadow that an earlier graph reads stays where it is."""
    import torch
    from dwim_b200 import B200, Tensor
    stream = torch.cuda.Stream()
    d = B200(0, stream=stream.cuda_stream)
    try:
        rng = np.random.default_rng(73)
        rows, cols, n = 96, 2048, 48
        blocks = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
        weight = d.upload(Tensor(fmt, (rows, cols), blocks))
        x = rng.standard_normal((3, n, cols)).astype(np.float32)
        want = [oracle.matmul(fmt, blocks, rows, cols, y).reshape(n, rows) for y in x]
        xb, out = d.buffer(x[0]), d.alloc(n * rows)
        d.resize(xb, 8 * cols)
        d.resize(out, 8 * rows)
        d.matmul(out, weight, xb)                         # eight tokens' planes: all that the first graph has
        d.resize(xb, n * cols)
        d.resize(out, n * rows)
        graphs = []
        for i in range(2):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                d.matmul(out, weight, xb)
            graphs.append(graph)
            d.write(xb, x[i])
            d.matmul(out, weight, xb)
            assert max_rel_err(d.read(out), want[i]) <= 2e-5
        for i, graph in ((1, graphs[0]), (2, graphs[1]), (0, graphs[0])):
            d.write(xb, x[i])
            with torch.cuda.stream(stream):
                graph.replay()
            assert max_rel_err(d.read(out), want[i]) <= 2e-5
        del graphs, graph
    finally:
        d.close()


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n", [5, 16, 48])
def test_a_captured_conversion_is_not_taken_for_a_made_one(oracle, fmt, n):
    """A conversion recorded into a graph has not run, and one that a graph makes again at another length of the buffer
    takes its place: an eager product multiplies the buffer's contents all the same.  A captured norm still spares its
    product the conversion."""
    import torch
    from dwim_b200 import B200, Tensor
    stream = torch.cuda.Stream()
    d = B200(0, stream=stream.cuda_stream)
    try:
        rng = np.random.default_rng(79)
        rows, cols, other = 96, 2048, n + 3      # (longer: no array that a graph reads is made anew)
        blocks = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
        weight = d.upload(Tensor(fmt, (rows, cols), blocks))
        x = rng.standard_normal((3, other, cols)).astype(np.float32)
        want = [oracle.matmul(fmt, blocks, rows, cols, y).reshape(-1, rows) for y in x]
        xb, out, gain = d.buffer(x[0]), d.alloc(other * rows), d.buffer(np.ones(cols, np.float32))

        def at(tokens):
            d.resize(xb, tokens * cols)
            d.resize(out, tokens * rows)

        def captured(call):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                call()
            return graph

        def product():
            d.matmul(out, weight, xb)

        def right(y, tokens):
            got = d.read(out).reshape(tokens, rows)
            d.write(out, np.zeros(tokens * rows, np.float32))
            return max_rel_err(got, want[y][:tokens]) <= 2e-5

        at(other)
        product()
        graphs = [captured(product)]                      # at the other length
        at(n)
        product()
        d.write(xb, x[1][:n])
        graphs.append(captured(product))
        product()
        assert right(1, n), "an eager product after a capture that has not run"
        for graph in (graphs[0], graphs[1], graphs[0]):
            with torch.cuda.stream(stream):
                graph.replay()
            product()
            assert right(1, n), "an eager product after a graph of another length"
        # the norm's operand: made by its launch under the capture, not there before the graph has run
        normed = d.alloc(n * cols)
        d.normalize(normed, xb, gain, n * cols, 1e-6)
        d.matmul(out, weight, normed)
        d.write(normed, x[0][:n])
        launches = d.launches
        graphs.append(captured(lambda: (d.normalize(normed, xb, gain, n * cols, 1e-6), d.matmul(out, weight, normed))))
        if fmt == "q4_k" or n != 16:                      # (groups of eight convert for themselves)
            assert d.launches - launches == 2, "the product ran a conversion of its own"
        d.matmul(out, weight, normed)
        assert right(0, n), "an eager product after a captured norm that has not run"
        for i in (2, 0):
            d.write(xb, x[i][:n])
            with torch.cuda.stream(stream):
                graphs[1].replay()
            assert right(i, n)
        at(other)
        d.write(xb, x[2])
        with torch.cuda.stream(stream):
            graphs[0].replay()
        assert right(2, other), "captured while an eager product's operand was there"
        del graphs, graph
    finally:
        d.close()


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n", [3, 16])
def test_a_graph_keeps_the_operand_that_it_reads(oracle, fmt, n):
    """A product captured at a few tokens, then eager ones of more and more, whose operand is longer: the graph's own stays
    where it is, whatever is allocated after it."""
    import torch
    from dwim_b200 import B200, Tensor
    stream = torch.cuda.Stream()
    d = B200(0, stream=stream.cuda_stream)
    try:
        rng = np.random.default_rng(89)
        rows, cols, most = 96, 2048, 300
        blocks = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
        weight = d.upload(Tensor(fmt, (rows, cols), blocks))
        x = rng.standard_normal((most, cols)).astype(np.float32)
        want = oracle.matmul(fmt, blocks, rows, cols, x).reshape(most, rows)
        xb, out = d.buffer(x), d.alloc(most * rows)

        def at(tokens):
            d.resize(xb, tokens * cols)
            d.resize(out, tokens * rows)

        def right(tokens):
            got = d.read(out).reshape(tokens, rows)
            d.write(out, np.zeros(tokens * rows, np.float32))
            return max_rel_err(got, want[:tokens]) <= 2e-5

        at(n)
        d.matmul(out, weight, xb)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            d.matmul(out, weight, xb)
        others = []
        for tokens in (n + 6, 100, most):
            at(tokens)
            d.matmul(out, weight, xb)
            assert right(tokens)
            others += [d.buffer(np.full(1 << k, 7.0, np.float32)) for k in range(12, 20)]
            at(n)
            with torch.cuda.stream(stream):
                graph.replay()
            assert right(n), tokens
            at(tokens)
            d.matmul(out, weight, xb)
            assert right(tokens)
        assert all((d.read(o) == 7.0).all() for o in others)
        del graph
    finally:
        d.close()


@pytest.mark.parametrize("fmt", ["q6_k", "q8_0"])
def test_dense_kernel_gives_its_bits_whatever_memory_there_is(oracle, fmt):
    """The products that the groups of eight tokens could take as well: captured before any eager one, by a buffer that
    was read as rows of another length first, and by one whose operand does not fit the device (a buffer of which the
    caller says that it is longer than any memory; a few rows are used), in as many launches as it takes."""
    import torch
    from dwim_b200 import B200, Tensor
    stream = torch.cuda.Stream()
    d = B200(0, stream=stream.cuda_stream)
    try:
        rng = np.random.default_rng(83)
        n, short, long = 70, 1024, 12544
        rows, tokens = {short: 96, long: 300}, {short: 64, long: n}
        blocks = {c: d.quantize(fmt, (0.02 * rng.standard_normal((rows[c], c))).astype(np.float32)).data for c in rows}
        weight = {c: d.upload(Tensor(fmt, (rows[c], c), blocks[c])) for c in rows}
        x = rng.standard_normal(n * long).astype(np.float32)

        def product(xb, c, graph=False):
            d.resize(xb, tokens[c] * c)
            d.write(xb, x[:tokens[c] * c])
            out = d.buffer(rng.standard_normal(tokens[c] * rows[c]).astype(np.float32))
            launches = d.launches
            if graph:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=stream):
                    d.matmul(out, weight[c], xb)
                with torch.cuda.stream(stream):
                    g.replay()
                    stream.synchronize()
                del g
            else:
                d.matmul(out, weight[c], xb)
            return d.read(out), d.launches - launches

        want = {c: product(d.alloc(n * long), c)[0] for c in rows}
        for c in rows:
            w = oracle.dequantize(fmt, blocks[c], rows[c], c).reshape(rows[c], c).astype(np.float64)
            y = x[:tokens[c] * c].reshape(-1, c).astype(np.float64) @ w.T
            assert np.linalg.norm(want[c].reshape(y.shape) - y) <= 3e-7 * np.linalg.norm(y)
            got, launches = product(d.alloc(n * long), c, graph=True)
            assert np.array_equal(got, want[c]) and launches == 2, "captured first"
        for order in ((short, long), (long, short)):
            xb = d.alloc(n * long)
            for c in order:
                got, launches = product(xb, c)
                assert np.array_equal(got, want[c]) and launches == 2, order
        with torch.cuda.stream(stream):
            real = torch.zeros(n * long, device="cuda")
        xb = d.wrap(real.data_ptr(), 1 << 36)
        got, launches = product(xb, long)
        assert np.array_equal(got, want[long]) and launches > 2, "no room for the operand"
        # an addend and a second product's values in the same pieces
        res, gated, scratch = d.buffer(want[long]), d.alloc(n * rows[long]), d.alloc(n * rows[long])
        d.matmul_add(res, weight[long], xb)
        assert np.array_equal(d.read(res), want[long] + want[long])
        d.swiglu(gated, weight[long], weight[long], xb, scratch)
        assert max_rel_err(d.read(gated), silu_times(want[long].astype(np.float64), want[long])) <= 1e-5
        del xb
    finally:
        d.close()


@pytest.mark.parametrize("fmt,n", [("q4_k", 16), ("q4_k", 40), ("q4_k", 150), ("q6_k", 40), ("q6_k", 80), ("q6_k", 150), ("q8_0", 40), ("q8_0", 150)])
def test_gemm_activations_at_the_ends_of_f32(dev, oracle, fmt, n):
    """Rows whose largest activation is near the ends of f32's exponents: the token's power of two reaches both, so that
    such a row's result is as exact as an ordinary one's (the smallest here a little above the subnormals)."""
    rng = np.random.default_rng(n)
    rows, cols = 129, 768
    weight, w, _, _ = random_pair(dev, oracle, fmt, rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    sizes = (1.0, 1e36, 1e-34, 8e34, 3e37, 1e-30)
    for i, size in enumerate(sizes):
        x[i::len(sizes)] *= np.float32(size)
    want = x.astype(np.float64) @ w.T
    out = dev.alloc(n * rows)
    dev.matmul(out, weight, dev.buffer(x))
    got = dev.read(out).reshape(n, rows)
    assert np.isfinite(got).all()
    for t in range(n):
        assert np.abs(got[t] - want[t]).max() <= 1e-5 * np.sqrt((want[t] ** 2).mean()), (t, sizes[t % len(sizes)])


@pytest.mark.parametrize("bf16", [True, False])
def test_gemm_fused_epilogues_at_256_columns(dev, oracle, bf16):
    """matmul_add and swiglu of 300 tokens of bf16 input, or 150 of f32 in two terms (in tiles of 192 columns, whose wave is
    the shorter one here; of 256: test_tiles_of_256_columns)."""
    rng = np.random.default_rng(3100 + bf16)
    rows, cols, n = 1030, 5120, 300 if bf16 else 150
    gate = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    up = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    xb = dev.alloc(n * cols)
    if bf16:
        bits, x = bf16_rows(oracle, rng, n, cols)
        dev.write_bf16(xb, bits)
    else:
        x = rng.standard_normal((n, cols)).astype(np.float32)
        dev.write(xb, x)
    wg, wu = upload(dev, "q4_k", rows, cols, gate), upload(dev, "q4_k", rows, cols, up)
    out, scratch = dev.alloc(n * rows), dev.alloc(n * rows)
    dev.swiglu(out, wg, wu, xb, scratch)
    assert max_rel_err(dev.read(out), oracle.swiglu("q4_k", gate, up, rows, cols, x)) <= 1e-4
    res = rng.standard_normal((n, rows)).astype(np.float32)
    acc = dev.buffer(res)
    dev.matmul_add(acc, wg, xb)
    got, want = dev.read(acc).reshape(n, rows), oracle.matmul_add("q4_k", gate, rows, cols, x, res)
    assert max_rel_err(got - res, want - res) <= 1e-4


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("bf16", [True, False])
def test_tiles_of_256_columns(dev, oracle, fmt, bf16):
    """76 row tiles by 255 tokens: one wave in tiles of 256 columns and two of 192, so these take it; the three epilogues,
    ragged rows and tokens.  2e-5 of the result's root mean square, as for the narrower tiles."""
    rng = np.random.default_rng(3200 + bf16)
    rows, cols, n = 9601, 512, 255
    weight, w, other, w2 = random_pair(dev, oracle, fmt, rows, cols, rng)
    x = rng.standard_normal((n, cols)).astype(np.float32)
    xb = dev.buffer(x)
    if bf16:
        bits = oracle.to_bf16(x)
        dev.write_bf16(xb, bits)
        x = oracle.bf16(bits).reshape(n, cols)
    want = x.astype(np.float64) @ w.T
    bar = 2e-5 * np.sqrt((want ** 2).mean())
    out, scratch, res = dev.alloc(n * rows), dev.alloc(n * rows), rng.standard_normal((n, rows)).astype(np.float32)
    acc = dev.buffer(res)
    dev.matmul(out, weight, xb)
    assert np.abs(dev.read(out).reshape(n, rows) - want).max() <= bar
    dev.matmul_add(acc, weight, xb)
    assert np.abs(dev.read(acc).reshape(n, rows) - (want + res)).max() <= bar + 1e-6
    dev.swiglu(out, weight, other, xb, scratch)
    silu = silu_times(want, x.astype(np.float64) @ w2.T)
    assert np.abs(dev.read(out).reshape(n, rows) - silu).max() <= 4 * bar * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("fmt", ["q6_k", "q8_0"])
@pytest.mark.parametrize("n,bf16", [(12, False), (33, False), (65, True), (130, False), (300, True)])
def test_dense_pair_gemm_for_q6_k_and_q8_0(dev, oracle, fmt, n, bf16):
    """Above the small-M kernel's eight tokens Q6_K and Q8_0 go in groups of eight
    (up to 24 tokens by f32 activations, 64 by bf16) and then through the dense kernel, whose weights are pairs of
    f16 terms: its narrower tiles, ragged rows, both activation forms, fused epilogues.
    Against the oracle's fp32 sums: 2e-5 for either path (4.2e-6 of the result's root
    mean square is the most the dense kernel was measured to be off, at any K)."""
    rng = np.random.default_rng(4000 + n)
    rows, cols = 1030, 2304
    gate = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    up = oracle.quantize(fmt, (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
    xb = dev.alloc(n * cols)
    if bf16:
        bits, x = bf16_rows(oracle, rng, n, cols)
        dev.write_bf16(xb, bits)
    else:
        x = rng.standard_normal((n, cols)).astype(np.float32)
        dev.write(xb, x)
    wg, wu = upload(dev, fmt, rows, cols, gate), upload(dev, fmt, rows, cols, up)
    out, scratch = dev.alloc(n * rows), dev.alloc(n * rows)
    dev.matmul(out, wg, xb)
    assert max_rel_err(dev.read(out), oracle.matmul(fmt, gate, rows, cols, x)) <= 2e-5
    dev.swiglu(out, wg, wu, xb, scratch)
    # either product's error times the other factor, at most 4.5 of its rms: 4.2e-6 * 4.5 * 2 over silu(g) u's smaller rms
    assert max_rel_err(dev.read(out), oracle.swiglu(fmt, gate, up, rows, cols, x)) <= 8e-5
    res = rng.standard_normal((n, rows)).astype(np.float32)
    acc = dev.buffer(res)
    dev.matmul_add(acc, wu, xb)
    got, want = dev.read(acc).reshape(n, rows), oracle.matmul_add(fmt, up, rows, cols, x, res)
    assert max_rel_err(got - res, want - res) <= 2e-5


@pytest.mark.parametrize("fmt,rows,cols,n", [("q6_k", 151936, 5120, 128), ("q8_0", 5120, 5120, 2048), ("q6_k", 20000, 5120, 512)])
def test_dense_pair_gemm_full_size(dev, oracle, fmt, rows, cols, n):
    """The head's and the projections' matrices at GEMM sizes through the dense kernel,
    against the oracle on sampled rows and every token."""
    rng = np.random.default_rng(4100 + n)
    srows = 2048                                      # distinct rows; the matrix repeats them (generation time)
    base = oracle.quantize(fmt, (0.02 * rng.standard_normal((srows, cols))).astype(np.float32))
    from dwim_b200 import Tensor, row_bytes
    reps = -(-rows // srows)
    blocks = np.tile(base.reshape(srows, -1), (reps, 1))[:rows].reshape(-1)
    weight = dev.upload(Tensor(fmt, (rows, cols), blocks))
    bits, x = bf16_rows(oracle, rng, n, cols)
    xb, out = dev.alloc(n * cols), dev.alloc(n * rows)
    dev.write_bf16(xb, bits)
    dev.matmul(out, weight, xb)
    got = dev.read(out).reshape(n, rows)
    sample = sampled_rows(rows, rng)
    rb = row_bytes(fmt, cols)
    want = oracle.matmul(fmt, blocks.reshape(rows, rb)[sample].reshape(-1), sample.size, cols, x)
    assert max_rel_err(got[:, sample], want) <= 2e-5


# ---- the boundary: a caller's stream, a caller's writes -----------------------------------------
def test_adopted_stream_and_touch(oracle):
    """The composition an engine would use: the library opened on the caller's
    stream, a buffer wrapped over the caller's memory, a kernel of the caller's
    (torch, on that stream) rewriting it between two products.  After touch the
    second product sees the new data; the stream orders everything."""
    import torch
    from dwim_b200 import B200, Tensor
    stream = torch.cuda.Stream()
    d = B200(0, stream=stream.cuda_stream)
    try:
        rng = np.random.default_rng(97)
        rows, cols, n = 640, 1024, 3
        blocks = oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32))
        weight = d.upload(Tensor("q4_k", (rows, cols), blocks))
        x1 = rng.standard_normal((n, cols)).astype(np.float32)
        x2 = rng.standard_normal((n, cols)).astype(np.float32)
        with torch.cuda.stream(stream):
            xt = torch.from_numpy(x1).cuda(non_blocking=False)
            x2t = torch.from_numpy(x2).cuda(non_blocking=False)
            ot = torch.empty(n * rows, dtype=torch.float32, device="cuda")
        stream.synchronize()
        xb, out = d.wrap(xt.data_ptr(), n * cols), d.wrap(ot.data_ptr(), n * rows)
        d.matmul(out, weight, xb)
        with torch.cuda.stream(stream):
            first = ot.clone()
            xt.copy_(x2t)                    # the caller's kernel, ordered by the shared stream
        d.touch(xb)
        d.matmul(out, weight, xb)
        with torch.cuda.stream(stream):
            second = ot.clone()
        stream.synchronize()
        d.sync()
        assert max_rel_err(first.cpu().numpy(), oracle.matmul("q4_k", blocks, rows, cols, x1)) <= 2e-5
        assert max_rel_err(second.cpu().numpy(), oracle.matmul("q4_k", blocks, rows, cols, x2)) <= 2e-5
    finally:
        d.close()


@pytest.mark.parametrize("n", [1, 6, 40])
def test_feed_forward_block_push_exchange_in_a_world_of_one(dev, oracle, n):
    """matmul_scatter, reduce_gather and the barriers with a single rank: the
    whole result is this rank's slice, its one slot the whole sum."""
    from dwim_b200 import Tensor, shard
    rng = np.random.default_rng(161 + n)
    hidden, inner = 512, 1024
    mk = lambda r, c: Tensor("q4_k", (r, c), oracle.quantize("q4_k", (0.05 * rng.standard_normal((r, c))).astype(np.float32)))
    gate, up, down = mk(inner, hidden), mk(inner, hidden), mk(hidden, inner)
    x = rng.standard_normal((n, hidden)).astype(np.float32)
    block = shard.ShardedFFN(dev, gate, up, down, exchange="push")
    got = dev.read(block.forward(dev.buffer(x))).reshape(n, hidden)
    h = oracle.swiglu("q4_k", gate.data, up.data, inner, hidden, x)
    want = oracle.matmul("q4_k", down.data, hidden, inner, h).reshape(n, hidden)
    assert max_rel_err(got, want) <= 5e-5


def test_shared_buffer_in_a_world_of_one(dev, oracle):
    """matmul_gather and the barrier with a single rank: two row shards written
    into one shared result at their offsets, as two ranks would."""
    rng = np.random.default_rng(99)
    rows, cols = 1000, 1024
    from dwim_b200 import Tensor
    t = Tensor("q4_k", (rows, cols), oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)))
    for n in (1, 5, 40):
        x = rng.standard_normal((n, cols)).astype(np.float32)
        out, handle = dev.shared_alloc(n * rows)
        dev.shared_connect(out, 1, 0, [handle])
        xb = dev.buffer(x)
        for b, e in ((0, 496), (496, 1000)):
            dev.matmul_gather(out, dev.upload(t.slice_rows(b, e)), xb, b, rows)
        dev.shared_barrier(out)
        assert max_rel_err(dev.read(out), oracle.matmul("q4_k", t.data, rows, cols, x)) <= 2e-5


def test_shared_result_of_two_ranks_on_one_gpu(dev, oracle):
    """Two ranks of one process (dwim_b200_shared_connect_local): each rank's matmul_gather must put
    its rows into BOTH copies of the shared result -- the small-M kernel's peer stores, the
    tensor-core kernel's TMA stores (slices on 16-byte boundaries) and its register stores (a slice
    that is not).  No barrier kernel: both ranks share the GPU, and the stream orders them."""
    from dwim_b200 import Tensor
    rng = np.random.default_rng(101)
    cols = 1024
    for rows, cut in ((1000, 496), (1002, 499)):          # aligned slices / a slice that starts on an odd row
        t = Tensor("q4_k", (rows, cols), oracle.quantize("q4_k", (0.02 * rng.standard_normal((rows, cols))).astype(np.float32)))
        shards = [(0, cut, dev.upload(t.slice_rows(0, cut))), (cut, rows, dev.upload(t.slice_rows(cut, rows)))]
        for n in (3, 40, 300):
            x = rng.standard_normal((n, cols)).astype(np.float32)
            want = oracle.matmul("q4_k", t.data, rows, cols, x)
            copies = [dev.shared_alloc(n * rows)[0] for _ in range(2)]
            for r in range(2):
                dev.shared_connect_local(copies[r], 2, r, copies)
            xb = dev.buffer(x)
            for r, (b, e, w) in enumerate(shards):
                dev.matmul_gather(copies[r], w, xb, b, rows)
            for r in range(2):
                assert max_rel_err(dev.read(copies[r]), want) <= 2e-5, (rows, n, r)


def test_activation_precision_f16(dev, oracle):
    """f32 activations as one f16 term on request (the reference device's own precision, `halves`,
    gpu/cuda/mod.rs:313-384): it passes the reference's gate for that device (rms error below 1e-3 of
    the typical magnitude and the worst below 1e-2, gpu/tests.rs:198-211), not this library's 1e-3
    on the worst element, and is really another path than the exact one."""
    from dwim_b200 import DeviceError
    g = np.random.default_rng(91)
    rows, cols, n = 384, 5120, 40
    blocks = oracle.quantize("q4_k", (0.02 * g.standard_normal((rows, cols))).astype(np.float32))
    weight = upload(dev, "q4_k", rows, cols, blocks)
    x = g.standard_normal((n, cols)).astype(np.float32)
    x[3] *= 1e4                                    # a token of another magnitude keeps its own scale
    want = oracle.matmul("q4_k", blocks, rows, cols, x)
    xb, out = dev.buffer(x), dev.alloc(n * rows)
    dev.matmul(out, weight, xb)
    exact = max_rel_err(dev.read(out), want)
    dev.activation_precision("f16")
    try:
        dev.matmul(out, weight, xb)
        got = dev.read(out).reshape(n, rows)
        half = max_rel_err(got, want)
        typical = np.sqrt((want.reshape(n, rows) ** 2).mean(axis=1, keepdims=True))      # per token: one is 1e4 times the others
        half_rms = float(np.sqrt((((got - want.reshape(n, rows)) / typical) ** 2).mean()))
    finally:
        dev.activation_precision("exact")
    dev.matmul(out, weight, xb)
    again = max_rel_err(dev.read(out), want)
    assert exact <= 1e-5 and again <= 1e-5, (exact, again)
    assert 1e-5 < half <= 1e-2 and half_rms <= 1e-3, (half, half_rms)
    with pytest.raises(DeviceError):
        dev._check(dev._L.dwim_b200_activation_precision(dev._ctx, 7))
