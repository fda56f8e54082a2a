"""Parity of the sm_100a kernels (through the C ABI) with the CPU oracle and, where the reference
library is present, with the reference's own kernels on the same inputs."""
import numpy as np
import pytest

import oracle_lib as O
import ref_lib as R

pytestmark = pytest.mark.gpu
L = O.lib()


def f16(a):
    return np.asarray(a, np.float32).astype(np.float16).view(np.uint16)


def f32(u):
    return np.asarray(u, np.uint16).view(np.float16).astype(np.float32)


def rel_to_max(x, gold):
    return float(np.abs(x - gold).max() / np.abs(gold).max())


# ------------------------------------------------------------------ generator
def test_synth_generator_bits_equal_oracle(lcu):
    for name, n, first in [("layers.0.attention.wq", 1 << 18, 0), ("output", 12345, 1 << 33)]:
        assert (lcu.synth_f16(n, 1234, name, 0.02, first) == O.synth_f16(n, 1234, name, 0.02, first)).all()


# ------------------------------------------------------------------ quantizer: bit exact
@pytest.mark.parametrize("h,w,bs", [(16, 256, 128), (7, 512, 64), (5, 128, 32), (33, 11008, 128), (4096, 4096, 128)])
def test_quantizer_bit_exact(lcu, h, w, bs):
    x = O.synth_f16(h * w, 1234, f"quant{h}x{w}", 0.02).reshape(h, w)
    if h >= 5:
        x[1, :bs] = 0          # all-zero block: 0/0
        x[2, :] = f16(np.linspace(-3, 3, w))
        x[3, :bs] = 0x0001     # smallest subnormal
    q, s, st = lcu.quantize(x, bs, stats=True)
    qo, so = O.quantize(x, h, w, bs)
    assert (s == so).all()
    assert (q == qo).all()
    if R.available():
        qr, sr, str_ = R.quantize(x, bs)
        assert (s == sr).all() and (q == qr).all()
        assert np.allclose(st, str_, rtol=1e-3, atol=1e-9)
    dq = lcu.dequantize(q, s, bs)
    do = np.empty_like(dq)
    L.orc_dequantize_absmax_uint8(do, s, q, h, w, bs)
    assert (dq == do).all()


@pytest.mark.parametrize("bs", [32, 64, 128, 256])
@pytest.mark.parametrize("blocks", [1, 3, 9, 517])
def test_quantizer_equal_on_every_alignment(lcu, bs, blocks):
    """The vector kernel (16-byte aligned input; whole and halved stores) against the plain one, which input at 8 bytes takes: any
    bit patterns, ordinary values, sparse rows, values half way between two bytes."""
    rng = np.random.default_rng(bs + blocks)
    x = rng.integers(0, 1 << 16, (blocks, bs)).astype(np.uint16)
    x[::3] = f16(rng.standard_normal(x[::3].shape) * 0.02)
    x[1::6] = f16(rng.standard_normal(x[1::6].shape) * (rng.random(x[1::6].shape) < 0.1))
    half = rng.integers(-127, 127, x[4::6].shape)  # (scale 1/64: every other value is a whole or a half number of scales)
    half[:, 0] = 255
    x[4::6] = f16(half / 128)
    raw = lcu.DeviceBuffer(x.nbytes + 32)
    outs = []
    for at, q_at in ((0, 0), (16, 8), (8, 0)):
        lcu.check(lcu.lib.lcu_memcpy_h2d(raw.ptr.value + at, x.ctypes.data, x.nbytes))
        q, s = lcu.DeviceBuffer(x.size + 32), lcu.DeviceBuffer(blocks * 2)
        lcu.check(lcu.lib.lcu_quantize_absmax_uint8(q.ptr.value + q_at, s.ptr, raw.ptr.value + at, blocks, bs, bs, None))
        lcu.check(lcu.lib.lcu_synchronize())
        outs.append((q.to_host(np.uint8, (x.size + 32,))[q_at:q_at + x.size], s.to_host(np.uint16, (blocks,))))
    for q, s in outs[:2]:
        assert (q == outs[2][0]).all() and (s == outs[2][1]).all()


def test_quantizer_empty_and_bad_block(lcu):
    q, s = lcu.quantize(np.zeros((0, 128), np.uint16), 128)
    assert q.shape == (0, 128) and s.shape == (0, 1)
    with pytest.raises(lcu.LcuError):
        lcu.quantize(np.zeros((2, 128), np.uint16), 96)


# ------------------------------------------------------------------ matmul: the single-layer configuration
def test_single_layer_fp16_4096(lcu):
    n = k = 4096
    w = O.synth_f16(n * k, 1234, "W", 0.02).reshape(n, k)
    x = O.synth_f16(k, 1234, "x", 1.0).reshape(1, k)
    y = lcu.matmul_nt(x, w)
    gold = np.zeros((1, n), np.float64)
    L.orc_matmul_nt_gold(gold.reshape(-1), x.reshape(-1), w.ctypes.data, None, None, 1, k, n, 0, 0)
    mine = rel_to_max(f32(y).astype(np.float64), gold)
    assert mine <= 1e-2, mine              # tolerance of the task: 1e-2 max relative error
    assert mine <= 1e-3, mine              # what fp32 accumulation + one fp16 rounding gives
    yo = np.zeros((1, n), np.uint16)
    L.orc_matmul_nt_f16(yo.reshape(-1), x.reshape(-1), w.reshape(-1), 1, k, n, 0.0, 0)
    assert np.abs(f32(y) - f32(yo)).max() <= 2 * 2.0 ** -8  # within 2 ulp of the oracle's fp32 evaluation at |y| < 8
    if R.available():
        for mtype in (4, 1):
            yr = R.matmul_f16(x, w, mtype=mtype)
            theirs = rel_to_max(f32(yr).astype(np.float64), gold)
            assert mine <= theirs * 1.5 + 1e-6, (mine, theirs, mtype)  # no worse than the reference's own kernels


def test_single_layer_int8_4096(lcu):
    n = k = 4096
    bs = 128
    w = O.synth_f16(n * k, 1234, "W", 0.02).reshape(n, k)
    x = O.synth_f16(k, 1234, "x", 1.0).reshape(1, k)
    q, s = lcu.quantize(w, bs)
    y = lcu.matmul_nt(x, q, s, bs)
    gold = np.zeros((1, n), np.float64)  # double accumulation over the half-rounded de-quantized weights
    L.orc_matmul_nt_gold(gold.reshape(-1), x.reshape(-1), None, q.ctypes.data, s.ctypes.data, 1, k, n, bs, 1)
    mine = rel_to_max(f32(y).astype(np.float64), gold)
    assert mine <= 1e-3, mine
    if R.available():
        yr = R.matmul_u8(x, q, s, bs, mtype=4)
        theirs = rel_to_max(f32(yr).astype(np.float64), gold)
        assert mine <= theirs * 1.5 + 1e-6, (mine, theirs)


@pytest.mark.parametrize("m,k,n,bs,beta", [(1, 256, 64, 0, 0.0), (1, 768, 256, 0, 1.0), (2, 512, 130, 0, 0.0), (5, 256, 64, 128, 1.0),
                                           (8, 1280, 96, 64, 0.0), (9, 512, 64, 32, 0.0), (16, 256, 32, 0, 1.0), (3, 11008, 64, 128, 0.0),
                                           (1, 22016, 34, 0, 0.0)])
def test_matmul_small_shapes(lcu, m, k, n, bs, beta):
    rng = np.random.default_rng(m * 1000 + n)
    x = f16(rng.standard_normal((m, k)))
    w = O.synth_f16(n * k, 99, f"w{n}x{k}", 0.05).reshape(n, k)
    prev = f16(rng.standard_normal((m, n)))
    yo = prev.copy()
    if bs == 0:
        y = lcu.matmul_nt(x, w, beta=beta, out_u16=prev)
        L.orc_matmul_nt_f16(yo.reshape(-1), x.reshape(-1), w.reshape(-1), m, k, n, beta, 1)
    else:
        q, s = O.quantize(w, n, k, bs)
        y = lcu.matmul_nt(x, q, s, bs, beta=beta, out_u16=prev)
        L.orc_matmul_nt_fp16u8(yo.reshape(-1), x.reshape(-1), q.reshape(-1), s.reshape(-1), m, k, n, bs, beta, 2)
    scale = max(1.0, float(np.abs(f32(yo)).max()))
    assert np.abs(f32(y) - f32(yo)).max() <= 2e-3 * scale, (m, k, n, bs)


@pytest.mark.parametrize("bs", [32, 64, 128])
@pytest.mark.parametrize("m,k,n,beta", [(3, 4096, 2, 0.0), (17, 256, 128, 1.0), (9, 512, 130, 0.0), (224, 512, 384, 0.0), (225, 1280, 96, 1.0),
                                        # K split over 2, 4 and 8 CTAs, ragged last tile
                                        (40, 1024, 1026, 1.0), (300, 2048, 200, 0.0), (9, 11008, 64, 1.0),
                                        # more tiles than SMs, several row tiles
                                        (460, 256, 9000, 0.0)])
def test_product_expands_8_bit_weights(lcu, m, k, n, beta, bs):
    """Several rows: 8-bit weights are expanded inside the tcgen05 product: against the product over the same half-rounded weights in 64
    bits, element by element, against the oracle's, and against the GEMV passes of 8 rows.  Bounds: the result's rounding to half, and
    for the sums (K / 16 tensor-core steps and the parts of a split K, each within 2^-22 of what it has summed) their count times 2^-22
    of sum|x w|; leaving out 64 of K shows in two thirds of the elements or more.  The GEMV does not round weights to half: 2^-11 of
    sum|x w| more."""
    rng = np.random.default_rng(m + n + bs)
    x = f16(rng.standard_normal((m, k)))
    w = O.synth_f16(n * k, 5, f"u8{n}x{k}", 0.05).reshape(n, k)
    q, s = O.quantize(w, n, k, bs)
    prev = f16(rng.standard_normal((m, n)))
    yo = prev.copy()
    L.orc_matmul_nt_fp16u8(yo.reshape(-1), x.reshape(-1), q.reshape(-1), s.reshape(-1), m, k, n, bs, beta, 2)
    y = lcu.matmul_nt(x, q, s, bs, beta=beta, out_u16=prev)
    assert np.array_equal(y, lcu.matmul_nt(x, q, s, bs, beta=beta, out_u16=prev))
    lcu.check(lcu.lib.lcu_set_tuning(b"prefill_u8_deq_min_rows", 1000000))
    try:
        y_gemv = lcu.matmul_nt(x, q, s, bs, beta=beta, out_u16=prev)
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"prefill_u8_deq_min_rows", 2))
    halves = ((q.reshape(n, -1, bs) - np.float32(127.5)) * f32(s).reshape(n, -1, 1)).astype(np.float16).astype(np.float64).reshape(n, k)
    xd = f32(x).astype(np.float64)
    exact = xd @ halves.T + beta * f32(prev)
    weight = np.abs(xd) @ np.abs(halves).T + abs(beta) * np.abs(f32(prev))
    half = 2.0 ** -11 * np.abs(exact) + 2.0 ** -25
    sums = (k / 16 + 16) * 2.0 ** -22 * weight
    assert (np.abs(f32(y) - exact) <= half + sums).all()
    assert (np.abs(f32(y) - f32(yo)) <= 2 * (half + sums)).all()
    assert (np.abs(f32(y_gemv) - exact) <= half + sums + 2.0 ** -11 * weight).all()


@pytest.mark.parametrize("m", [48, 100, 200])  # tiles of 48, 112 and 208 rows: seven, five and three stages
def test_product_with_8_bit_weights_from_a_cold_cache(lcu, m):
    """Loads that arrive out of order: three copies of a matrix, more than the L2 cache holds, give the same bits every time."""
    torch = pytest.importorskip("torch")
    k, n, bs = 4096, 11008, 64
    g = torch.Generator().manual_seed(m)
    x = torch.randn((m, k), generator=g).half().cuda()
    q = torch.randint(0, 256, (n, k), generator=g, dtype=torch.uint8).cuda()
    s = (torch.rand((n, k // bs), generator=g) * 1e-3 + 1e-4).half().cuda()
    copies = [(q.clone(), s.clone()) for _ in range(3)]
    stream, first = torch.cuda.current_stream().cuda_stream, None
    for i in range(30):
        out = torch.full((m, n), float("nan"), dtype=torch.half, device="cuda")
        cq, cs = copies[i % 3]
        lcu.check(lcu.lib.lcu_matmul_nt_fp16u8(out.data_ptr(), x.data_ptr(), cq.data_ptr(), cs.data_ptr(), m, k, n, bs, 0.0, stream))
        first = out if first is None else first
        assert bool(torch.isfinite(out).all()) and torch.equal(out, first)


@pytest.mark.parametrize("m,k,n", [(200, 512, 384), (9, 4096, 256)])  # one CTA per tile, and K split over a cluster
def test_product_with_8_bit_weights_behind_an_earlier_error(lcu, m, k, n):
    """A code that another operator's launch left in the error word does not keep a product from its results, and is reported."""
    import ctypes as C
    rng = np.random.default_rng(m)
    x = f16(rng.standard_normal((m, k)))
    q, s = O.quantize(f16(rng.standard_normal((n, k)) * 0.05), n, k, 64)
    want = lcu.matmul_nt(x, q, s, 64)
    word, code = C.c_void_p(), C.c_int(-1)
    lcu.check(lcu.lib.lcu_operator_error_word(C.byref(word)))
    assert lcu.lib.lcu_operator_status(C.byref(code)) == 0 and code.value == 0
    stale = np.array([0x103], np.int32)
    lcu.check(lcu.lib.lcu_memcpy_h2d(word, stale.ctypes.data, 4))
    try:
        got = lcu.matmul_nt(x, q, s, 64)
    finally:
        rc = lcu.lib.lcu_operator_status(C.byref(code))
    assert np.array_equal(got, want)
    assert rc == 4 and code.value == 0x103
    assert lcu.lib.lcu_operator_status(C.byref(code)) == 0 and code.value == 0


@pytest.mark.parametrize("m,k,n,beta,tile", [(9, 64, 32, 0.0, 0), (16, 256, 32, 1.0, 0), (128, 64, 128, 0.0, 128), (129, 512, 192, 1.0, 0),
                                             (200, 1024, 256, 1.0, 64), (77, 4096, 1024, 0.0, 32), (300, 11008, 128, 0.0, 0),
                                             (257, 4096, 4096, 1.0, 0),
                                             # more pair tiles than SM pairs: the persistent loop takes several tiles per pair
                                             (300, 256, 22016, 1.0, 0), (257, 320, 12288, 0.0, 0),
                                             # tile widths that do not divide N: the last tile hangs over the matrix
                                             (16, 512, 22016, 1.0, 160), (100, 256, 1024, 0.0, 96), (128, 512, 4096, 1.0, 224),
                                             (33, 1024, 2560, 0.0, 192), (64, 256, 1536, 1.0, 256), (9, 64, 32, 0.0, 96),
                                             # the widths the dispatch picks for short prompts by itself (7B shapes, short K)
                                             (16, 512, 12288, 0.0, 0), (128, 512, 22016, 1.0, 0),
                                             # K steps that do not fill the last stage of two or four k-blocks (its rest arrives as zeros)
                                             (50, 320, 1024, 1.0, 0), (20, 192, 4096, 0.0, 0), (120, 704, 4096, 1.0, 128), (2, 4096, 4096, 0.0, 0)])
def test_prefill_tensor_core_gemm(lcu, m, k, n, beta, tile):
    """fp16 weights with more than 8 rows run on tcgen05 with the accumulator in tensor memory: compared with
    the oracle's binary64-accumulated product (tolerance 2e-3 of the largest output: fp32 accumulation in a
    different order plus one rounding to half) and with the 8-row GEMV passes it replaces."""
    rng = np.random.default_rng(m * 7 + n)
    x = f16(rng.standard_normal((m, k)))
    w = O.synth_f16(n * k, 5, f"tc{n}x{k}", 0.05).reshape(n, k)
    prev = f16(rng.standard_normal((m, n)))
    yo = prev.copy()
    L.orc_matmul_nt_f16(yo.reshape(-1), x.reshape(-1), w.reshape(-1), m, k, n, beta, 1)
    lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_tile_n", tile))
    try:
        y = lcu.matmul_nt(x, w, beta=beta, out_u16=prev)
        lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_min_rows", 0))
        y_gemv = lcu.matmul_nt(x, w, beta=beta, out_u16=prev) if k % 256 == 0 else None
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_tile_n", 0))
        lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_min_rows", 2))
    scale = max(1.0, float(np.abs(f32(yo)).max()))
    assert np.abs(f32(y) - f32(yo)).max() <= 2e-3 * scale
    if y_gemv is not None:
        assert np.abs(f32(y) - f32(y_gemv)).max() <= 2e-3 * scale


@pytest.mark.parametrize("tile", [256, 512])
@pytest.mark.parametrize("m,k,n,beta", [(129, 512, 512, 0.0), (200, 1024, 1024, 1.0), (300, 4096, 1536, 0.0), (512, 11008, 4096, 1.0),
                                        # fewer tiles than SM pairs: every tile is shared by several pairs
                                        (257, 2048, 512, 1.0),
                                        # whole waves first, then the shared tiles (2 x 86 tiles for 74 pairs)
                                        (512, 320, 22016, 0.0), (1000, 2048, 2560, 1.0),
                                        # smallest legal K and N, ragged rows
                                        (131, 64, 512, 1.0), (515, 128, 1024, 0.0),
                                        # short prompts: only the rows that exist are handed over between pairs
                                        (16, 4096, 1536, 1.0), (100, 2048, 2560, 0.0), (1, 512, 512, 1.0)])
def test_prefill_gemm_with_balanced_k_steps(lcu, m, k, n, beta, tile):
    """The tcgen05 GEMM that deals the K steps of the last wave's tiles evenly over the SM pairs (partial sums through a
    workspace, added in pair order): against the oracle's binary64-accumulated product, same tolerance as the whole-tile
    kernel, for both tile widths; and twice in a row with equal bits (the order of the sums does not depend on timing)."""
    if n % tile:
        pytest.skip("tile width does not divide N")
    rng = np.random.default_rng(m * 11 + n + tile)
    x = f16(rng.standard_normal((m, k)))
    w = O.synth_f16(n * k, 5, f"sk{n}x{k}", 0.05).reshape(n, k)
    prev = f16(rng.standard_normal((m, n)))
    yo = prev.copy()
    L.orc_matmul_nt_f16(yo.reshape(-1), x.reshape(-1), w.reshape(-1), m, k, n, beta, 1)
    lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_sk", tile))
    try:
        y = lcu.matmul_nt(x, w, beta=beta, out_u16=prev)
        y2 = lcu.matmul_nt(x, w, beta=beta, out_u16=prev)
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_sk", -1))
    scale = max(1.0, float(np.abs(f32(yo)).max()))
    assert np.abs(f32(y) - f32(yo)).max() <= 2e-3 * scale
    assert np.array_equal(y, y2)


@pytest.mark.parametrize("tile", [256, 512])
@pytest.mark.parametrize("m,k,f", [(512, 4096, 11008), (2000, 1024, 2816), (129, 64, 256), (515, 512, 1280),
                                   # fewer tiles than SM pairs: every tile is shared by several pairs
                                   (700, 4096, 5632), (300, 2048, 128)])
def test_gated_gemm_equals_the_stacked_product_followed_by_silu(lcu, m, k, f, tile):
    """w1|w3 and the SiLU gate as one launch (both products of a tile in tensor memory, the gate in the epilogue) against
    the two-step path the reference takes (llama_cu.cu:1180-1183): the stacked product stored as halves, then silu on
    those halves.  The one launch rounds the products to half before the gate exactly as the store does, and the balanced
    kernel with the same tile width adds partial sums in the same order, so only the gate's quotient can differ."""
    if f % (tile // 2):
        pytest.skip("tile width does not divide the output")
    rng = np.random.default_rng(m + 3 * f)
    x = f16(rng.standard_normal((m, k)))
    w13 = O.synth_f16(2 * f * k, 9, f"gate{f}x{k}", 0.05).reshape(2 * f, k)
    # the two-step path with the same tile shape and K split: half a tile of columns of w1 beside the same of w3
    hw = tile // 2
    order = np.concatenate([np.concatenate([np.arange(c, c + hw), f + np.arange(c, c + hw)]) for c in range(0, f, hw)])
    lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_sk", tile))
    try:
        h = lcu.matmul_nt(x, np.ascontiguousarray(w13[order]))
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"prefill_tc_sk", -1))
    stacked = np.empty((m, 2 * f), np.uint16)
    stacked[:, order] = h
    want = lcu.silu(np.ascontiguousarray(stacked[:, :f]), np.ascontiguousarray(stacked[:, f:]))
    got = lcu.matmul_nt_gated(x, w13, tile)
    # the fused gate's quotient is within two binary32 units of the division's: now and then one unit of the half result
    off = np.abs(got.astype(np.int32) - want.astype(np.int32))
    assert off.max() <= 1 and (off > 0).mean() < 0.01
    # and against the oracle's product + gate (binary64 accumulation), at the GEMM's tolerance
    ref = np.zeros((m, f), np.uint16)
    L.orc_matmul_nt_f16_gated(ref.reshape(-1), x.reshape(-1), w13.reshape(-1), m, k, f, 1)
    scale = max(1.0, float(np.abs(f32(ref)).max()))
    assert np.abs(f32(got) - f32(ref)).max() <= 4e-3 * scale


def test_gate_arithmetic_against_the_division_for_every_half(lcu):
    """The one-launch w1|w3 + gate forms a / (1 + expf(-a)) with __fdividef (two units of binary32 off the division,
    llama_cu.cu:533-539 divides): rounded to half, all but a few of the 65536 half-precision a give the same value."""
    import ctypes as C
    checked, diff = C.c_uint64(0), C.c_uint64(0)
    lcu.check(lcu.lib.lcu_selftest_silu_arithmetic(C.byref(checked), C.byref(diff)))
    assert checked.value == 65536
    assert diff.value <= 64


def test_quantizer_arithmetic_on_its_whole_domain(lcu):
    """The quantizer truncates x / scale + 128, the quotient formed from the block's 1 / scale, instead of rounding
    127.5f + x / scale (transform.cu:60-80).  The device compares the two for every pair the quantizer can meet - every positive finite half as scale, every finite half within
    the absmax that rounds to it: about two billion pairs - and must find no differing byte."""
    import ctypes as C
    checked, diff = C.c_uint64(0), C.c_uint64(0)
    lcu.check(lcu.lib.lcu_selftest_quantizer_arithmetic(C.byref(checked), C.byref(diff)))
    assert checked.value > 1_000_000_000
    assert diff.value == 0


def test_matmul_rejects_bad_shapes(lcu):
    with pytest.raises(lcu.LcuError, match="multiple of 256"):
        lcu.matmul_nt(np.zeros((1, 100), np.uint16), np.zeros((4, 100), np.uint16))


# ------------------------------------------------------------------ row-wise operators
def test_rms_norm_silu(lcu):
    rng = np.random.default_rng(5)
    x, w = f16(rng.standard_normal((6, 4096)) * 2), f16(1 + 0.1 * rng.standard_normal(4096))
    y = lcu.rms_norm(x, w, 1e-6)
    yo = np.zeros_like(x)
    L.orc_rms_norm(yo.reshape(-1), x.reshape(-1), w, 6, 4096, 1e-6)
    ulp_diff = np.abs(y.astype(np.int32) - yo.astype(np.int32))
    assert ulp_diff.max() <= 1 and (ulp_diff > 0).mean() < 0.02  # rsqrt: device intrinsic vs libm
    if R.available():
        yr = np.zeros_like(x)
        assert R.lib().ref_rms_norm(yr, x, w, 6, 4096, 1e-6) == 0
        assert (y == yr).all()  # same summation order, same intrinsics: bit exact
    a, b = f16(rng.standard_normal(11008) * 3), f16(rng.standard_normal(11008))
    o = lcu.silu(a, b)
    oo = np.zeros_like(a)
    L.orc_silu(oo, a, b, a.size)
    d = np.abs(o.astype(np.int32) - oo.astype(np.int32))
    assert d.max() <= 1 and (d > 0).mean() < 0.02  # expf: device vs libm
    if R.available():
        orf = np.zeros_like(a)
        assert R.lib().ref_silu(orf, a, b, a.size) == 0
        assert (o == orf).all()


def test_rope_scatter(lcu):
    rng = np.random.default_rng(6)
    m, dim, H, pos0, ctx = 5, 256, 2, 9, 32
    q, k, v = (f16(rng.standard_normal((m, dim))) for _ in range(3))
    qr, kc, vc = lcu.rope_scatter(q, k, v, H, pos0, ctx)
    qo, ko = np.zeros_like(q), np.zeros_like(k)
    L.orc_rotary(qo.reshape(-1), q.reshape(-1), m, dim, H, pos0, 10000.0)
    L.orc_rotary(ko.reshape(-1), k.reshape(-1), m, dim, H, pos0, 10000.0)
    hd = dim // H
    k_rows = kc[:, pos0:pos0 + m, :].transpose(1, 0, 2).reshape(m, dim)
    v_rows = vc[:, pos0:pos0 + m, :].transpose(1, 0, 2).reshape(m, dim)
    assert (v_rows == v).all()
    assert (kc[:, :pos0] == 0).all() and (kc[:, pos0 + m:] == 0).all()
    for mine, want in ((qr, qo), (k_rows, ko)):
        assert np.abs(f32(mine) - f32(want)).max() <= 4e-3  # powf/sinf/cosf: device vs libm
    if R.available():
        rr = np.zeros_like(q)
        assert R.lib().ref_rotary(rr, q, m, dim, H, pos0) == 0
        assert (qr == rr).all()  # same libdevice calls as the reference kernel: bit exact


@pytest.mark.parametrize("m,T0,H,cluster", [(1, 0, 2, 1), (1, 1, 2, 8), (1, 37, 2, 4), (1, 383, 4, 8), (1, 2047, 2, 8), (7, 5, 2, 1),
                                            (16, 0, 3, 1), (1, 100, 2, 2),
                                            # cluster 0 = the prompt kernel (64-row query tiles on tensor cores)
                                            (7, 5, 2, 0), (64, 0, 2, 0), (65, 37, 1, 0), (200, 0, 2, 0), (130, 300, 2, 0), (1, 77, 2, 0),
                                            # cluster -1 = the prompt path on tcgen05 (scores, softmax, probabilities x V)
                                            (7, 5, 2, -1), (128, 0, 1, -1), (200, 0, 2, -1), (130, 300, 2, -1), (512, 0, 4, -1), (1, 77, 2, -1),
                                            # cluster -2 = the same path in one kernel (scores in tensor memory, no score buffer)
                                            (7, 5, 2, -2), (128, 0, 1, -2), (200, 0, 2, -2), (130, 300, 2, -2), (512, 0, 4, -2), (1, 77, 2, -2),
                                            (129, 127, 2, -2), (1000, 24, 2, -2), (300, 1700, 1, -2), (65, 0, 1, -2), (100, 1948, 1, -2),
                                            (66, 3, 3, -2)])
def test_attention_against_oracle(lcu, m, T0, H, cluster):
    rng = np.random.default_rng(T0 + m)
    dim = H * 128
    T = T0 + m
    q, k, v = f16(rng.standard_normal((m, dim))), f16(rng.standard_normal((T, dim))), f16(rng.standard_normal((T, dim)))
    out = lcu.attention(q, k, v, H, T0, cluster)
    oo = np.zeros_like(q)
    L.orc_attention(oo.reshape(-1), q.reshape(-1), k.reshape(-1), v.reshape(-1), m, T, dim, H, T0, 0)
    # identical rounding points; only the order of fp32 sums and expf ulps differ
    assert np.abs(f32(out) - f32(oo)).max() <= 4e-3, (m, T0, H, cluster)
    # The reference's score kernel writes rows with stride m while its softmax / PV kernels read them
    # with stride T (llama_cu.cu:418 vs 437, 526); the two agree only for m == 1 or start_pos == 0,
    # which are the only cases its own client produces - the comparison is limited to those.
    if R.available() and (m == 1 or T0 == 0):
        orf = np.zeros_like(q)
        assert R.lib().ref_attention(orf, q, k, v, m, T, dim, H, T0) == 0
        assert np.abs(f32(out) - f32(orf)).max() <= 4e-3


@pytest.mark.parametrize("T0,H,hd,cluster", [(0, 2, 128, 1), (37, 2, 128, 4), (383, 4, 128, 8), (2047, 2, 128, 8), (600, 1, 128, 2), (1500, 3, 64, 8),
                                              (129, 2, 128, 1)])
def test_attention_streaming_kernel_gives_the_same_bits(lcu, T0, H, hd, cluster):
    """Long slices come through a shared-memory ring of bulk copies instead of per-thread loads; thread-to-row
    assignment and summation order are the same, so the two kernels must agree bit for bit."""
    rng = np.random.default_rng(T0 + H)
    dim, T = H * hd, T0 + 1
    q, k, v = f16(rng.standard_normal((1, dim))), f16(rng.standard_normal((T, dim))), f16(rng.standard_normal((T, dim)))
    outs = []
    try:
        for mode in (0, 1):
            lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", mode))
            outs.append(lcu.attention(q, k, v, H, T0, cluster))
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", -1))
    assert (outs[0] == outs[1]).all()
    oo = np.zeros_like(q)
    L.orc_attention(oo.reshape(-1), q.reshape(-1), k.reshape(-1), v.reshape(-1), 1, T, dim, H, T0, 0)
    assert np.abs(f32(outs[1]) - f32(oo)).max() <= 4e-3


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("T0", [0, 7, 8, 63, 64, 127, 510, 511, 512, 1023, 1024])
def test_attention_slices_at_the_edges_of_chunks(lcu, T0, hd):
    """One query row over slices that are empty, end with a chunk of 64 rows or one row behind it, through both decode kernels, for every
    cluster size: equal bits of the two, and the oracle's row.  Bound: the oracle rounds every probability to half (2^-11 of it), so
    its row may be off by 2^-11 max|v| < 2.5e-3 here, and both round the result (|row| < 4.5: 2^-9)."""
    H = 2
    rng = np.random.default_rng(T0 + hd)
    dim, T = H * hd, T0 + 1
    q, k, v = f16(rng.standard_normal((1, dim))), f16(rng.standard_normal((T, dim))), f16(rng.standard_normal((T, dim)))
    oo = np.zeros_like(q)
    L.orc_attention(oo.reshape(-1), q.reshape(-1), k.reshape(-1), v.reshape(-1), 1, T, dim, H, T0, 0)
    for cluster in (1, 2, 4, 8):
        outs = []
        try:
            for mode in (0, 1):
                lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", mode))
                outs.append(lcu.attention(q, k, v, H, T0, cluster))
        finally:
            lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", -1))
        assert (outs[0] == outs[1]).all()
        assert np.abs(f32(outs[0]) - f32(oo)).max() <= 2.5e-3 + 2.0**-9, cluster


@pytest.mark.parametrize("hd,T", [(128, 73632), (64, 87968), (64, 110000)])
def test_attention_over_more_positions_than_ever_fitted_in_shared_memory(lcu, hd, T):
    """Nothing is kept per position: one CTA takes any slice, in both decode kernels, with equal bits.  Against binary64; bound: the result's
    rounding to half (2^-11 of it); scores that round to another half (one of a thousand, by 2^-9 of its weight) and binary32 sums move a
    row by less than 1e-6, a chunk of 64 rows too few by 1e-4."""
    rng = np.random.default_rng(T)
    q, k, v = f16(rng.standard_normal((1, hd))), f16(rng.standard_normal((T, hd))), f16(rng.standard_normal((T, hd)))
    s = ((f32(k).astype(np.float64) @ f32(q)[0]) / np.sqrt(hd)).astype(np.float16).astype(np.float64)
    e = np.exp(s - s.max())
    want = (e / e.sum()) @ f32(v).astype(np.float64)
    outs = []
    try:
        for mode in (0, 1):
            lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", mode))
            outs.append(lcu.attention(q, k, v, 1, T - 1, 1))
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", -1))
    assert (outs[0] == outs[1]).all() and 1e-3 < np.abs(want).max() < 0.1
    assert np.abs(f32(outs[0])[0] - want).max() <= 2.0**-11 * np.abs(want).max() + 1e-6


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("score", [np.nan, -np.inf])
def test_attention_of_a_key_whose_score_is_no_number(lcu, hd, score):
    """A cached key that overflowed, at every place of short slices and alone in its warp and CTA or not: a score that is NaN makes the whole
    row NaN, as in the formula and in prompt attention; a score of -inf weighs nothing, unless there is no other (0 / 0).  Values stay
    finite.  Bound of the rows that are numbers: as in the test of chunk edges."""
    H = 2
    rng = np.random.default_rng(hd)
    for T0 in (0, 1, 6, 15, 38):
        T, dim = T0 + 1, H * hd
        q, k, v = rng.standard_normal((1, dim)), rng.standard_normal((T, dim)), f16(rng.standard_normal((T, dim)))
        q[0, :2] = 1.0, -1.0
        want = np.zeros((T, dim))  # by place of the key
        for at in range(T):
            kk = k.copy()
            kk[at, :2] = (np.inf, np.inf) if np.isnan(score) else (-np.inf, 0.0)
            qh, kh, vh = f32(f16(q)).reshape(H, hd), f32(f16(kk)).reshape(T, H, hd), f32(v).reshape(T, H, hd)
            with np.errstate(invalid="ignore"):
                s = (np.einsum("hd,thd->ht", qh, kh) / np.sqrt(hd)).astype(np.float16).astype(np.float64)
                e = np.exp(s - s.max(1, keepdims=True))
                want[at] = np.einsum("ht,thd->hd", e / e.sum(1, keepdims=True), vh).reshape(-1)
            assert np.isnan(want[at, :hd]).all() == (np.isnan(score) or T == 1) and np.isfinite(want[at, hd:]).all()
            got = [lcu.attention(f16(q), f16(kk), v, H, T0, 0)] if np.isnan(score) else []  # (prompt attention)
            try:
                for mode in (0, 1):
                    lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", mode))
                    got += [lcu.attention(f16(q), f16(kk), v, H, T0, cluster) for cluster in (1, 2, 8)]
            finally:
                lcu.check(lcu.lib.lcu_set_tuning(b"attn_stream", -1))
            for i, g in enumerate(got):
                g = f32(g)[0]
                assert (np.isnan(g) == np.isnan(want[at])).all(), (T, at, i)
                assert np.nanmax(np.abs(g - want[at]), initial=0) <= 2.5e-3 + 2.0**-9, (T, at, i)


@pytest.mark.parametrize("m,T0,cluster", [(1, 50, 4), (70, 9, 0), (70, 9, -1), (300, 100, -1), (70, 9, -2), (300, 100, -2)])
def test_attention_head_dim_64(lcu, m, T0, cluster):
    rng = np.random.default_rng(8)
    H, dim = 4, 256
    T = T0 + m
    q, k, v = f16(rng.standard_normal((m, dim))), f16(rng.standard_normal((T, dim))), f16(rng.standard_normal((T, dim)))
    out = lcu.attention(q, k, v, H, T0, cluster)
    oo = np.zeros_like(q)
    L.orc_attention(oo.reshape(-1), q.reshape(-1), k.reshape(-1), v.reshape(-1), m, T, dim, H, T0, 0)
    assert np.abs(f32(out) - f32(oo)).max() <= 4e-3


@pytest.mark.parametrize("vocab", [200, 255, 256, 1000, 32000])  # one CTA below 256, a cluster from there on
def test_logits_head_of_rows_without_a_number(lcu, vocab):
    """No probability is a number where a logit is NaN or infinite, or all are -inf: token 0, as std::max_element over such a row gives
    (a chained step feeds it back, so it has to lie inside the embedding table)."""
    rng = np.random.default_rng(vocab)
    rows = [np.full(vocab, np.nan), np.full(vocab, -np.inf)]
    for value in (np.nan, np.inf):
        for at in (0, vocab // 2, vocab - 1):
            rows.append(rng.standard_normal(vocab))
            rows[-1][at] = value
    for row in rows:
        token, probs = lcu.logits_head(f16(row), 0.8)
        assert token == 0 and np.isnan(f32(probs)).all()
    row = rng.standard_normal(vocab)
    row[vocab // 3:] = -np.inf  # (some of them: no reason to worry)
    token, probs = lcu.logits_head(f16(row), 0.8)
    assert token == f16(row).view(np.float16).argmax() and np.isfinite(f32(probs)).all()


def test_logits_head_first_maximum_and_ties(lcu):
    rng = np.random.default_rng(9)
    V = 32000
    lg = f16(rng.standard_normal(V) * 1.3)
    tok, probs = lcu.logits_head(lg, 0.8)
    po = np.zeros(V, np.uint16)
    L.orc_softmax_rows(po, lg, 1, V, 0.8)
    assert np.abs(probs.astype(np.int32) - po.astype(np.int32)).max() <= 1
    assert tok == int(np.argmax(f32(probs)))  # numpy argmax = first maximum, like std::max_element
    # exact ties in the logits and ties created by the fp16 rounding of the probabilities
    lg2 = lg.copy()
    top = int(np.argmax(f32(lg2)))
    lg2[[17, 4000, 31999]] = lg2[top]
    tok2, probs2 = lcu.logits_head(lg2, 0.8)
    assert tok2 == min(17, top) and tok2 == int(np.argmax(f32(probs2)))
    flat = np.full(1000, f16(0.25), np.uint16)
    tok3, _ = lcu.logits_head(flat, 1.0)
    assert tok3 == 0


def test_bounded_wait_reports_and_leaves_the_context_usable(lcu):
    """Every mbarrier wait in the kernels is bounded.  A probe kernel waits on a barrier that nothing completes: the
    wait runs out (about a second), the kernel ends, the host gets status 4 with the device code, and the next
    operation on the same context works."""
    import ctypes as C
    import time
    code = C.c_int(0)
    t0 = time.perf_counter()
    rc = lcu.lib.lcu_selftest_bounded_wait(C.byref(code))
    dt = time.perf_counter() - t0
    assert rc == 4 and code.value == 0x101, (rc, hex(code.value))
    assert b"bounded wait" in lcu.lib.lcu_last_error()
    assert 0.3 < dt < 10.0, dt
    x = f16(np.ones((1, 256)))
    w = f16(np.full((64, 256), 0.5))
    y = lcu.matmul_nt(x, w)
    assert (f32(y) == 128.0).all()
