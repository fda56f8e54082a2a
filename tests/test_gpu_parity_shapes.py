"""Parity where the decode kernels actually run: the single-row (batch-1) weight-streaming GEMV in every weight mode
(fp16; u8 with the reference's per-weight rounding, llama_cu.cu:287-289; u8 with factored scales), every block size,
ragged last chunks, and the row lengths of the 13B and 65B models; attention at 40 and 64 heads over ~2100 cached
positions; one-layer models at 13B / 65B widths so that the fused RMSNorm / RoPE / SiLU epilogues run at those shapes;
and the pedantic kernels of matmul_type 1.  Everything goes through the C ABI and is compared with the CPU oracle and,
where the reference library is present and its kernels accept the shape, with the reference's own kernels."""
import contextlib
import functools

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


@contextlib.contextmanager
def tuning(lcu, key, value, default):
    lcu.check(lcu.lib.lcu_set_tuning(key, value))
    try:
        yield
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(key, default))


@contextlib.contextmanager
def matmul_type(lcu, value):
    lcu.check(lcu.lib.lcu_set_matmul_type(value))
    try:
        yield
    finally:
        lcu.check(lcu.lib.lcu_set_matmul_type(4))


def gold(x, w=None, q=None, s=None, bs=0, rounded=1):
    m, k = x.shape
    n = (w if w is not None else q).shape[0]
    out = np.zeros((m, n), np.float64)
    L.orc_matmul_nt_gold(out.reshape(-1), x.reshape(-1), None if w is None else w.ctypes.data, None if q is None else q.ctypes.data,
                         None if s is None else s.ctypes.data, m, k, n, bs, rounded)
    return out


# ------------------------------------------------------------------ single-row u8 GEMV, both weight modes
U8_SHAPES = [(256, 64), (4096, 4096), (11008, 4096), (8192, 128), (22016, 34)]  # (K, N): short rows, the single-layer shape,
                                                                                 # a ragged last chunk (11008 = 2.69 chunks),
                                                                                 # 65B row lengths


@functools.lru_cache(maxsize=1)
def weights_for(k, n, bs, seed, scale):
    """Seeded weights (and their quantization) of one shape; the parametrisation keeps the shape as the slowest-varying
    argument, so the CPU work is done once per shape."""
    w = O.synth_f16(n * k, seed, f"w.{n}x{k}", scale).reshape(n, k)
    q, s = O.quantize(w, n, k, bs) if bs else (None, None)
    return w, q, s


@pytest.mark.parametrize("factored", [0, 1])
@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("bs", [32, 64, 128])
@pytest.mark.parametrize("k,n", U8_SHAPES)
def test_gemv_single_row_u8(lcu, factored, bs, k, n, beta):
    """m = 1 with u8 weights.  int8_factored = 0 is the mode that keeps the reference's rounding (every weight rounded
    to half((q - 127.5) * scale) before the product); 1 factors the scale out of each block (block size >= 64; at 32 the
    library falls back to the exact kernel).  Both are checked against the binary64 evaluation over the half-rounded
    weights (the arithmetic the reference's tensor-core kernel defines) within 1e-3 of the largest output - the task's
    bar is 1e-2 - and the exact mode additionally against the oracle's binary32 restatement of that kernel."""
    rng = np.random.default_rng(k + n + bs)
    x = f16(rng.standard_normal((1, k)))
    w, q, s = weights_for(k, n, bs, 31, 0.03)
    prev = f16(rng.standard_normal((1, n)))
    with tuning(lcu, b"int8_factored", factored, 1):
        y = f32(lcu.matmul_nt(x, q, s, bs, beta=beta, out_u16=prev))
    g = gold(x, q=q, s=s, bs=bs, rounded=1) + beta * f32(prev)
    scale = max(1.0, float(np.abs(g).max()))
    assert np.abs(y - g).max() <= 1e-3 * scale + 2.0 ** -11 * scale, (factored, bs, k, n, beta)
    yo = prev.copy()
    L.orc_matmul_nt_fp16u8(yo.reshape(-1), x.reshape(-1), q.reshape(-1), s.reshape(-1), 1, k, n, bs, beta, 0)
    assert np.abs(y - f32(yo)).max() <= 2e-3 * scale
    if R.available() and n % 128 == 0 and k % 256 == 0:  # the reference's tile kernel needs whole 128-row / 256-column tiles
        yr = f32(R.matmul_u8(x, q, s, bs, beta=beta, out=prev, mtype=4))
        mine, theirs = np.abs(y - g).max(), np.abs(yr - g).max()
        assert mine <= theirs * 1.5 + 2.0 ** -10 * scale, (mine, theirs)  # no worse than the reference's own kernel


# ------------------------------------------------------------------ 13B / 65B row lengths, fp16 and u8
BIG_SHAPES = [(5120, 5120), (5120, 2 * 13824), (13824, 5120), (8192, 3 * 8192), (22016, 8192)]  # (K, N) of wo / w1|w3 / w2 (13B), wq|wk|wv / w2 (65B)


@pytest.mark.parametrize("mode", ["f16", "u8_exact", "u8_factored"])
@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("k,n", BIG_SHAPES)
def test_gemv_single_row_large_models(lcu, k, n, mode, beta):
    rng = np.random.default_rng(k + n)
    x = f16(rng.standard_normal((1, k)))
    w, q, s = weights_for(k, n, 128, 32, 0.02)
    prev = f16(rng.standard_normal((1, n)))
    if mode == "f16":
        y = f32(lcu.matmul_nt(x, w, beta=beta, out_u16=prev))
        g = gold(x, w=w) + beta * f32(prev)
    else:
        with tuning(lcu, b"int8_factored", int(mode == "u8_factored"), 1):
            y = f32(lcu.matmul_nt(x, q, s, 128, beta=beta, out_u16=prev))
        g = gold(x, q=q, s=s, bs=128, rounded=1) + beta * f32(prev)
    scale = max(1.0, float(np.abs(g).max()))
    assert np.abs(y - g).max() <= 1e-3 * scale + 2.0 ** -11 * scale, (k, n, mode, beta)
    if R.available() and beta == 0.0:
        yr = f32(R.matmul_f16(x, w, mtype=4)) if mode == "f16" else f32(R.matmul_u8(x, q, s, 128, mtype=4))
        mine, theirs = np.abs(y - g).max(), np.abs(yr - g).max()
        assert mine <= theirs * 1.5 + 2.0 ** -10 * scale, (mine, theirs)


# ------------------------------------------------------------------ attention at 13B / 65B head counts, long context
@pytest.mark.parametrize("m,T0,H,cluster", [(1, 2099, 40, 8), (1, 2099, 64, 8), (1, 2175, 40, 8), (1, 640, 64, 8),
                                            (260, 1840, 40, -1), (130, 1970, 64, 0)])
def test_attention_at_large_model_head_counts(lcu, m, T0, H, cluster):
    rng = np.random.default_rng(T0 + H)
    dim, T = H * 128, T0 + m
    q, k, v = f16(rng.standard_normal((m, dim))), f16(rng.standard_normal((T, dim))), f16(rng.standard_normal((T, dim)))
    out = lcu.attention(q, k, v, H, T0, cluster)
    oo = np.zeros_like(q)
    L.orc_attention(oo.reshape(-1), q.reshape(-1), k.reshape(-1), v.reshape(-1), m, T, dim, H, T0, 0)
    assert np.abs(f32(out) - f32(oo)).max() <= 4e-3, (m, T0, H, cluster)
    if R.available() and m == 1:
        orf = np.zeros_like(q)
        assert R.lib().ref_attention(orf, q, k, v, m, T, dim, H, T0) == 0
        assert np.abs(f32(out) - f32(orf)).max() <= 4e-3


# ------------------------------------------------------------------ fused epilogues at 13B / 65B widths
@pytest.mark.parametrize("dim,n_heads", [(5120, 40), (8192, 64)])
@pytest.mark.parametrize("mode", ["f16", "u8_exact", "u8_factored"])
def test_one_layer_model_at_large_widths(lcu, dim, n_heads, mode):
    """One layer + head at the 13B / 65B widths: the decode kernels with their fused prologues and epilogues (RMSNorm,
    RoPE + cache write at 40 / 64 heads, SiLU gate over w1|w3 of 13824 / 22016 rows, residual adds) against the oracle's
    forward pass on identical weights.  Teacher-forced on the oracle's tokens."""
    bs = 0 if mode == "f16" else 128
    cfg = dict(dim=dim, n_heads=n_heads, n_layers=1, n_vocab=2000)
    scale = 0.02
    model = lcu.Model.synthetic(block_size=bs, seed=77, scale=scale, **cfg)
    om = O.OracleModel(multiple_of=256, block_size=bs, seed=77, scale=scale, context_len=48, temperature=0.8, **cfg)
    prompt = O.synth_tokens(5, 77, lo=3, hi=2000)  # a 5-row prompt goes through the multi-row GEMV
    with tuning(lcu, b"int8_factored", int(mode != "u8_exact"), 1):
        ctx = lcu.Context(model, context_len=48, temperature=0.8)
        t, to = ctx.next_token(prompt), om.next_token(prompt)
        agree = []
        for step in range(10):
            h, ho = f32(ctx.hidden()), f32(om.last_hidden())
            assert np.abs(h - ho).max() <= 0.02 * np.abs(ho).max(), (step, mode)
            p, po = f32(ctx.probs()), f32(om.probs())
            assert np.abs(p - po).max() <= 0.02 * po.max() + 1e-4, (step, mode)
            agree.append(t == to)
            t, to = ctx.next_token([to]), om.next_token([to])
        chained, _ = ctx.decode_chained(t, 4)  # the captured graph at these shapes
        assert len(chained) == 4
        ctx.close()
    assert np.mean(agree) >= 0.8, agree
    om.close()
    model.close()


@pytest.mark.parametrize("dim", [4096, 4352, 6400, 8192, 8448])
def test_norm_weights_of_rows_longer_than_the_first_vectors(lcu, dim):
    """wq|wk|wv, w1|w3 and the output matrix with every norm weight of its own, where a thread's norm weights are its first four vectors of the
    row, a fifth, all eight, and more: against the kernel that shares no code with it (16-row blocks).  Bound: between the two, sums differ
    in their order only, so that halves rounded on the way move by one unit at most, three roundings in a chain - 2^-9 of the logits'
    RMS; norm weights of one vector that belong to another move them by 1e-2."""
    model = lcu.Model.synthetic(dim=dim, n_heads=dim // 128, n_layers=1, n_vocab=512, seed=7, scale=0.02)
    rng = np.random.default_rng(dim)
    for name in ("layers.0.attention_norm", "layers.0.ffn_norm", "norm"):
        w = f16(rng.choice([-1.0, 1.0], dim) * rng.uniform(0.5, 1.5, dim))
        ptr, size, _ = model.tensor(name, 0)
        assert size == w.nbytes
        lcu.check(lcu.lib.lcu_memcpy_h2d(ptr, w.ctypes.data, size))
    rows = []
    for variant in (0, 1):
        with tuning(lcu, b"gemv_variant", variant, 1):
            ctx = lcu.Context(model, context_len=16, temperature=0.8)
            rows.append(np.concatenate([ctx.step([t], [0]) for t in (5, 9, 300)]).astype(np.float64))
            ctx.close()
    error = np.sqrt(((rows[1] - rows[0]) ** 2).mean(1)) / np.sqrt((rows[0] ** 2).mean(1))
    assert np.isfinite(rows[1]).all() and error.max() <= 2.0 ** -9, error
    model.close()


# ------------------------------------------------------------------ matmul_type 1: the pedantic kernels
@pytest.mark.parametrize("m,k,n,bs,beta", [(1, 256, 64, 0, 0.0), (3, 768, 130, 0, 1.0), (1, 4096, 512, 128, 0.0), (5, 512, 96, 64, 1.0),
                                           (2, 256, 33, 32, 0.0)])
def test_pedantic_kernels_are_the_reference_naive_pair(lcu, m, k, n, bs, beta):
    """matmul_type 1 adds the K terms in index order (binary32 sum; u8: binary64 terms, the sum rounded to binary32
    after each addition, llama_cu.cu:111-145): bit-identical to the oracle's restatement of those kernels and to the
    reference's own matmul_type 1."""
    rng = np.random.default_rng(m + k + n)
    x = f16(rng.standard_normal((m, k)))
    w = O.synth_f16(n * k, 33, f"ped.{n}x{k}", 0.05).reshape(n, k)
    prev = f16(rng.standard_normal((m, n)))
    yo = prev.copy()
    with matmul_type(lcu, 1):
        if bs == 0:
            y = lcu.matmul_nt(x, w, beta=beta, out_u16=prev)
            L.orc_matmul_nt_f16(yo.reshape(-1), x.reshape(-1), w.reshape(-1), m, k, n, beta, 0)
        else:
            q, s = O.quantize(w, n, k, bs)
            y = lcu.matmul_nt(x, q, s, bs, beta=beta, out_u16=prev)
            L.orc_matmul_nt_fp16u8(yo.reshape(-1), x.reshape(-1), q.reshape(-1), s.reshape(-1), m, k, n, bs, beta, 1)
    assert (y == yo).all(), np.abs(f32(y) - f32(yo)).max()
    if R.available():
        yr = R.matmul_f16(x, w, beta=beta, out=prev, mtype=1) if bs == 0 else R.matmul_u8(x, q, s, bs, beta=beta, out=prev, mtype=1)
        assert (y == yr).all()


@pytest.mark.parametrize("bs", [0, 128])
def test_pedantic_context_against_oracle_naive_mode(lcu, bs):
    """With matmul_type 1 every product of next_token runs on the pedantic kernels; the oracle in its naive-matmul mode
    evaluates the same sums in the same order, so the two forward passes differ only by libm / device ulps of exp, rsqrt,
    sin and cos and by the summation order inside attention: the residual stream must agree far tighter than between
    the fast kernels and the oracle."""
    cfg = dict(dim=256, n_heads=2, n_layers=3, n_vocab=1000)
    model = lcu.Model.synthetic(block_size=bs, seed=1234, scale=0.08, **cfg)
    om = O.OracleModel(multiple_of=256, block_size=bs, seed=1234, scale=0.08, context_len=64, temperature=0.8, **cfg)
    om.set_modes(wmma_rounding=0)
    prompt = O.synth_tokens(12, 1234, lo=3, hi=1000)
    with matmul_type(lcu, 1):
        ctx = lcu.Context(model, context_len=64, temperature=0.8)
        t, to = ctx.next_token(prompt), om.next_token(prompt)
        same = []
        for step in range(12):
            h, ho = f32(ctx.hidden()), f32(om.last_hidden())
            assert np.abs(h - ho).max() <= 4e-3 * np.abs(ho).max(), step
            same.append(t == to)
            t, to = ctx.next_token([to]), om.next_token([to])
        with pytest.raises(lcu.LcuError, match="matmul_type 1"):
            ctx.decode_chained(t, 2)
        ctx.close()
    assert np.mean(same) >= 0.9, same
    # the fast kernels on the same context length agree with the pedantic run on the tokens where the margin is clear
    om.close()
    model.close()


def test_context_memory_matches_the_partitioners_figures(lcu):
    """context_memory_usage = scratch arena + K/V caches, exactly the two figures the memory-based partitioner packs with."""
    cfg = dict(dim=512, n_heads=4, n_layers=4, n_vocab=2000)
    for bs in (0, 128):
        model = lcu.Model.synthetic(block_size=bs, seed=3, scale=0.05, **cfg)
        ctx = lcu.Context(model, context_len=512, temperature=0.8)
        raw = lcu.pack_params(512, 256, 4, 4, 2000, 1e-6, bs)
        want = lcu.lib.lcu_context_scratch_bytes(raw, 512) + 4 * lcu.lib.lcu_context_kv_bytes_per_layer(raw, 512)
        assert ctx.memory_usage() == want
        ctx.close()
        model.close()
