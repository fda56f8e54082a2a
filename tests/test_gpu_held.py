"""Small matrices of a single activation row are held in registers instead of streamed through a ring of shared memory: the two
kernels form every sum in the same order, so their results are compared bit for bit; each is compared with the oracle elsewhere."""
import numpy as np
import pytest

import block_cases as B
import oracle_lib as O
from block_runs import run  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu


def f16(a):
    return np.ascontiguousarray(np.asarray(a, np.float16)).view(np.uint16)


def both_kernels(lcu, fn):
    out = []
    try:
        for mode in (0, -1):
            lcu.check(lcu.lib.lcu_set_tuning(b"gemv_held", mode))
            out.append(fn())
    finally:
        lcu.check(lcu.lib.lcu_set_tuning(b"gemv_held", -1))
    return out


# rows of half a chunk (two row pairs per warp from 592 pairs on), of one chunk, of one and a part, of a half segment (u8), past the rule
@pytest.mark.parametrize("bs", [0, 64, 128])
@pytest.mark.parametrize("k,n", [(256, 2), (256, 2400), (512, 1186), (768, 34), (1024, 2816), (1024, 1182), (1280, 1536), (2048, 2048), (2304, 256),
                                 (2816, 1024), (3072, 3552), (4096, 130), (4352, 96), (5632, 2048), (6144, 514)])
def test_products_have_the_same_bits(lcu, k, n, bs):
    rng = np.random.default_rng(k + n)
    x, prev = f16(rng.standard_normal((1, k))), f16(rng.standard_normal((1, n)))
    w = O.synth_f16(n * k, 99, f"w{n}x{k}", 0.05).reshape(n, k)
    q, s = O.quantize(w, n, k, bs) if bs else (w, None)
    ring, held = both_kernels(lcu, lambda: lcu.matmul_nt(x, q, s, bs, beta=1.0, out_u16=prev.copy()) if bs else lcu.matmul_nt(x, q, beta=1.0, out_u16=prev.copy()))
    assert np.isfinite(ring.view(np.float16).astype(np.float32)).all() and np.array_equal(ring, held)


@pytest.mark.parametrize("k,n", [(1280, 888), (1280, 890), (1536, 600), (1792, 1792), (2304, 1184), (2304, 1186), (3072, 1000)])
def test_fp16_products_on_both_sides_of_the_rule(lcu, k, n):
    test_products_have_the_same_bits(lcu, k, n, 0)


@pytest.mark.parametrize("dim,heads,bs", [(256, 2, 0), (512, 8, 64), (1024, 8, 0), (1024, 16, 128), (1280, 10, 0), (2048, 16, 128), (2048, 16, 0)])
def test_decode_steps_have_the_same_bits(lcu, dim, heads, bs):
    """Norms, rotation and cache rows, gate and residual of a step: greedy tokens and the last probabilities."""
    model = lcu.Model.synthetic(dim=dim, n_heads=heads, n_layers=2, n_vocab=1000, block_size=bs, seed=5, scale=0.08)

    def go():
        ctx = lcu.Context(model, context_len=64, temperature=0.8)
        t = ctx.next_token(list(range(3, 12)))
        toks = ctx.decode_chained(t, 6)[0]
        probs = ctx.probs().copy()
        ctx.close()
        return toks, probs

    (t0, p0), (t1, p1) = both_kernels(lcu, go)
    assert np.array_equal(t0, t1) and np.array_equal(p0, p1)
    model.close()


@pytest.mark.parametrize("name", ["routed", "recurrent"])
def test_block_model_steps_have_the_same_bits(lcu, run, name):  # noqa: F811
    """Batches of matrices, gated pairs, picked experts in bfloat16."""
    if name == "routed":
        cfg, W = B.latent_case(seed=3, layers=2, width=384, experts=6, top=2, ff=128, mixer=dict(heads=6, dim=64, rot_dim=32, vdim=64, kv_rank=192, window=40))
    else:
        cfg, W = B.case(seed=3)
    t = B.tokens(cfg, 20, 1)
    ring, held = both_kernels(lcu, lambda: run(cfg, W, "bfloat16").feed(t, [1]))
    assert np.isfinite(ring).all() and np.array_equal(ring, held)
