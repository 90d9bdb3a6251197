"""Operator-level parity on the GPU: every method of the Backend mirror, the dequantisers and the
quantised matmuls against the CPU oracle, through the C ABI."""
import numpy as np
import pytest

from conftest import assert_close

pytestmark = pytest.mark.gpu

ALL_TYPES = [0, 1, 2, 8, 12, 13, 14, 20]


def rng(seed):
    return np.random.default_rng(seed)


def test_matmul_f32_is_bit_exact(gpu, oracle):
    be = gpu.B200Backend()
    r = rng(1)
    for (m, k, n) in [(2, 2, 2), (2, 3, 3), (16, 32, 24), (5, 77, 41), (128, 256, 128), (1, 512, 40)]:
        a = r.standard_normal(m * k).astype(np.float32)
        b = r.standard_normal(k * n).astype(np.float32)
        got = be.matmul(a, b, m, k, n)
        want = oracle.matmul(a, b, m, k, n)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (m, k, n)


def test_vector_ops_are_bit_exact(gpu, oracle):
    be = gpu.B200Backend()
    r = rng(2)
    for n in [1, 5, 1000, 4097]:
        a = r.standard_normal(n).astype(np.float32)
        b = r.standard_normal(n).astype(np.float32)
        assert np.array_equal(be.vec_add(a, b), oracle.vec_add(a, b))
        assert np.array_equal(be.vec_mul(a, b), oracle.vec_mul(a, b))
        assert np.array_equal(be.vec_scale(a, 0.37), oracle.vec_scale(a, np.float32(0.37)))
        assert np.array_equal(be.vec_scale_mul(a, 1.7, b), oracle.vec_scale_mul(a, np.float32(1.7), b))


def test_rms_norm_silu_softmax_sum_sq(gpu, oracle):
    be = gpu.B200Backend()
    r = rng(3)
    for hidden, rows in [(3, 1), (64, 4), (2048, 3), (4096, 2), (11008, 1)]:
        x = (r.standard_normal(hidden * rows) * 2).astype(np.float32)
        w = r.standard_normal(hidden).astype(np.float32)
        # sum of squares: different association than the reference's 4 strided lanes -> a few ulp of the sum
        assert_close(be.rms_norm(x, w, 1e-5, hidden), oracle.rms_norm(x, w, 1e-5, hidden), 1e-6, 2e-6, "rms_norm")
        assert_close(be.silu(x), oracle.silu(x), 1e-6, 1e-6, "silu")
        assert_close(be.softmax(x, hidden), oracle.softmax(x, hidden), 1e-8, 2e-6, "softmax")
        assert abs(be.sum_sq(x) - oracle.sum_sq(x)) <= 2e-6 * oracle.sum_sq(x)
    y = be.softmax(np.array([1.0, 2.0, 3.0], np.float32), 3)  # rust/src/model/tensor.rs:211-216
    assert abs(y.sum() - 1.0) < 1e-5


@pytest.mark.parametrize("typ", ALL_TYPES)
def test_dequantize_bit_exact_on_random_bytes(gpu, oracle, typ):
    be_elems, bb = gpu.QUANT_GEOMETRY[typ]
    r = rng(100 + typ)
    nblocks = 257 if be_elems > 1 else 4099
    raw = r.integers(0, 256, nblocks * bb, dtype=np.uint8)
    n = nblocks * be_elems
    got = gpu.dequantize(typ, raw, n)
    want = oracle.dequantize(typ, raw, n)
    g, w = got.view(np.uint32), want.view(np.uint32)
    nan_both = np.isnan(got) & np.isnan(want)
    assert np.array_equal(g[~nan_both], w[~nan_both])


@pytest.mark.parametrize("typ", [2, 8, 12])
def test_dequantize_bit_exact_on_synthetic_weights(gpu, oracle, typ):
    from leafcutterllm_b200 import synth
    n = 256 * 1024
    raw = synth.host_tensor(typ, 7, "t", n)
    assert np.array_equal(gpu.dequantize(typ, raw, n).view(np.uint32), oracle.dequantize(typ, raw, n).view(np.uint32))


def test_dequantize_rejects_ragged_and_unknown(gpu):
    with pytest.raises((ValueError, gpu.LeafcutterError)):
        gpu.dequantize(12, np.zeros(144, np.uint8), 255)
    with pytest.raises(gpu.LeafcutterError):
        gpu.dequantize(3, np.zeros(32, np.uint8), 32)  # Q4_1 has no kernel in the reference either


QM_CASES = [
    # typ, m, k, n
    (12, 1, 256, 32), (12, 1, 4096, 4096), (12, 1, 11008, 4096), (12, 1, 4096, 1000), (12, 3, 2048, 96), (12, 8, 512, 33),
    (12, 9, 1024, 64), (12, 2, 11008, 128),
    (2, 1, 2048, 2048), (2, 1, 5632, 2048), (2, 4, 256, 100), (2, 1, 96, 64),
    (8, 1, 2048, 3200), (8, 5, 512, 70), (8, 1, 64, 48),
    # Q4_0 / Q8_0 on the int8 tensor-core kernel: two to four tokens, rows of one to 43 units, row counts off the 32-row tile
    (2, 2, 1024, 77), (2, 3, 2304, 40), (2, 4, 11008, 33), (8, 2, 1024, 50), (8, 3, 768, 100), (8, 4, 4096, 33), (8, 1, 11008, 65),
    (13, 1, 512, 40), (14, 2, 512, 40), (20, 1, 128, 40), (0, 2, 100, 24), (1, 1, 100, 24),
    (13, 1, 4096, 300), (13, 5, 2816, 64), (13, 8, 256, 19), (14, 1, 4096, 300), (14, 3, 11008, 40), (14, 8, 768, 21),
    (20, 1, 4096, 300), (20, 2, 2816, 33), (0, 3, 512, 40), (1, 1, 4096, 300), (1, 8, 256, 19), (1, 2, 11008, 33),
    # Q6_K on the int8 tensor-core kernel (a multiple of 16 rows, one to four tokens): one unit, an odd number of units (every
    # other row's blocks then start two bytes off a word), more units than warps, several tiles per CTA
    (14, 1, 256, 16), (14, 1, 4096, 4096), (14, 1, 11008, 4096), (14, 2, 2816, 64), (14, 3, 11008, 48), (14, 4, 768, 160), (14, 4, 8192, 32),
    (14, 1, 4096, 32000),
    # Q5_K on the Q4_K kernel's fifth-bit variant (one to four tokens)
    (13, 1, 11008, 4096), (13, 2, 2816, 77), (13, 3, 11008, 40), (13, 4, 4096, 33), (13, 1, 256, 8),
    # five to eight tokens of these types: two passes of the tensor-core kernels
    (14, 8, 4096, 64), (14, 6, 11008, 32), (14, 5, 512, 48), (13, 7, 11008, 40), (13, 8, 4096, 96),
]


@pytest.mark.parametrize("typ,m,k,n", QM_CASES)
def test_qmatmul_vs_oracle(gpu, oracle, typ, m, k, n):
    from leafcutterllm_b200 import synth
    r = rng(k * 7 + n)
    if typ in (2, 8, 12, 0, 1):
        w = synth.host_tensor(typ, 99, f"w{typ}_{k}_{n}", n * k)
    else:  # no quantiser for these: random bytes with sane f16 scales
        be_elems, bb = gpu.QUANT_GEOMETRY[typ]
        w = r.integers(0, 256, n * k // be_elems * bb, dtype=np.uint8).reshape(-1, bb)
        sc = np.float16(r.uniform(0.001, 0.01, w.shape[0])).view(np.uint16)
        off = {13: 0, 14: 208, 20: 0}[typ]
        w[:, off] = sc & 0xFF
        w[:, off + 1] = sc >> 8
        if typ == 13:
            w[:, 2] = sc & 0xFF
            w[:, 3] = sc >> 8
        w = w.ravel()
    a = r.standard_normal(m * k).astype(np.float32)
    got = gpu.qmatmul(typ, a, w, m, k, n)
    want = oracle.qmatmul(typ, a, w, m, k, n)
    scale = np.abs(want).max()
    # the reference's own tolerance for its quantised GEMMs is 1e-3 absolute (int8_gemm.rs:394-511)
    assert_close(got, want, 2e-5 * scale, 1e-4, f"qmatmul typ={typ} {m}x{k}x{n}")


@pytest.mark.parametrize("typ", [12, 13])
@pytest.mark.parametrize("m,k,n", [(9, 256, 128), (16, 512, 128), (64, 4096, 512), (40, 2816, 300), (130, 1024, 256), (200, 11008, 128)])
def test_qmatmul_q4k_many_tokens_tensor_core_gemm(gpu, oracle, monkeypatch, typ, m, k, n):
    """Q4_K and Q5_K (the same unit with a fifth bit per element).  Five tokens and more go through a tcgen05 product (up to 64: integers in tensor memory, drained
    per unit; more: weights as f16 high/low halves; activations as swizzled f16 high/low tiles): one k unit, token counts that are not a multiple of 16 or of
    the token tiles, rows that are not a multiple of 128, a long k.  Activations carry a wide dynamic range so that the
    per-token power-of-two scale matters."""
    from leafcutterllm_b200 import synth
    w = synth.host_tensor(typ, 43, f"gemm_{k}_{n}", n * k)
    r = rng(k + n + m)
    a = (r.standard_normal((m, k)) * np.exp(r.uniform(-6, 6, (m, 1)))).astype(np.float32).ravel()
    got = gpu.qmatmul(typ, a, w, m, k, n).reshape(m, n)
    want = oracle.qmatmul(typ, a, w, m, k, n).reshape(m, n)
    for t in range(m):  # per token: its own scale
        assert_close(got[t], want[t], 2e-5 * np.abs(want[t]).max(), 1e-4, f"gemm {m}x{k}x{n} token {t}")
    if m > 64:  # another kernel, which has no such form
        return
    monkeypatch.setenv("LC_GEMM_TERMS", "1")  # plain f16 operands: 2^-11 per factor
    fast = gpu.qmatmul(typ, a, w, m, k, n).reshape(m, n)
    for t in range(m):
        assert_close(fast[t], want[t], 4e-3 * np.abs(want[t]).max(), 0, f"one-term gemm token {t}")


# one unit, odd numbers of units (rows of Q6_K blocks then start two bytes off a word), token counts on both sides of the 16-token steps
# and of the tiles of 64 and 128, row counts off the 128-row tile, k cut over several CTAs (few tiles) and not
@pytest.mark.parametrize("m,k,n", [(5, 256, 1), (17, 768, 130), (64, 4096, 256), (65, 2816, 100), (128, 1024, 384), (129, 11008, 129), (300, 1280, 4100)])
@pytest.mark.parametrize("typ", [2, 8, 12, 13, 14])
def test_many_token_product_vs_oracle(gpu, oracle, typ, m, k, n):
    """Weights of both signs whose block scales differ by 2^12 inside a row and by 2^24 between rows, tokens that differ by e^12.
    A weight and an activation keep 22 bits each, and 256 products are added with truncation before each rounded sum (measured 3.5e-7 of the
    sum of squares' root before its mean is corrected): 2e-5 of that root for every single result leaves fifty times that."""
    r = rng(typ * 1000 + k + n + m)
    be, bb = gpu.QUANT_GEOMETRY[typ]
    w = r.integers(0, 256, n * k // be * bb, dtype=np.uint8).reshape(n, -1, bb)
    size = np.exp2(r.uniform(-18, 6, (n, 1))) * np.exp2(r.uniform(-12, 0, w.shape[:2])) / {2: 8, 8: 128, 12: 945, 13: 1953, 14: 4064}[typ]
    sc = (np.maximum(size, 2.0 ** -24) * r.choice([-1, 1], w.shape[:2])).astype(np.float16).view(np.uint16)
    at = 208 if typ == 14 else 0
    w[..., at], w[..., at + 1] = sc & 0xFF, sc >> 8
    if typ in (12, 13):
        w[..., 2], w[..., 3] = sc & 0xFF, sc >> 8
    w = w.ravel()
    a = (r.standard_normal((m, k)) * np.exp(r.uniform(-6, 6, (m, 1)))).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    dense = gpu.dequantize(typ, w, n * k).reshape(n, k).astype(np.float64)  # bit-exact with the oracle's (tested above)
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2))  # per result: the root of the products' sum of squares
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()
    rows = r.choice(n, min(n, 8), replace=False)
    rb = w.size // n
    sub = np.concatenate([w[i * rb:(i + 1) * rb] for i in rows])
    assert_close(want[:5, rows], oracle.qmatmul(typ, a[:5].ravel(), sub, 5, k, len(rows)).reshape(5, len(rows)), 2e-5 * np.abs(want[:5, rows]).max(), 1e-4, "oracle sample")


def scaled_blocks(gpu, typ, n, k, size, r):
    """Random blocks whose largest weight is about `size` [n, blocks of a row] (offsets as large), and the weights in 64 bits."""
    be, bb = gpu.QUANT_GEOMETRY[typ]
    w = r.integers(0, 256, n * k // be * bb, dtype=np.uint8).reshape(n, -1, bb)
    sc = np.broadcast_to(size / {2: 8, 8: 128, 12: 945, 13: 1953, 14: 4064}[typ], w.shape[:2]).astype(np.float16).view(np.uint16)
    at = 208 if typ == 14 else 0
    w[..., at], w[..., at + 1] = sc & 0xFF, sc >> 8
    if typ in (12, 13):
        w[..., 2], w[..., 3] = sc & 0xFF, sc >> 8
    w = w.ravel()
    return w, gpu.dequantize(typ, w, n * k).reshape(n, k).astype(np.float64)


@pytest.mark.parametrize("m", [16, 70])  # the tiles of up to 64 tokens and of more
@pytest.mark.parametrize("typ", [2, 8, 12, 13, 14])
def test_many_token_product_at_the_ends_of_f32(gpu, typ, m):
    """Tokens whose largest element is a denormal, just above 2^-126, or just below f32's end: the power of two that brings them to f16's range has
    an inverse in f32, and results are as exact as any (the bound of the test above, and half a denormal's step for each of the few roundings)."""
    k, n = 512, 70
    r = rng(typ + m)
    w, dense = scaled_blocks(gpu, typ, n, k, np.exp2(r.uniform(-12, -8, (n, 1))), r)
    a = r.uniform(-1, 1, (m, k))
    power = np.resize([-140, -130, -127, -126, -116, 0, 110, 126, 127], m)
    a = (a * np.exp2(power.astype(np.float64))[:, None]).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2)) + 2.0 ** -147
    assert np.isfinite(got).all()
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max(1)


@pytest.mark.parametrize("m", [16, 70])
@pytest.mark.parametrize("typ", [2, 8, 14])
def test_many_token_product_of_infinities(gpu, typ, m):
    """A token with one infinity gives infinities of the weights' signs (NaN where the weight is zero), one with a NaN gives NaN, the others what they always give."""
    k, n = 512, 70
    r = rng(typ + m + 1)
    w, dense = scaled_blocks(gpu, typ, n, k, np.ones((n, 1)), r)
    a = r.standard_normal((m, k)).astype(np.float32)
    a[0, 300], a[2, 7], a[m - 1, 511] = np.inf, -np.inf, np.nan
    a[0, 301] = 1e30  # finite, and past f16's largest
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    with np.errstate(invalid="ignore"):
        for t, c in ((0, 300), (2, 7)):
            want = a[t, c] * dense[:, c]
            assert np.array_equal(got[t], want.astype(np.float32), equal_nan=True), t
    assert np.isnan(got[m - 1]).all()
    rest = [t for t in range(m) if t not in (0, 2, m - 1)]
    want = a[rest].astype(np.float64) @ dense.T
    assert (np.abs(got[rest] - want) <= 2e-5 * np.sqrt((a[rest].astype(np.float64) ** 2) @ (dense.T ** 2))).all()


@pytest.mark.parametrize("typ", [12, 13])
@pytest.mark.parametrize("m,k,n", [(65, 256, 70), (129, 512, 300), (97, 768, 1), (70, 4352, 130), (200, 11008, 64)])
def test_many_token_product_in_pairs_of_ctas(gpu, typ, m, k, n):
    """Q4_K and Q5_K: one, two and three units (the offsets come ahead of the last), seventeen (two runs of offsets), shares of k that begin at any unit;
    row counts that leave the second CTA of a pair few rows or none, token counts that leave it few tokens.  One token holds an infinity: its results have the weights' signs."""
    r = rng(typ + m + k)
    w, dense = scaled_blocks(gpu, typ, n, k, np.exp2(r.uniform(-1, 0, (n, k // 256))), r)
    a = r.standard_normal((m, k)).astype(np.float32)
    a[3, k - 100] = -np.inf
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    with np.errstate(invalid="ignore"):
        assert np.array_equal(got[3], (a[3, k - 100] * dense[:, k - 100]).astype(np.float32), equal_nan=True)
    rest = [t for t in range(m) if t != 3]
    want = a[rest].astype(np.float64) @ dense.T
    assert np.linalg.norm(got[rest] - want) <= 4e-7 * np.linalg.norm(want)
    # 22 bits of an activation and sums that lose up to 2^-22 of a run, the offsets' as large: 1.7e-7 of the root of the products' squares in a result on average, up to
    # 2.9e-7 where eight shares of k are added; the largest of ten thousand results is up to eight times that (2.2e-6 measured): the bound of the tests above, 2e-5, leaves room
    assert (np.abs(got[rest] - want) <= 2e-5 * np.sqrt((a[rest].astype(np.float64) ** 2) @ (dense.T ** 2))).all()


@pytest.mark.parametrize("typ", [12, 13])
@pytest.mark.parametrize("m,k,n,bound", [(70, 512, 512, 1.4e-7), (70, 14336, 512, 8e-8), (300, 11008, 512, 5.5e-8), (300, 4096, 4096, 3.4e-7), (300, 8192, 4096, 1.45e-7)])
def test_many_token_product_of_positive_activations(gpu, typ, m, k, n, bound):
    """Q4_K and Q5_K, offsets of one sign times positive activations: what the matrix unit cuts off all points one way.  Shares of two, seven, five, sixteen and eleven units.  The bounds lie above
    what the product of three halves gave where it was nearer (5.5e-8 - 5.8e-8, 5.9e-8 - 6.9e-8, 3.5e-7 - 3.9e-7, 1.3e-7 - 1.4e-7) and below what one correction for all runs of
    offsets did (1.2e-7, 7.0e-8 - 7.6e-8, 3.7e-7 - 3.9e-7, 1.5e-7 - 1.7e-7); the first holds too much put back in short ones."""
    r = rng([typ, k, m, n])
    w, dense = scaled_blocks(gpu, typ, n, k, np.exp2(r.uniform(-1, 0, (n, k // 256))), r)
    a = np.abs(r.standard_normal((m, k))).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ dense.T
    assert np.linalg.norm(got - want) <= bound * np.linalg.norm(want), np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("m", [16, 70])
@pytest.mark.parametrize("typ", [2, 8, 12, 13, 14])
def test_many_token_product_beside_a_large_activation(gpu, typ, m):
    """One element 2^12 times the size of the others, over blocks of zeros: the others keep their 22 bits, and results the bound that they have without it."""
    k, n = 1024, 70
    r = rng(typ + m + 2)
    blocks = k // gpu.QUANT_GEOMETRY[typ][0]
    w, dense = scaled_blocks(gpu, typ, n, k, np.where(np.arange(blocks) == 0, 0.0, 1.0)[None], r)
    a = r.standard_normal((m, k)).astype(np.float32)
    a[:, 3] = 4096 * r.choice([-1, 1], m)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2))
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


@pytest.mark.parametrize("typ,m,runs", [(2, 5, 8), (8, 16, 8), (14, 30, 8), (2, 70, 8), (8, 70, 8), (8, 40, 16), (14, 70, 16), (12, 70, 16), (13, 70, 16)])
def test_many_token_product_is_centred(gpu, typ, m, runs):
    """The tensor cores cut off toward zero: uncorrected, results are 1.6e-7 (eight additions to a run) or 2.8e-7 (sixteen) too small on average.  Corrected
    to one or two 2^-23, 5e-8 of that is left; 1e-7 is asked for.  Around the mean an addition is off by a unit's length, 2^-23 or less of its run, divided by
    the root of twelve: 1e-7 or 1.4e-7 for all of a run, 1e-7 more where up to 16 runs are added: twice that is asked for, and three times where offsets
    come in as sums of their own."""
    k, n = 2048, 256
    r = rng(typ + m + 3)
    # block scales of many bits: with one power of two for all, sums would need little cutting
    w, dense = scaled_blocks(gpu, typ, n, k, np.exp2(r.uniform(-1, 0, (n, k // gpu.QUANT_GEOMETRY[typ][0]))), r)
    a = r.standard_normal((m, k)).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n).astype(np.float64)
    want = a.astype(np.float64) @ dense.T
    off = got - want
    mean = (off * want).sum() / (want * want).sum()
    assert abs(mean) <= (1.6e-7 if typ in (12, 13) else 1e-7), mean  # the offsets of eight units are a run of eight additions, corrected as if sixteen: 8e-8 more
    assert np.linalg.norm(off) <= (3 if typ in (12, 13) else 2) * np.sqrt(runs / 12 + 0.7) * 2.0 ** -23 * np.linalg.norm(want), np.linalg.norm(off) / np.linalg.norm(want)


@pytest.mark.parametrize("typ,k", [(12, 2048), (12, 11008), (13, 2048), (13, 11008)])
def test_many_token_product_of_positive_activations(gpu, typ, k):
    """Weights d sc q - dmin m of both signs against positive activations: the two parts are sums of one sign each, far larger than their difference.  Taken
    about c = 8 or 16 the parts are half a step (the middle of q's range is 7.5 or 15.5) times the sum of the activations: with a step of 0.4 of the weights'
    deviation and a mean activation of 0.8, 0.16 sqrt(k) times the result.  2e-7 of each part is cut off; twice that is asked for."""
    from leafcutterllm_b200 import synth
    m, n = 70, 256
    w = synth.host_tensor(typ, 5, f"positive_{k}", n * k)
    a = np.abs(rng(k + typ).standard_normal((m, k))).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ gpu.dequantize(typ, w, n * k).reshape(n, k).astype(np.float64).T
    assert np.linalg.norm(got - want) <= 4e-7 * (1 + 0.16 * np.sqrt(k)) * np.linalg.norm(want), np.linalg.norm(got - want) / np.linalg.norm(want)


@pytest.mark.parametrize("m", [16, 70])
@pytest.mark.parametrize("typ", [2, 8, 12, 13, 14])
def test_many_token_product_of_small_blocks_beside_large_ones(gpu, typ, m):
    """Rows in which every other block is 2^20 times smaller, and no activations but over those: a weight is off by 2^-25 beside a row's largest of
    2^13 and more, i.e. by 2^-38 of that at most (uniformly, so results by its share of the activations' root of squares: four times that, seven
    deviations, is asked for), beside what every result is off by."""
    k, n = 2048, 70
    r = rng(typ + m + 4)
    be = gpu.QUANT_GEOMETRY[typ][0]
    small = np.arange(k // be) % 2 == 1
    # block scales of 2^6 ... 2^7 and 2^-14 ... 2^-13, where f16 still has all its bits
    w, dense = scaled_blocks(gpu, typ, n, k, {2: 8, 8: 128, 12: 945, 13: 1953, 14: 4064}[typ] * np.exp2(r.uniform(6, 7, (n, k // be)) - 20.0 * small), r)
    a = (r.standard_normal((m, k)) * np.repeat(small, be)).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2)) + 4 * 2.0 ** -38 * np.linalg.norm(a.astype(np.float64), axis=1)[:, None] * np.abs(dense).max(1)
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


@pytest.mark.parametrize("m", [16, 70])
@pytest.mark.parametrize("typ", [2, 8, 12, 13, 14])
def test_many_token_product_into_an_unaligned_output(gpu, typ, m):
    """Two row tiles over a long k, which several CTAs share where the summing kernel may write four results at once: an output on a word boundary takes the
    way without it, to the same results but for the order of the sums."""
    import ctypes as C
    lib, chk = gpu.load(), gpu._capi.check
    k, n = 4096, 256
    r = rng(typ + m + 5)
    w, dense = scaled_blocks(gpu, typ, n, k, np.ones((n, 1)), r)
    a = r.standard_normal((m, k)).astype(np.float32)
    ptr = [C.c_void_p() for _ in range(3)]
    for p, size in zip(ptr, (a.nbytes, w.nbytes, 4 * m * n + 16)):
        chk(lib.lc_dev_alloc(size, C.byref(p)))
    chk(lib.lc_dev_upload(ptr[0], a.ctypes.data_as(C.c_void_p), a.nbytes))
    chk(lib.lc_dev_upload(ptr[1], w.ctypes.data_as(C.c_void_p), w.nbytes))
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2))
    for off in (0, 4, 8):
        out = C.c_void_p(ptr[2].value + off)
        got = np.empty((m, n), np.float32)
        chk(lib.lc_qmatmul_dev(typ, ptr[0], ptr[1], m, k, n, out))
        chk(lib.lc_dev_download(got.ctypes.data_as(C.c_void_p), out, got.nbytes))
        assert (np.abs(got - want) <= bound).all(), (off, (np.abs(got - want) / bound).max())
    for p in ptr:
        lib.lc_dev_free(p)


@pytest.mark.parametrize("k", [57856, 58112, 65536])  # the longest row but one unit that the preparation holds in shared memory; the first past it; far past it
@pytest.mark.parametrize("typ", [2, 8, 12, 13, 14])
def test_rows_past_the_many_token_product(gpu, typ, k):
    """Tokens whose rows are too long for its preparation take the matrix-vector kernels.  A sum of k f32 products in any order is off by sqrt(k) 2^-24
    of the products' root of squares at most on average: 2e-5 is more than that."""
    m, n = 16, 12
    r = rng(typ + k)
    w, dense = scaled_blocks(gpu, typ, n, k, np.ones((n, 1)), r)
    a = r.standard_normal((m, k)).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2))
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


@pytest.mark.parametrize("m", [4, 5, 8, 9, 12, 13, 516, 521])  # both sides of where either type changes from the matrix-vector kernels, alone and behind 512 rows
@pytest.mark.parametrize("typ", [8, 14])
def test_few_rows_on_both_sides_of_the_switch(gpu, typ, m):
    k, n = 768, 130
    r = rng(typ + m + 6)
    w, dense = scaled_blocks(gpu, typ, n, k, np.ones((n, 1)), r)
    a = r.standard_normal((m, k)).astype(np.float32)
    got = gpu.qmatmul(typ, a.ravel(), w, m, k, n).reshape(m, n)
    want = a.astype(np.float64) @ dense.T
    bound = 2e-5 * np.sqrt((a.astype(np.float64) ** 2) @ (dense.T ** 2))  # either way's rounding, as above
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


def test_many_token_products_from_several_threads(gpu):
    """Four threads queue products of different types, row lengths and token counts on device buffers of their own: each finds its own results, to the bit,
    whatever the others' need of the workspace that they share."""
    import ctypes as C
    import threading
    lib, chk = gpu.load(), gpu._capi.check
    jobs = []
    for i, (typ, m, k, n) in enumerate([(2, 16, 2048, 256), (8, 70, 4352, 384), (14, 40, 1024, 130), (12, 100, 8192, 256)]):
        r = rng(typ + m + 7)
        w, _ = scaled_blocks(gpu, typ, n, k, np.ones((n, 1)), r)
        a = r.standard_normal((m, k)).astype(np.float32)
        ptr = [C.c_void_p() for _ in range(3)]
        for p, size in zip(ptr, (a.nbytes, w.nbytes, 4 * m * n)):
            chk(lib.lc_dev_alloc(size, C.byref(p)))
        chk(lib.lc_dev_upload(ptr[0], a.ctypes.data_as(C.c_void_p), a.nbytes))
        chk(lib.lc_dev_upload(ptr[1], w.ctypes.data_as(C.c_void_p), w.nbytes))
        jobs.append((typ, m, k, n, ptr))

    def run(job):
        typ, m, k, n, ptr = job
        chk(lib.lc_qmatmul_dev(typ, ptr[0], ptr[1], m, k, n, ptr[2]))
        out = np.empty((m, n), np.float32)
        chk(lib.lc_dev_download(out.ctypes.data_as(C.c_void_p), ptr[2], out.nbytes))
        return out
    alone = [run(j) for j in jobs]
    wrong = []

    def work(i):
        chk(lib.lc_dev_sync())  # brings the device's context to this thread: without it tensor maps cannot be encoded, and the first call takes another kernel
        for _ in range(60):
            if not np.array_equal(run(jobs[i]), alone[i]):
                wrong.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for *_, ptr in jobs:
        for p in ptr:
            lib.lc_dev_free(p)
    assert not wrong


NO_ROOM = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
import leafcutterllm_b200 as gpu
from leafcutterllm_b200 import synth
lib, typ, m, k, n = gpu.load(), {typ}, 16, 4096, 64
w = synth.host_tensor(typ, 5, "room", n * k)
a = np.random.default_rng(2).standard_normal((m, k)).astype(np.float32)
gpu.qmatmul(typ, np.zeros((4, 4 * k), np.float32), synth.host_tensor(typ, 6, "more", 16 * n * k), 4, 4 * k, 4 * n)  # room for the call's own inputs
held, size, at = [], 16 << 30, ctypes.c_void_p()
while size >= 32 << 20:
    if lib.lc_dev_alloc(size, ctypes.byref(at)) == 0:
        held.append(at.value)
    else:
        size >>= 1
full = gpu.qmatmul(typ, a, w, m, k, n).reshape(m, n)
for p in held:
    lib.lc_dev_free(ctypes.c_void_p(p))
free = gpu.qmatmul(typ, a, w, m, k, n).reshape(m, n)
want = a.astype(np.float64) @ gpu.dequantize(typ, w, n * k).reshape(n, k).T.astype(np.float64)
for got in (full, free):  # 4096 products in f32 or better
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max(), np.abs(got - want).max()
"""


@pytest.mark.parametrize("typ", [2, 14])
def test_qmatmul_without_room_for_the_many_token_product(gpu, typ):
    """Sixteen rows while the device has no memory left for the product's workspace (64 MB and more) run through the matrix-vector kernels; afterwards, with
    room again, through the product.  In a process of its own, whose workspace no other test has made."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", NO_ROOM.format(root=root, typ=typ)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_qmatmul_linearity_full_size(gpu, oracle):
    """7B-shape matrices: A(x+y) = Ax + Ay and a sample of rows against the oracle."""
    from leafcutterllm_b200 import synth
    for (k, n) in [(4096, 4096), (11008, 4096), (4096, 11008)]:
        w = synth.host_tensor(12, 5, f"full_{k}_{n}", n * k)
        r = rng(k + n)
        x = r.standard_normal(k).astype(np.float32)
        y = r.standard_normal(k).astype(np.float32)
        ax, ay, axy = (gpu.qmatmul(12, v, w, 1, k, n).ravel() for v in (x, y, x + y))
        assert_close(axy, ax + ay, 1e-4 * np.abs(axy).max(), 1e-4, "linearity")
        rows = r.choice(n, 64, replace=False)
        rb = k // 256 * 144
        sub = np.concatenate([w[i * rb:(i + 1) * rb] for i in rows])
        want = oracle.qmatmul(12, x, sub, 1, k, 64).ravel()
        assert_close(ax[rows], want, 2e-5 * np.abs(want).max(), 1e-4, "row sample")


def test_shard_order_gemms_are_bit_exact(gpu, oracle):
    # generators of rust/src/kernels/int8_gemm.rs:377-392 and :455-472
    for (m, k, n) in [(4, 8, 32), (8, 16, 64)]:
        bpr = n // 32
        scales = np.array([[0.01 * (row + 1)] * bpr for row in range(k)], np.float32)
        q8 = np.array([[b * 32 + jj - 16 for b in range(bpr) for jj in range(32)] for _ in range(k)], np.int8)
        a = (np.arange(m * k, dtype=np.float32) * np.float32(0.1)) if n == 32 else (np.arange(m * k, dtype=np.float32) * np.float32(0.01) - np.float32(0.5))
        got = gpu.q8_0_matmul(a, gpu.Q8Matrix(k, n, scales, q8), m, k, n)
        want = oracle.q8_0_matmul_shard(a, scales, q8, m, k, n)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
        deq = (q8.astype(np.float32) * np.repeat(scales, 32, axis=1)).astype(np.float32)
        assert_close(got, oracle.matmul(a, deq, m, k, n), 1e-3, 0, "q8 vs dequant->f32 (reference test bound)")
        q4 = np.zeros((k, n // 2), np.uint8)
        for row in range(k):
            for b in range(bpr):
                for jj in range(16):
                    low = min(8 + (b * 32 + jj * 2) % 8, 15)
                    high = min(8 + (b * 32 + jj * 2 + 1) % 8, 15)
                    q4[row, b * 16 + jj] = (high << 4) | low
        got4 = gpu.q4_0_matmul(a, gpu.Q4Matrix(k, n, scales, q4), m, k, n)
        want4 = oracle.q4_0_matmul_shard(a, scales, q4, m, k, n)
        assert np.array_equal(got4.view(np.uint32), want4.view(np.uint32))
    with pytest.raises(gpu.LeafcutterError):
        gpu.q8_0_matmul(np.zeros(8, np.float32), gpu.Q8Matrix(8, 33, np.zeros((8, 1), np.float32), np.zeros((8, 33), np.int8)), 1, 8, 33)


def test_rope_and_argmax(gpu, oracle):
    r = rng(9)
    for (seq, heads, hd, theta, pos0) in [(1, 4, 64, 10000.0, 0), (7, 32, 128, 10000.0, 0), (5, 8, 64, 500000.0, 2043)]:
        x = r.standard_normal(seq * heads * hd).astype(np.float32)
        got = gpu.apply_rotary_emb(x, seq, heads, hd, theta, pos0)
        want = oracle.rope(x, seq, heads, hd, theta, pos0)
        # powf/sinf/cosf of the device and of glibc differ by ulps; at angle ~2000 rad that is ~1e-4 of |x|
        assert_close(got, want, 4e-4 * (1 + pos0 / 500.0), 1e-5, "rope")
    assert np.array_equal(gpu.apply_rotary_emb(x[:64 * 4], 1, 4, 64, 10000.0, 0), x[:64 * 4])  # position 0 is the identity
    assert gpu.sample_top_p(np.array([0.1, 0.5, 0.3], np.float32), 0.0, 0.9) == 1  # rust/src/inference/sampler.rs:56-61
    v = np.zeros(32000, np.float32)
    v[[5, 31000, 17]] = 3.0
    assert gpu.sample_top_p(v, 0.0, 1.0) == 31000 == oracle.argmax(v)  # last of equal maxima
    v = r.standard_normal(128256).astype(np.float32)
    assert gpu.sample_top_p(v, 0.0, 1.0) == oracle.argmax(v)


def test_tcgen05_probe_runs(gpu):
    """The diagnostic that times the building blocks of the many-token product: it must come back (every wait inside is
    bounded) with a positive cycle count for each of its fourteen measurements."""
    import ctypes as C
    out = (C.c_double * 16)()
    gpu._capi.check(gpu.load().lc_tcgen05_probe(out))
    vals = [out[i] for i in range(14)]
    assert all(v > 0 for v in vals), vals
    assert out[15] == 0.0
