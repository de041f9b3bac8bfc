"""fprop_pool / bprop_pool: bit-exact against the reference's numpy path (B200 only)."""
import numpy as np
import pytest

from oracle import reference_math as rm
from tests._util import golden, golden_names

pytestmark = pytest.mark.gpu


def _run(ng, cfg, I, E, dtype=np.float16):
    layer = ng.pool_layer(dtype, "max", *cfg)
    dI, dE = ng.array(I, dtype=dtype), ng.array(E, dtype=dtype)
    dO, dB = ng.empty(layer.dimO, dtype=dtype), ng.empty(layer.dimI, dtype=dtype)
    ng.fprop_pool(layer, dI, dO)
    ng.bprop_pool(layer, dI, dE, dB)
    return layer, dO.get(), dB.get()


@pytest.mark.parametrize("name", golden_names("pool_"))
def test_golden_vectors_of_the_reference_numpy_path(ng, name):
    g = golden(name)
    cfg = [int(v) for v in g["cfg"]]
    # the reference script back-propagates its own output
    layer, O, B = _run(ng, cfg, g["I"], g["O"].astype(np.float16))
    assert np.array_equal(O.astype(np.float32), g["O"])
    assert np.array_equal(B, g["gradI"].astype(np.float16))


CASES = {
    # (N, C, D, H, W, J, T, R, S, pad_j, pad_d, pad_h, pad_w, str_j, str_d, str_h, str_w)
    "alexnet_3x3_s2_n64": (64, 8, 1, 13, 13, 1, 1, 3, 3, 0, 0, 0, 0, 1, 1, 2, 2),
    "vgg_2x2_n32": (32, 8, 1, 8, 8, 1, 1, 2, 2, 0, 0, 0, 0, 1, 1, 2, 2),
    "config5_jtrs_2222": (32, 8, 4, 6, 6, 2, 2, 2, 2, 0, 0, 0, 0, 2, 2, 2, 2),
    "padded_overlapping": (16, 5, 1, 9, 9, 2, 1, 3, 3, 1, 0, 1, 1, 1, 1, 2, 2),
    "n4_scalar_lanes": (4, 3, 1, 7, 7, 1, 1, 3, 3, 0, 0, 0, 0, 1, 1, 2, 2),
    "stride_larger_than_window": (8, 2, 1, 9, 9, 1, 1, 2, 2, 0, 0, 0, 0, 1, 1, 3, 3),
    "maxout_over_feature_maps": (64, 16, 1, 1, 1, 4, 1, 1, 1, 0, 0, 0, 0, 4, 1, 1, 1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_bit_exact_against_oracle(ng, name):
    cfg = CASES[name]
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(1005)
    # few distinct values: plenty of ties, so the first-maximum rule is exercised
    I = (rng.integers(0, 12, pd.dimI) / 8.0).astype(np.float16)
    E = rng.uniform(-1, 1, pd.dimO).astype(np.float16)
    refO, refB = rm.pool_max(pd, I, E)
    layer, O, B = _run(ng, cfg, I, E)
    assert layer.dimO == pd.dimO
    assert np.array_equal(O, refO.astype(np.float16))
    assert np.array_equal(B, refB.astype(np.float16))


@pytest.mark.parametrize("name", sorted(CASES))
def test_fused_relu_mask_equals_bprop_then_mask(ng, name):
    cfg = CASES[name]
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(31)
    # a ReLU output: about half zeros (whole windows of zeros included), ties among the rest
    I = (np.maximum(rng.integers(-8, 6, pd.dimI), 0) / 4.0).astype(np.float16)
    E = rng.uniform(-1, 1, pd.dimO).astype(np.float16)
    _, refB = rm.pool_max(pd, I, E)
    ref = (refB * (I > 0)).astype(np.float16)           # Layer.bprop_relu on the pool's deltas
    layer = ng.pool_layer(np.float16, "max", *cfg)
    dI, dE, dB = ng.array(I), ng.array(E), ng.empty(layer.dimI)
    ng.bprop_pool(layer, dI, dE, dB, relu_mask=True)
    assert np.array_equal(dB.get(), ref)
    assert (ref != refB.astype(np.float16)).any() or not (I[refB != 0] <= 0).any()


@pytest.mark.parametrize("name", ["alexnet_3x3_s2_n64", "vgg_2x2_n32", "stride_larger_than_window"])
@pytest.mark.parametrize("mask", [False, True])
def test_recorded_argmax_gives_the_same_backward_pass(ng, name, mask):
    cfg = CASES[name]
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(77)
    I = (np.maximum(rng.integers(-8, 6, pd.dimI), 0) / 4.0).astype(np.float16)
    E = rng.uniform(-1, 1, pd.dimO).astype(np.float16)
    layer = ng.pool_layer(np.float16, "max", *cfg)
    nbytes = ng.pool_argmax_bytes(layer)
    if name == "stride_larger_than_window":
        assert nbytes == 0                      # no specialised path: callers fall back
        return
    assert nbytes == int(np.prod(pd.dimO))
    dI, dE = ng.array(I), ng.array(E)
    O1, O2 = ng.empty(layer.dimO), ng.empty(layer.dimO)
    B1, B2 = ng.empty(layer.dimI), ng.empty(layer.dimI)
    rec = ng.empty((nbytes,), dtype=np.uint8)
    ng.fprop_pool(layer, dI, O1)
    ng.fprop_pool(layer, dI, O2, argmax=rec)
    ng.bprop_pool(layer, dI, dE, B1, relu_mask=mask)
    dI.fill(0)                                  # the recorded pass must not need the input
    ng.bprop_pool(layer, dI, dE, B2, relu_mask=mask, argmax=rec)
    assert np.array_equal(O1.get(), O2.get())
    assert np.array_equal(B1.get(), B2.get())


def test_fp32_pooling(ng):
    cfg = CASES["alexnet_3x3_s2_n64"]
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(2)
    I = rng.uniform(0, 1, pd.dimI).astype(np.float32)
    E = rng.uniform(-1, 1, pd.dimO).astype(np.float32)
    refO, refB = rm.pool_max(pd, I, E)
    _, O, B = _run(ng, cfg, I, E, dtype=np.float32)
    assert np.array_equal(O, refO)
    assert np.array_equal(B, refB)


def test_full_size_alexnet_pool1_properties(ng):
    """pool1 at BASELINE size (N=128, C=64, 55x55 -> 27x27, 3x3 stride 2): size-independent checks.
    Every output is >= each tap of its window and equals one of them; bprop conserves the sum of E
    (each error lands on exactly one input) and puts nothing where the input is not a window max."""
    cfg = (128, 64, 1, 55, 55, 1, 1, 3, 3, 0, 0, 0, 0, 1, 1, 2, 2)
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(1003)
    I = rng.uniform(0, 1, pd.dimI).astype(np.float16)
    E = (rng.integers(1, 5, pd.dimO) / 4.0).astype(np.float16)
    _, O, B = _run(ng, cfg, I, E)
    taps = np.stack([I[:, :, r:r + 53:2, s:s + 53:2, :] for r in range(3) for s in range(3)])
    assert np.array_equal(O, taps.max(axis=0))
    assert abs(float(B.astype(np.float64).sum()) - float(E.astype(np.float64).sum())) <= 1e-6 * E.size
    assert (B >= 0).all() and (B[:, :, 55 - 0:, :, :] == 0).all()
    # sampled channels against the oracle, bit for bit
    sub = rm.PoolDims(128, 2, 1, 55, 55, 1, 1, 3, 3, 0, 0, 0, 0, 1, 1, 2, 2)
    refO, refB = rm.pool_max(sub, I[5:7], E[5:7])
    assert np.array_equal(O[5:7], refO.astype(np.float16))
    assert np.array_equal(B[5:7], refB.astype(np.float16))


@pytest.mark.parametrize("op", ["avg", "l2"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_avg_and_l2_pooling_against_oracle(ng, name, op):
    """The ops the reference defines in numpy only (benchmarks/pool_test.py:141-146). Forward: the
    fp32 result rounded to fp16 (one ulp of slack for the order of the fp32 additions); backward:
    the derivative of the forward definition, tolerance 2 fp16 ulps of the largest term sum."""
    cfg = CASES[name]
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(77)
    I = rng.uniform(-1, 1, pd.dimI).astype(np.float16)
    E = rng.uniform(-1, 1, pd.dimO).astype(np.float16)
    refO, refB = rm.pool_avg_l2(pd, I, op, E)
    layer = ng.pool_layer(np.float16, op, *cfg)
    dI, dE = ng.array(I), ng.array(E)
    dO, dB = ng.empty(layer.dimO), ng.empty(layer.dimI)
    ng.fprop_pool(layer, dI, dO)
    ng.bprop_pool(layer, dI, dE, dB)
    O, B = dO.get().astype(np.float32), dB.get().astype(np.float32)
    assert np.all(np.abs(O - refO) <= 2.0 ** -10 * np.maximum(np.abs(refO), 2.0 ** -14))
    windows = np.prod(pd.JTRS)
    assert np.all(np.abs(B - refB) <= 2.0 ** -9 * np.maximum(np.abs(refB), 1.0) * max(1, windows // 4))
    assert np.abs(B).sum() > 0


def test_avg_and_l2_refuse_the_max_only_extensions(ng):
    cfg = CASES["vgg_2x2_n32"]
    layer = ng.pool_layer(np.float16, "avg", *cfg)
    dI, dE, dB = ng.empty(layer.dimI), ng.empty(layer.dimO), ng.empty(layer.dimI)
    with pytest.raises(ValueError):
        ng.bprop_pool(layer, dI, dE, dB, relu_mask=True)


WINDOWS = {"3x3_s2": (3, 2, 0), "2x2_s2": (2, 2, 0), "3x3_s3": (3, 3, 0), "3x3_s1_p1": (3, 1, 1), "3x3_s2_p1": (3, 2, 1)}


@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("size", ["single_rows", "strips"])
@pytest.mark.parametrize("name", sorted(WINDOWS))
def test_window_shapes_with_kernels_of_their_own(ng, name, size, dtype):
    """Maximum (bit for bit) and mean of the window shapes that are compiled in, few outputs (one row
    per thread) and many (strips of rows), map sizes that leave ragged strips and borders."""
    R, st, pad = WINDOWS[name]
    lanes = 8 if dtype is np.float16 else 4
    n, c, h, w = 16, 3, 7, 10
    if size == "strips":      # over 4096 threads of one output each per SM
        n, c, h, w = 72 * lanes, 40, 14 * st + 5, 15 * st + 4
    cfg = (n, c, 1, h, w, 1, 1, R, R, 0, 0, pad, pad, 1, 1, st, st)
    pd = rm.PoolDims(*cfg)
    rng = np.random.default_rng(5 + R + st)
    I = (rng.integers(0, 12, pd.dimI) / 8.0).astype(dtype)      # plenty of ties
    E = rng.uniform(-1, 1, pd.dimO).astype(dtype)
    refO, refB = rm.pool_max_fast(pd, I, E)
    layer, O, B = _run(ng, cfg, I, E, dtype)
    assert np.array_equal(O, refO.astype(dtype))
    assert np.array_equal(B, refB.astype(dtype))
    if size == "strips":
        return
    refO, refB = rm.pool_avg_l2(pd, I, "avg", E)
    layer = ng.pool_layer(dtype, "avg", *cfg)
    dI, dE = ng.array(I, dtype=dtype), ng.array(E, dtype=dtype)
    dO, dB = ng.empty(layer.dimO, dtype=dtype), ng.empty(layer.dimI, dtype=dtype)
    ng.fprop_pool(layer, dI, dO)
    ng.bprop_pool(layer, dI, dE, dB)
    # nine fp32 additions of values up to 1.5 in another order, then one rounding to the stored type
    unit = 2.0 ** -11 if dtype is np.float16 else 2.0 ** -24
    assert np.all(np.abs(dO.get() - refO) <= unit * np.abs(refO) + 9 * 2.0 ** -24 * 1.5)
    assert np.all(np.abs(dB.get() - refB) <= unit * np.abs(refB) + 9 * 2.0 ** -24)


@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("kind", ["nan", "inf", "lowest"])
@pytest.mark.parametrize("shape", [(3, 2, 0, 1), (2, 2, 0, 1), (3, 1, 1, 1), (3, 3, 0, 1), (3, 2, 1, 1), (2, 2, 0, 2)])
def test_windows_without_a_largest_value(ng, dtype, kind, shape):
    """Windows of NaN, minus infinity or the lowest number: the vectorised kernels leave the bits of the
    general ones, which tensors one element off a 16-byte boundary run on."""
    R, st, pad, T = shape
    if dtype is np.float16 and pad == 0 and T == 1:
        pytest.skip("these windows keep their first tap")
    rng = np.random.default_rng(5)
    D = 4 if T == 2 else 1
    L = ng.pool_layer(dtype, "max", 16, 3, D, 8, 8, 1, T, R, R, 0, 0, pad, pad, 1, T, st, st)
    x = rng.integers(-2, 3, L.dimI).astype(dtype)
    bad = rng.random(L.dimI) < 0.7
    x[bad] = {"nan": np.nan, "inf": -np.inf, "lowest": np.finfo(dtype).min}[kind]
    x[0, 0, :4, :4] = -np.inf
    e = rng.normal(0, 1, L.dimO).astype(dtype)

    def place(shape, shift, values=None):
        n = int(np.prod(shape))
        t = ng.empty((n + 8,), dtype=dtype)[shift:shift + n].reshape(shape)
        return t if values is None else t.set(values)

    got = []
    for shift in (0, 1):
        I, O, E, B = place(L.dimI, shift, x), place(L.dimO, shift), place(L.dimO, shift, e), place(L.dimI, shift)
        ng.fprop_pool(L, I, O)
        ng.bprop_pool(L, I, E, B)
        got.append((O.get(), B.get()))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("shape", [(3, 2, 0, 1), (2, 2, 0, 1), (3, 1, 1, 1), (3, 3, 0, 1), (3, 2, 1, 1), (2, 2, 0, 2)])
def test_zeros_of_both_signs_keep_the_first(ng, dtype, shift, shape):
    """-0 and +0 are equal: the first of a window's largest values is stored, sign included, by the
    vectorised kernels and (tensors one element off a 16-byte boundary) by the general ones."""
    R, st, pad, T = shape
    rng = np.random.default_rng(6)
    L = ng.pool_layer(dtype, "max", 16, 3, 4 if T == 2 else 1, 9, 9, 1, T, R, R, 0, 0, pad, pad, 1, T, st, st)
    x = rng.choice(np.array([-0.0, 0.0, -1.0], dtype), L.dimI)
    C, D, H, W, N = L.dimI
    K, M, P, Q, _ = L.dimO
    padded = np.full((C, D, H + 2 * pad + st, W + 2 * pad + st, N), -np.inf, dtype)
    padded[:, :, pad:pad + H, pad:pad + W] = x
    taps = np.stack([padded[:, t::T, r:r + P * st:st, s:s + Q * st:st][:, :M, :P, :Q]
                     for t in range(T) for r in range(R) for s in range(R)])
    ref = np.take_along_axis(taps, taps.argmax(axis=0)[None], axis=0)[0]     # (argmax: the first of equal values)
    assert (np.signbit(ref) & (ref == 0)).any() and (~np.signbit(ref) & (ref == 0)).any()
    n_in, n_out = int(np.prod(L.dimI)), int(np.prod(L.dimO))
    I = ng.empty((n_in + 8,), dtype=dtype)[shift:shift + n_in].reshape(L.dimI).set(x)
    O = ng.empty((n_out + 8,), dtype=dtype)[shift:shift + n_out].reshape(L.dimO)
    ng.fprop_pool(L, I, O)
    bits = np.uint16 if dtype is np.float16 else np.uint32
    assert np.array_equal(O.get().view(bits), ref.view(bits))


@pytest.mark.parametrize("dtype", [np.float16, np.float32])
@pytest.mark.parametrize("name", sorted(WINDOWS))
def test_mean_passes_errors_on_as_the_general_kernel_does(ng, dtype, name):
    """Bit for bit, and without an infinity from errors whose sum is out of range while their shares are not."""
    R, st, pad = WINDOWS[name]
    L = ng.pool_layer(dtype, "avg", 16, 3, 1, 11, 12, 1, 1, R, R, 0, 0, pad, pad, 1, 1, st, st)
    rng = np.random.default_rng(8)
    largest = float(np.finfo(dtype).max)
    e = (rng.uniform(0.4, 0.9, L.dimO) * largest).astype(dtype)
    e[1] = rng.normal(0, 1, L.dimO[1:]).astype(dtype)
    n_in, n_out = int(np.prod(L.dimI)), int(np.prod(L.dimO))
    got = []
    for shift in (0, 1):       # tensors one element off a 16-byte boundary run on the general kernel
        I = ng.empty((n_in + 8,), dtype=dtype)[shift:shift + n_in].reshape(L.dimI)
        I.fill(0)
        B = ng.empty((n_in + 8,), dtype=dtype)[shift:shift + n_in].reshape(L.dimI)
        E = ng.empty((n_out + 8,), dtype=dtype)[shift:shift + n_out].reshape(L.dimO).set(e)
        ng.bprop_pool(L, I, E, B)
        got.append(B.get())
    assert np.isfinite(got[1]).all()
    bits = np.uint16 if dtype is np.float16 else np.uint32
    assert np.array_equal(got[0].view(bits), got[1].view(bits))
