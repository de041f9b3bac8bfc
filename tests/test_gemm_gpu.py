"""ng.dot / the hgemm C entry points against the numpy oracle (B200 only)."""
import ctypes

import numpy as np
import pytest

from oracle import reference_math as rm
from tests._util import assert_close, ref_percent_error, rn16_tol

pytestmark = pytest.mark.gpu


def _operands(rng, m, n, k, op, std=1.0):
    A = rng.normal(0, std, (k, m) if op[0] == "t" else (m, k)).astype(np.float16)
    B = rng.normal(0, std, (n, k) if op[1] == "t" else (k, n)).astype(np.float16)
    return A, B


def _dot(ng, A, B, op, C0=None, **kw):
    dA, dB = ng.array(A), ng.array(B)
    m = A.shape[1] if op[0] == "t" else A.shape[0]
    n = B.shape[0] if op[1] == "t" else B.shape[1]
    dC = ng.array(C0) if C0 is not None else ng.empty((m, n))
    ng.dot(dA.T if op[0] == "t" else dA, dB.T if op[1] == "t" else dB, dC, **kw)
    return dC.get()


@pytest.mark.parametrize("size", [257, 256, 255, 129, 128, 127, 65, 64, 17, 16, 15])
@pytest.mark.parametrize("op", ["nn", "nt", "tn"])
def test_known_answers_all_ones_and_zeros(ng, size, op):
    """The reference's C smoke test (kernels/C_interface/test.cu:27-55,70): edge tiles, aligned and
    unaligned leading dimensions (the latter are packed, and run on the SIMT kernel when very short)."""
    ones = np.ones((size, size), dtype=np.float16)
    assert (_dot(ng, ones, ones, op) == size).all()
    zeros = np.zeros((size, size), dtype=np.float16)
    assert (_dot(ng, zeros, zeros, op) == 0).all()


def test_config1_tn_2048_relu(ng):
    """C = relu(A^T B), A k x m, B k x n, m=n=k=2048, N(0,1), seed 1001."""
    rng = np.random.default_rng(1001)
    k = m = n = 2048
    A = rng.standard_normal((k, m)).astype(np.float16)
    B = rng.standard_normal((k, n)).astype(np.float16)
    got = _dot(ng, A, B, "tn", relu=True)
    ref = rm.gemm(A, B, a_t=True, relu=True)
    assert_close(got, ref, rn16_tol(ref, rm.gemm_abs(A, B, a_t=True), k), "cfg1")
    assert ref_percent_error(got, ref) <= 0.7   # the reference's fp16 threshold, cublas_test.py:96


@pytest.mark.parametrize("op", ["nn", "nt", "tn"])
@pytest.mark.parametrize("mnk", [(4096, 128, 9216), (4096, 128, 4096), (1000, 128, 4096), (9216, 4096, 128),
                                 (3072, 3072, 3072)])
def test_config2_fc_sweep(ng, op, mnk):
    """BASELINE config 2 shapes, inputs N(0, 0.1), round to nearest."""
    m, n, k = mnk
    if m * n * k > 2 ** 34:
        m, n, k = 1024, 1024, 3072      # full 3072^3 is covered by the linearity test below
    rng = np.random.default_rng(1002 + m + k)
    A, B = _operands(rng, m, n, k, op, std=0.1)
    got = _dot(ng, A, B, op)
    ref = rm.gemm(A, B, a_t=op[0] == "t", b_t=op[1] == "t")
    assert_close(got, ref, rn16_tol(ref, rm.gemm_abs(A, B, op[0] == "t", op[1] == "t"), k), "cfg2 %s %s" % (op, mnk))


@pytest.mark.parametrize("op", ["nn", "nt", "tn"])
def test_ragged_shapes_alpha_beta_relu(ng, op):
    """Odd sizes of the reference's gemm_test.py lists (:27-29), aligned to 8 where TMA needs it
    and not aligned otherwise; epilogue order alpha -> relu -> beta."""
    rng = np.random.default_rng(7)
    for (m, n, k) in [(136, 72, 200), (778, 192, 1536), (65, 127, 9), (1, 64, 192), (8, 8, 8), (785, 16, 72)]:
        A, B = _operands(rng, m, n, k, op)
        C0 = rng.standard_normal((m, n)).astype(np.float16)
        got = _dot(ng, A, B, op, C0=C0, alpha=0.5, beta=0.25, relu=True)
        ref = rm.gemm(A, B, op[0] == "t", op[1] == "t", alpha=0.5, beta=0.25, relu=True, C=C0)
        tol = rn16_tol(ref, rm.gemm_abs(A, B, op[0] == "t", op[1] == "t"), k) + 2.0 ** -11 * np.abs(C0.astype(np.float32))
        assert_close(got, ref, tol, "%s %s" % (op, (m, n, k)))


def test_simt_and_tensor_paths_agree(ng, lib):
    """Both kernels accumulate in fp32 and round once: results agree to one fp16 ulp."""
    rng = np.random.default_rng(3)
    m, n, k = 384, 256, 512
    A, B = _operands(rng, m, n, k, "nn")
    dA, dB = ng.array(A), ng.array(B)
    c1, c2 = ng.empty((m, n)), ng.empty((m, n))
    for fn, c in ((lib.ng_hgemm, c1), (lib.ng_hgemm_simt, c2)):
        assert fn(dA.ptr, dB.ptr, c.ptr, 0, 0, m, n, k, k, n, n, 1.0, 0.0, 0, 0, 0, 0, None) == 0
    a, b = c1.get().astype(np.float32), c2.get().astype(np.float32)
    # different summation orders: allow the fp32 accumulation slack on top of one fp16 ulp
    assert (np.abs(a - b) <= rn16_tol(a, rm.gemm_abs(A, B), k)).all()


def test_large_size_property_linearity(ng):
    """3072^3 at full size: dot(A, B1 + B2) == dot(A, B1) + dot(A, B2) within rounding, plus a
    sampled exact check of 64 rows against the oracle."""
    rng = np.random.default_rng(11)
    n = 3072
    A = rng.normal(0, 0.1, (n, n)).astype(np.float16)
    B1 = (rng.integers(-8, 9, (n, n)) / 16.0).astype(np.float16)
    B2 = (rng.integers(-8, 9, (n, n)) / 16.0).astype(np.float16)
    c1, c2, c12 = _dot(ng, A, B1, "nn"), _dot(ng, A, B2, "nn"), _dot(ng, A, (B1 + B2).astype(np.float16), "nn")
    s = c1.astype(np.float32) + c2.astype(np.float32)
    assert (np.abs(c12.astype(np.float32) - s) <= 3 * 2.0 ** -10 * (np.abs(s) + np.abs(c1) + np.abs(c2)) + 1e-3).all()
    rows = rng.choice(n, 64, replace=False)
    ref = rm.gemm(A[rows], B1)
    assert_close(c1[rows], ref, rn16_tol(ref, rm.gemm_abs(A[rows], B1), n), "sampled rows")


def test_batched_dot(ng):
    rng = np.random.default_rng(5)
    b, m, n, k = 4, 128, 256, 64
    A = rng.standard_normal((b, m, k)).astype(np.float16)
    B = rng.standard_normal((b, k, n)).astype(np.float16)
    dA, dB, dC = ng.array(A), ng.array(B), ng.empty((b, m, n))
    ng.batched_dot(dA, dB, dC)
    ref = np.einsum("bmk,bkn->bmn", A.astype(np.float32), B.astype(np.float32))
    assert_close(dC.get(), ref, 2.0 ** -10 * np.abs(ref) + 1e-2, "batched grid")
    # 2-D C: the products are summed over the batch
    dS = ng.empty((m, n))
    ng.batched_dot(dA, dB, dS)
    refs = ref.sum(axis=0)
    assert_close(dS.get(), refs, 2.0 ** -10 * np.abs(refs) + 2e-2, "batched loops")


@pytest.mark.parametrize("op", ["nn", "nt", "tn"])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (7, 9, 8), (127, 129, 63), (130, 250, 65), (257, 31, 1030)])
def test_operands_at_odd_addresses(ng, op, mnk):
    """Views whose rows start at every even address: bases one to seven elements behind a 16-byte
    boundary and odd leading dimensions. The copies that TMA reads and the products equal the oracle."""
    m, n, k = mnk
    rng = np.random.default_rng(13 + m)
    for shift in (1, 2, 5, 7):
        A, B = _operands(rng, m, n, k, op)
        bigA = np.full((A.shape[0], A.shape[1] + 9), np.nan, np.float16)
        bigB = np.full((B.shape[0], B.shape[1] + 9 - shift), np.nan, np.float16)
        bigA[:, shift:shift + A.shape[1]] = A
        bigB[:, :B.shape[1]] = B
        dA = ng.array(bigA)[:, shift:shift + A.shape[1]]
        dB = ng.array(bigB)[:, :B.shape[1]]
        C0 = rng.standard_normal((m, n)).astype(np.float16)
        C = ng.array(C0)
        ng.dot(dA.T if op[0] == "t" else dA, dB.T if op[1] == "t" else dB, C, alpha=0.5, beta=0.25)
        ref = rm.gemm(A, B, op[0] == "t", op[1] == "t", alpha=0.5, beta=0.25, C=C0)
        tol = rn16_tol(ref, rm.gemm_abs(A, B, op[0] == "t", op[1] == "t"), k) + 2.0 ** -11 * np.abs(C0.astype(np.float32))
        assert_close(C.get(), ref, tol, "%s %s +%d" % (op, mnk, shift))


@pytest.mark.parametrize("op", ["nn", "nt", "tn"])
@pytest.mark.parametrize("mnk", [(1, 1, 1), (7, 9, 8), (65, 63, 16), (33, 129, 17), (33, 128, 17), (65, 300, 32), (65, 300, 33)])
def test_short_products_of_odd_operands_packed_and_unpacked(ng, lib, op, mnk):
    """Both sides of the line between the CUDA-core kernel and the packed product, and the rule itself."""
    m, n, k = mnk
    rng = np.random.default_rng(19 + m)
    A, B = _operands(rng, m, n, k, op)
    bigA, bigB = (np.pad(x, ((0, 0), (0, 1 + x.shape[1] % 2))) for x in (A, B))      # odd leading dimensions
    dA, dB = ng.array(bigA)[:, :A.shape[1]], ng.array(bigB)[:, :B.shape[1]]
    C0 = rng.standard_normal((m, n)).astype(np.float16)
    ref = rm.gemm(A, B, op[0] == "t", op[1] == "t", alpha=0.5, beta=0.25, C=C0)
    tol = rn16_tol(ref, rm.gemm_abs(A, B, op[0] == "t", op[1] == "t"), k) + 2.0 ** -11 * np.abs(C0.astype(np.float32))
    before, after = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    launches = []
    try:
        for form in (0, 2, -1):
            assert lib.ng_tune(b"pack_odd", form) == 0
            C = ng.array(C0)
            assert lib.ng_launch_count(ctypes.byref(before)) == 0
            ng.dot(dA.T if op[0] == "t" else dA, dB.T if op[1] == "t" else dB, C, alpha=0.5, beta=0.25)
            assert lib.ng_launch_count(ctypes.byref(after)) == 0
            launches.append(after.value - before.value)
            assert_close(C.get(), ref, tol, "%s %s form %d" % (op, mnk, form))
    finally:
        assert lib.ng_tune(b"pack_odd", -1) == 0
    assert launches[0] == 1 and launches[1] >= 2
    assert launches[2] == launches[0 if k <= 16 or (k <= 32 and n > 128) else 1]


@pytest.mark.parametrize("dims", [(2, 8, 8, 8), (3, 129, 72, 65), (5, 33, 17, 130), (17, 128, 128, 64), (1, 40, 24, 72)])
@pytest.mark.parametrize("shared", [None, "A", "B"])
def test_batched_dot_forms(ng, dims, shared):
    """Independent products and products summed over the batch, either operand shared by all of
    them, reductions that end inside a 64-wide block of every product, odd sizes."""
    b, m, n, k = dims
    rng = np.random.default_rng(17 + b)
    A = rng.standard_normal((m, k) if shared == "A" else (b, m, k)).astype(np.float16)
    B = rng.standard_normal((k, n) if shared == "B" else (b, k, n)).astype(np.float16)
    a3, b3 = (np.broadcast_to(x.astype(np.float32), (b,) + x.shape[-2:]) for x in (A, B))
    each = np.matmul(a3, b3)
    mag = np.matmul(np.abs(a3), np.abs(b3))
    C, S = ng.empty((b, m, n)), ng.empty((m, n))
    ng.batched_dot(ng.array(A), ng.array(B), C)
    assert_close(C.get(), each, rn16_tol(each, mag, k), "independent %s" % (dims,))
    ng.batched_dot(ng.array(A), ng.array(B), S, relu=True)
    total = np.maximum(each.sum(axis=0), 0)
    assert_close(S.get(), total, rn16_tol(total, mag.sum(axis=0), k * b), "summed %s" % (dims,))


def test_reference_c_interface(ng, lib):
    """nervana_hgemm / nervana_hgemm_colmajor keep the reference's signatures and conventions."""
    rng = np.random.default_rng(9)
    m, n, k = 128, 64, 256
    A, B = _operands(rng, m, n, k, "nn")
    dA, dB, dC = ng.array(A), ng.array(B), ng.empty((m, n))
    assert lib.nervana_loadKernels(b"unused")
    assert lib.nervana_randStateSizeBytes() == 2048 * 32 * 4
    assert lib.nervana_hgemm(dA.ptr, dB.ptr, dC.ptr, False, False, m, n, k, k, n, n, 1.0, 0.0, None, False, True, None, -1)
    ref = rm.gemm(A, B, relu=True)
    assert_close(dC.get(), ref, rn16_tol(ref, rm.gemm_abs(A, B), k), "nervana_hgemm")
    # column-major view of the same buffers: C^T (n x m col-major == m x n row-major) = B^T A^T
    dCt = ng.empty((m, n))
    assert lib.nervana_hgemm_colmajor(dB.ptr, dA.ptr, dCt.ptr, False, False, n, m, k, n, k, n, 1.0, 0.0, None,
                                      False, True, None, -1)
    assert np.array_equal(dCt.get(), dC.get())
    assert not lib.nervana_sgemm(dA.ptr, dB.ptr, dC.ptr, False, False, m, n, k, k, n, n, 1.0, 0.0, None, False, False,
                                 None, -1)


def test_dot_argument_errors(ng):
    A, B, C = ng.empty((16, 8)), ng.empty((8, 16)), ng.empty((16, 16))
    with pytest.raises(AssertionError):
        ng.dot(A.T, B.T, C)                      # "tt" is not supported
    with pytest.raises(AssertionError):
        ng.dot(A, ng.empty((9, 16)), C)          # inner dimensions differ
    with pytest.raises(TypeError):
        ng.dot(ng.empty((4, 4), dtype=np.float32), ng.empty((4, 4), dtype=np.float32),
               ng.empty((4, 4), dtype=np.float32))
    with pytest.raises(TypeError):
        ng.dot(ng.empty((4, 4), dtype=np.int8), ng.empty((4, 4), dtype=np.int8), ng.empty((4, 4), dtype=np.int8))


@pytest.mark.parametrize("op", ["nn", "nt", "tn"])
def test_cta_pair_instances_match_the_oracle(ng, lib, op):
    """The two-SM form of the tensor-core kernel (tcgen05 cta_group::2, switched on with the
    "pair_mma" tuning field): a 256-row tile is shared by the two CTAs of a cluster, each of which
    loads its own half of the B columns. Same results as the one-CTA kernel up to summation order."""
    rng = np.random.default_rng(31)
    try:
        assert lib.ng_tune(b"pair_mma", 1) == 0
        for (m, n, k) in [(512, 512, 256), (384, 256, 1024), (1000, 136, 520), (256, 128, 64)]:
            A, B = _operands(rng, m, n, k, op, std=0.1)
            C0 = rng.standard_normal((m, n)).astype(np.float16)
            got = _dot(ng, A, B, op, C0=C0, alpha=0.5, beta=0.25, relu=True)
            ref = rm.gemm(A, B, op[0] == "t", op[1] == "t", alpha=0.5, beta=0.25, relu=True, C=C0)
            tol = rn16_tol(ref, rm.gemm_abs(A, B, op[0] == "t", op[1] == "t"), k) + 2.0 ** -11 * np.abs(C0.astype(np.float32))
            assert_close(got, ref, tol, "pair %s %s" % (op, (m, n, k)))
            plain = _dot(ng, A, B, op)
            ref = rm.gemm(A, B, op[0] == "t", op[1] == "t")
            assert_close(plain, ref, rn16_tol(ref, rm.gemm_abs(A, B, op[0] == "t", op[1] == "t"), k), "pair plain")
    finally:
        assert lib.ng_tune(b"pair_mma", -1) == 0
    assert lib.ng_sync() == 0


@pytest.mark.parametrize("bits", [10, 7, 4])
@pytest.mark.parametrize("scale", [0, -12, -20])
@pytest.mark.parametrize("mnk", [(256, 256, 64), (130, 264, 40), (130, 131, 40), (64, 72, 1024)])
def test_stochastic_rounding_forms_agree_bit_for_bit(ng, lib, mnk, scale, bits):
    """Small integers times a power of two: every sum is exact whatever its order, so the vectorised,
    the ragged and the split-K output stages must round each element with the same random bits as the
    element-by-element form of the CUDA-core kernel. Scales put the results in the normal and in the
    subnormal fp16 range; zeros occur in all of them."""
    m, n, k = mnk
    rng = np.random.default_rng(3)
    A = rng.integers(-3, 4, (m, k)).astype(np.float16)
    B = (rng.integers(-3, 4, (k, n)) * 2.0 ** scale * (1 + 2.0 ** -4)).astype(np.float16)
    A[5], B[:, 7] = 0, 0
    dA, dB, c1, c2 = ng.array(A), ng.array(B), ng.empty((m, n)), ng.empty((m, n))
    for fn, c in ((lib.ng_hgemm, c1), (lib.ng_hgemm_simt, c2)):
        assert fn(dA.ptr, dB.ptr, c.ptr, 0, 0, m, n, k, k, n, n, 1.0, 0.0, 0, bits, 99, 7, None) == 0
    a, b = c1.get(), c2.get()
    assert np.array_equal(a, b)
    assert (a[5] == 0).all() and (a[:, 7] == 0).all() and (a != 0).sum() > a.size // 2
