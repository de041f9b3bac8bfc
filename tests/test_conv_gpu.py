"""fprop_conv / bprop_conv / update_conv against the reference's numpy path (B200 only)."""
import numpy as np
import pytest

from nervanagpu_b200 import _lib
from oracle import reference_math as rm
from tests._util import assert_close, f32_tol, golden, golden_names, rn16_tol

pytestmark = pytest.mark.gpu

PATHS = {"auto": _lib.NG_PATH_AUTO, "tensor": _lib.NG_PATH_TENSOR, "simt": _lib.NG_PATH_SIMT,
         "im2col": _lib.NG_PATH_IM2COL}


def _layer(ng, cfg, path="auto"):
    layer = ng.conv_layer(np.float16, *cfg)
    layer.path = PATHS[path]
    return layer


def _abs_terms(cd, I, F, E):
    """sum |a||b| of each output's dot product, for the accumulation-error bound."""
    aI, aF, aE = np.abs(I.astype(np.float32)), np.abs(F.astype(np.float32)), np.abs(E.astype(np.float32))
    return rm.conv_fprop_fast(cd, aI, aF), rm.conv_bprop_fast(cd, aF, aE), rm.conv_update_fast(cd, aI, aE)


def _run_all(ng, layer, I, F, E, relu=False, alpha=1.0, ops="fbu"):
    dI, dF, dE = ng.array(I), ng.array(F), ng.array(E)
    out = {}
    if "f" in ops:
        dO = ng.empty(layer.dimO)
        ng.fprop_conv(layer, dI, dF, dO, alpha=alpha, relu=relu)
        out["O"] = dO.get()
    if "b" in ops:
        dB = ng.empty(layer.dimI)
        ng.bprop_conv(layer, dF, dE, dB, alpha=alpha)
        out["gradI"] = dB.get()
    if "u" in ops:
        dU = ng.empty(layer.dimF, dtype=np.float32)
        ng.update_conv(layer, dI, dE, dU, alpha=alpha)
        out["gradF"] = dU.get()
    return out


def _check(cd, got, I, F, E, ref, what):
    T, R, S = cd.TRS
    aO, aB, aU = _abs_terms(cd, I, F, E)
    M, P, Q = cd.MPQ
    if "O" in got:
        assert_close(got["O"], ref["O"], rn16_tol(ref["O"], aO, cd.C * T * R * S), what + " fprop")
    if "gradI" in got:
        assert_close(got["gradI"], ref["gradI"], rn16_tol(ref["gradI"], aB, cd.K * T * R * S), what + " bprop")
    if "gradF" in got:
        assert_close(got["gradF"], ref["gradF"], f32_tol(aU, M * P * Q * cd.N), what + " update")


@pytest.mark.parametrize("name", golden_names("conv_"))
@pytest.mark.parametrize("path", ["auto", "simt"])
def test_golden_vectors_of_the_reference_numpy_path(ng, name, path):
    g = golden(name)
    cfg = [int(v) for v in g["cfg"]]
    cd = rm.ConvDims(*cfg)
    got = _run_all(ng, _layer(ng, cfg, path), g["I"], g["F"], g["E"])
    _check(cd, got, g["I"], g["F"], g["E"], g, "%s/%s" % (name, path))


CASES = {
    # name: (N, C, K, D, H, W, T, R, S, pad_d, pad_h, pad_w, str_d, str_h, str_w)
    "c64_3x3_n64": (64, 64, 128, 1, 8, 8, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "c3_3x3_n64_first_layer": (64, 3, 64, 1, 12, 12, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "c16_5x5_stride2_n128": (128, 16, 32, 1, 13, 13, 1, 5, 5, 0, 2, 2, 1, 2, 2),
    "c96_3x3_n32_flattened": (32, 96, 64, 1, 8, 8, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "c64_3d_n32": (32, 64, 64, 4, 6, 6, 3, 3, 3, 1, 1, 1, 1, 1, 1),
    "c3_11x11_stride4_n64_alexnet1": (64, 3, 64, 1, 35, 35, 1, 11, 11, 0, 2, 2, 1, 4, 4),
    "c130_k200_ragged_channels": (64, 130, 200, 1, 7, 7, 1, 3, 3, 0, 0, 0, 1, 1, 1),
    "c32_1x1": (64, 32, 48, 1, 5, 5, 1, 1, 1, 0, 0, 0, 1, 1, 1),
    "c8_n16_flattened_q8": (16, 8, 16, 1, 8, 8, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "stride_h_only": (64, 16, 16, 1, 9, 8, 1, 3, 3, 0, 1, 1, 1, 2, 1),
    # update: two 48-row taps stacked per accumulator, 192-column tiles
    "c48_k384_stacked_taps": (64, 48, 384, 1, 6, 6, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "c64_k192_5x5_n128": (128, 64, 192, 1, 7, 7, 1, 5, 5, 0, 2, 2, 1, 1, 1),
    # tap blocks with two image groups per pixel (one box per pixel), update with exchanged operands
    "c3_11x11_stride4_n128": (128, 3, 64, 1, 27, 27, 1, 11, 11, 0, 2, 2, 1, 4, 4),
    # 256 output rows: filter halves as single boxes, column tiles as single boxes (N = 64),
    # and a width (6) that makes some tiles straddle image rows
    "c64_k256_w6_merged_boxes": (64, 64, 256, 1, 6, 6, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    # K = 96: the first-layer update keeps the filters on the MMA rows (K <= 128), one column tile
    "c3_7x7_stride2_k96": (64, 3, 96, 1, 21, 21, 1, 7, 7, 0, 3, 3, 1, 2, 2),
}


# Per-GPU shapes of a minibatch that is split over 2 / 4 / 8 GPUs (AlexNet 128 -> 64/32/16, VGG model A
# 64 -> 32/16/8): with fewer than 64 images a 64-element chunk is several pixels of one image row, and
# rows that are not a multiple of 64 elements (13 x 32, 27 x 16, 14 x 8, ...) are padded to whole chunks.
SHARDED = {
    "alexnet_conv2_n32": (32, 64, 192, 1, 27, 27, 1, 5, 5, 0, 2, 2, 1, 1, 1),
    "alexnet_conv2_n16": (16, 64, 192, 1, 27, 27, 1, 5, 5, 0, 2, 2, 1, 1, 1),
    "alexnet_conv3_n32": (32, 192, 384, 1, 13, 13, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "alexnet_conv3_n16": (16, 192, 384, 1, 13, 13, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "alexnet_conv4_n16": (16, 384, 256, 1, 13, 13, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "alexnet_conv5_n32": (32, 256, 256, 1, 13, 13, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "vgg_64_128_n8_w20": (8, 64, 128, 1, 20, 20, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "vgg_256_512_28_n8": (8, 256, 512, 1, 28, 28, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "vgg_512_512_14_n8": (8, 512, 512, 1, 14, 14, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "vgg_512_512_14_n16": (16, 512, 512, 1, 14, 14, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "vgg_512_512_14_n32": (32, 512, 512, 1, 14, 14, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    # no padding (Q < W): the tail of a row's last chunk reads real pixels of the next columns
    "valid_conv_n24_q9": (24, 32, 64, 1, 11, 11, 1, 3, 3, 0, 0, 0, 1, 1, 1),
    # 3-D, one image row shorter than a chunk
    "c32_3d_n8_w5": (8, 32, 32, 3, 5, 5, 3, 3, 3, 1, 1, 1, 1, 1, 1),
}


def _inputs(cd, seed):
    rng = np.random.default_rng(seed)
    I = rng.uniform(0, 1, cd.dimI).astype(np.float16)
    F = rng.normal(0, 0.1, cd.dimF).astype(np.float16)
    E = (rng.uniform(-1, 1, cd.dimO) * 0.125).astype(np.float16)
    return I, F, E


@pytest.mark.parametrize("name", sorted(CASES))
def test_tensor_core_path_matches_oracle(ng, name):
    cfg = CASES[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1003)
    ref = {"O": rm.conv_fprop_fast(cd, I, F, alpha=0.5, relu=True), "gradI": rm.conv_bprop_fast(cd, F, E, alpha=0.5),
           "gradF": rm.conv_update_fast(cd, I, E, alpha=0.5)}
    got = _run_all(ng, _layer(ng, cfg, "tensor"), I, F, E, relu=True, alpha=0.5)
    _check(cd, got, I, F, E, ref, name)
    assert (got["O"] >= 0).all()


BLOCKED = ["c64_3x3_n64", "c96_3x3_n32_flattened", "c64_3d_n32", "c130_k200_ragged_channels", "stride_h_only",
           "c48_k384_stacked_taps", "c64_k192_5x5_n128", "c64_k256_w6_merged_boxes"]


@pytest.mark.parametrize("name", BLOCKED)
def test_channel_blocked_copies_change_nothing(ng, lib, name):
    """Activation tensors whose channel planes are larger than a page are read through a copy in
    (z, y, channel, x, n) order (the "chan_block" tuning field: 2 = every shape, 0 = never). The
    product reads the same values in the same order either way: results are equal bit for bit,
    for every kind of tensor map (per pixel, flattened rows, merged boxes, strided rows)."""
    cfg = CASES[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1005)
    try:
        assert lib.ng_tune(b"chan_block", 0) == 0
        plain = _run_all(ng, _layer(ng, cfg, "tensor"), I, F, E, relu=True, alpha=0.5)
        assert lib.ng_tune(b"chan_block", 2) == 0
        blocked = _run_all(ng, _layer(ng, cfg, "tensor"), I, F, E, relu=True, alpha=0.5)
    finally:
        assert lib.ng_tune(b"chan_block", -1) == 0
    for key in ("O", "gradI", "gradF"):
        np.testing.assert_array_equal(blocked[key], plain[key], err_msg="%s %s" % (name, key))
    ref = {"O": rm.conv_fprop_fast(cd, I, F, alpha=0.5, relu=True), "gradI": rm.conv_bprop_fast(cd, F, E, alpha=0.5),
           "gradF": rm.conv_update_fast(cd, I, E, alpha=0.5)}
    _check(cd, blocked, I, F, E, ref, name + " (blocked)")


STRIDED_FIRST_LAYERS = {
    # AlexNet conv1 on the shard of one of 4 / 8 / 16 GPUs (smaller image, same filter geometry)
    "alexnet_conv1_n32": (32, 3, 64, 1, 35, 35, 1, 11, 11, 0, 2, 2, 1, 4, 4),
    "alexnet_conv1_n16": (16, 3, 64, 1, 39, 37, 1, 11, 11, 0, 2, 2, 1, 4, 4),
    "alexnet_conv1_n8": (8, 3, 64, 1, 35, 35, 1, 11, 11, 0, 2, 2, 1, 4, 4),
    # stride 2, 7x7 (a filter that is not a multiple of the stride), odd padding, 4 channels
    "c4_7x7_stride2_n24": (24, 4, 96, 1, 21, 23, 1, 7, 7, 0, 3, 3, 1, 2, 2),
    # stride 3 with a 5x5 filter and no padding: the last window ends before the image does
    "c3_5x5_stride3_n40": (40, 3, 32, 1, 20, 20, 1, 5, 5, 0, 0, 0, 1, 3, 3),
}


@pytest.mark.parametrize("name", sorted(STRIDED_FIRST_LAYERS))
def test_strided_first_layers_of_small_minibatches_run_as_space_to_depth(ng, lib, name):
    """Fewer than 64 images, fewer than 16 channels, stride > 1: the layer is rewritten as a
    unit-stride layer over st*st times the channels (copies of the input and the filters) and runs
    on the tensor-core path; the weight gradient is gathered back into the filter's own shape."""
    import ctypes
    cfg = STRIDED_FIRST_LAYERS[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1006)
    ref = {"O": rm.conv_fprop_fast(cd, I, F, alpha=0.5, relu=True), "gradF": rm.conv_update_fast(cd, I, E, alpha=0.5)}
    before = ctypes.c_ulonglong(0)
    after = ctypes.c_ulonglong(0)
    assert lib.ng_fallback_launch_count(ctypes.byref(before)) == 0
    got = _run_all(ng, _layer(ng, cfg, "auto"), I, F, E, relu=True, alpha=0.5, ops="fu")
    assert lib.ng_fallback_launch_count(ctypes.byref(after)) == 0
    assert after.value == before.value, "left the tensor-core path"
    _check(cd, got, I, F, E, ref, name)
    # the same through the im2col form it replaces (switch off): same sums, other order
    try:
        assert lib.ng_tune(b"space_to_depth", 0) == 0
        old = _run_all(ng, _layer(ng, cfg, "auto"), I, F, E, relu=True, alpha=0.5, ops="fu")
    finally:
        assert lib.ng_tune(b"space_to_depth", -1) == 0
    _check(cd, old, I, F, E, ref, name + " (im2col)")
    # fp16 weight gradient
    layer = _layer(ng, cfg, "auto")
    dU = ng.empty(layer.dimF)
    ng.update_conv(layer, ng.array(I), ng.array(E), dU, alpha=0.5)
    aU = _abs_terms(cd, I, F, E)[2]
    M, P, Q = cd.MPQ
    assert_close(dU.get(), ref["gradF"], f32_tol(aU, M * P * Q * cd.N) + 2.0 ** -11 * np.abs(ref["gradF"]), name + " fp16 dW")


@pytest.mark.parametrize("name", sorted(STRIDED_FIRST_LAYERS))
@pytest.mark.parametrize("warm", [False, True])
def test_space_to_depth_update_with_exchanged_operands_and_copies(ng, lib, name, warm):
    """The update of the rewritten layer in its exchanged form, with channel-blocked copies of its operands: its
    scratch and the outer call's must not share memory, on a stream without scratch buffers and on one whose
    buffers are large already."""
    cfg = STRIDED_FIRST_LAYERS[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1021)
    ref = {"O": rm.conv_fprop_fast(cd, I, F), "gradF": rm.conv_update_fast(cd, I, E)}
    layer = _layer(ng, cfg)
    dI, dF, dE, dO, dU = ng.array(I), ng.array(F), ng.array(E), ng.empty(layer.dimO), ng.empty(layer.dimF, dtype=np.float32)
    ng.synchronize()
    default, ng.stream = ng.stream, ng.new_stream()
    try:
        for key in (b"update_swap", b"chan_block"):
            assert lib.ng_tune(key, 2) == 0
        for _ in range(3 if warm else 1):
            dU.fill(0.0)
            ng.update_conv(layer, dI, dE, dU)
            ng.fprop_conv(layer, dI, dF, dO)
        ng.synchronize()
        got = {"O": dO.get(), "gradF": dU.get()}
    finally:
        for key in (b"update_swap", b"chan_block"):
            assert lib.ng_tune(key, -1) == 0
        ng.stream = default
    _check(cd, got, I, F, E, ref, name)


@pytest.mark.parametrize("name", sorted(SHARDED))
def test_sharded_minibatch_shapes_run_on_the_tensor_core_path(ng, name):
    cfg = SHARDED[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1004)
    ref = {"O": rm.conv_fprop_fast(cd, I, F, relu=True), "gradI": rm.conv_bprop_fast(cd, F, E),
           "gradF": rm.conv_update_fast(cd, I, E)}
    # guard cells around the outputs: columns of the padded chunk space must not be stored anywhere
    layer = _layer(ng, cfg, "tensor")
    dI, dF, dE = ng.array(I), ng.array(F), ng.array(E)
    pad = 4096
    bufO = ng.empty((layer.sizeO + 2 * pad,))
    bufB = ng.empty((layer.sizeI + 2 * pad,))
    bufO.fill(7.0)
    bufB.fill(7.0)
    dO = bufO[pad:pad + layer.sizeO].reshape(layer.dimO)
    dB = bufB[pad:pad + layer.sizeI].reshape(layer.dimI)
    dU = ng.empty(layer.dimF, dtype=np.float32)
    ng.fprop_conv(layer, dI, dF, dO, relu=True)
    ng.bprop_conv(layer, dF, dE, dB)
    ng.update_conv(layer, dI, dE, dU)
    got = {"O": dO.get(), "gradI": dB.get(), "gradF": dU.get()}
    _check(cd, got, I, F, E, ref, name)
    for buf, size in ((bufO, layer.sizeO), (bufB, layer.sizeI)):
        h = buf.get()
        assert (h[:pad] == 7.0).all() and (h[pad + size:] == 7.0).all(), name + ": wrote outside the tensor"


@pytest.mark.parametrize("name", ["c3_3x3_n64_first_layer", "c3_11x11_stride4_n64_alexnet1", "c64_3x3_n64"])
def test_update_im2col_path(ng, name):
    cfg = CASES[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 77)
    got = _run_all(ng, _layer(ng, cfg, "im2col"), I, F, E, ops="u")
    _check(cd, got, I, F, E, {"gradF": rm.conv_update_fast(cd, I, E)}, name + "/im2col")


def test_shapes_outside_the_tensor_path_run_on_simt(ng):
    # N = 8 with a W stride: no 64-element chunks in place. The forward pass reads a copy that has them, the small
    # update a patch matrix, and the small backward pass runs on the CUDA cores.
    cfg = (8, 24, 16, 1, 5, 5, 1, 3, 3, 0, 1, 1, 1, 2, 2)
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 5)
    ref = {"O": rm.conv_fprop(cd, I, F), "gradI": rm.conv_bprop(cd, F, E), "gradF": rm.conv_update(cd, I, E)}
    _check(cd, _run_all(ng, _layer(ng, cfg, "auto"), I, F, E), I, F, E, ref, "auto->simt")
    with pytest.raises(_lib.NervanaError):
        _run_all(ng, _layer(ng, cfg, "tensor"), I, F, E, ops="f")


def test_update_fp16_output_and_determinism(ng):
    cfg = CASES["c64_3x3_n64"]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 9)
    layer = _layer(ng, cfg)
    dI, dE = ng.array(I), ng.array(E)
    u16 = ng.empty(layer.dimF, dtype=np.float16)
    ng.update_conv(layer, dI, dE, u16)
    ref = rm.conv_update_fast(cd, I, E)
    assert_close(u16.get(), ref, 2.0 ** -10 * np.abs(ref) + 1e-3, "fp16 dW")
    a, b = ng.empty(layer.dimF, dtype=np.float32), ng.empty(layer.dimF, dtype=np.float32)
    ng.update_conv(layer, dI, dE, a)
    ng.update_conv(layer, dI, dE, b)
    assert np.array_equal(a.get(), b.get())     # fixed summation order, unlike atomics


def test_full_size_alexnet_layer_properties(ng):
    """AlexNet conv3 at BASELINE size (N=128, 192->384, 13x13): the oracle is too slow for every
    output, so check (a) linearity in the filter, (b) an exact sample of output pixels."""
    cfg = (128, 192, 384, 1, 13, 13, 1, 3, 3, 0, 1, 1, 1, 1, 1)
    cd = rm.ConvDims(*cfg)
    rng = np.random.default_rng(1003)
    I = rng.uniform(0, 1, cd.dimI).astype(np.float16)
    F1 = (rng.integers(-8, 9, cd.dimF) / 256.0).astype(np.float16)
    F2 = (rng.integers(-8, 9, cd.dimF) / 256.0).astype(np.float16)
    layer = _layer(ng, cfg)
    dI = ng.array(I)
    outs = []
    for F in (F1, F2, (F1 + F2).astype(np.float16)):
        dO = ng.empty(layer.dimO)
        ng.fprop_conv(layer, dI, ng.array(F), dO)
        outs.append(dO.get().astype(np.float32))
    s = outs[0] + outs[1]
    assert (np.abs(outs[2] - s) <= 3 * 2.0 ** -10 * (np.abs(s) + np.abs(outs[0]) + np.abs(outs[1])) + 1e-3).all()
    # exact sample: 6 output pixels through the per-pixel oracle arithmetic
    F2d = F1.astype(np.float32).reshape(-1, cd.K)
    I2 = np.zeros((cd.C * 169 + 1, cd.N), np.float32)
    I2[:-1] = I.astype(np.float32).reshape(-1, cd.N)
    for (p, q) in [(0, 0), (0, 12), (6, 6), (12, 0), (12, 12), (3, 9)]:
        rows = rm._conv_pixel_rows(cd, 0, p - 1, q - 1)
        ref = np.dot(F2d.T, I2[rows, :])
        absd = np.dot(np.abs(F2d).T, np.abs(I2[rows, :]))
        assert_close(outs[0][:, 0, p, q, :], ref, rn16_tol(ref, absd, cd.C * 9), "pixel %d,%d" % (p, q))


FULL_SIZE = {
    # BASELINE configs at their real sizes: (N, C, K, D, H, W, T, R, S, pads, strides)
    "alexnet_conv1_tap_blocks": (128, 3, 64, 1, 224, 224, 1, 11, 11, 0, 2, 2, 1, 4, 4),
    "alexnet_conv2_stacked_update": (128, 64, 192, 1, 27, 27, 1, 5, 5, 0, 2, 2, 1, 1, 1),
    "vgg_conv4_256_rows": (64, 256, 256, 1, 56, 56, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "config5_3d_conv": (32, 64, 64, 16, 56, 56, 3, 3, 3, 1, 1, 1, 1, 1, 1),
}


@pytest.mark.parametrize("name", sorted(FULL_SIZE))
def test_full_size_adjoint_identity(ng, name):
    """At full size the three passes are checked against each other: they are the three partial
    derivatives of one bilinear form, so <fprop(I, F), E> = <I, bprop(F, E)> = <F, update(I, E)>."""
    cfg = FULL_SIZE[name]
    cd = rm.ConvDims(*cfg)
    rng = np.random.default_rng(1004)
    I = rng.uniform(0, 1, cd.dimI).astype(np.float16)
    F = rng.normal(0, 0.05, cd.dimF).astype(np.float16)
    E = (rng.uniform(-1, 1, cd.dimO) * 0.125).astype(np.float16)
    got = _run_all(ng, _layer(ng, cfg), I, F, E)
    f64 = np.float64
    via_fprop = np.sum(got["O"].astype(f64) * E.astype(f64))
    via_bprop = np.sum(got["gradI"].astype(f64) * I.astype(f64))
    via_update = np.sum(got["gradF"].astype(f64) * F.astype(f64))
    scale = np.sum(np.abs(got["O"].astype(f64)) * np.abs(E.astype(f64)))
    assert np.isfinite([via_fprop, via_bprop, via_update]).all() and scale > 0
    # fp16 rounding of O and gradI: relative 2^-11 per element, random in sign; a dropped tap or a
    # misplaced tile would show at the percent level
    assert abs(via_fprop - via_update) <= 1e-3 * scale, (via_fprop, via_update, scale)
    assert abs(via_fprop - via_bprop) <= 1e-3 * scale, (via_fprop, via_bprop, scale)
    assert abs(via_bprop - via_update) <= 1e-3 * scale, (via_bprop, via_update, scale)


def test_layer_argument_checks(ng):
    with pytest.raises(AssertionError):
        ng.conv_layer(np.float16, 12, 3, 8, 1, 8, 8, 1, 3, 3)       # N % 8
    with pytest.raises(AssertionError):
        ng.conv_layer(np.float16, 16, 3, 12, 1, 8, 8, 1, 3, 3)      # K % 8
    layer = ng.conv_layer(np.float16, 16, 3, 8, 1, 8, 8, 1, 3, 3)
    with pytest.raises(AssertionError):
        ng.fprop_conv(layer, ng.empty((3, 1, 8, 8, 8)), ng.empty(layer.dimF), ng.empty(layer.dimO))   # sizeI
    with pytest.raises(TypeError):
        ng.fprop_conv(layer, ng.empty(layer.dimI, dtype=np.float32), ng.empty(layer.dimF, dtype=np.float32),
                      ng.empty(layer.dimO, dtype=np.float32))


STRIDED = {
    # minibatches that are no multiple of 64 (split copies of the input), and multiples of it (phases of
    # the backward pass alone); filters shorter than the stride, padding larger than a phase, 3-D
    "n8_3x3_s2": (8, 24, 16, 1, 5, 5, 1, 3, 3, 0, 1, 1, 1, 2, 2),
    "n24_5x5_s3": (24, 40, 72, 1, 17, 14, 1, 5, 5, 0, 2, 2, 1, 3, 3),
    "n88_7x7_s2_c96": (88, 96, 72, 1, 13, 15, 1, 7, 7, 0, 3, 3, 1, 2, 2),
    "n16_1x1_s2": (16, 64, 136, 1, 9, 8, 1, 1, 1, 0, 0, 0, 1, 2, 2),
    "n40_2x3_s3_h1": (40, 17, 64, 1, 8, 16, 1, 2, 3, 0, 0, 1, 1, 1, 3),
    "n32_3d_s222": (32, 32, 32, 5, 6, 7, 3, 3, 3, 1, 1, 1, 2, 2, 2),
    "n16_c3_5x5_s2": (16, 3, 24, 1, 12, 11, 1, 5, 5, 0, 2, 2, 1, 2, 2),
    "n64_3x3_s2": (64, 130, 72, 1, 9, 12, 1, 3, 3, 0, 1, 1, 1, 2, 2),
    "n128_1x1_s2": (128, 64, 64, 1, 7, 7, 1, 1, 1, 0, 0, 0, 1, 2, 2),
    "n64_4x4_s4_pad3": (64, 16, 32, 1, 10, 9, 1, 4, 4, 0, 3, 3, 1, 4, 4),
    "n64_2x2_s3": (64, 48, 64, 1, 11, 10, 1, 2, 2, 0, 1, 0, 1, 3, 3),
}


@pytest.mark.parametrize("name", sorted(STRIDED))
def test_strided_layers_run_on_the_tensor_core_path(ng, lib, name):
    import ctypes
    cfg = STRIDED[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1007)
    ref = {"O": rm.conv_fprop_fast(cd, I, F, relu=True), "gradI": rm.conv_bprop_fast(cd, F, E),
           "gradF": rm.conv_update_fast(cd, I, E)}
    before, after = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    assert lib.ng_fallback_launch_count(ctypes.byref(before)) == 0
    got = _run_all(ng, _layer(ng, cfg, "auto"), I, F, E, relu=True)
    assert lib.ng_fallback_launch_count(ctypes.byref(after)) == 0
    assert after.value == before.value
    _check(cd, got, I, F, E, ref, name)


EXCHANGED = {
    # few channels and filters, many taps: whole and last, partly filled column tiles of taps; rows per tap
    # that are and are not a divisor of 256; ragged image rows; a phase-split input; 3-D
    "c64_k64_3d": (32, 64, 64, 4, 14, 14, 3, 3, 3, 1, 1, 1, 1, 1, 1),
    "c33_k72_5x5": (64, 33, 72, 1, 12, 11, 1, 5, 5, 0, 2, 2, 1, 1, 1),
    "c17_k128_7x7_n8": (8, 17, 128, 1, 13, 13, 1, 7, 7, 0, 3, 3, 1, 1, 1),
    "c64_k8_3x3": (128, 64, 8, 1, 9, 9, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "c48_k128_5x5_s2_n24": (24, 48, 128, 1, 17, 15, 1, 5, 5, 0, 2, 2, 1, 2, 2),
    "c16_k16_1x1": (64, 16, 16, 1, 8, 8, 1, 1, 1, 0, 0, 0, 1, 1, 1),
}


@pytest.mark.parametrize("name", sorted(EXCHANGED))
@pytest.mark.parametrize("half", [False, True])
def test_update_with_exchanged_operands(ng, lib, name, half):
    cfg = EXCHANGED[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1011)
    layer = _layer(ng, cfg, "auto")
    dI, dE = ng.array(I), ng.array(E)
    ref = rm.conv_update_fast(cd, I, E)
    got = []
    try:
        for form in (2, 0):
            assert lib.ng_tune(b"update_swap", form) == 0
            dU = ng.empty(layer.dimF, dtype=np.float16 if half else np.float32)
            ng.update_conv(layer, dI, dE, dU)
            got.append(dU.get().astype(np.float64))
    finally:
        assert lib.ng_tune(b"update_swap", -1) == 0
    # 16 2^-24 |a|_2 |b|_2 (as for the full-size layers), the norms of n values bounded by the largest;
    # fp16 results are rounded once more
    n = int(np.prod(cd.MPQ)) * cd.N
    tol = 16 * 2.0 ** -24 * n * float(np.abs(I).max()) * float(np.abs(E).max())
    if half:
        tol = tol + 2.0 ** -11 * np.abs(ref) + 2.0 ** -25
    for g in got:
        assert (np.abs(g - ref) <= tol).all(), name


ROW_PAIRS = {
    # at most 64 output channels in one pass or both: odd and even numbers of rows, filters of two rows and
    # more, ragged image rows, planes, phases of a strided backward pass, tap blocks, a phase-split input
    "c64_k64_h7": (64, 64, 64, 1, 7, 9, 1, 3, 3, 0, 1, 1, 1, 1, 1),
    "c33_k24_2x3_n8": (8, 33, 24, 1, 6, 5, 1, 2, 3, 0, 0, 1, 1, 1, 1),
    "c16_k72_5x5_n128": (128, 16, 72, 1, 9, 8, 1, 5, 5, 0, 2, 2, 1, 1, 1),
    "c32_k48_3d": (32, 32, 48, 3, 5, 6, 3, 3, 3, 1, 1, 1, 1, 1, 1),
    "c130_k64_valid": (64, 130, 64, 1, 9, 9, 1, 3, 3, 0, 0, 0, 1, 1, 1),
    "c40_k72_5x5_s2": (64, 40, 72, 1, 12, 11, 1, 5, 5, 0, 2, 2, 1, 2, 2),
    "c40_k64_3x5_s3_n24": (24, 40, 64, 1, 11, 10, 1, 3, 5, 0, 1, 2, 1, 1, 3),
    "c3_k64_11x11_s4_n128": (128, 3, 64, 1, 23, 23, 1, 11, 11, 0, 3, 3, 1, 4, 4),
    "c3_k40_11x11_s4_n64": (64, 3, 40, 1, 27, 23, 1, 11, 11, 0, 3, 3, 1, 4, 4),
}


@pytest.mark.parametrize("name", sorted(ROW_PAIRS))
def test_two_image_rows_per_tile(ng, lib, name):
    cfg = ROW_PAIRS[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1013)
    ref = {"O": rm.conv_fprop_fast(cd, I, F, relu=True), "gradI": rm.conv_bprop_fast(cd, F, E),
           "gradF": rm.conv_update_fast(cd, I, E)}
    layer = _layer(ng, cfg, "auto")
    # an infinity reaches the outputs under the filter and no others
    I2, E2 = I.copy(), E.copy()
    I2[1, 0, I.shape[2] // 2, 3, 5] = np.inf
    E2[2, 0, E.shape[2] // 2, 1, 4] = -np.inf
    got, finite = {}, []
    try:
        for form in (0, 2):
            assert lib.ng_tune(b"row_stack", form) == 0
            pad = 4096              # guard cells around the outputs
            bufs = [ng.empty((n + 2 * pad,)) for n in (layer.sizeO, layer.sizeI)]
            views = []
            for buf, n, dim in zip(bufs, (layer.sizeO, layer.sizeI), (layer.dimO, layer.dimI)):
                buf.fill(7.0)
                views.append(buf[pad:pad + n].reshape(dim))
            dU = ng.empty(layer.dimF, dtype=np.float32)
            ng.fprop_conv(layer, ng.array(I), ng.array(F), views[0], relu=True)
            ng.bprop_conv(layer, ng.array(F), ng.array(E), views[1])
            ng.update_conv(layer, ng.array(I), ng.array(E), dU)
            got = {"O": views[0].get(), "gradI": views[1].get(), "gradF": dU.get()}
            _check(cd, got, I, F, E, ref, name)
            for buf in bufs:
                h = buf.get()
                assert (h[:pad] == 7.0).all() and (h[-pad:] == 7.0).all(), name + ": wrote outside the tensor"
            ng.fprop_conv(layer, ng.array(I2), ng.array(F), views[0])
            ng.bprop_conv(layer, ng.array(F), ng.array(E2), views[1])
            finite.append([np.isfinite(v.get()) for v in views])
    finally:
        assert lib.ng_tune(b"row_stack", -1) == 0
    for one, two in zip(*finite):
        assert np.array_equal(one, two), name
        assert not one.all()


@pytest.mark.parametrize("name", sorted(ROW_PAIRS))
def test_two_image_rows_per_tile_give_the_bits_of_one(ng, lib, name):
    """Every output sums its products in the order of the plain form (unsplit reductions in both)."""
    cfg = ROW_PAIRS[name]
    cd = rm.ConvDims(*cfg)
    rng = np.random.default_rng(1019)
    I, F, E = (rng.normal(0, 1, dim).astype(np.float16) for dim in (cd.dimI, cd.dimF, cd.dimO))
    layer = _layer(ng, cfg, "auto")
    got = []
    try:
        assert lib.ng_tune(b"conv_splits", 1) == 0
        for form in (0, 2):
            assert lib.ng_tune(b"row_stack", form) == 0
            got.append(_run_all(ng, layer, I, F, E, relu=True, ops="fb"))
    finally:
        assert lib.ng_tune(b"row_stack", -1) == 0
        assert lib.ng_tune(b"conv_splits", -1) == 0
    for key in ("O", "gradI"):
        assert np.array_equal(got[0][key].view(np.uint16), got[1][key].view(np.uint16)), (name, key)


@pytest.mark.parametrize("name", ["n24_5x5_s3", "n40_2x3_s3_h1", "n8_3x3_s2", "n24_odd_rows_s2"])
def test_strided_update_keeps_nan_to_the_taps_it_meets(ng, name):
    """Rows of no whole number of chunks: a NaN in the input reaches the taps that the oracle's reach."""
    cfg = STRIDED.get(name, (24, 17, 24, 1, 9, 8, 1, 3, 3, 0, 1, 1, 1, 2, 2))
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1017)
    for y, x in ((0, 0), (2, I.shape[3] - 1), (3, I.shape[3] - 2), (4, 3)):
        I2 = I.copy()
        I2[3, 0, y, x, 5] = np.nan
        dU = ng.empty(cd.dimF, dtype=np.float32)
        ng.update_conv(_layer(ng, cfg, "auto"), ng.array(I2), ng.array(E), dU)
        assert np.array_equal(np.isnan(dU.get()), np.isnan(rm.conv_update_fast(cd, I2, E))), (name, y, x)


def test_operand_copies_of_all_passes_share_one_scratch_buffer(ng, lib):
    """Channel-blocked copies: a pass finds room in the buffer that the pass before it left."""
    import ctypes
    layer = _layer(ng, (32, 64, 64, 8, 28, 28, 3, 3, 3, 1, 1, 1, 1, 1, 1))
    copy_bytes = 2 * layer.sizeI                  # 26 MB; the error tensor has the same size
    I, F, E = ng.zeros(layer.dimI), ng.zeros(layer.dimF), ng.zeros(layer.dimO)
    O, gI, gF = ng.empty(layer.dimO), ng.empty(layer.dimI), ng.empty(layer.dimF, dtype=np.float32)

    def free():
        ng.synchronize()
        f, t = ctypes.c_size_t(0), ctypes.c_size_t(0)
        assert lib.ng_mem_info(ctypes.byref(f), ctypes.byref(t)) == 0
        return f.value
    ng.synchronize()
    default, ng.stream = ng.stream, ng.new_stream()
    try:
        assert lib.ng_tune(b"chan_block", 2) == 0
        ng.update_conv(layer, I, E, gF)           # copies of both operands
        before = free()
        ng.fprop_conv(layer, I, F, O)
        ng.bprop_conv(layer, F, E, gI)
        assert before - free() < copy_bytes // 2
    finally:
        assert lib.ng_tune(b"chan_block", -1) == 0
        ng.stream = default


@pytest.fixture
def by_phases(lib):
    """Strided layers of every size in their forms by phases."""
    assert lib.ng_tune(b"stride_phases", 2) == 0
    yield
    assert lib.ng_tune(b"stride_phases", -1) == 0


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("name", ["n24_5x5_s3", "n88_7x7_s2_c96", "n40_2x3_s3_h1", "n32_3d_s222", "n16_1x1_s2", "n8_3x3_s2"])
def test_strided_layers_keep_infinities_from_outputs_that_do_not_meet_them(ng, lib, by_phases, name, value):
    """Minibatches that are no multiple of 64: an infinity or NaN reaches what it reaches on the CUDA-core
    kernels, which skip the pixels outside the tensors that the tensor cores multiply as zeros."""
    cfg = STRIDED[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1023)
    C, T, R, S, K = F.shape

    def check(I, F, E, ops):
        got = [_run_all(ng, _layer(ng, cfg, path), I, F, E, relu=True, ops=ops) for path in ("auto", "simt")]
        for key in got[0]:
            a, b = got[0][key].astype(np.float64), got[1][key].astype(np.float64)
            assert not np.isfinite(b).all() and np.isfinite(b).any()
            for what in (np.isnan, np.isposinf, np.isneginf):
                assert np.array_equal(what(a), what(b)), (name, key)

    for t, r, s in ((0, 0, 0), (T - 1, R - 1, S - 1)):           # corner taps: most outputs at a border miss one
        bad = F.copy()
        bad[C // 2, t, r, s, 1] = value
        got = [_run_all(ng, _layer(ng, cfg, path), I, bad, E, ops="fb") for path in ("auto", "simt")]
        for key in ("O", "gradI"):
            np.testing.assert_array_equal(got[0][key], got[1][key])
            assert not np.isfinite(got[1][key]).all()
        if value > 0:      # (negative ones and NaN are gone after a ReLU)
            check(I, bad, E, "f")
    P, Q = E.shape[2:4]
    for p, q in ((0, 0), (P - 1, Q - 1)):
        bad = E.copy()
        bad[3, 0, p, q, 2] = value
        check(I, F, bad, "b")
        try:                    # (updates whose patch matrix is too large; smaller ones multiply patches, zeros included)
            assert lib.ng_tune(b"stride_phases", 3) == 0
            check(I, F, bad, "u")
        finally:
            assert lib.ng_tune(b"stride_phases", 2) == 0
    bad = I.copy()
    bad[1, 0, 0, I.shape[3] - 1, 5] = value
    if R > 1:              # (a 1x1 filter steps over that pixel)
        check(bad, F, E, "u")


def test_strided_update_in_fp16_keeps_infinities_apart_too(ng, lib, by_phases):
    assert lib.ng_tune(b"stride_phases", 3) == 0
    cfg = STRIDED["n24_5x5_s3"]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1025)
    E[3, 0, 0, 0, 2] = np.inf
    got = []
    for path in ("auto", "simt"):
        layer = _layer(ng, cfg, path)
        dU = ng.empty(layer.dimF)
        ng.update_conv(layer, ng.array(I), ng.array(E), dU)
        got.append(dU.get())
    for what in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(what(got[0]), what(got[1]))
    assert np.isfinite(got[1][:, :, 0]).all() and not np.isfinite(got[1]).all()


@pytest.mark.parametrize("form", [0, 2])
@pytest.mark.parametrize("name", sorted(STRIDED) + ["n64_3d_s222", "n24_1x3_s_h2"])
def test_strided_layers_in_both_forms(ng, lib, name, form):
    """Phase by phase, and in one launch: the size of the layer decides, the results do not show it."""
    cfg = STRIDED.get(name) or {"n64_3d_s222": (64, 32, 40, 4, 6, 7, 2, 3, 3, 1, 1, 1, 2, 2, 2),
                                "n24_1x3_s_h2": (24, 32, 40, 1, 9, 7, 1, 3, 3, 0, 1, 1, 1, 2, 1)}[name]
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1027)
    ref = {"gradI": rm.conv_bprop_fast(cd, F, E, alpha=0.5), "gradF": rm.conv_update_fast(cd, I, E, alpha=0.5)}
    layer = _layer(ng, cfg)
    pad = 4096                  # guard cells
    buf = ng.empty((layer.sizeI + 2 * pad,))
    buf.fill(7.0)
    dB, dU = buf[pad:pad + layer.sizeI].reshape(layer.dimI), ng.empty(layer.dimF, dtype=np.float32)
    try:
        assert lib.ng_tune(b"stride_phases", form) == 0
        ng.bprop_conv(layer, ng.array(F), ng.array(E), dB, alpha=0.5)
        ng.update_conv(layer, ng.array(I), ng.array(E), dU, alpha=0.5)
    finally:
        assert lib.ng_tune(b"stride_phases", -1) == 0
    _check(cd, {"gradI": dB.get(), "gradF": dU.get()}, I, F, E, ref, "%s form %d" % (name, form))
    guard = buf.get()
    assert (guard[:pad] == 7.0).all() and (guard[-pad:] == 7.0).all()


@pytest.mark.parametrize("cfg, launches", [
    ((64, 64, 64, 1, 32, 32, 1, 4, 4, 0, 0, 0, 1, 4, 4), 1), ((128, 96, 96, 1, 55, 55, 1, 3, 3, 0, 1, 1, 1, 2, 2), 4),
    ((8, 16, 16, 1, 8, 8, 1, 4, 4, 0, 0, 0, 1, 4, 4), 1), ((48, 64, 64, 1, 56, 56, 1, 3, 3, 0, 1, 1, 1, 2, 2), 6)])
def test_small_strided_backward_passes_take_one_launch(ng, lib, cfg, launches):
    import ctypes
    layer = _layer(ng, cfg)
    F, E, gI = ng.zeros(layer.dimF), ng.zeros(layer.dimO), ng.empty(layer.dimI)
    before, after = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    assert lib.ng_launch_count(ctypes.byref(before)) == 0
    ng.bprop_conv(layer, F, E, gI)
    assert lib.ng_launch_count(ctypes.byref(after)) == 0
    assert after.value - before.value == launches


STRIDED_SUMS = {
    # name: layer, longest partition of its sums in k-blocks of 64: patches (at most 3), a phase-split copy (294 k-blocks
    # in 32 partitions)
    "c64_3x3_n16_patches": ((16, 64, 64, 1, 14, 14, 1, 3, 3, 0, 1, 1, 1, 2, 2), 3),
    "c128_1x1_n24_patches": ((24, 128, 128, 1, 28, 28, 1, 1, 1, 0, 0, 0, 1, 2, 2), 3),
    "c24_3x3_n96_patches": ((96, 24, 512, 1, 13, 13, 1, 3, 3, 0, 1, 1, 1, 2, 2), 3),
    "c128_3x3_n40_phases": ((40, 128, 256, 1, 41, 41, 1, 3, 3, 0, 1, 1, 1, 2, 2), 10),
}


@pytest.mark.parametrize("name", sorted(STRIDED_SUMS))
def test_strided_gradients_are_summed_in_short_partitions(ng, name):
    """Against sums in 64 bits. Each of the four MMAs of a k-block cuts its sum to 24 bits: 0.36 2^-23 of it on average. A
    partition's sum grows like a random walk, so that the sums cut are two thirds of its end on average, and the
    partitions' errors, like their ends, add as a random walk: 4 * 0.36 * 2/3 * 2^-23 of the result per k-block."""
    cfg, longest = STRIDED_SUMS[name]
    cd = rm.ConvDims(*cfg)
    rng = np.random.default_rng(1029)
    I = rng.uniform(0, 1, cd.dimI).astype(np.float16)
    E = rng.normal(0, 0.1, cd.dimO).astype(np.float16)
    layer = _layer(ng, cfg)
    dU = ng.empty(layer.dimF, dtype=np.float32)
    ng.update_conv(layer, ng.array(I), ng.array(E), dU)
    N, C, K, _, H, W, _, R, S = cfg[:9]
    pad, st = cfg[10], cfg[13]
    _, P, Q = cd.MPQ
    padded = np.zeros((C, H + 2 * pad + st, W + 2 * pad + st, N))
    padded[:, pad:pad + H, pad:pad + W] = I[:, 0]
    e = E.astype(np.float64).reshape(K, -1)
    ref = np.empty((C, 1, R, S, K))
    for r in range(R):
        for s in range(S):
            ref[:, 0, r, s] = padded[:, r:r + P * st:st, s:s + Q * st:st][:, :P, :Q].reshape(C, -1) @ e.T
    got = dU.get().astype(np.float64)
    assert np.linalg.norm(got - ref) <= 4 * 0.36 * 2 / 3 * 2.0 ** -23 * longest * np.linalg.norm(ref)


@pytest.mark.parametrize("name", sorted(STRIDED))
def test_strided_layers_by_phases(ng, lib, by_phases, name):
    test_strided_layers_run_on_the_tensor_core_path(ng, lib, name)


@pytest.mark.parametrize("name", ["c40_k72_5x5_s2", "c40_k64_3x5_s3_n24"])
def test_two_image_rows_per_tile_by_phases(ng, lib, by_phases, name):
    test_two_image_rows_per_tile(ng, lib, name)
    test_two_image_rows_per_tile_give_the_bits_of_one(ng, lib, name)


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("name", ["c48_k128_5x5_s2_n24"])
def test_update_with_exchanged_operands_by_phases(ng, lib, by_phases, name, half):
    test_update_with_exchanged_operands(ng, lib, name, half)


@pytest.mark.parametrize("name", ["n24_5x5_s3", "n40_2x3_s3_h1", "n8_3x3_s2", "n24_odd_rows_s2"])
def test_strided_update_keeps_nan_to_the_taps_it_meets_by_phases(ng, by_phases, name):
    test_strided_update_keeps_nan_to_the_taps_it_meets(ng, name)


@pytest.mark.parametrize("swap", [0, 2])
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("name", ["n88_7x7_s2_c96", "n24_5x5_s3", "n32_3d_s222", "n40_2x3_s3_h1", "n24_c48_5x5_s2"])
def test_strided_sums_in_several_launches(ng, lib, name, half, swap):
    """The form of updates beyond the patch matrix, forced on small layers: partitions of six k-blocks, two to a launch."""
    cfg = STRIDED.get(name, (24, 48, 128, 1, 17, 15, 1, 5, 5, 0, 2, 2, 1, 2, 2))
    cd = rm.ConvDims(*cfg)
    I, F, E = _inputs(cd, 1031)
    ref = rm.conv_update_fast(cd, I, E, alpha=0.5)
    layer = _layer(ng, cfg)
    pad = 4096                  # guard cells
    buf = ng.empty((layer.sizeF + 2 * pad,), dtype=np.float16 if half else np.float32)
    buf.fill(7.0)
    try:
        for key, value in ((b"stride_phases", 3), (b"conv_splits", 2), (b"update_swap", swap)):
            assert lib.ng_tune(key, value) == 0
        ng.update_conv(layer, ng.array(I), ng.array(E), buf[pad:pad + layer.sizeF].reshape(layer.dimF), alpha=0.5)
    finally:
        for key in (b"stride_phases", b"conv_splits", b"update_swap"):
            assert lib.ng_tune(key, -1) == 0
    got = buf.get()
    assert (got[:pad] == 7.0).all() and (got[-pad:] == 7.0).all()
    tol = f32_tol(_abs_terms(cd, I, F, E)[2], int(np.prod(cd.MPQ)) * cd.N)
    if half:
        tol = tol + 2.0 ** -11 * np.abs(ref) + 2.0 ** -25
    assert_close(got[pad:-pad].reshape(layer.dimF), ref, tol, name)
