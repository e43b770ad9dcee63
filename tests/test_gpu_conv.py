"""GPU parity of the three convolution entry points (through the C ABI) against the CPU oracle.

DCG_PREC_FP32 keeps the reference CPU's summation order with unfused multiply/add and must
reproduce the oracle bit for bit.  DCG_PREC_TF32 (tcgen05, fp32 accumulate) must stay within
1e-2 * max|ref| per output tensor - the tolerance stated for the TF32 tensor-core path.
"""
import ctypes
import threading

import numpy as np
import pytest
import torch

import oracle
from conftest import seeded

pytestmark = pytest.mark.gpu

TF32_TOL = 1e-2  # max abs error <= TF32_TOL * max|ref|
X3_TOL = 1e-5    # 3xTF32 (operand = TF32 part + residual, three MMAs per K step), same norm

# N, H, W, C, K, O, stride.  Small / ragged shapes the reference's unit tests use, odd sizes,
# channel counts below and above one 32-wide K chunk, and DCGAN layer shapes at batch 2.
SHAPES = [
    (2, 4, 4, 2, 2, 2, 2), (2, 3, 5, 3, 3, 2, 2), (1, 7, 9, 3, 5, 4, 2), (2, 6, 6, 2, 3, 3, 1),
    (3, 3, 5, 1, 2, 3, 1), (2, 9, 9, 5, 5, 2, 2), (1, 1, 1, 1, 1, 1, 1),
    (2, 8, 8, 4, 5, 8, 2), (2, 16, 16, 32, 5, 64, 2), (2, 12, 20, 36, 5, 40, 2),
    (2, 64, 64, 3, 5, 64, 2), (2, 32, 32, 64, 5, 128, 2), (2, 16, 16, 128, 5, 256, 2),
    (2, 8, 8, 256, 5, 512, 2),
    # narrow-channel paths (<= 4 input channels, O a multiple of 32): window-map forward, one-tile
    # kernel gradient over pixel partitions, GEMM + gather input gradient; stride 1, even kernel
    (3, 20, 12, 1, 3, 32, 1), (2, 16, 16, 4, 5, 96, 2), (5, 32, 32, 2, 4, 64, 2), (2, 10, 14, 3, 5, 160, 2),
]


def _check(got, ref, prec, pkg, what):
    got = got.cpu().numpy()
    assert got.shape == ref.shape, (what, got.shape, ref.shape)
    if prec == pkg.PREC_FP32:
        assert np.array_equal(got, ref), "%s: fp32 path differs from the oracle, max err %g" % (
            what, np.abs(got - ref).max())
    else:
        lim = (X3_TOL if prec == pkg.PREC_3XTF32 else TF32_TOL) * max(np.abs(ref).max(), 1e-30)
        err = np.abs(got - ref).max()
        assert err <= lim, "%s: max err %g > %g" % (what, err, lim)


PRECS = {"fp32": "PREC_FP32", "tf32": "PREC_TF32", "3xtf32": "PREC_3XTF32"}


@pytest.mark.parametrize("prec_name", ["fp32", "tf32", "3xtf32"])
@pytest.mark.parametrize("shape", SHAPES)
def test_conv_fwd_dx_dk(pkg, dev, orc, shape, prec_name):
    F = pkg.functional
    prec = getattr(pkg, PRECS[prec_name])
    N, H, W, C, K, O, s = shape
    x = seeded((N, H, W, C), 234)
    k = seeded((K, K, C, O), 235) * np.float32(0.1)
    pad = (oracle.same_pad(H, K, s), oracle.same_pad(W, K, s))
    y_ref = orc.conv2d(x, k, (s, s))
    dy = seeded(y_ref.shape, 236)
    xd, kd, dyd = (torch.from_numpy(a).to(dev) for a in (x, k, dy))
    y = F.conv2d_fwd(xd, kd, (s, s), precision=prec)
    dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=prec)
    dk = F.conv2d_dk(xd, dyd, (K, K), (s, s), precision=prec)
    torch.cuda.synchronize()
    _check(y, y_ref, prec, pkg, "fwd")
    _check(dx, orc.conv2d_input_grad(dy, k, s, (H, W)), prec, pkg, "dx")
    _check(dk, orc.conv2d_kernel_grad(dy, x, s, pad), prec, pkg, "dk")


# stride 2 (four parity classes): the shapes the class-fused input gradient takes - tiles narrower and wider than
# 64 columns, a ragged channel chunk (40 = 32 + 8), two channel
# tiles (256 = 2 x 128), odd extents (a class with fewer rows / columns), 3x3 and 4x4 kernels
FUSED_DX_SHAPES = [
    (2, 16, 16, 32, 5, 64, 2), (2, 12, 20, 36, 5, 40, 2), (2, 32, 32, 64, 5, 128, 2), (2, 16, 16, 128, 5, 256, 2),
    (2, 8, 8, 256, 5, 512, 2), (1, 7, 9, 8, 5, 12, 2), (2, 9, 9, 8, 3, 8, 2), (3, 32, 32, 8, 4, 64, 2),
    # channel counts that rule out 16-byte stores (element-wise epilogue)
    (2, 16, 16, 6, 5, 32, 2), (2, 10, 14, 9, 5, 160, 2),
]


@pytest.mark.parametrize("shape", FUSED_DX_SHAPES)
def test_dx_with_parity_classes_fused(pkg, dev, orc, shape):
    """The input gradient that gives one CTA all parity classes of a pixel tile (planned by default only where
    one CTA per tile fills the GPU; forced here) against the reference's CPU code: plain, gated by the previous
    layer's activation with the raw gradient kept, and as a generator layer (bias, pre-activation, activation)."""
    F, L = pkg.functional, pkg.lib
    N, H, W, C, K, O, s = shape
    k = seeded((K, K, C, O), 235) * np.float32(0.1)
    y_shape = orc.conv2d(seeded((N, H, W, C), 234), k, (s, s)).shape
    dy = seeded(y_shape, 236)
    z = seeded((N, H, W, C), 237)
    b = seeded((C,), 238)
    dx_ref = orc.conv2d_input_grad(dy, k, s, (H, W))
    kd, dyd, zd, bd = (torch.from_numpy(a).to(dev) for a in (k, dy, z, b))
    before = L.dcg_debug_fused_dx_launches()
    try:
        L.dcg_debug_set_dx_mode(2)
        dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_TF32)
        raw = torch.empty(dx_ref.shape, device=dev)
        gated = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_TF32,
                            epilogue=F.make_epilogue(gate=zd, gate_act=pkg.ACT_LEAKY, gate_alpha=0.2, raw_out=raw))
        pre = torch.empty(dx_ref.shape, device=dev)
        act = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_TF32,
                          epilogue=F.make_epilogue(bias=bd, act=pkg.ACT_RELU, pre_act=pre))
        torch.cuda.synchronize()
    finally:
        L.dcg_debug_set_dx_mode(-1)
    assert L.dcg_device_status() == 0, L.dcg_last_error()
    assert L.dcg_debug_fused_dx_launches() - before == 3, "the fused kernel did not take this shape"
    _check(dx, dx_ref, pkg.PREC_TF32, pkg, "dx")
    _check(raw, dx_ref, pkg.PREC_TF32, pkg, "raw dx")
    _check(gated, orc.leaky_relu_grad(z, dx_ref, 0.2), pkg.PREC_TF32, pkg, "gated dx")
    pre_ref = orc.mvrow_add(dx_ref.reshape(-1, C), b).reshape(dx_ref.shape)
    _check(pre, pre_ref, pkg.PREC_TF32, pkg, "pre-activation")
    _check(act, orc.vect_relu(pre_ref), pkg.PREC_TF32, pkg, "activation")
    # and the same call planned the other way gives the same numbers up to TF32 summation order
    L.dcg_debug_set_dx_mode(0)
    try:
        dx0 = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_TF32)
        torch.cuda.synchronize()
    finally:
        L.dcg_debug_set_dx_mode(-1)
    assert L.dcg_debug_fused_dx_launches() - before == 3
    _check(dx0, dx_ref, pkg.PREC_TF32, pkg, "dx, one tile per class")


# one shape or more for every thread tile of the ordered fp32 kernels (few / some / many outputs per lane, RGB input gradient,
# kernel gradient with the images over 1, 4 and 16 thread groups), with and without 16-byte copies of either operand, tap
# counts with and without an unrolled form, tiles and channel quads that are not full, and a kernel too large for them
ORDERED_SHAPES = [
    (2, 96, 101, 5, 3, 36, 1), (2, 64, 80, 68, 3, 6, 1), (3, 5, 6, 164, 5, 156, 1), (2, 9, 7, 36, 5, 44, 2), (5, 9, 7, 36, 5, 44, 2),
    (17, 6, 5, 3, 4, 34, 2), (2, 33, 65, 12, 1, 20, 1), (4, 24, 40, 33, 5, 40, 2), (1, 11, 9, 2, 7, 3, 2), (1, 5, 4, 7, 2, 3, 3),
]


@pytest.mark.parametrize("shape", ORDERED_SHAPES)
def test_fp32_ordered_kernels_match_oracle_bit_for_bit(pkg, dev, orc, shape):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    x, k = seeded((N, H, W, C), 234), seeded((K, K, C, O), 235)
    pad = (oracle.same_pad(H, K, s), oracle.same_pad(W, K, s))
    y_ref = orc.conv2d(x, k, (s, s))
    dy, b = seeded(y_ref.shape, 236), seeded((O,), 237)
    xd, kd, dyd, bd = (torch.from_numpy(a).to(dev) for a in (x, k, dy, b))
    y = F.conv2d_fwd(xd, kd, (s, s), epilogue=F.make_epilogue(bias=bd, act=pkg.ACT_LEAKY), precision=pkg.PREC_FP32)
    dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_FP32)
    dk = F.conv2d_dk(xd, dyd, (K, K), (s, s), precision=pkg.PREC_FP32)
    torch.cuda.synchronize()
    _check(y, orc.vect_relu_leaky(orc.mvrow_add(y_ref.reshape(-1, O), b), 0.2).reshape(y_ref.shape), pkg.PREC_FP32, pkg, "fwd")
    _check(dx, orc.conv2d_input_grad(dy, k, s, (H, W)), pkg.PREC_FP32, pkg, "dx")
    _check(dk, orc.conv2d_kernel_grad(dy, x, s, pad), pkg.PREC_FP32, pkg, "dk")


@pytest.mark.parametrize("shape", ORDERED_SHAPES + [(2, 20, 20, 6, 7, 10, 1)])
def test_fp32_taps_outside_the_image_are_skipped(pkg, dev, orc, shape):
    """Infinite and NaN factors of taps (pixels) that some outputs do not have: those outputs stay finite, as in the oracle."""
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    pad = (oracle.same_pad(H, K, s), oracle.same_pad(W, K, s))
    ho, wo = -(-H // s), -(-W // s)
    x, k, dy = seeded((N, H, W, C), 240), seeded((K, K, C, O), 241), seeded((N, ho, wo, O), 242)
    k_bad, dy_bad = k.copy(), dy.copy()
    k_bad[0, :, 0, 0], k_bad[K - 1, K - 1, C - 1, O - 1] = np.inf, np.nan
    dy_bad[0, 0, :, 0], dy_bad[N - 1, ho - 1, wo - 1, O - 1] = -np.inf, np.nan
    xd, kd, dyd, dy_badd = (torch.from_numpy(a).to(dev) for a in (x, k_bad, dy, dy_bad))
    y = F.conv2d_fwd(xd, kd, (s, s), precision=pkg.PREC_FP32)
    dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_FP32)
    dk = F.conv2d_dk(xd, dy_badd, (K, K), (s, s), precision=pkg.PREC_FP32)
    with np.errstate(invalid="ignore"):
        refs = orc.conv2d(x, k_bad, (s, s)), orc.conv2d_input_grad(dy, k_bad, s, (H, W)), orc.conv2d_kernel_grad(dy_bad, x, s, pad)
    for name, got, ref in zip(("fwd", "dx", "dk"), (y, dx, dk), refs):
        assert np.array_equal(got.cpu().numpy(), ref, equal_nan=True), name


# more column tiles and more parity classes than a grid has rows and layers of blocks
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1, 4200000, 1), (1, 1, 1, 2100000, 1, 2, 1), (1, 300, 300, 2, 1, 3, 300)])
def test_fp32_extents_beyond_a_grid(pkg, dev, orc, shape):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    x, k = seeded((N, H, W, C), 243), seeded((K, K, C, O), 244)
    dy = seeded((N, -(-H // s), -(-W // s), O), 245)
    xd, kd, dyd = (torch.from_numpy(a).to(dev) for a in (x, k, dy))
    y = F.conv2d_fwd(xd, kd, (s, s), precision=pkg.PREC_FP32)
    dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_FP32)
    dk = F.conv2d_dk(xd, dyd, (K, K), (s, s), precision=pkg.PREC_FP32)
    _check(y, orc.conv2d(x, k, (s, s)), pkg.PREC_FP32, pkg, "fwd")
    dx_ref = np.zeros((N, H, W, C), np.float32)   # one tap: the gradient of the pixels that were read
    dx_ref[:, ::s, ::s] = orc.conv2d_input_grad(dy, k, 1, dy.shape[1:3])
    _check(dx, dx_ref, pkg.PREC_FP32, pkg, "dx")
    _check(dk, orc.conv2d_kernel_grad(dy, x, s, (0, 0))[:K, :K], pkg.PREC_FP32, pkg, "dk")


@pytest.mark.parametrize("shape", [(40, 64, 64, 3, 5, 64, 2), (40, 60, 52, 3, 5, 64, 2), (37, 64, 64, 4, 5, 32, 2)])
def test_three_channel_layers_with_persistent_ctas(pkg, dev, orc, shape):
    """More tiles than SMs: the forward of a <= 4-channel layer and the GEMM of its input gradient run as
    persistent CTAs that walk several tiles each (weights resident, accumulator double-buffered).  Forward with
    the whole fused chain, input gradient with bias + tanh (a generator's last layer), against the CPU code;
    tile counts that do and do not divide by the grid, output extents that do not fill the pixel tiles."""
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    x = seeded((N, H, W, C), 234)
    k = seeded((K, K, C, O), 235) * np.float32(0.1)
    b = seeded((O,), 303)
    raw_ref = orc.conv2d(x, k, (s, s))
    z_ref = orc.mvrow_add(raw_ref, b)
    xd, kd, bd = (torch.from_numpy(a).to(dev) for a in (x, k, b))
    raw = torch.empty(raw_ref.shape, device=dev)
    z = torch.empty(raw_ref.shape, device=dev)
    y = F.conv2d_fwd(xd, kd, (s, s), precision=pkg.PREC_TF32,
                     epilogue=F.make_epilogue(bias=bd, act=pkg.ACT_LEAKY, alpha=0.2, pre_act=z, raw_out=raw))
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0, pkg.lib.dcg_last_error()
    _check(raw, raw_ref, pkg.PREC_TF32, pkg, "raw")
    _check(z, z_ref, pkg.PREC_TF32, pkg, "pre-activation")
    _check(y, orc.vect_relu_leaky(z_ref, 0.2), pkg.PREC_TF32, pkg, "activation")
    dy = seeded(raw_ref.shape, 236)
    bc = seeded((C,), 304)
    dyd, bcd = torch.from_numpy(dy).to(dev), torch.from_numpy(bc).to(dev)
    dx_ref = orc.conv2d_input_grad(dy, k, s, (H, W))
    dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_TF32)
    t = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=pkg.PREC_TF32, epilogue=F.make_epilogue(bias=bcd, act=pkg.ACT_TANH))
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0, pkg.lib.dcg_last_error()
    _check(dx, dx_ref, pkg.PREC_TF32, pkg, "dx")
    np.testing.assert_allclose(t.cpu().numpy(), orc.vect_tanh(orc.mvrow_add(dx_ref, bc)), rtol=0,
                               atol=TF32_TOL * max(np.abs(dx_ref).max(), 1.0))


@pytest.mark.parametrize("prec_name", ["fp32", "tf32"])
def test_golden_reference_cases(pkg, dev, golden, prec_name):
    """The reference's own unit-test tensors (tests/test_conv2d*.cu) through the C ABI."""
    F = pkg.functional
    prec = pkg.PREC_FP32 if prec_name == "fp32" else pkg.PREC_TF32
    for case in ("conv2d", "conv2d_padding"):
        x, k = (torch.from_numpy(golden[case + "/" + n]).to(dev) for n in ("x", "k"))
        _check(F.conv2d_fwd(x, k, precision=prec), golden[case + "/y"], prec, pkg, case)
    for case in ("conv2d_grad", "conv2d_padding_grad"):
        x, k, dy = (torch.from_numpy(golden[case + "/" + n]).to(dev) for n in ("x", "k", "dy_hat"))
        _check(F.conv2d_dx(dy, k, x.shape[1:3], precision=prec), golden[case + "/dx"], prec, pkg, case + " dx")
        _check(F.conv2d_dk(x, dy, k.shape[:2], precision=prec), golden[case + "/dk"], prec, pkg, case + " dk")
    # conv2d_transpose = dx of the mirrored conv; its gradients = fwd / dk with roles swapped
    c = "conv2d_transpose_grad"
    x, k, dy = (torch.from_numpy(golden[c + "/" + n]).to(dev) for n in ("x", "k", "dy_hat"))
    _check(F.conv2d_dx(x, k, (8, 8), pad=(0, 0), precision=prec), golden[c + "/y_hat"], prec, pkg, "convT fwd")
    _check(F.conv2d_fwd(dy, k, pad=(0, 0), precision=prec), golden[c + "/dx"], prec, pkg, "convT dx")
    _check(F.conv2d_dk(dy, x, (2, 2), pad=(0, 0), precision=prec), golden[c + "/dk"], prec, pkg, "convT dk")


@pytest.mark.parametrize("prec_name", ["fp32", "tf32"])
@pytest.mark.parametrize("shape", [(2, 9, 9, 5, 5, 6, 2), (2, 16, 16, 32, 5, 64, 2), (2, 16, 16, 3, 5, 64, 2)])
def test_fused_epilogues(pkg, dev, orc, shape, prec_name):
    F = pkg.functional
    prec = pkg.PREC_FP32 if prec_name == "fp32" else pkg.PREC_TF32
    N, H, W, C, K, O, s = shape
    x = seeded((N, H, W, C), 301)
    k = seeded((K, K, C, O), 302) * np.float32(0.1)
    b = seeded((O,), 303)
    raw_ref = orc.conv2d(x, k, (s, s))
    z_ref = orc.mvrow_add(raw_ref, b)
    xd, kd, bd = (torch.from_numpy(a).to(dev) for a in (x, k, b))
    for act, fn in ((pkg.ACT_LEAKY, lambda a: orc.vect_relu_leaky(a, 0.2)), (pkg.ACT_RELU, orc.vect_relu),
                    (pkg.ACT_TANH, orc.vect_tanh), (pkg.ACT_SIGMOID, orc.vect_sigmoid), (pkg.ACT_NONE, lambda a: a)):
        raw = torch.empty(raw_ref.shape, device=dev)
        z = torch.empty(raw_ref.shape, device=dev)
        ep = F.make_epilogue(bias=bd, act=act, alpha=0.2, pre_act=z, raw_out=raw)
        y = F.conv2d_fwd(xd, kd, (s, s), epilogue=ep, precision=prec)
        torch.cuda.synchronize()
        _check(raw, raw_ref, prec, pkg, "raw")
        _check(z, z_ref, prec, pkg, "pre_act")
        a_ref = fn(z_ref)
        if prec == pkg.PREC_FP32 and act in (pkg.ACT_TANH, pkg.ACT_SIGMOID):
            # device expf is not glibc's: a few ulp on the exponential
            np.testing.assert_allclose(y.cpu().numpy(), a_ref, rtol=0, atol=2e-6)
        else:
            _check(y, a_ref, prec, pkg, "act %d" % act)

    # input gradient gated by the derivative of the previous layer's activation
    dy = seeded(raw_ref.shape, 304)
    zprev = seeded((N, H, W, C), 305)
    dyd, zd = torch.from_numpy(dy).to(dev), torch.from_numpy(zprev).to(dev)
    dx_ref = orc.conv2d_input_grad(dy, k, s, (H, W))
    for gact, fn in ((pkg.ACT_LEAKY, lambda g, d: orc.leaky_relu_grad(g, d, 0.2)), (pkg.ACT_RELU, orc.relu_grad),
                     (pkg.ACT_TANH, orc.tanh_grad)):
        raw = torch.empty(dx_ref.shape, device=dev)
        ep = F.make_epilogue(gate=zd, gate_act=gact, gate_alpha=0.2, raw_out=raw)
        dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), epilogue=ep, precision=prec)
        torch.cuda.synchronize()
        _check(raw, dx_ref, prec, pkg, "dx raw")
        ref_g = fn(zprev, dx_ref)
        if prec == pkg.PREC_FP32:
            assert np.array_equal(dx.cpu().numpy(), ref_g)
        else:
            _check(dx, ref_g, prec, pkg, "gated dx")


def test_transposed_conv_roles(pkg, dev, orc):
    """Generator layer [2,4,4,64] -> [2,8,8,32] (5x5, stride 2, SAME): forward is the dx entry
    point, its input gradient the fwd entry point, its kernel gradient dk with roles swapped."""
    F = pkg.functional
    x = seeded((2, 4, 4, 64), 401)
    k = seeded((5, 5, 32, 64), 402) * np.float32(0.05)   # [kh, kw, Cout, Cin]
    dy = seeded((2, 8, 8, 32), 403)
    xd, kd, dyd = (torch.from_numpy(a).to(dev) for a in (x, k, dy))
    for prec in (pkg.PREC_FP32, pkg.PREC_TF32):
        y = F.conv2d_dx(xd, kd, (8, 8), precision=prec)
        dx = F.conv2d_fwd(dyd, kd, precision=prec)
        dk = F.conv2d_dk(dyd, xd, (5, 5), precision=prec)
        torch.cuda.synchronize()
        _check(y, orc.conv2d_transpose(x, k, (2, 8, 8, 32), 2), prec, pkg, "convT")
        _check(dx, orc.conv2d_transpose_input_grad(dy, k, 2, (4, 4)), prec, pkg, "convT dx")
        _check(dk, orc.conv2d_transpose_kernel_grad(dy, x, 2, (5, 5)), prec, pkg, "convT dk")


@pytest.mark.parametrize("layer", [(64, 32, 32, 64, 128), (64, 16, 16, 128, 256), (64, 8, 8, 256, 512),
                                   (64, 64, 64, 3, 64)])
def test_full_batch_layers_tf32_vs_fp32_path(pkg, dev, layer):
    """Batch-64 DCGAN layers: too slow for the scalar oracle, so the tensor path is compared with
    the fp32 CUDA-core path (itself bit-exact with the oracle at small sizes), and the three
    operators are tied together by the adjoint identity <conv(x,k),dy> = <x,dx> = <k,dk>."""
    F = pkg.functional
    N, H, W, C, O = layer
    g = torch.Generator(device="cpu").manual_seed(5)
    x = (torch.rand((N, H, W, C), generator=g) * 2 - 1).to(dev)
    k = (torch.randn((5, 5, C, O), generator=g) * 0.02).to(dev)
    dy = (torch.rand((N, H // 2, W // 2, O), generator=g) * 2 - 1).to(dev)
    outs = {}
    for prec in (pkg.PREC_FP32, pkg.PREC_TF32):
        outs[prec] = (F.conv2d_fwd(x, k, precision=prec), F.conv2d_dx(dy, k, (H, W), precision=prec),
                      F.conv2d_dk(x, dy, (5, 5), precision=prec))
    torch.cuda.synchronize()
    for name, a, b in zip(("fwd", "dx", "dk"), outs[pkg.PREC_FP32], outs[pkg.PREC_TF32]):
        lim = TF32_TOL * a.abs().max().item()
        assert (a - b).abs().max().item() <= lim, name
    # 3xTF32 is held to 1e-5 * max|ref| against a float64 evaluation (torch, same SAME padding: 1 before,
    # 2 after): at these sizes the fp32 paths themselves carry ~sqrt(K) * 2^-24 = 1.5e-5 of summation
    # noise in the longest reductions (65 536 pixels per kernel-gradient element), which the yardstick
    # must not
    x3 = (F.conv2d_fwd(x, k, precision=pkg.PREC_3XTF32), F.conv2d_dx(dy, k, (H, W), precision=pkg.PREC_3XTF32),
          F.conv2d_dk(x, dy, (5, 5), precision=pkg.PREC_3XTF32))
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    x64 = x.double().permute(0, 3, 1, 2).contiguous().requires_grad_(True)
    k64 = k.double().permute(3, 2, 0, 1).contiguous().requires_grad_(True)
    y64 = torch.nn.functional.conv2d(torch.nn.functional.pad(x64, (1, 2, 1, 2)), k64, stride=2)
    dx64, dk64 = torch.autograd.grad(y64, (x64, k64), dy.double().permute(0, 3, 1, 2).contiguous())
    ref64 = (y64.detach().permute(0, 2, 3, 1), dx64.permute(0, 2, 3, 1), dk64.permute(2, 3, 1, 0))
    for name, a, b in zip(("fwd", "dx", "dk"), ref64, x3):
        assert (a - b.double()).abs().max().item() <= X3_TOL * a.abs().max().item(), "3xTF32 " + name
    for name, a, b in zip(("fwd", "dx", "dk"), ref64, outs[pkg.PREC_FP32]):   # the yardstick agrees with the fp32 path
        assert (a - b.double()).abs().max().item() <= 1e-4 * a.abs().max().item(), "fp32 vs float64 " + name
    y, dx, dk = (t.double() for t in outs[pkg.PREC_TF32])
    terms = y * dy.double()
    lhs = terms.sum().item()
    # the inner product is a sum of ~1e6 signed terms that largely cancel; TF32 rounding (~5e-4 per
    # term, random sign) perturbs it by about 5e-4 * sqrt(sum of squared terms)
    tol = 5e-3 * terms.pow(2).sum().sqrt().item() + 1e-3
    assert abs(lhs - (dx * x.double()).sum().item()) <= tol
    assert abs(lhs - (dk * k.double()).sum().item()) <= tol


# six kernel rows fill one column tile of the kernel gradient in 3xTF32, seven and eight take two; also with K partitions and
# without, more than 128 output channels, and a count that comes in pieces of 32
@pytest.mark.parametrize("prec_name", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", [(2, 20, 18, 3, 6, 32, 2), (3, 21, 17, 3, 7, 64, 2), (2, 16, 19, 4, 8, 36, 1), (9, 33, 30, 1, 7, 160, 2),
                                   (1, 9, 7, 3, 8, 32, 1)])
def test_tall_kernels_of_rgb_layers(pkg, dev, orc, shape, prec_name):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    prec = getattr(pkg, PRECS[prec_name])
    x, k = seeded((N, H, W, C), 234), seeded((K, K, C, O), 235) * np.float32(0.1)
    pad = (oracle.same_pad(H, K, s), oracle.same_pad(W, K, s))
    y_ref = orc.conv2d(x, k, (s, s))
    dy = seeded(y_ref.shape, 236)
    xd, kd, dyd = (torch.from_numpy(a).to(dev) for a in (x, k, dy))
    y = F.conv2d_fwd(xd, kd, (s, s), precision=prec)
    dx = F.conv2d_dx(dyd, kd, (H, W), (s, s), precision=prec)
    dk = F.conv2d_dk(xd, dyd, (K, K), (s, s), precision=prec)
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    _check(y, y_ref, prec, pkg, "fwd")
    _check(dx, orc.conv2d_input_grad(dy, k, s, (H, W)), prec, pkg, "dx")
    _check(dk, orc.conv2d_kernel_grad(dy, x, s, pad), prec, pkg, "dk")


# accumulators 64, 96, 160 and 256 columns wide, one CTA per SM with and without K partitions, two MMA warps on one, two and
# an odd number of stages, pixel boxes that do not fill their tile, and kernel gradients with the channels of two or four
# taps in one tile, the last one part empty
TILING_SHAPES = [
    (13, 75, 51, 96, 3, 160, 1), (160, 16, 16, 128, 5, 256, 2), (4, 16, 16, 192, 3, 320, 1), (3, 22, 18, 64, 3, 96, 1),
    (5, 13, 11, 32, 3, 224, 2), (1, 7, 5, 32, 1, 32, 1), (1, 7, 9, 64, 1, 64, 1), (2, 17, 9, 32, 5, 64, 1), (70, 9, 9, 64, 2, 128, 2),
]


@pytest.mark.parametrize("prec_name", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", TILING_SHAPES)
def test_tile_widths_and_pixel_boxes(pkg, dev, shape, prec_name):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    x, k, dy = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in
                ((51, (N, H, W, C)), (52, (K, K, C, O)), (53, (N, -(-H // s), -(-W // s), O))))
    got, ref = ([F.conv2d_fwd(x, k, (s, s), precision=p), F.conv2d_dx(dy, k, (H, W), (s, s), precision=p),
                 F.conv2d_dk(x, dy, (K, K), (s, s), precision=p)] for p in (getattr(pkg, PRECS[prec_name]), pkg.PREC_FP32))
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    tol = TF32_TOL if prec_name == "tf32" else 1e-4   # the fp32 path sums tens of thousands of pixels one by one
    for name, a, b in zip(("fwd", "dx", "dk"), got, ref):
        assert (a - b).abs().max().item() <= tol * b.abs().max().item(), name


# channel counts that are no multiple of 32 on either side or both: one piece of 32 channels and several, the last of them
# nearly empty and nearly full, more than one tile along each axis, K partitions and none
RAGGED_SHAPES = [
    (2, 12, 20, 36, 5, 40, 2), (3, 9, 11, 16, 3, 20, 1), (2, 16, 16, 132, 5, 100, 2), (5, 13, 11, 68, 3, 260, 2),
    (1, 7, 9, 188, 1, 28, 1), (4, 20, 14, 32, 3, 36, 1), (4, 20, 14, 36, 3, 32, 1), (16, 24, 24, 60, 3, 156, 1),
    # <= 4 input channels: dy in pieces, weights padded to 32; fewer images than a pixel box holds
    (20, 33, 30, 3, 5, 36, 2), (9, 40, 40, 4, 3, 140, 1), (1, 200, 180, 1, 5, 12, 1), (3, 4, 4, 64, 5, 96, 2),
]


@pytest.mark.parametrize("prec_name", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", RAGGED_SHAPES)
def test_ragged_channel_counts(pkg, dev, shape, prec_name):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    x, k, dy = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in
                ((54, (N, H, W, C)), (55, (K, K, C, O)), (56, (N, -(-H // s), -(-W // s), O))))
    got, ref = ([F.conv2d_fwd(x, k, (s, s), precision=p), F.conv2d_dx(dy, k, (H, W), (s, s), precision=p),
                 F.conv2d_dk(x, dy, (K, K), (s, s), precision=p)] for p in (getattr(pkg, PRECS[prec_name]), pkg.PREC_FP32))
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    tol = TF32_TOL if prec_name == "tf32" else 3e-5
    for name, a, b in zip(("fwd", "dx", "dk"), got, ref):
        assert (a - b).abs().max().item() <= tol * b.abs().max().item(), name


# the last column tile has fewer channels than columns; the bias ends where the channels do, not where the tile does
@pytest.mark.parametrize("prec_name", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", [(2, 12, 20, 36, 5, 40, 2), (1, 7, 9, 36, 1, 36, 1), (40, 24, 24, 60, 3, 260, 1), (5, 13, 11, 68, 3, 260, 2)])
def test_ragged_channel_counts_with_epilogue(pkg, dev, shape, prec_name):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    ho, wo = -(-H // s), -(-W // s)
    x, k, dy, gate = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in
                      ((57, (N, H, W, C)), (58, (K, K, C, O)), (59, (N, ho, wo, O)), (60, (N, H, W, C))))
    bias_o, bias_c = (torch.full((n + 512,), float("nan"), device=dev) for n in (O, C))
    bias_o[:O], bias_c[:C] = torch.from_numpy(seeded((O,), 61)), torch.from_numpy(seeded((C,), 62))
    got = {}
    for prec in (getattr(pkg, PRECS[prec_name]), pkg.PREC_FP32):
        z, raw = torch.empty((N, ho, wo, O), device=dev), torch.empty((N, H, W, C), device=dev)
        y = F.conv2d_fwd(x, k, (s, s), epilogue=F.make_epilogue(bias=bias_o[:O], act=pkg.ACT_TANH, pre_act=z), precision=prec)
        dx = F.conv2d_dx(dy, k, (H, W), (s, s), precision=prec,
                         epilogue=F.make_epilogue(bias=bias_c[:C], raw_out=raw, gate=gate, gate_act=pkg.ACT_TANH))
        got[prec] = (y, z, dx, raw)
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    tol = TF32_TOL if prec_name == "tf32" else 3e-5
    for name, a, b in zip(("y", "z", "dx", "raw"), *got.values()):
        assert (a - b).abs().max().item() <= tol * b.abs().max().item(), name


def test_ragged_channel_counts_without_scratch(pkg, dev):
    """They ran on the CUDA cores before they took the tensor path, and still do where there is no scratch for that - as
    operators and as nodes of a context with little scratch of its caller; counts that always needed scratch ask for it."""
    F, L, N = pkg.functional, pkg.lib, pkg.nodes
    x, k, dy = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in ((1, (4, 32, 32, 36)), (2, (3, 3, 36, 40)), (3, (4, 32, 32, 40))))
    y, dk = torch.zeros_like(dy), torch.zeros_like(k)
    d = F.conv_desc(x.shape, k.shape, (1, 1))
    assert all(L.dcg_conv_workspace_bytes(ctypes.byref(d), kind, pkg.PREC_TF32) > 256 for kind in (pkg._lib.KIND_FWD, pkg._lib.KIND_DK))
    refs = F.conv2d_fwd(x, k, (1, 1), precision=pkg.PREC_FP32), F.conv2d_dk(x, dy, (3, 3), (1, 1), precision=pkg.PREC_FP32)
    stream, scratch = torch.cuda.current_stream().cuda_stream, torch.empty((256,), dtype=torch.uint8, device=dev)
    for ws, size in ((None, 0), (scratch.data_ptr(), 256)):
        y.zero_(), dk.zero_()
        pkg._lib.check(L.dcg_conv2d_fwd(ctypes.byref(d), x.data_ptr(), k.data_ptr(), y.data_ptr(), None, pkg.PREC_TF32, ws, size, stream))
        pkg._lib.check(L.dcg_conv2d_dk(ctypes.byref(d), x.data_ptr(), dy.data_ptr(), dk.data_ptr(), pkg.PREC_TF32, ws, size, stream))
        assert torch.equal(y, refs[0]) and torch.equal(dk, refs[1])
    y.zero_(), dk.zero_()
    ctx = ctypes.c_void_p()
    pkg._lib.check(L.dcg_context_create(ctypes.byref(ctx), pkg.PREC_TF32, scratch.data_ptr(), 256, stream))
    nodes = [N.op_conv2d(x, k, (1, 1), 2, 2, y, x.shape, k.shape), N.op_conv2d_kernel_grad(dy, x, (1, 1), dk, dy.shape, x.shape, (2, 2))]
    pkg._lib.check(L.dcg_run_nodes(ctx, (pkg._lib.Node * 2)(*nodes), 2, 1))
    torch.cuda.synchronize()
    L.dcg_context_destroy(ctx)
    assert torch.equal(y, refs[0]) and torch.equal(dk, refs[1])
    d2 = F.conv_desc((2, 16, 16, 128), (5, 5, 128, 256))
    x2, k2, y2 = torch.zeros((2, 16, 16, 128), device=dev), torch.zeros((5, 5, 128, 256), device=dev), torch.zeros((2, 8, 8, 256), device=dev)
    assert L.dcg_conv2d_fwd(ctypes.byref(d2), x2.data_ptr(), k2.data_ptr(), y2.data_ptr(), None, pkg.PREC_TF32, None, 0, stream) == pkg._lib.ERR_WORKSPACE


@pytest.mark.parametrize("threads", [1, 2])
def test_calls_on_two_streams_do_not_share_scratch(pkg, dev, threads):
    """K partitions, padded images and column sums of two streams in flight together, from one thread and from two."""
    F = pkg.functional

    def work(i):
        x, k, dy = (torch.from_numpy(seeded(t, 70 + i)).to(dev) for t in ((4 + i, 16, 16, 192), (3, 3, 192, 320), (4 + i, 8, 8, 320)))
        rgb, k3, dy3 = (torch.from_numpy(seeded(t, 80 + i)).to(dev) for t in ((9 + i, 32, 32, 3), (5, 5, 3, 64), (9 + i, 16, 16, 64)))
        rows = torch.from_numpy(seeded((5000 + i, 37), 90 + i)).to(dev)
        return lambda: [F.conv2d_fwd(x, k), F.conv2d_dk(x, dy, (3, 3)), F.conv2d_fwd(rgb, k3), F.conv2d_dk(rgb, dy3, (5, 5)), F.colsum(rows)]

    calls = [work(0), work(1)]
    alone = [call() for call in calls]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream(), torch.cuda.Stream()], [[], []]

    def run(indexes):
        for _ in range(20):
            for i in indexes:
                with torch.cuda.stream(streams[i]):
                    got[i].append(calls[i]())

    if threads == 1:
        run([0, 1])
    else:
        workers = [threading.Thread(target=run, args=([i],)) for i in (0, 1)]
        for w in workers:
            w.start()
        for w in workers:
            w.join()
    torch.cuda.synchronize()
    assert [len(g) for g in got] == [20, 20]
    for i in (0, 1):
        for again in got[i]:
            assert all(torch.equal(a, b) for a, b in zip(alone[i], again))


@pytest.mark.parametrize("batch", [20, 28, 40, 56, 100])
def test_k_partition_counts(pkg, dev, batch):
    """The number of K partitions of a tile (= thread-block cluster size) follows the tile count:
    these batches give clusters of 8, 8/7, 7/5, 5/4 and 2/3 CTAs on a 148-SM part for the
    128 -> 256 channel layer, odd sizes included.  Each must agree with the fp32 path and with itself."""
    F = pkg.functional
    g = torch.Generator(device="cpu").manual_seed(11)
    x = (torch.rand((batch, 16, 16, 128), generator=g) * 2 - 1).to(dev)
    k = (torch.randn((5, 5, 128, 256), generator=g) * 0.02).to(dev)
    dy = (torch.rand((batch, 8, 8, 256), generator=g) * 2 - 1).to(dev)
    bias = torch.randn((256,), generator=g).to(dev)
    ref = (F.conv2d_fwd(x, k, precision=pkg.PREC_FP32) + bias, F.conv2d_dx(dy, k, (16, 16), precision=pkg.PREC_FP32),
           F.conv2d_dk(x, dy, (5, 5), precision=pkg.PREC_FP32))
    run = lambda: (F.conv2d_fwd(x, k, epilogue=F.make_epilogue(bias=bias)), F.conv2d_dx(dy, k, (16, 16)),
                   F.conv2d_dk(x, dy, (5, 5)))
    a, b = run(), run()
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    for name, r, u, v in zip(("fwd+bias", "dx", "dk"), ref, a, b):
        assert (r - u).abs().max().item() <= TF32_TOL * r.abs().max().item(), name
        assert torch.equal(u, v), name


def _form(pkg, shape, op, precision):
    """What a call takes: dcg_conv_form, whether a second launch adds the K partitions, how many those are."""
    import ctypes
    N, H, W, C, K, O, s = shape
    kh, kw = K if isinstance(K, tuple) else (K, K)
    d, form, plan = pkg.functional.conv_desc((N, H, W, C), (kh, kw, C, O), (s, s)), (ctypes.c_int * 4)(), (ctypes.c_int * 6)()
    kind = {"fwd": pkg._lib.KIND_FWD, "dx": pkg._lib.KIND_DX, "dk": pkg._lib.KIND_DK}[op]
    if pkg.lib.dcg_debug_conv_form(ctypes.byref(d), kind, precision, form) or pkg.lib.dcg_debug_conv_plan(ctypes.byref(d), kind, precision, plan):
        return None
    return form[0], form[1], plan[2]


# kernel gradients of few tiles, whose partitions a second launch adds: one tap and nine, four taps to a tile, the channel
# roles swapped, ragged channels, a last partition tile that is nearly empty
@pytest.mark.parametrize("prec_name", ["tf32", "3xtf32"])
@pytest.mark.parametrize("shape", [(4, 60, 60, 64, 1, 128, 1), (8, 40, 40, 32, 3, 64, 1), (6, 64, 64, 256, 1, 64, 1), (16, 50, 50, 40, 3, 44, 1),
                                   (20, 64, 64, 8, 1, 16, 1), (13, 75, 51, 96, 3, 160, 1), (5, 61, 47, 132, 1, 260, 2), (9, 61, 47, 100, 1, 132, 2)])
def test_kernel_gradients_of_many_partitions(pkg, dev, shape, prec_name):
    import ctypes
    F, L = pkg.functional, pkg.lib
    N, H, W, C, K, O, s = shape
    prec = getattr(pkg, PRECS[prec_name])
    # (two of them stay with a cluster at one of the precisions)
    if (C, prec_name) not in ((132, "tf32"), (96, "3xtf32")):
        assert _form(pkg, shape, "dk", prec)[:2] == (0, 1) and _form(pkg, shape, "dk", prec)[2] > 8
    x, dy = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in ((57, (N, H, W, C)), (58, (N, -(-H // s), -(-W // s), O))))
    pt, pl = (max((-(-e // s) - 1) * s + K - e, 0) for e in (H, W))
    xp = torch.nn.functional.pad(x.double().permute(0, 3, 1, 2), (pl // 2, pl - pl // 2, pt // 2, pt - pt // 2))
    ref = torch.nn.grad.conv2d_weight(xp, (O, C, K, K), dy.double().permute(0, 3, 1, 2), stride=s).permute(2, 3, 1, 0)
    # operands of 11 bits: 2^-10 of each product at most, which average out; else the rounding of a fp32 sum
    tol = TF32_TOL if prec_name == "tf32" else 1e-5
    got = [F.conv2d_dk(x, dy, (K, K), (s, s), precision=prec) for _ in range(2)]
    assert torch.equal(*got)
    # with less scratch than asked for: fewer partitions
    d = F.conv_desc(x.shape, (K, K, C, O), (s, s), None, None)
    need = L.dcg_conv_workspace_bytes(ctypes.byref(d), pkg._lib.KIND_DK, prec)
    small, less = torch.empty(need - 256, dtype=torch.uint8, device=dev), torch.zeros_like(got[0])
    assert L.dcg_conv2d_dk(ctypes.byref(d), x.data_ptr(), dy.data_ptr(), less.data_ptr(), prec, small.data_ptr(), small.numel(),
                           torch.cuda.current_stream().cuda_stream) == 0, L.dcg_last_error()
    torch.cuda.synchronize()
    assert L.dcg_device_status() == 0
    for dk in (got[0], less):
        assert (dk - ref).abs().max().item() <= tol * ref.abs().max().item()


# <= 4 input channels straight from the image: patches by TMA and by 4-byte copies (rows that are no 16 bytes), 16 and 32 places
# per kernel row, even and odd pixel distances, tiles of several images, one and many tiles per CTA, one to four column slabs
@pytest.mark.parametrize("shape", [(1, 64, 64, 3, 5, 64, 2), (130, 64, 64, 3, 5, 64, 2), (3, 63, 61, 3, 5, 32, 2), (4, 20, 20, 1, 5, 32, 2),
                                   (6, 40, 30, 3, 3, 96, 1), (2, 50, 64, 2, 4, 128, 2), (3, 17, 19, 3, 7, 64, 1), (40, 9, 7, 3, 3, 32, 1),
                                   (2, 40, 200, 3, 5, 64, 1), (1, 5, 5, 3, 5, 64, 2), (9, 30, 28, 4, 8, 32, 2), (2, 64, 64, 3, 1, 64, 1),
                                   (3, 40, 38, 3, (3, 7), 64, 2), (5, 33, 40, 3, (4, 7), 32, 1), (2, 50, 64, 4, (2, 5), 128, 2), (9, 24, 20, 3, (3, 8), 96, 1),
                                   (3, 21, 23, 3, (3, 6), 64, 1), (70, 40, 40, 3, (4, 7), 32, 2), (20, 64, 64, 4, 5, 64, 2)])
def test_forward_of_rgb_layers(pkg, dev, shape):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    kh, kw = K if isinstance(K, tuple) else (K, K)
    # two whole operand tiles of every kernel row have to fit: 7 x 7 x 3, 8 x 8 x 4 and 5 x 5 x 4 keep the window form
    kernel = {(7, 3): 0, (8, 4): 0, (5, 4): 5}.get((K, C), 2)
    assert _form(pkg, shape, "fwd", pkg.PREC_TF32)[0] == kernel
    ho, wo = -(-H // s), -(-W // s)
    x, k, bias, gate = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in
                        ((61, (N, H, W, C)), (62, (kh, kw, C, O)), (63, (O,)), (64, (N, ho, wo, O))))
    ref = F.conv2d_fwd(x, k, (s, s), precision=pkg.PREC_FP32)
    tol = TF32_TOL * ref.abs().max().item()
    assert (F.conv2d_fwd(x, k, (s, s)) - ref).abs().max().item() <= tol
    # the whole chain: every tensor it writes, a gate beside the bias, and nothing beyond the ragged border
    for gated in (None, gate):
        raw, pre, out = (torch.full((N + 1, ho, wo, O), 7.0, device=dev) for _ in range(3))
        ep = F.make_epilogue(bias=bias, act=pkg.ACT_LEAKY, alpha=0.2, pre_act=pre[:N], raw_out=raw[:N], gate=gated, gate_act=pkg.ACT_RELU if gated is not None else pkg.ACT_NONE)
        F.conv2d_fwd(x, k, (s, s), epilogue=ep, out=out[:N])
        torch.cuda.synchronize()
        assert pkg.lib.dcg_device_status() == 0
        assert (raw[:N] - ref).abs().max().item() <= tol
        assert torch.equal(pre[:N], raw[:N] + bias)
        y = torch.where(pre[:N] < 0, pre[:N] * 0.2, pre[:N])
        assert torch.equal(out[:N], y if gated is None else torch.where(gate > 0, y, torch.zeros_like(y)))
        assert all(bool((t[N] == 7.0).all()) for t in (raw, pre, out))


def test_repeated_calls_encode_no_tensor_maps(pkg, dev):
    """Of a call on the same tensors none; of an RGB forward with another output that one's, and the results follow the tensors."""
    F, encoded = pkg.functional, pkg.lib.dcg_debug_maps_encoded
    for shape in ((8, 64, 64, 3, 5, 64, 2), (80, 32, 32, 32, 5, 64, 2)):   # (neither takes scratch, which has a new address each time)
        N, H, W, C, K, O, s = shape
        x, k, gate = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in ((68, (N, H, W, C)), (69, (K, K, C, O)), (70, (N, H // s, W // s, O))))
        raw, pre, out, other = (torch.empty_like(gate) for _ in range(4))
        ep = F.make_epilogue(act=pkg.ACT_LEAKY, raw_out=raw, pre_act=pre, gate=gate, gate_act=pkg.ACT_RELU)
        F.conv2d_fwd(x, k, (s, s), epilogue=ep, out=out)
        first = [t.clone() for t in (raw, pre, out)]
        before = encoded()
        for t in (raw, pre, out):
            t.zero_()
        F.conv2d_fwd(x, k, (s, s), epilogue=ep, out=out)
        assert encoded() == before
        assert all(torch.equal(a, b) for a, b in zip(first, (raw, pre, out)))
        out.zero_()
        F.conv2d_fwd(x, k, (s, s), epilogue=ep, out=other)
        F.conv2d_fwd(x, k, (s, s), out=raw)
        assert encoded() - before == (2 if C == 3 else 0)
        assert torch.equal(other, first[2]) and not out.any() and torch.equal(raw, first[0])
    assert pkg.lib.dcg_device_status() == 0


def test_rgb_forward_into_one_tensor(pkg, dev):
    """Results of the chain that go to the same tensor: the last one stays, as it does in every other kernel."""
    F = pkg.functional
    x, k, bias = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in ((65, (40, 64, 64, 3)), (66, (5, 5, 3, 64)), (67, (64,))))

    def call(**chain):
        return F.conv2d_fwd(x, k, (2, 2), epilogue=F.make_epilogue(bias=bias, act=pkg.ACT_TANH, **chain), out=out)

    out = torch.empty((40, 32, 32, 64), device=dev)
    raw, pre = torch.empty_like(out), torch.empty_like(out)
    y = call(raw_out=raw, pre_act=pre).clone()
    assert pkg.lib.dcg_device_status() == 0 and torch.equal(pre, raw + bias)
    for _ in range(5):
        for first, second in ((out, out), (pre, out), (out, pre), (pre, pre)):   # raw and pre-activation
            pre.zero_()
            call(raw_out=first, pre_act=second)
            assert torch.equal(out, y)
            if second is pre:
                assert torch.equal(pre, raw + bias)
            elif first is pre:
                assert torch.equal(pre, raw)


# more tiles than SMs, walked by persistent CTAs: one to three tiles each and a last round that is nearly empty, widths of 16 to 192
# columns, the last column tile partly beyond the channels, parity classes, channels that are no multiple of four, one stage a tile
@pytest.mark.parametrize("shape", [(24, 48, 48, 32, 1, 192, 1), (13, 75, 51, 96, 3, 160, 1), (32, 40, 40, 64, 3, 96, 1), (37, 60, 60, 20, 5, 64, 2),
                                   (40, 33, 35, 6, 3, 32, 1), (150, 12, 11, 32, 3, 288, 1), (20, 64, 64, 8, 1, 32, 1), (16, 50, 50, 40, 3, 44, 1)])
def test_more_tiles_than_sms(pkg, dev, shape):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    ho, wo = -(-H // s), -(-W // s)
    x, k, dy, bias, gate = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in
                            ((65, (N, H, W, C)), (66, (K, K, C, O)), (67, (N, ho, wo, O)), (68, (O,)), (69, (N, H, W, C))))
    pkg.lib.dcg_debug_set_dx_mode(0)
    forms = [_form(pkg, shape, op, pkg.PREC_TF32) for op in ("fwd", "dx")]
    pkg.lib.dcg_debug_set_dx_mode(-1)
    assert forms == [(1, 0, 1) if C % 4 == 0 else None, (1, 0, 1)]   # (forwards of 6 channels are on the CUDA cores)
    pre = [torch.empty((N, ho, wo, O), device=dev) for _ in range(2)]
    results = []
    pkg.lib.dcg_debug_set_dx_mode(0)
    try:
        for i, prec in enumerate((pkg.PREC_TF32, pkg.PREC_FP32)):
            results.append([F.conv2d_fwd(x, k, (s, s), epilogue=F.make_epilogue(bias=bias, act=pkg.ACT_LEAKY, pre_act=pre[i]), precision=prec), pre[i],
                            F.conv2d_dx(dy, k, (H, W), (s, s), epilogue=F.make_epilogue(gate=gate, gate_act=pkg.ACT_RELU), precision=prec)])
    finally:
        pkg.lib.dcg_debug_set_dx_mode(-1)
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    for name, a, b in zip(("fwd", "pre-activation", "dx"), *results):
        assert (a - b).abs().max().item() <= TF32_TOL * b.abs().max().item(), name


# parity classes together where their tiles fit the layer, as tiles of their own where they would be half empty
@pytest.mark.parametrize("shape,fused", [((64, 32, 32, 64, 5, 128, 2), True), ((30, 33, 47, 192, 3, 64, 2), False), ((9, 96, 96, 192, 3, 64, 2), False)])
def test_parity_classes_together_or_apart(pkg, dev, shape, fused):
    F = pkg.functional
    N, H, W, C, K, O, s = shape
    k, dy = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in ((71, (K, K, C, O)), (72, (N, -(-H // s), -(-W // s), O))))
    before = pkg.lib.dcg_debug_fused_dx_launches()
    got, ref = (F.conv2d_dx(dy, k, (H, W), (s, s), precision=p) for p in (pkg.PREC_TF32, pkg.PREC_FP32))
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    assert pkg.lib.dcg_debug_fused_dx_launches() - before == int(fused)
    assert (got - ref).abs().max().item() <= TF32_TOL * ref.abs().max().item()


def test_deterministic(pkg, dev):
    """Two runs of every operator give identical bits (fixed-order split-K reduction)."""
    F = pkg.functional
    g = torch.Generator(device="cpu").manual_seed(9)
    x = (torch.rand((8, 16, 16, 128), generator=g) * 2 - 1).to(dev)
    k = (torch.randn((5, 5, 128, 256), generator=g) * 0.02).to(dev)
    dy = (torch.rand((8, 8, 8, 256), generator=g) * 2 - 1).to(dev)
    a = (F.conv2d_fwd(x, k), F.conv2d_dx(dy, k, (16, 16)), F.conv2d_dk(x, dy, (5, 5)))
    b = (F.conv2d_fwd(x, k), F.conv2d_dx(dy, k, (16, 16)), F.conv2d_dk(x, dy, (5, 5)))
    torch.cuda.synchronize()
    for u, v in zip(a, b):
        assert torch.equal(u, v)


def test_workspace_and_alignment_contract(pkg, dev, orc):
    """What the entry points promise about their operands: a tensor-path call that needs scratch
    refuses a buffer that is too small (nothing is launched, the output stays untouched) and says how
    much it wants; operands that are not 16-byte aligned (which TMA cannot address) silently take the
    CUDA-core path, whose result is the oracle's bit for bit."""
    import ctypes
    F, L = pkg.functional, pkg.lib
    # 128 -> 256 channels at batch 8: few tiles, so the K partitions need scratch
    g = torch.Generator(device="cpu").manual_seed(41)
    x = (torch.rand((8, 16, 16, 128), generator=g) * 2 - 1).to(dev)
    k = (torch.randn((5, 5, 128, 256), generator=g) * 0.02).to(dev)
    d = F.conv_desc(x.shape, k.shape, (2, 2), None, None)
    need = L.dcg_conv_workspace_bytes(ctypes.byref(d), pkg._lib.KIND_FWD, pkg.PREC_TF32)
    assert need > 0
    y = torch.full((8, 8, 8, 256), 7.0, device=dev)
    small = torch.empty(need // 2, dtype=torch.uint8, device=dev)
    st = L.dcg_conv2d_fwd(ctypes.byref(d), x.data_ptr(), k.data_ptr(), y.data_ptr(), None, pkg.PREC_TF32,
                          small.data_ptr(), small.numel(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert st == pkg._lib.ERR_WORKSPACE and b"workspace" in L.dcg_last_error()
    assert bool((y == 7.0).all())
    assert L.dcg_conv_workspace_bytes(ctypes.byref(d), pkg._lib.KIND_FWD, pkg.PREC_FP32) == 0

    # the same small layer from a buffer that starts 4 bytes off a 16-byte boundary
    xs = seeded((2, 8, 8, 32), 42)
    ks = seeded((5, 5, 32, 64), 43) * np.float32(0.1)
    raw = torch.empty(xs.size + 1, device=dev)
    xo = raw[1:].view(2, 8, 8, 32)
    xo.copy_(torch.from_numpy(xs))
    assert xo.data_ptr() % 16 == 4
    y_off = F.conv2d_fwd(xo, torch.from_numpy(ks).to(dev), precision=pkg.PREC_TF32)
    torch.cuda.synchronize()
    assert np.array_equal(y_off.cpu().numpy(), orc.conv2d(xs, ks, (2, 2)))



# (batch, H, Cin, Cout): the four DCGAN layers at the batch the benchmark runs (64) and at the 128
# images of the discriminator's single pass over [fake | real]
BENCH_LAYERS = [(b, h, c, o) for b in (64, 128) for (h, c, o) in ((64, 3, 64), (32, 64, 128), (16, 128, 256), (8, 256, 512))]


@pytest.mark.parametrize("layer", BENCH_LAYERS)
def test_benchmark_shapes_vs_reference_cpu_code(pkg, dev, ref, layer):
    """The shapes bench.py times - with their K partitions, cluster shapes and two-wave grids -
    against the reference's own CPU code (oracle/_ref = src/cpu/ops.hxx compiled from its sources) on
    xorshift inputs (seed 234 as tests/test_conv_s1.cu:31).  The scalar CPU code needs minutes for a
    whole batch-64 layer, so it is run on what is independent: forward and input gradient on the
    first and last image (images do not interact), the kernel gradient over the WHOLE batch on
    two 4-channel slices of x and dy (dk[:, :, c, o] only reads x[..., c] and dy[..., o]; the slice
    keeps the reference's (n, i, j) summation order, src/cpu/ops.hxx:754-772).
    Bounds: fp32 path bit-equal, TF32 path 1e-2 * max|ref|."""
    F = pkg.functional
    B, H, C, O = layer
    Ho = H // 2
    x = seeded((B, H, H, C), 234)
    k = (seeded((5, 5, C, O), 235) * np.float32(0.05)).astype(np.float32)
    dy = seeded((B, Ho, Ho, O), 236)
    xd, kd, dyd = (torch.from_numpy(a).to(dev) for a in (x, k, dy))
    ends = [0, B - 1]
    y_ref = ref.conv2d(x[ends], k, (2, 2))
    dx_ref = ref.conv2d_input_grad(dy[ends], k, 2, (H, H))
    slices = [(0, 0), (max(C - 4, 0), O - 4)]
    pad = (oracle.same_pad(H, 5, 2), oracle.same_pad(H, 5, 2))
    dk_refs = [ref.conv2d_kernel_grad(np.ascontiguousarray(dy[..., o0:o0 + 4]), np.ascontiguousarray(x[..., c0:c0 + 4]), 2, pad)
               for c0, o0 in slices]
    for prec in (pkg.PREC_FP32, pkg.PREC_TF32):
        y = F.conv2d_fwd(xd, kd, precision=prec)
        dx = F.conv2d_dx(dyd, kd, (H, H), precision=prec)
        dk = F.conv2d_dk(xd, dyd, (5, 5), precision=prec)
        torch.cuda.synchronize()
        assert pkg.lib.dcg_device_status() == 0
        _check(y[ends], y_ref, prec, pkg, "fwd images 0 and %d" % (B - 1))
        _check(dx[ends], dx_ref, prec, pkg, "dx images 0 and %d" % (B - 1))
        for (c0, o0), dk_ref in zip(slices, dk_refs):
            got = dk[:, :, c0:c0 + 4, o0:o0 + 4].contiguous()
            if prec == pkg.PREC_FP32:
                _check(got, dk_ref, prec, pkg, "dk slice c%d o%d" % (c0, o0))
            else:   # the bound is on the operator's output tensor: scale by the whole dk
                lim = TF32_TOL * float(dk.abs().max())
                assert float(np.abs(got.cpu().numpy() - dk_ref).max()) <= lim, "dk slice c%d o%d" % (c0, o0)


def test_bounded_wait_runs_out_and_the_context_survives(pkg, dev):
    """Failure detection without a fault: the producer is told to leave one pipeline stage out, so
    the MMA warp's wait on that stage can never complete; with the wait limit lowered to about a
    millisecond the kernel gives up, records (block, role, stage) in the device status word, still
    reaches its final barrier and frees TMEM.  dcg_device_status() then reports DCG_ERR_DEVICE, and a
    normal call right after passes - the context stays usable."""
    F, L = pkg.functional, pkg.lib
    x = seeded((80, 32, 32, 32), 501)         # 160 tiles of 128 pixels: more tiles than SMs, so no K partitions, no cluster
    k = seeded((5, 5, 32, 64), 502) * np.float32(0.1)
    xd, kd = torch.from_numpy(x).to(dev), torch.from_numpy(k).to(dev)
    assert L.dcg_device_status() == 0
    try:
        L.dcg_debug_set_wait_limit(2_000_000)   # ~1 ms of SM clocks
        L.dcg_debug_skip_stage(3)
        F.conv2d_fwd(xd, kd, precision=pkg.PREC_TF32)
        torch.cuda.synchronize()                # returns: every wait in the kernel is bounded
    finally:
        L.dcg_debug_skip_stage(-1)
        L.dcg_debug_set_wait_limit(0)
    assert L.dcg_device_status() == pkg._lib.ERR_DEVICE
    assert b"gave up waiting" in L.dcg_last_error()
    assert L.dcg_device_status() == 0           # reading clears the word
    y = F.conv2d_fwd(xd, kd, precision=pkg.PREC_TF32)
    torch.cuda.synchronize()
    assert L.dcg_device_status() == 0
    y32 = F.conv2d_fwd(xd, kd, precision=pkg.PREC_FP32)   # bit-equal to the oracle (test_conv_fwd_dx_dk)
    torch.cuda.synchronize()
    assert (y - y32).abs().max().item() <= TF32_TOL * y32.abs().max().item()


# one stage of the pipeline never comes: kernel (dcg_conv_form), operator, precision, shape (n, h, w, c, k, o, s), the stage
GIVE_UP = [(2, "fwd", "tf32", (64, 64, 64, 3, 5, 64, 2), 1), (1, "fwd", "tf32", (80, 32, 32, 32, 5, 64, 2), 3),
           (1, "dx", "tf32", (37, 60, 60, 20, 1, 64, 1), 1), (0, "fwd", "tf32", (8, 48, 48, 64, 3, 128, 1), 3),
           (0, "dx", "tf32", (8, 48, 48, 64, 3, 128, 1), 3), (0, "fwd", "3xtf32", (8, 48, 48, 64, 3, 128, 1), 3),
           (0, "fwd", "3xtf32", (80, 32, 32, 32, 5, 64, 2), 9)]


@pytest.mark.parametrize("form,op,prec_name,shape,stage", GIVE_UP)
def test_a_wait_that_runs_out_in_each_kernel(pkg, dev, form, op, prec_name, shape, stage):
    """As above, without K partitions: every wait ends, the status tells, a call right after is clean - with a gate, whose values
    an RGB forward fetches while it waits."""
    import ctypes
    F, L = pkg.functional, pkg.lib
    n, h, w, c, k, o, s = shape
    prec, kind = getattr(pkg, PRECS[prec_name]), {"fwd": pkg._lib.KIND_FWD, "dx": pkg._lib.KIND_DX}[op]
    d, plan, got = F.conv_desc((n, h, w, c), (k, k, c, o), (s, s)), (ctypes.c_int * 6)(), (ctypes.c_int * 4)()
    assert L.dcg_debug_conv_form(ctypes.byref(d), kind, prec, got) == 0 and got[0] == form
    assert L.dcg_debug_conv_plan(ctypes.byref(d), kind, prec, plan) == 0 and plan[2] == 1
    x, kk, dy = (torch.from_numpy(seeded(t, i)).to(dev) for i, t in ((81, (n, h, w, c)), (82, (k, k, c, o)), (83, (n, -(-h // s), -(-w // s), o))))
    gate = dy if op == "fwd" else x
    ep = F.make_epilogue(gate=gate, gate_act=pkg.ACT_RELU)

    def call(p):
        return F.conv2d_fwd(x, kk, (s, s), epilogue=ep, precision=p) if op == "fwd" else F.conv2d_dx(dy, kk, (h, w), (s, s), epilogue=ep, precision=p)

    assert L.dcg_device_status() == 0
    try:
        L.dcg_debug_set_wait_limit(2_000_000)   # ~1 ms of SM clocks
        L.dcg_debug_skip_stage(stage)
        call(prec)
        torch.cuda.synchronize()
    finally:
        L.dcg_debug_skip_stage(-1)
        L.dcg_debug_set_wait_limit(0)
    assert L.dcg_device_status() == pkg._lib.ERR_DEVICE
    got, ref = call(prec), call(pkg.PREC_FP32)
    torch.cuda.synchronize()
    assert L.dcg_device_status() == 0
    assert (got - ref).abs().max().item() <= TF32_TOL * ref.abs().max().item()
