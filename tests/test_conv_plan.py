"""Planning of the tensor-path convolutions on the host: what a launch asks of an SM has to exist."""
import ctypes

import pytest


def _plans(pkg, shapes, precision):
    plan = (ctypes.c_int * 6)()
    for n, h, w, c, k, o, s in shapes:
        desc = pkg.functional.conv_desc((n, h, w, c), (k, k, c, o), (s, s))
        for kind in (pkg._lib.KIND_FWD, pkg._lib.KIND_DX, pkg._lib.KIND_DK):
            if pkg.lib.dcg_debug_conv_plan(ctypes.byref(desc), kind, precision, plan) == 0:
                yield (n, h, w, c, k, o, s, kind), list(plan)


@pytest.mark.parametrize("precision", ["PREC_TF32", "PREC_3XTF32"])
def test_accumulators_fit(pkg, precision):
    """512 columns of TMEM, 227 KB of shared memory; 3xTF32 sums 192 columns in registers."""
    shapes = [(n, 40, 36, c, k, o, s) for n in (1, 8, 256) for c in (1, 3, 4, 32, 36, 64, 96, 100, 160, 256, 260) for k in range(1, 9)
              for o in (8, 32, 36, 64, 96, 160, 224, 256, 260, 512) for s in (1, 2)]
    x3 = precision == "PREC_3XTF32"
    planned = 0
    for call, (width, tiles, splits, stages, tmem, smem) in _plans(pkg, shapes, getattr(pkg, precision)):
        assert 0 < width <= (192 if x3 else 256) and tmem <= 512 and smem <= 227 * 1024 and stages >= 2, call
        planned += 1
    assert planned > len(shapes)


def test_tall_kernels_of_rgb_layers_in_3xtf32(pkg):
    """Kernel gradients of seven and eight kernel rows, 32 columns each, in two tiles on the tensor path."""
    for k in range(1, 9):
        plans = [p for call, p in _plans(pkg, [(4, 40, 36, 3, k, 64, 2)], pkg.PREC_3XTF32) if call[-1] == pkg._lib.KIND_DK]
        assert len(plans) == 1 and plans[0][:2] == ([32 * k, 1] if k <= 6 else [128, 2])
