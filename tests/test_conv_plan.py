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


def _ambiguous_waits(stages, groups, slots, looks, steps=120):
    """Waits of the groups of warps that take 3xTF32 stages apart that a parity does not decide: the barrier may still be in the
    phase before the one waited for (the wait passes at once, on the one before that), or may be beyond it (it never passes).  What
    a group knows is what it has waited for: loads that have landed (its own stages, and all whose MMAs are done), MMAs that are
    done (they end in order).  What it holds up is the MMAs from its next stage on."""
    found = []
    for g in range(groups):
        landed, done, turn = set(), -1, g   # turn: its next stage
        for it in range(steps):
            def full(i):       # the load of stage i, between those of i - stages and i + stages
                nonlocal done
                if (i >= stages and i - stages not in landed and i - stages > done) or turn > i:
                    found.append((g, i))
                landed.add(i)
                done = max(done, i - stages)   # whoever loaded it waited for the stage's release

            def released(i):   # the MMAs of stage i
                nonlocal done
                if i < 0:
                    return
                if i - stages > done or turn > i + stages:
                    found.append((g, i))
                done = max(done, i)

            if it % groups == g:
                if looks:
                    released(it - stages)
                full(it)
                released(it - (4 if stages >= 4 else 2))
                released(it - slots)
                turn = it + groups
            if it % 4 == 1 and it > 4:   # the sums of a block of four stages are taken over
                done = max(done, it - 2)
    return found


def test_3xtf32_waits_are_unambiguous(pkg):
    """Every plan's ring, groups of warps and kept residuals.  Rings of one stage more than groups have such waits unless a group
    looks at the release of its stage first, as the three groups of the wide tiles do."""
    assert _ambiguous_waits(5, 4, 2, False) and _ambiguous_waits(4, 3, 2, False)
    form, seen = (ctypes.c_int * 4)(), set()
    shapes = [(n, 40, 36, c, k, o, s) for n in (1, 8, 64) for c in (3, 8, 16, 32, 64, 80, 100, 128, 256) for k in range(1, 9)
              for o in (8, 32, 48, 64, 96, 100, 112, 128, 160, 192, 256) for s in (1, 2)]
    for call, (width, _, _, stages, _, _) in _plans(pkg, shapes, pkg.PREC_3XTF32):
        n, h, w, c, k, o, s, kind = call
        desc = pkg.functional.conv_desc((n, h, w, c), (k, k, c, o), (s, s))
        assert pkg.lib.dcg_debug_conv_form(ctypes.byref(desc), kind, pkg.PREC_3XTF32, form) == 0
        if form[0] == 0:
            seen.add((stages, form[2], form[3]))
    assert {groups for _, groups, _ in seen} == {3, 4}
    for plan in seen:
        assert not _ambiguous_waits(*plan, plan[1] == 3), plan


def test_class_fused_input_gradients_are_planned_once(pkg):
    """Where the parity classes stay together the general kernel is planned for the comparison only, once a shape and not with
    every call on other tensors; where they do not, once a call is what it takes."""
    form = (ctypes.c_int * 4)()
    for shape, kernel, each in (((64, 32, 32, 64, 5, 128, 2), 3, 0), ((30, 33, 47, 192, 3, 64, 2), 1, 1)):
        n, h, w, c, k, o, s = shape
        desc = pkg.functional.conv_desc((n, h, w, c), (k, k, c, o), (s, s))
        counts = []
        for _ in range(3):
            before = pkg.lib.dcg_debug_dx_plans()
            assert pkg.lib.dcg_debug_conv_form(ctypes.byref(desc), pkg._lib.KIND_DX, pkg.PREC_TF32, form) == 0 and form[0] == kernel
            counts.append(pkg.lib.dcg_debug_dx_plans() - before)
        assert counts[1:] == [each] * 2


def test_persistent_kernels_report_both_accumulators(pkg):
    """An RGB forward and a walked one: two accumulators, in the power of two of columns that is allocated."""
    form = (ctypes.c_int * 4)()
    for shape, kernel, columns in (((64, 64, 64, 3, 5, 64, 2), 2, 128), ((8, 64, 64, 3, 3, 96, 1), 2, 256), ((130, 64, 64, 3, 5, 128, 2), 2, 256),
                                   ((16, 96, 96, 64, 1, 192, 1), 1, 256), ((37, 60, 60, 20, 5, 64, 2), 1, 128)):
        plans = [p for call, p in _plans(pkg, [shape], pkg.PREC_TF32) if call[-1] == pkg._lib.KIND_FWD]
        n, h, w, c, k, o, s = shape
        desc = pkg.functional.conv_desc((n, h, w, c), (k, k, c, o), (s, s))
        assert pkg.lib.dcg_debug_conv_form(ctypes.byref(desc), pkg._lib.KIND_FWD, pkg.PREC_TF32, form) == 0 and form[0] == kernel, shape
        assert plans[0][0] == (96 if o == 192 else o) and plans[0][4] == columns, shape
