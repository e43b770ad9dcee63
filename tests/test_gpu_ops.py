"""GPU parity of the memory-bound operators and the dense layers against the CPU oracle."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import seeded

pytestmark = pytest.mark.gpu


def _t(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _s():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("rows,cols", [(8, 2), (64 * 16 * 16, 128), (1000, 3), (77, 36), (64, 8192), (5, 1)])
def test_bias_act_and_colsum(pkg, dev, orc, rows, cols):
    L = pkg.lib
    a = seeded((rows, cols), 500)
    b = seeded((cols,), 501)
    ad, bd = _t(a, dev), _t(b, dev)
    z, act = torch.empty_like(ad), torch.empty_like(ad)
    pkg._lib.check(L.dcg_bias_act(ad.data_ptr(), bd.data_ptr(), z.data_ptr(), act.data_ptr(), rows, cols,
                                  pkg.ACT_LEAKY, 0.2, _s()))
    torch.cuda.synchronize()
    z_ref = orc.mvrow_add(a, b)
    assert np.array_equal(z.cpu().numpy(), z_ref)
    assert np.array_equal(act.cpu().numpy(), orc.vect_relu_leaky(z_ref, 0.2))
    got = pkg.functional.colsum(ad).cpu().numpy()
    ref = orc.mat_sum_cols(a)
    # different (tree) summation order than the sequential reference loop
    np.testing.assert_allclose(got, ref, rtol=0, atol=1e-6 * rows ** 0.5 + 1e-5 * np.abs(ref).max())
    rs = torch.empty((rows,), device=dev)
    pkg._lib.check(L.dcg_rowsum(ad.data_ptr(), rs.data_ptr(), rows, cols, _s()))
    np.testing.assert_allclose(rs.cpu().numpy(), orc.mat_sum_rows(a), rtol=0, atol=1e-5 * max(1, cols) ** 0.5)


@pytest.mark.parametrize("n", [1, 12, 4099, 1 << 20])
def test_activations_and_grads(pkg, dev, orc, n):
    L = pkg.lib
    a = seeded((n,), 510, -4, 4)
    d = seeded((n,), 511)
    ad, dd = _t(a, dev), _t(d, dev)
    out = torch.empty_like(ad)
    for act, fn, exact in ((pkg.ACT_LEAKY, lambda v: orc.vect_relu_leaky(v, 0.3), True),
                           (pkg.ACT_RELU, orc.vect_relu, True), (pkg.ACT_TANH, orc.vect_tanh, False),
                           (pkg.ACT_SIGMOID, orc.vect_sigmoid, False)):
        pkg._lib.check(L.dcg_act_fwd(ad.data_ptr(), out.data_ptr(), n, act, 0.3, _s()))
        got = out.cpu().numpy()
        if exact:
            assert np.array_equal(got, fn(a))
        else:
            np.testing.assert_allclose(got, fn(a), rtol=0, atol=2e-6)
    t = orc.vect_tanh(a)
    sg = orc.vect_sigmoid(a)
    for act, gate, fn in ((pkg.ACT_LEAKY, a, lambda g, x: orc.leaky_relu_grad(g, x, 0.3)),
                          (pkg.ACT_RELU, a, orc.relu_grad), (pkg.ACT_TANH, t, orc.tanh_grad),
                          (pkg.ACT_SIGMOID, sg, orc.sigmoid_grad)):
        gd = _t(gate, dev)
        pkg._lib.check(L.dcg_act_grad(gd.data_ptr(), dd.data_ptr(), out.data_ptr(), n, act, 0.3, _s()))
        assert np.array_equal(out.cpu().numpy(), fn(gate, d)), act
    pkg._lib.check(L.dcg_add(ad.data_ptr(), dd.data_ptr(), out.data_ptr(), n, _s()))
    assert np.array_equal(out.cpu().numpy(), orc.vect_add(a, d))
    coeff = torch.tensor([-0.37], device=dev)
    var = ad.clone()
    pkg._lib.check(L.dcg_update(dd.data_ptr(), var.data_ptr(), coeff.data_ptr(), n, _s()))
    assert np.array_equal(var.cpu().numpy(), orc.vect_update(d, a, -0.37))


@pytest.mark.parametrize("rows,cols", [(1, 7), (3, 4), (100, 10), (100, 100), (128, 512), (256, 36), (257, 128), (513, 10), (120, 40), (31, 8200)])
def test_colsum_of_a_few_hundred_rows(pkg, dev, rows, cols):
    """One block per column tile up to 32 rows per thread row, partial sums beyond: both sides of that line."""
    a = seeded((rows, cols), 515)
    got = pkg.functional.colsum(_t(a, dev)).cpu().numpy()
    np.testing.assert_allclose(got, a.astype(np.float64).sum(axis=0), rtol=0, atol=2e-6 * rows ** 0.5)


def _column_sums_in_order(a, sms):
    """The column sums with every fp32 addition where dcg_colsum has it: slabs of rows, in each a halving tree over lanes that
    take every lanes-th row, then the slabs (sixteen at a time, where the column tiles are few) over lanes again."""
    rows, cols = a.shape
    groups = cols // 4 if cols % 4 == 0 else cols
    tx = 1
    while tx < 32 and tx < groups:
        tx *= 2
    lanes, tiles = 256 // tx, -(-groups // tx)
    want = max(1, min(-(-4 * sms // tiles), 1008, -(-rows // (4 * lanes))))
    per_slab = -(-rows // want)

    def lane_sums(r, n):
        acc = np.zeros((n, cols), np.float32)
        for i in range(0, len(r), n):
            acc[:len(r[i:i + n])] += r[i:i + n]
        return acc

    def add_slabs(r, n):
        acc = lane_sums(r, n)
        total = acc[0].copy()
        for lane in acc[1:]:
            total += lane
        return total

    slabs = []
    for r0 in range(0, rows, per_slab):
        acc, h = lane_sums(a[r0:min(r0 + per_slab, rows)], lanes), lanes // 2
        while h:
            acc[:h] += acc[h:2 * h]
            h //= 2
        slabs.append(acc[0].copy())
    if len(slabs) == 1:
        return slabs[0]
    if tiles > 16:
        return add_slabs(np.stack(slabs), 8)
    while len(slabs) > 1:
        slabs = [add_slabs(np.stack(slabs[g:g + 16]), lanes) for g in range(0, len(slabs), 16)]
    return slabs[0]


# one lane to 256 of them, slabs that one block adds up and slabs that meet through memory, more column tiles than have a ticket
@pytest.mark.parametrize("cols", [1, 3, 4, 10, 33, 36, 64, 100, 128, 512, 2052, 8200])
def test_colsum_order_of_additions(pkg, dev, cols):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for rows in (1, 2, 7, 31, 32, 33, 63, 64, 65, 100, 127, 128, 129, 200, 255, 256, 257, 300, 400, 511, 512, 513):
        a = seeded((rows, cols), 516)
        got = pkg.functional.colsum(_t(a, dev)).cpu().numpy()
        assert np.array_equal(got, _column_sums_in_order(a, sms)), (rows, cols)


# more than sixteen groups of sixteen slabs, whose sums a lane adds with four sums that take turns: 8, 16 and 256 lanes, a last
# slab and a last group that are short, rows that are no float4s
@pytest.mark.parametrize("rows,cols", [(65536, 64), (49725, 160), (40000, 128), (300001, 10), (524288, 4), (262144, 64)])
def test_colsum_order_of_many_slabs(pkg, dev, rows, cols):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    a = seeded((rows, cols), 517)
    groups = cols // 4 if cols % 4 == 0 else cols
    tx = 1
    while tx < 32 and tx < groups:
        tx *= 2
    lanes, tiles = 256 // tx, -(-groups // tx)
    per_slab = -(-rows // max(1, min(-(-4 * sms // tiles), 1008, -(-rows // (4 * lanes)))))

    def tree(r):   # one slab
        acc, h = np.zeros((lanes, cols), np.float32), lanes // 2
        for i in range(0, len(r), lanes):
            acc[:len(r[i:i + lanes])] += r[i:i + lanes]
        while h:
            acc[:h] += acc[h:2 * h]
            h //= 2
        return acc[0].copy()

    def in_turns(r):   # lane l: rows l, l + lanes, ... in four sums; then the lanes in order
        t = np.zeros((4, lanes, cols), np.float32)
        for n, i in enumerate(range(0, len(r), lanes)):
            t[n & 3, :len(r[i:i + lanes])] += r[i:i + lanes]
        acc = (t[0] + t[1]) + (t[2] + t[3])
        total = acc[0].copy()
        for lane in acc[1:]:
            total += lane
        return total

    slabs = np.stack([tree(a[r:r + per_slab]) for r in range(0, rows, per_slab)])
    assert len(slabs) > 256 and tiles <= 16
    ref = in_turns(np.stack([in_turns(slabs[g:g + 16]) for g in range(0, len(slabs), 16)]))
    assert np.array_equal(pkg.functional.colsum(_t(a, dev)).cpu().numpy(), ref)


def test_golden_small_ops(pkg, dev, golden):
    """The reference's unit-test tensors for bias add, activation gradients, losses, argmax."""
    L, g = pkg.lib, golden
    x, b = _t(g["conv2d_bias_add/x"], dev), _t(g["conv2d_bias_add/bias"], dev)
    out = torch.empty_like(x)
    pkg._lib.check(L.dcg_bias_act(x.data_ptr(), b.data_ptr(), out.data_ptr(), None, 8, 2, 0, 0.0, _s()))
    assert np.array_equal(out.cpu().numpy(), g["conv2d_bias_add/out"])
    assert np.array_equal(pkg.functional.colsum(_t(g["conv2d_bias_add_grad/dy_hat"], dev)).cpu().numpy(),
                          g["conv2d_bias_add_grad/db"])
    for case, act, gate_key in (("leaky_relu_grad", pkg.ACT_LEAKY, "x"), ("relu_grad", pkg.ACT_RELU, "x"),
                                ("tanh_grad", pkg.ACT_TANH, "y_hat")):
        gate, d = _t(g[case + "/" + gate_key], dev), _t(g[case + "/dy_hat"], dev)
        o = torch.empty_like(d)
        pkg._lib.check(L.dcg_act_grad(gate.data_ptr(), d.data_ptr(), o.data_ptr(), d.numel(), act, 0.3, _s()))
        assert np.array_equal(o.cpu().numpy(), g[case + "/dx"]), case
    x, y = _t(g["sigmoid_cross_entropy/x"], dev), _t(g["sigmoid_cross_entropy/y"], dev)
    loss = torch.empty((1,), device=dev)
    pkg._lib.check(L.dcg_sigmoid_xent(y.data_ptr(), x.data_ptr(), loss.data_ptr(), 15, _s()))
    assert abs(loss.item() - float(g["sigmoid_cross_entropy/loss"])) < 1e-6
    dx = torch.empty_like(x)
    pkg._lib.check(L.dcg_sigmoid_xent_grad(y.data_ptr(), x.data_ptr(), dx.data_ptr(), 15, _s()))
    np.testing.assert_allclose(dx.cpu().numpy(), g["sigmoid_cross_entropy_grad/dx"], rtol=0, atol=1e-7)
    ya, yh = _t(g["argmax/y"], dev), _t(g["argmax/y_hat"], dev)
    acc = torch.empty((1,), device=dev)
    pkg._lib.check(L.dcg_argmax_acc(ya.data_ptr(), yh.data_ptr(), acc.data_ptr(), 10, 3, _s()))
    assert acc.item() == float(g["argmax/acc"])  # bit-exact integer count


def test_argmax_first_max_wins_and_is_exact(pkg, dev, orc):
    rows, cols = 5000, 10
    a = np.round(seeded((rows, cols), 520) * 3).astype(np.float32)  # many ties
    b = np.round(seeded((rows, cols), 521) * 3).astype(np.float32)
    acc = torch.empty((1,), device=dev)
    ad, bd = _t(a, dev), _t(b, dev)
    pkg._lib.check(pkg.lib.dcg_argmax_acc(ad.data_ptr(), bd.data_ptr(), acc.data_ptr(), rows, cols, _s()))
    assert acc.item() == float(orc.argmax_acc(a, b))


@pytest.mark.parametrize("m,n,p", [(64, 100, 8192), (64, 8192, 1), (3, 5, 7), (100, 64, 130), (64, 784, 100)])
def test_dense(pkg, dev, orc, m, n, p):
    L = pkg.lib
    a = seeded((m, n), 530)
    b = seeded((n, p), 531) * np.float32(0.1)
    bias = seeded((p,), 532)
    ad, bd, biasd = _t(a, dev), _t(b, dev), _t(bias, dev)
    out = torch.empty((m, p), device=dev)
    pkg._lib.check(L.dcg_matmul(ad.data_ptr(), bd.data_ptr(), biasd.data_ptr(), out.data_ptr(), m, n, p, _s()))
    ref = orc.mat_mul_add(a, b, bias)
    tol = 1e-6 * n ** 0.5 * max(1.0, np.abs(ref).max())
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0, atol=tol)
    pkg._lib.check(L.dcg_matmul(ad.data_ptr(), bd.data_ptr(), None, out.data_ptr(), m, n, p, _s()))
    np.testing.assert_allclose(out.cpu().numpy(), orc.mm_mul(a, b), rtol=0, atol=tol)
    # dW = x^T dy  (x [m, n] stored, dy [m, p]) -> [n, p]
    dy = seeded((m, p), 533)
    dyd = _t(dy, dev)
    dw = torch.empty((n, p), device=dev)
    pkg._lib.check(L.dcg_matmul_tn(ad.data_ptr(), dyd.data_ptr(), dw.data_ptr(), n, m, p, _s()))
    assert np.array_equal(dw.cpu().numpy(), orc.tmm_mul(a, dy))
    # dx = dy W^T  (dy [m, p], W [n, p]) -> [m, n]
    dx = torch.empty((m, n), device=dev)
    pkg._lib.check(L.dcg_matmul_nt(dyd.data_ptr(), bd.data_ptr(), dx.data_ptr(), m, p, n, _s()))
    assert np.array_equal(dx.cpu().numpy(), orc.mtm_mul(dy, b))


# every tile of the ordered kernel (flat for a few rows, 1 x 1 / 2 x 2 / 4 x 4 outputs per thread), its edges and reduction
# remainders, with and without 16-byte copies, and the outer product of n == 1
@pytest.mark.parametrize("m,n,p", [(1, 100, 8192), (8, 37, 513), (17, 784, 100), (100, 10, 784), (130, 65, 800), (300, 33, 1281),
                                   (640, 130, 602), (5, 1, 44), (3, 1, 7), (33, 3, 8193)])
def test_dense_is_bit_exact(pkg, dev, orc, m, n, p):
    L = pkg.lib
    a, b, bias, dy = seeded((m, n), 530), seeded((n, p), 531), seeded((p,), 532), seeded((m, p), 533)
    ad, bd, biasd, dyd = (_t(t, dev) for t in (a, b, bias, dy))
    out, dw, dx = torch.empty((m, p), device=dev), torch.empty((n, p), device=dev), torch.empty((m, n), device=dev)
    pkg._lib.check(L.dcg_matmul(ad.data_ptr(), bd.data_ptr(), biasd.data_ptr(), out.data_ptr(), m, n, p, _s()))
    pkg._lib.check(L.dcg_matmul_tn(ad.data_ptr(), dyd.data_ptr(), dw.data_ptr(), n, m, p, _s()))
    pkg._lib.check(L.dcg_matmul_nt(dyd.data_ptr(), bd.data_ptr(), dx.data_ptr(), m, p, n, _s()))
    assert np.array_equal(out.cpu().numpy(), orc.mat_mul_add(a, b, bias))
    assert np.array_equal(dw.cpu().numpy(), orc.tmm_mul(a, dy))
    assert np.array_equal(dx.cpu().numpy(), orc.mtm_mul(dy, b))


def test_dense_with_an_axis_of_two_to_the_thirty(pkg, dev):
    L, P = pkg.lib, (1 << 30) + 5
    if torch.cuda.mem_get_info()[0] < 20 * P:
        pytest.skip("needs %d GB" % (20 * P >> 30))
    a, bias = torch.tensor([0.75, -1.25], device=dev), None
    b = torch.empty((2 * P,), device=dev).uniform_(-1, 1)
    out = torch.empty((P,), device=dev)
    at = torch.tensor([0, 1, 2, 12345, (1 << 29) + 1, P - 2, P - 1], device=dev)

    def check(x, y):
        ref = (x * 0.75) + (y * -1.25)
        assert torch.equal(out[at], ref)

    pkg._lib.check(L.dcg_matmul(a.data_ptr(), b.data_ptr(), bias, out.data_ptr(), 1, 2, P, _s()))
    check(b[:P][at], b[P:][at])
    pkg._lib.check(L.dcg_matmul_tn(a.data_ptr(), b.data_ptr(), out.data_ptr(), 1, 2, P, _s()))
    check(b[:P][at], b[P:][at])
    pkg._lib.check(L.dcg_matmul_nt(a.data_ptr(), b.data_ptr(), out.data_ptr(), 1, 2, P, _s()))
    check(b[2 * at], b[2 * at + 1])


# the form for a few reduction steps and its limits, the outer product from either storage, stores of whole words and of single
# ones, unaligned operands and results
@pytest.mark.parametrize("m,n,p,off", [(700, 1, 640, 0), (700, 2, 641, 0), (650, 15, 642, 0), (650, 16, 644, 0), (650, 17, 644, 0),
                                       (700, 7, 644, 1), (130, 1, 600, 1), (1300, 16, 301, 0)])
def test_dense_with_a_short_reduction(pkg, dev, orc, m, n, p, off):
    L = pkg.lib

    def put(t):
        buf = torch.empty((t.size + off,), device=dev)
        buf[off:] = torch.from_numpy(t.reshape(-1)).to(dev)
        return buf[off:]

    a, b, bias, at, bt = (seeded(s, 534 + i) for i, s in enumerate([(m, n), (n, p), (p,), (n, m), (p, n)]))
    ad, bd, biasd, atd, btd = (put(t) for t in (a, b, bias, at, bt))
    out, tn, nt = (put(np.zeros((m, p), np.float32)) for _ in range(3))
    pkg._lib.check(L.dcg_matmul(ad.data_ptr(), bd.data_ptr(), biasd.data_ptr(), out.data_ptr(), m, n, p, _s()))
    pkg._lib.check(L.dcg_matmul_tn(atd.data_ptr(), bd.data_ptr(), tn.data_ptr(), m, n, p, _s()))
    pkg._lib.check(L.dcg_matmul_nt(ad.data_ptr(), btd.data_ptr(), nt.data_ptr(), m, n, p, _s()))
    assert np.array_equal(out.cpu().numpy().reshape(m, p), orc.mat_mul_add(a, b, bias))
    assert np.array_equal(tn.cpu().numpy().reshape(m, p), orc.tmm_mul(at, b))
    assert np.array_equal(nt.cpu().numpy().reshape(m, p), orc.mtm_mul(a, bt))


def test_losses(pkg, dev, orc):
    L = pkg.lib
    for n in (64, 1000):
        x = seeded((n,), 540, -5, 5)
        y = (seeded((n,), 541) > 0).astype(np.float32)
        xd, yd = _t(x, dev), _t(y, dev)
        loss = torch.empty((1,), device=dev)
        pkg._lib.check(L.dcg_sigmoid_xent(yd.data_ptr(), xd.data_ptr(), loss.data_ptr(), n, _s()))
        assert abs(loss.item() - float(orc.sigmoid_cross_entropy(y, x))) < 2e-6 * max(1, abs(loss.item()))
        g = torch.empty_like(xd)
        pkg._lib.check(L.dcg_sigmoid_xent_grad(yd.data_ptr(), xd.data_ptr(), g.data_ptr(), n, _s()))
        np.testing.assert_allclose(g.cpu().numpy(), orc.sigmoid_cross_entropy_grad(y, x), rtol=0, atol=1e-7)
    a, b = seeded((32, 10), 542), seeded((32, 10), 543)
    ad, bd = _t(a, dev), _t(b, dev)
    out = torch.empty((1,), device=dev)
    pkg._lib.check(L.dcg_mse(ad.data_ptr(), bd.data_ptr(), out.data_ptr(), 32, 10, _s()))
    assert abs(out.item() - float(orc.mse(a, b))) < 1e-6
    g = torch.empty_like(ad)
    pkg._lib.check(L.dcg_mse_grad(ad.data_ptr(), bd.data_ptr(), g.data_ptr(), 320, _s()))
    assert np.array_equal(g.cpu().numpy(), orc.mse_grad(a, b))
    # softmax family against torch (MNIST example operators)
    sm = torch.empty_like(ad)
    pkg._lib.check(L.dcg_softmax(ad.data_ptr(), sm.data_ptr(), 32, 10, _s()))
    assert torch.allclose(sm, torch.softmax(ad, 1), atol=1e-6)
    pkg._lib.check(L.dcg_log_softmax(ad.data_ptr(), sm.data_ptr(), 32, 10, _s()))
    assert torch.allclose(sm, torch.log_softmax(ad, 1), atol=1e-5)
    onehot = torch.zeros_like(ad)
    onehot[torch.arange(32), torch.arange(32) % 10] = 1
    pkg._lib.check(L.dcg_softmax_xent(onehot.data_ptr(), ad.data_ptr(), out.data_ptr(), 32, 10, _s()))
    want = -(onehot * torch.log_softmax(ad, 1)).sum() / 32
    assert abs(out.item() - want.item()) < 1e-5
    pkg._lib.check(L.dcg_softmax_xent_grad(onehot.data_ptr(), ad.data_ptr(), sm.data_ptr(), 32, 10, _s()))
    assert torch.allclose(sm, (torch.softmax(ad, 1) - onehot) / 32, atol=1e-6)


@pytest.mark.parametrize("sizes", [[5000], [3, 64, 4800, 512, 204800, 1], [4096 * 3 + 5, 7]])
def test_adam_multi_bit_exact(pkg, dev, orc, sizes):
    """Fused multi-tensor Adam == the reference's moment/moment2/adam node triple, bit for bit,
    over several steps (lr 2e-4, beta1 0.5, beta2 0.999, eps 1e-8 as dcgan/main.cu:35-36)."""
    F = pkg.functional
    ps = [seeded((n,), 600 + i) for i, n in enumerate(sizes)]
    ms = [np.zeros_like(p) for p in ps]
    vs = [np.zeros_like(p) for p in ps]
    pd, md, vd = ([_t(a, dev) for a in lst] for lst in (ps, ms, vs))
    t_ref = 0.0
    t = ctypes.c_float(0)
    for step in range(3):
        gs = [seeded((n,), 700 + 10 * step + i) for i, n in enumerate(sizes)]
        gd = [_t(g, dev) for g in gs]
        lr_t = F.adam_lr_t(t, 2e-4, 0.5, 0.999)
        F.adam_multi(pd, gd, md, vd, lr_t, 0.5, 0.999, 1e-8)
        torch.cuda.synchronize()
        for i in range(len(sizes)):
            ps[i], ms[i], vs[i], t_new, lr_ref = orc.adam_step(ps[i], gs[i], ms[i], vs[i], t_ref, 2e-4, 0.5, 0.999, 1e-8)
            assert lr_t == float(lr_ref)
            assert np.array_equal(pd[i].cpu().numpy(), ps[i]), (step, i)
            assert np.array_equal(md[i].cpu().numpy(), ms[i]) and np.array_equal(vd[i].cpu().numpy(), vs[i])
        t_ref = t_new
        assert t.value == t_ref


def test_adam_grad_scale_and_second_path(pkg, dev, orc):
    """grad_scale (the 1/world of data-parallel averaging) and the optional second gradient path."""
    F = pkg.functional
    n = 10000
    p, g1, g2 = seeded((n,), 801), seeded((n,), 802), seeded((n,), 803)
    pd, g1d, g2d = _t(p, dev), _t(g1, dev), _t(g2, dev)
    md, vd = torch.zeros_like(pd), torch.zeros_like(pd)
    F.adam_multi([pd], [g1d], [md], [vd], 1e-3, 0.5, 0.999, 1e-8, grad_scale=0.25, grads2=[g2d])
    g = (g1 + g2) * np.float32(0.25)
    ref, _, _, _, _ = orc.adam_step(p, g, np.zeros_like(p), np.zeros_like(p), 0.0, 2e-4, 0.5, 0.999, 1e-8)
    # same update with lr_t = 1e-3 instead of the schedule's value: recompute by hand
    m = np.float32(0.5) * g
    v = (np.float32(1) - np.float32(0.999)) * g * g
    want = p - np.float32(1e-3) * m / (np.sqrt(v) + np.float32(1e-8))
    np.testing.assert_allclose(pd.cpu().numpy(), want, rtol=0, atol=1e-6)
