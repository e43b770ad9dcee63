"""The DCGAN training step (dcg_trainer, node lists + fusion) against the CPU restatement of
dcgan/main.cu built from oracle operators, on identical parameters and inputs."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from conftest import seeded
from oracle import dcgan_model as M

pytestmark = pytest.mark.gpu


def _load_state(tr, st):
    for i in range(10):
        tr.tensor("g_param%d" % i).copy_(torch.from_numpy(st["g"][i].reshape(-1)))
        tr.tensor("d_param%d" % i).copy_(torch.from_numpy(st["d"][i].reshape(-1)))


def _maxrel(got, ref):
    return float(np.abs(got - ref).max() / max(np.abs(ref).max(), 1e-30))


def _l2rel(got, ref):
    return float(np.linalg.norm(got.astype(np.float64) - ref) / max(np.linalg.norm(ref.astype(np.float64)), 1e-30))


@pytest.mark.parametrize("prec_name,tol", [("fp32", 2e-5), ("tf32", 1e-1), ("3xtf32", 1e-2)])
@pytest.mark.parametrize("fuse", [False, True])
def test_gradients_match_cpu_model(pkg, dev, orc, prec_name, tol, fuse):
    """Every weight gradient of the D run and the G run, per layer.
    fp32 path: max abs error <= 2e-5 * max|ref| (summation-order noise only; measured 0).
    TF32 tensor path: each operator meets 1e-2 * max|ref| on identical inputs (tests/test_gpu_conv.py).
    Through the whole graph a pre-activation within rounding distance of zero can land on the other
    side of a leaky-relu / relu kink, which moves that element's gradient by a finite step; at
    batch 2 a kernel gradient sums as few as 32 pixels, so single flips show up at the percent level
    element-wise.  The whole-graph check therefore bounds the relative L2 error of each gradient
    and holds the losses to 1e-4.  3xTF32 (operators within 1e-5) sits in between: kink flips become
    rare (measured: 1e-6 on most gradients, 2.5e-3 where one pre-activation flipped), the relative L2
    bound tightens to 1e-2."""
    B = 2
    rng = np.random.default_rng(3)
    st = M.init_state(rng, B)
    for i in (1, 3, 5, 7, 9):   # non-zero biases make the bias path visible
        st["g"][i] = (rng.standard_normal(st["g"][i].shape) * 0.05).astype(np.float32)
        st["d"][i] = (rng.standard_normal(st["d"][i].shape) * 0.05).astype(np.float32)
    x = rng.uniform(-1, 1, (B, 64, 64, 3)).astype(np.float32)
    z = rng.uniform(-1, 1, (B, 100)).astype(np.float32)
    prec = {"fp32": pkg.PREC_FP32, "tf32": pkg.PREC_TF32, "3xtf32": pkg.PREC_3XTF32}[prec_name]
    err = _maxrel if prec_name == "fp32" else _l2rel
    loss_tol = 2e-5 if prec_name == "fp32" else 1e-4
    tr = pkg.Trainer(batch=B, precision=prec, fuse=fuse)
    _load_state(tr, st)
    tr.x.copy_(torch.from_numpy(x))
    tr.z.copy_(torch.from_numpy(z))

    d_loss, gf, gr = M.run(M.d_gradients(orc, st, x, z))
    tr.d_backward()
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    assert abs(tr.d_loss.item() - float(d_loss)) <= loss_tol * abs(float(d_loss)) + 1e-6
    for i in range(10):
        got_f, got_r = tr.tensor("d_grad%d" % i).cpu().numpy(), tr.tensor("d_gradb%d" % i).cpu().numpy()
        if prec_name == "fp32":   # the reference's two passes, one gradient set each
            assert err(got_f, gf[i].reshape(-1)) <= tol, ("fake", i)
            assert err(got_r, gr[i].reshape(-1)) <= tol, ("real", i)
        else:   # tensor path: one pass over [fake | real]; d_grad holds the sum, d_gradb stays zero
            assert not got_r.any()
            assert err(got_f, (gf[i] + gr[i]).reshape(-1)) <= tol, ("fake + real", i)

    g_loss, gg = M.run(M.g_gradients(orc, st, z))
    tr.g_backward()
    torch.cuda.synchronize()
    assert pkg.lib.dcg_device_status() == 0
    assert abs(tr.g_loss.item() - float(g_loss)) <= loss_tol * abs(float(g_loss)) + 1e-6
    for i in range(10):
        assert err(tr.tensor("g_grad%d" % i).cpu().numpy(), gg[i].reshape(-1)) <= tol, ("gen", i)
    tr.close()


@pytest.mark.parametrize("fuse", [False, True])
@pytest.mark.parametrize("net", ["d", "g"])
def test_smallest_negative_pre_activations_close_the_gate(pkg, dev, orc, net, fuse):
    """Pre-activations of -1 and -2 times 2^-149, whose leaky activation is -0: the fp32 path gates their gradients as the
    CPU model does, in the discriminator's first layer and in a leaky generator's dense layer."""
    B = 2
    rng = np.random.default_rng(11)
    st = M.init_state(rng, B)
    layer = 0 if net == "d" else 4   # its pre-activations are its bias
    st[net][2 * layer][...] = 0
    st[net][2 * layer + 1] = (np.float32(-2.0 ** -149) * (1 + np.arange(st[net][2 * layer + 1].size) % 2)).astype(np.float32)
    assert (st[net][2 * layer + 1] < 0).all()
    x = rng.uniform(-1, 1, (B, 64, 64, 3)).astype(np.float32)
    z = rng.uniform(-1, 1, (B, 100)).astype(np.float32)
    tr = pkg.Trainer(batch=B, precision=pkg.PREC_FP32, fuse=fuse, g_leaky=True)
    _load_state(tr, st)
    tr.x.copy_(torch.from_numpy(x))
    tr.z.copy_(torch.from_numpy(z))
    if net == "d":
        _, gf, gr = M.run(M.d_gradients(orc, st, x, z, True))
        tr.d_backward()
        pairs = [("d_grad1", gf[1]), ("d_gradb1", gr[1])]
    else:
        _, gg = M.run(M.g_gradients(orc, st, z, True))
        tr.g_backward()
        pairs = [("g_grad9", gg[9])]
    torch.cuda.synchronize()
    # (through an open gate five times as much; the bound is that of test_gradients_match_cpu_model)
    for name, ref in pairs:
        assert np.abs(ref).max() > 0 and _maxrel(tr.tensor(name).cpu().numpy(), ref.reshape(-1)) <= 2e-5, name
    tr.close()


def test_iteration_matches_cpu_model(pkg, dev, orc):
    """Two whole iterations (D update + 2 G updates each) on the fp32 path: parameters after the
    Adam updates follow the CPU model (Adam itself is bit-exact; the gradients carry reduction-order
    noise, so parameters are compared to a few 1e-6)."""
    B = 2
    rng = np.random.default_rng(5)
    st = M.init_state(rng, B)
    tr = pkg.Trainer(batch=B, precision=pkg.PREC_FP32, fuse=True)
    _load_state(tr, st)
    for it in range(2):
        x = rng.uniform(-1, 1, (B, 64, 64, 3)).astype(np.float32)
        z = rng.uniform(-1, 1, (B, 100)).astype(np.float32)
        d_ref, g_ref = M.run(M.train_iteration(orc, st, x, z))
        d_got, g_got = tr.step_host(x, z)
        assert abs(d_got - float(d_ref)) < 1e-4 and abs(g_got - float(g_ref)) < 1e-4
    for i in range(10):
        for net in ("g", "d"):
            got = tr.tensor("%s_param%d" % (net, i)).cpu().numpy()
            ref = st[net][i].reshape(-1)
            # Adam's first steps move each weight by ~lr whatever the gradient's size, so a sign flip
            # of a near-zero gradient shows up as 2*lr per update (4 generator updates so far)
            assert np.abs(got - ref).max() <= 2 * 2e-4 * 4 + 1e-6, (net, i)
            # ... and such flips feed back through the next forward pass; on average the two runs stay
            # within a fraction of one step
            assert np.mean(np.abs(got - ref)) <= 0.25 * 2e-4, (net, i)
    tr.close()


def test_fused_and_unfused_steps_are_identical(pkg, dev):
    B = 4
    g = torch.Generator().manual_seed(1)
    x = torch.rand((B, 64, 64, 3), generator=g) * 2 - 1
    z = torch.rand((B, 100), generator=g) * 2 - 1
    params = {}
    for fuse in (False, True):
        tr = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, fuse=fuse, seed=77)
        before = pkg.launches_total()
        losses = tr.step_host(x.numpy(), z.numpy())
        launches = pkg.launches_total() - before
        params[fuse] = (torch.cat([tr.tensor("d_params"), tr.tensor("g_params")]).cpu(), losses, launches)
        tr.close()
    assert torch.equal(params[False][0], params[True][0])
    assert params[False][1] == params[True][1]
    assert params[True][2] < params[False][2]


def test_generate_matches_cpu_model(pkg, dev, orc):
    """Config 0 of the benchmark set: generator forward, leaky-relu(0.2) between layers, tanh out."""
    B = 2
    rng = np.random.default_rng(9)
    st = M.init_state(rng, B)
    z = rng.uniform(-1, 1, (B, 100)).astype(np.float32)
    ref, _ = M.run(M.generator_forward(orc, st["g"], z, g_leaky=True))
    for prec, tol in ((pkg.PREC_FP32, 1e-5), (pkg.PREC_TF32, 1e-2)):
        tr = pkg.Trainer(batch=B, precision=prec, g_leaky=True)
        _load_state(tr, st)
        tr.z.copy_(torch.from_numpy(z))
        out = tr.generate()
        torch.cuda.synchronize()
        assert _maxrel(out.cpu().numpy(), ref) <= tol
        tr.close()


def test_graph_replay_equals_eager(pkg, dev, monkeypatch):
    """After two eager runs every node list is captured into a CUDA graph and replayed.  The replay
    launches the same kernels with the same arguments in the same order, so five iterations with and
    without graphs must leave bit-identical parameters and losses."""
    B = 4
    g = torch.Generator(device="cpu").manual_seed(21)
    xs = [(torch.rand((B, 64, 64, 3), generator=g) * 2 - 1).numpy() for _ in range(5)]
    zs = [(torch.rand((B, 100), generator=g) * 2 - 1).numpy() for _ in range(5)]
    results = []
    for eager in ("1", "0"):
        monkeypatch.setenv("DCG_TRAINER_EAGER", eager)
        tr = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, fuse=True, seed=77)
        losses = [tr.step_host(x, z) for x, z in zip(xs, zs)]
        torch.cuda.synchronize()
        assert pkg.lib.dcg_device_status() == 0
        results.append((losses, tr.tensor("d_params").clone(), tr.tensor("g_params").clone()))
        tr.close()
    (l0, d0, g0), (l1, d1, g1) = results
    assert l0 == l1
    assert torch.equal(d0, d1) and torch.equal(g0, g1)


@pytest.mark.parametrize("streams", [1, 2])
def test_replay_on_the_callers_stream_equals_eager(pkg, dev, monkeypatch, streams):
    """Captured graphs run on the stream the trainer was last called from, and in order when the calls change streams."""
    runs = {}
    for replay in (True, False):
        if not replay:
            monkeypatch.setattr(pkg.Trainer, "_replay", lambda self, what: False)
        tr = pkg.Trainer(batch=4, seed=7, precision=pkg.PREC_FP32)
        tr.x.copy_(torch.from_numpy(seeded((4, 64, 64, 3), 1)))
        callers = [torch.cuda.current_stream(), torch.cuda.Stream()][:streams]
        images, losses = [], []
        for i in range(12):
            stream = callers[i // 2 % streams]
            stream.wait_stream(callers[(i // 2 - 1) % streams])   # the inputs and outputs below are the caller's to order
            with torch.cuda.stream(stream):
                tr.z.copy_(torch.from_numpy(seeded((4, 100), i)), non_blocking=True)
                images.append(tr.generate().clone())
                tr.step()
                losses.append(tr.d_loss.clone())
        torch.cuda.synchronize()
        runs[replay] = [t.cpu() for t in images + losses + [tr.tensor("d_params"), tr.tensor("g_params")]]
        tr.close()
    assert all(torch.equal(a, b) for a, b in zip(runs[True], runs[False]))


def test_a_callers_stream_may_be_destroyed_between_calls(pkg, dev):
    """On streams that torch does not own the trainer keeps to its own stream, so that it never has to go back to one."""
    rt = torch.cuda.cudart()
    finals = []
    for external in (False, True):
        tr = pkg.Trainer(batch=4, seed=7, precision=pkg.PREC_FP32)
        tr.x.copy_(torch.from_numpy(seeded((4, 64, 64, 3), 1)))
        tr.z.copy_(torch.from_numpy(seeded((4, 100), 2)))
        torch.cuda.synchronize()
        for _ in range(3):
            handle = ctypes.c_size_t()
            if external:
                assert int(rt.cudaStreamCreate(ctypes.addressof(handle))) == 0
            with torch.cuda.stream(torch.cuda.ExternalStream(handle.value) if external else torch.cuda.current_stream()):
                for _ in range(4):
                    tr.step()
                    tr.generate()
                torch.cuda.current_stream().synchronize()
            if external:
                assert tr._joined is None
                assert int(rt.cudaStreamDestroy(handle.value)) == 0
            tr.step()
        torch.cuda.synchronize()
        finals.append([tr.tensor(n).cpu() for n in ("d_params", "g_params", "g_out")])
        tr.close()
    assert all(torch.equal(a, b) for a, b in zip(*finals))


def test_g_backward_in_two_parts(pkg, dev):
    """dcg_trainer_g_backward_part(0) then (1) - the split the data-parallel step uses to overlap the
    discriminator's all-reduce with the generator's forward pass - leaves the same gradients and loss
    as the one-call form, bit for bit, also once the parts replay as graphs."""
    B = 4
    g = torch.Generator(device="cpu").manual_seed(31)
    z = (torch.rand((B, 100), generator=g) * 2 - 1).to(dev)
    out = []
    for split in (False, True):
        tr = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, fuse=True, seed=99)
        tr.z.copy_(z)
        for _ in range(4):   # two eager runs, capture, replay
            if split:
                with tr._on_stream():
                    pkg._lib.check(pkg.lib.dcg_trainer_g_backward_part(tr._h, 0))
                    pkg._lib.check(pkg.lib.dcg_trainer_g_backward_part(tr._h, 1))
            else:
                tr.g_backward()
        torch.cuda.synchronize()
        assert pkg.lib.dcg_device_status() == 0
        out.append((tr.g_loss.clone(), tr.g_grads.clone()))
        tr.close()
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])



def test_batch64_tensor_path_vs_fp32_path(pkg, dev):
    """The benchmarked configuration (batch 64: the discriminator's single pass over 128 images, side
    streams, K-partition clusters at the shapes bench.py times) on the TF32 tensor path against the
    fp32 CUDA-core path on identical parameters and inputs; the fp32 path is itself pinned to the
    CPU oracle at batch 2 (test_gradients_match_cpu_model).  Losses to 1e-4; every gradient by
    relative L2 within 1e-1.  Measured: discriminator conv weights 0.016-0.032, its dense weight 0.0033,
    dense bias 2e-4; generator weights 0.012-0.018, its last conv weight 0.048, last bias 0.015 - TF32
    rounding moves single pre-activations across a leaky-relu / relu kink, a finite step per flip that
    no operator-level bound covers.  The test prints what it measured."""
    B = 64
    g = torch.Generator().manual_seed(17)
    x = torch.rand((B, 64, 64, 3), generator=g) * 2 - 1
    z = torch.rand((B, 100), generator=g) * 2 - 1
    grads, losses = {}, {}
    for name, prec in (("fp32", pkg.PREC_FP32), ("tf32", pkg.PREC_TF32)):
        tr = pkg.Trainer(batch=B, precision=prec, fuse=True, seed=234)
        tr.x.copy_(x)
        tr.z.copy_(z)
        for i in (1, 3, 5, 7):   # biases away from zero so that the bias path carries signal
            tr.tensor("d_param%d" % i).copy_(0.05 * torch.randn(tr.tensor("d_param%d" % i).shape, generator=torch.Generator().manual_seed(100 + i)))
            tr.tensor("g_param%d" % i).copy_(0.05 * torch.randn(tr.tensor("g_param%d" % i).shape, generator=torch.Generator().manual_seed(200 + i)))
        tr.d_backward()
        torch.cuda.synchronize()
        d = [tr.tensor("d_grad%d" % i).clone() for i in range(10)]
        if name == "fp32":   # the two passes of the fp32 path: fake + real
            d = [a + tr.tensor("d_gradb%d" % i) for i, a in enumerate(d)]
        dl = tr.d_loss.item()
        tr.g_backward()
        torch.cuda.synchronize()
        assert pkg.lib.dcg_device_status() == 0
        grads[name] = (d, [tr.tensor("g_grad%d" % i).clone() for i in range(10)])
        losses[name] = (dl, tr.g_loss.item())
        tr.close()
    for a, b in zip(losses["fp32"], losses["tf32"]):
        assert abs(a - b) <= 1e-4 * max(1.0, abs(a))
    worst = {}
    for net, idx in (("d", 0), ("g", 1)):
        for i in range(10):
            r, t = grads["fp32"][idx][i].double(), grads["tf32"][idx][i].double()
            worst["%s%d" % (net, i)] = float((r - t).norm() / max(float(r.norm()), 1e-30))
    print("batch-64 relative L2 of the TF32 gradients against the fp32 path:", worst)
    for name, rel in worst.items():
        assert rel <= 1e-1, (name, rel, worst)


def test_checkpoint_resume_is_bit_exact(pkg, dev, tmp_path):
    """save -> continue training equals save -> load into a fresh trainer -> continue training: the
    checkpoint carries the variables, Adam's moments and the step counters (the reference's
    save_vars / load_vars, src/ops/graph.cu:326-361, carries the variables only).  The file is written
    by a host thread while the next iterations are already enqueued."""
    B = 4
    g = torch.Generator(device="cpu").manual_seed(51)
    xs = [(torch.rand((B, 64, 64, 3), generator=g) * 2 - 1).numpy() for _ in range(4)]
    zs = [(torch.rand((B, 100), generator=g) * 2 - 1).numpy() for _ in range(4)]
    path = tmp_path / "ckpt.bin"
    a = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=77)
    for i in range(2):
        a.step_host(xs[i], zs[i])
    a.save(path)                        # returns at once; steps 2 and 3 run while the file is written
    la = [a.step_host(xs[i], zs[i]) for i in (2, 3)]
    a.save_wait()
    b = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=1234)   # different initial weights
    b.load(path)
    lb = [b.step_host(xs[i], zs[i]) for i in (2, 3)]
    torch.cuda.synchronize()
    assert la == lb
    for name in ("d_params", "g_params", "d_m0", "d_v8", "g_m0", "g_v8"):
        assert torch.equal(a.tensor(name), b.tensor(name)), name
    # the first 20 tensors are the variables, readable without knowing about the optimiser state
    import struct
    raw = open(path, "rb").read()
    assert raw[:4] == b"DCGT" and struct.unpack("<II", raw[4:12]) == (1, 61)
    assert struct.unpack("<I", raw[12:16])[0] == 4 and struct.unpack("<4I", raw[16:32]) == (5, 5, 256, 512)
    a.close()
    b.close()


def test_discriminator_forward_backward_matches_cpu_model(pkg, dev, orc):
    """BASELINE configs[1] (discriminator forward + backward on real images against labels of ones,
    dx and dk of every layer) at batch 2 against the oracle's real-image pass of the D run."""
    B = 2
    rng = np.random.default_rng(13)
    st = M.init_state(rng, B)
    x = rng.uniform(-1, 1, (B, 64, 64, 3)).astype(np.float32)
    z = rng.uniform(-1, 1, (B, 100)).astype(np.float32)
    _, _, gr = M.run(M.d_gradients(orc, st, x, z))    # gr: gradients of the real-image pass
    for prec, tol, err in ((pkg.PREC_FP32, 2e-5, _maxrel), (pkg.PREC_TF32, 1e-1, _l2rel)):
        tr = pkg.Trainer(batch=B, precision=prec)
        _load_state(tr, st)
        tr.x.copy_(torch.from_numpy(x))
        tr.d_fwd_bwd()
        torch.cuda.synchronize()
        assert pkg.lib.dcg_device_status() == 0
        for i in range(10):
            assert err(tr.tensor("d_gradb%d" % i).cpu().numpy(), gr[i].reshape(-1)) <= tol, i
        tr.close()


def test_pipelined_submit_equals_blocking_steps(pkg, dev):
    """submit_host / result with several iterations in flight (the host -> device copies of iteration
    i+1 overlap the compute of iteration i, losses are collected with a lag) gives the same losses and
    parameters as blocking step_host calls on the same host batches."""
    B = 4
    g = torch.Generator(device="cpu").manual_seed(81)
    xs = [(torch.rand((B, 64, 64, 3), generator=g) * 2 - 1).pin_memory() for _ in range(7)]
    zs = [(torch.rand((B, 100), generator=g) * 2 - 1).numpy() for _ in range(7)]   # pinned and pageable sources
    a = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=77)
    la = [a.step_host(x, z) for x, z in zip(xs, zs)]
    b = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=77)
    tickets, lb = [], []
    for x, z in zip(xs, zs):
        tickets.append(b.submit_host(x, z))
        if len(tickets) > 3:
            lb.append(b.result(tickets.pop(0)))
    lb += [b.result(t) for t in tickets]
    torch.cuda.synchronize()
    assert la == lb
    assert torch.equal(a.tensor("d_params"), b.tensor("d_params")) and torch.equal(a.tensor("g_params"), b.tensor("g_params"))
    a.close()
    b.close()


def test_uint8_images_are_decoded_on_the_device_like_the_reference(pkg, dev):
    """celeba::load scales bytes to [-1, 1] on the host: img = float(p) / 127.5 - 1. in double, stored
    as float (src/datasets/celeba.cu:29).  submit_host with uint8 images copies the bytes and runs that
    expression on the device: all 256 values bit-equal, and a step fed with bytes equals a step fed
    with the host-scaled floats."""
    import ctypes
    vals = torch.arange(256, dtype=torch.uint8).repeat(4)            # 1024 values, 16-byte multiples
    want = torch.from_numpy((vals.numpy().astype(np.float32).astype(np.float64) / 127.5 - 1.).astype(np.float32))
    src, dst = vals.to(dev), torch.empty(vals.numel(), device=dev)
    pkg._lib.check(pkg.lib.dcg_u8_to_unit(src.data_ptr(), dst.data_ptr(), src.numel(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(dst.cpu(), want)
    B = 4
    g = torch.Generator(device="cpu").manual_seed(91)
    px = torch.randint(0, 256, (B, 64, 64, 3), generator=g, dtype=torch.uint8)
    z = (torch.rand((B, 100), generator=g) * 2 - 1).numpy()
    xf = torch.from_numpy((px.numpy().astype(np.float32).astype(np.float64) / 127.5 - 1.).astype(np.float32))
    a = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=77)
    b = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=77)
    assert a.step_host(px, z) == b.step_host(xf, z)
    assert torch.equal(a.tensor("g_params"), b.tensor("g_params"))
    a.close()
    b.close()


def test_shared_generator_forward_gives_the_same_numbers(pkg, dev):
    """share_g_forward: the first G run of an iteration re-uses the generator activations of the D run
    (the generator's parameters are unchanged in between).  Same losses and parameters, bit for bit,
    as the recomputing form, before and after the iteration replays as a CUDA graph; fewer launches."""
    B = 4
    g = torch.Generator(device="cpu").manual_seed(33)
    xs = [(torch.rand((B, 64, 64, 3), generator=g) * 2 - 1).numpy() for _ in range(5)]
    zs = [(torch.rand((B, 100), generator=g) * 2 - 1).numpy() for _ in range(5)]
    out = []
    for share in (False, True):
        tr = pkg.Trainer(batch=B, precision=pkg.PREC_TF32, seed=77, share_g_forward=share)
        losses = [tr.step_host(x, z) for x, z in zip(xs, zs)]
        torch.cuda.synchronize()
        out.append((losses, tr.tensor("d_params").clone(), tr.tensor("g_params").clone(), tr.launches_per_step()))
        tr.close()
    assert out[0][0] == out[1][0]
    assert torch.equal(out[0][1], out[1][1]) and torch.equal(out[0][2], out[1][2])
    assert out[1][3] < out[0][3]
