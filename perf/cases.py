"""Performance cases: the work that users of this framework have it do, through its public entry points.

    step      one DCGAN training iteration, inputs resident on the device (Trainer.step)
    host      the same iteration fed from pinned host memory, uint8 images in, losses out (Trainer.step_host)
    grads     discriminator forward + backward with every layer's gradients (Trainer.d_fwd_bwd)
    generate  images from noise (Trainer.generate)
    layer     one convolution layer called directly: forward with its fused bias + activation, input gradient, kernel
              gradient, bias gradient (functional.conv2d_fwd / conv2d_dx / conv2d_dk / colsum)
    mlp       one training step of a dense classifier as a runtime node list (nodes.Context.run)
"""
import math

import torch

import __graft_entry__

_pkg = None
PRECISIONS = {"tf32": "PREC_TF32", "3xtf32": "PREC_3XTF32", "fp32": "PREC_FP32"}
D_PARAMS, G_PARAMS = 4314753, 5133443      # variables of the two networks
CONV_FLOPS_EDGE = 2 * 32 * 32 * 25 * 3 * 64       # one convolution operator of the image-side layer, per image
CONV_FLOPS_MID = 2 * 16 * 16 * 25 * 64 * 128      # ... of any of the three other layers, per image
IMAGE = 64 * 64 * 3
Z = 100


def _package():
    global _pkg
    if _pkg is None:
        _pkg = __graft_entry__.load_package()
    return _pkg


def listed():
    return [
        # the training iteration at the batch size the model is trained with (dcgan/main.cu), and the benchmark's workload
        {"name": "step_b64", "kind": "step", "precision": "tf32", "batch": 64},
        # a small batch: many short launches in a row
        {"name": "step_b8", "kind": "step", "precision": "tf32", "batch": 8},
        # a large batch, as throughput-minded training uses
        {"name": "step_b256", "kind": "step", "precision": "tf32", "batch": 256},
        # training with near-fp32 products on the tensor cores
        {"name": "step_b64_3xtf32", "kind": "step", "precision": "3xtf32", "batch": 64},
        # training bit-comparable with the CPU code: debugging runs, checks of a port
        {"name": "step_b8_fp32", "kind": "step", "precision": "fp32", "batch": 8},
        # the training loop of a user whose images come from a decoder on the host, waiting for each step's losses
        {"name": "host_u8_b64", "kind": "host", "precision": "tf32", "batch": 64},
        # discriminator alone, all gradients (the second configuration of the benchmark)
        {"name": "grads_b64", "kind": "grads", "precision": "tf32", "batch": 64},
        # one sampled image: latency
        {"name": "generate_b1", "kind": "generate", "precision": "tf32", "batch": 1},
        # a batch of samples, as for a dataset or an evaluation
        {"name": "generate_b512", "kind": "generate", "precision": "tf32", "batch": 512},
        # a layer of somebody else's network: extents that fill no tile, channels that are no multiple of 32
        {"name": "layer_small", "kind": "layer", "precision": "tf32", "n": 2, "h": 12, "w": 20, "c": 36, "k": 5, "o": 40, "s": 2},
        # a larger one, odd extents, 3x3 and stride 1
        {"name": "layer_odd", "kind": "layer", "precision": "tf32", "n": 13, "h": 75, "w": 51, "c": 96, "k": 3, "o": 160, "s": 1},
        # the dense classifier of the reference's second example program (784-100-10, Adam) as nodes
        {"name": "mlp_b100", "kind": "mlp", "batch": 100, "hidden": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "host", "grads", "generate", "generate", "layer", "layer", "mlp"])
    if kind == "step":
        precision = rng.choice(["tf32", "tf32", "tf32", "3xtf32", "fp32"])
        lo, hi = {"tf32": (4, 256), "3xtf32": (4, 64), "fp32": (1, 8)}[precision]
        return {"kind": kind, "precision": precision, "batch": _log_int(rng, lo, hi)}
    if kind in ("host", "grads"):
        return {"kind": kind, "precision": "tf32", "batch": _log_int(rng, 4 if kind == "host" else 16, 256)}
    if kind == "generate":
        return {"kind": kind, "precision": rng.choice(["tf32", "tf32", "3xtf32"]), "batch": _log_int(rng, 1, 512)}
    if kind == "mlp":
        return {"kind": kind, "batch": _log_int(rng, 10, 1000), "hidden": _log_int(rng, 32, 512)}
    k = rng.choice([1, 3, 3, 4, 5, 5])
    case = {"kind": kind, "precision": rng.choice(["tf32", "tf32", "3xtf32"]), "n": _log_int(rng, 1, 32),
            "h": _log_int(rng, 8, 96), "w": _log_int(rng, 8, 96), "c": 4 * _log_int(rng, 1, 48) if rng.random() < 0.8 else 3,
            "k": k, "o": 4 * _log_int(rng, 4, 48) if rng.random() < 0.5 else 32 * rng.randint(1, 6), "s": rng.choice([1, 2, 2]) if k > 1 else 1}
    while _layer_flops(case) > 30e9:
        longest = "n" if case["n"] > 1 else "h"
        case[longest] //= 2
    return case


# ---- geometry and work of a layer --------------------------------------------------------------------------------------
def _layer_sizes(case):
    ho, wo = -(-case["h"] // case["s"]), -(-case["w"] // case["s"])   # SAME padding
    x = case["n"] * case["h"] * case["w"] * case["c"]
    y = case["n"] * ho * wo * case["o"]
    return ho, wo, x, y, case["k"] * case["k"] * case["c"] * case["o"]


def _layer_flops(case):
    ho, wo, _, _, _ = _layer_sizes(case)
    return 3 * 2.0 * case["n"] * ho * wo * case["k"] * case["k"] * case["c"] * case["o"]


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: the convolutions and dense products."""
    kind = case["kind"]
    if kind in ("step", "host"):
        # per image 17 passes over all four convolutions of a network, less the two image gradients nobody needs
        flops = case["batch"] * (17.0 * (CONV_FLOPS_EDGE + 3 * CONV_FLOPS_MID) - 2 * CONV_FLOPS_EDGE)
        return {"bytes": 24.0 * (D_PARAMS + G_PARAMS) + case["batch"] * (2 * IMAGE + Z) * 4.0, "flops": flops}
    if kind == "grads":
        return {"bytes": 8.0 * D_PARAMS + case["batch"] * 2 * IMAGE * 4.0,
                "flops": case["batch"] * 3.0 * (CONV_FLOPS_EDGE + 3 * CONV_FLOPS_MID)}
    if kind == "generate":
        return {"bytes": 4.0 * G_PARAMS + case["batch"] * (IMAGE + Z) * 4.0,
                "flops": case["batch"] * (CONV_FLOPS_EDGE + 3.0 * CONV_FLOPS_MID + 2.0 * Z * 8192)}
    if kind == "layer":
        _, _, x, y, k = _layer_sizes(case)
        return {"bytes": 4.0 * (2 * x + 3 * y + 2 * k + 2 * case["o"]), "flops": _layer_flops(case)}
    b, h = case["batch"], case["hidden"]
    params = 784 * h + h + 10 * h + 10
    return {"bytes": 4.0 * (b * (784 + 10) + 7 * params), "flops": b * (4.0 * 784 * h + 6.0 * h * 10)}


def tolerance(case):
    if case["kind"] == "mlp":
        return {"rel": 1e-5, "max": 1e-3}
    if case["precision"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "layer":
        # TF32 operands keep 10 mantissa bits: up to 1e-3 of each factor is cut off
        return {"rel": 1e-5, "max": 1e-4} if case["precision"] == "3xtf32" else {"rel": 2e-3, "max": 2e-2}
    if case["kind"] == "generate":   # four layers, one after the other
        return {"rel": 1e-5, "max": 1e-4} if case["precision"] == "3xtf32" else {"rel": 5e-3, "max": 5e-2}
    # a pre-activation within rounding distance of a leaky-relu kink may land on either side of it, which moves the
    # gradients of a small batch by a percent; an Adam step moves a weight by its full step size whichever the sign of a
    # gradient that is close to zero
    if case["kind"] == "grads":
        return {"rel": 2e-2, "max": 0.9}
    return {"rel": 3e-3 if case["precision"] == "3xtf32" else 1e-2, "max": 0.5}


class Outputs(dict):
    """Tensors that are views of a trainer's own memory, and the trainer, which has to live as long as they are read."""

    def __init__(self, trainer, **tensors):
        super().__init__(tensors)
        self.trainer = trainer


# ---- states and passes -------------------------------------------------------------------------------------------------
def _uniform(shape, gen, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo


def _normal(shape, gen, sd):
    return torch.randn(shape, generator=gen, device="cuda") * sd


def prepare(case, seed):
    pkg = _package()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "layer":
        return _prepare_layer(case, gen, pkg)
    if kind == "mlp":
        return _prepare_mlp(case, gen, pkg)
    trainer = pkg.Trainer(batch=case["batch"], precision=getattr(pkg, PRECISIONS[case["precision"]]), seed=1 + seed % 100003,
                          g_leaky=kind == "generate")
    state = {"kind": kind, "trainer": trainer}
    trainer.z.copy_(_uniform(trainer.z.shape, gen))
    if kind != "host":
        trainer.x.copy_(_uniform(trainer.x.shape, gen))
    else:
        state["x"] = torch.randint(0, 256, tuple(trainer.x.shape), generator=gen, device="cuda").to(torch.uint8).cpu().pin_memory()
        state["z"] = trainer.z.cpu().pin_memory()
    if kind in ("step", "host"):
        # the variables after the pass; the summation order of the fp32 path is fixed, so there the gradients, moments and
        # images of a second pass can be compared too (elsewhere they follow every gradient sign that an Adam step takes up)
        names = ["d_params", "g_params"] + (["d_loss", "g_loss"] if kind == "step" else [])
        if case["precision"] == "fp32":
            names += ["g_out", "d_grads", "g_grads"] + ["%s_%s%d" % (net, m, i) for net in "dg" for m in "mv" for i in range(10)]
    elif kind == "grads":
        names = ["d_gradb%d" % i for i in range(10)] + ["logits_real"]
    else:
        names = ["g_out"]
    state["out"] = Outputs(trainer, **{name: trainer.tensor(name) for name in names})
    return state


def _prepare_layer(case, gen, pkg):
    ho, wo, _, _, _ = _layer_sizes(case)
    n, h, w, c, k, o = (case[key] for key in ("n", "h", "w", "c", "k", "o"))
    return {"kind": "layer", "s": (case["s"], case["s"]), "precision": getattr(pkg, PRECISIONS[case["precision"]]),
            "x": _uniform((n, h, w, c), gen), "k": _normal((k, k, c, o), gen, 0.02), "b": _normal((o,), gen, 0.02),
            "dz": _normal((n, ho, wo, o), gen, 1e-2), "z": torch.empty((n, ho, wo, o), device="cuda")}


def _prepare_mlp(case, gen, pkg):
    import ctypes
    b, h = case["batch"], case["hidden"]
    sizes = {"w1": (784, h), "b1": (h,), "w2": (h, 10), "b2": (10,)}
    s = {"kind": "mlp", "x": _uniform((b, 784), gen, 0.0, 1.0),
         "y": torch.nn.functional.one_hot(torch.randint(0, 10, (b,), generator=gen, device="cuda"), 10).float().contiguous()}
    for name, shape in sizes.items():
        s[name] = _normal(shape, gen, 0.05) if len(shape) == 2 else torch.zeros(shape, device="cuda")
        for moment in ("m_", "v_"):
            s[moment + name] = torch.zeros(shape, device="cuda")
        s["g_" + name] = torch.empty(shape, device="cuda")
        s["t_" + name] = ctypes.c_float(0.0)
    for name, shape in {"z1": (b, h), "a1": (b, h), "logits": (b, 10), "loss": (1,), "dlogits": (b, 10), "da1": (b, h), "dz1": (b, h)}.items():
        s[name] = torch.empty(shape, device="cuda")
    N = pkg.nodes
    s["nodes"] = [
        N.op_mat_mul_add(s["x"], s["w1"], s["b1"], s["z1"], b, 784, h),
        N.op_relu(s["z1"], s["a1"], b * h),
        N.op_mat_mul_add(s["a1"], s["w2"], s["b2"], s["logits"], b, h, 10),
        N.op_softmax_cross_entropy(s["y"], s["logits"], s["loss"], b, 10),
        N.op_softmax_cross_entropy_grad(s["y"], s["logits"], s["dlogits"], b, 10),
        N.op_tmat_mat_mul(s["a1"], s["dlogits"], s["g_w2"], h, b, 10),
        N.op_mat_sum_cols(s["dlogits"], s["g_b2"], b, 10),
        N.op_mat_tmat_mul(s["dlogits"], s["w2"], s["da1"], b, 10, h),
        N.op_relu_grad(s["z1"], s["da1"], s["dz1"], b * h),
        N.op_tmat_mat_mul(s["x"], s["dz1"], s["g_w1"], 784, b, h),
        N.op_mat_sum_cols(s["dz1"], s["g_b1"], b, h),
    ]
    for name, shape in sizes.items():
        count = math.prod(shape)
        s["nodes"] += [N.op_moment_update(s["m_" + name], s["g_" + name], 0.9, 0.1, count),
                       N.op_moment_update2(s["v_" + name], s["g_" + name], 0.999, 0.001, count),
                       N.op_adam_update(s[name], s["t_" + name], s["m_" + name], s["v_" + name], 1e-3, 0.9, 0.999, 1e-8, count)]
    s["context"] = pkg.Context()
    s["out"] = {key: s[key] for key in ["loss", "logits"] + [p + q for p in ("", "g_", "m_", "v_") for q in sizes]}
    return s


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["trainer"].step()
        return state["out"]
    if kind == "host":
        d_loss, g_loss = state["trainer"].step_host(state["x"], state["z"])
        return Outputs(state["trainer"], **state["out"], d_loss=d_loss, g_loss=g_loss)
    if kind == "grads":
        state["trainer"].d_fwd_bwd()
        return state["out"]
    if kind == "generate":
        state["trainer"].generate()
        return state["out"]
    if kind == "mlp":
        state["context"].run(state["nodes"], fuse=True)
        return state["out"]
    pkg = _package()
    F = pkg.functional
    x, k, dz, prec, s = state["x"], state["k"], state["dz"], state["precision"], state["s"]
    epilogue = F.make_epilogue(bias=state["b"], act=pkg.ACT_LEAKY, alpha=0.2, pre_act=state["z"])
    y = F.conv2d_fwd(x, k, s, epilogue=epilogue, precision=prec)
    dx = F.conv2d_dx(dz, k, x.shape[1:3], s, precision=prec)
    dk = F.conv2d_dk(x, dz, k.shape[:2], s, precision=prec)
    return {"y": y, "z": state["z"], "dx": dx, "dk": dk, "db": F.colsum(dz)}
