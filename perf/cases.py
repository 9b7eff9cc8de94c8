"""Performance cases of the MLP training step and its GEMM entry point, through the public API.

Four kinds of program use this package, and a case is one of them at one size:

  train    weights, inputs and targets are on the GPU; `MLP.step(iters)`, then the loss and every
           layer's updated weights are read back (training with periodic checkpoints; the
           reference's own main runs a fixed number of iterations and then reads the weights)
  stream   a data loader: every step copies a new batch from pinned host memory and returns its
           loss (`train_step_host_async` / `wait_loss`, two steps in flight), then the weights
  online   one blocking `train_step_host` call on one small batch: a latency-bound caller
  sgemm    `b2_sgemm` on device buffers the caller owns (the replacement of cblas_sgemm)

Each kind covers the precisions it is used with. Forward, weight gradient, input gradient and
update are all inside every training case. Nothing is cached between passes: training passes go
on from the weights of the pass before.
"""
import ctypes as C

import numpy as np
import torch

from tbb_test_b200 import _capi as K
from tbb_test_b200.mlp import MLP

PREC = {"fp32": K.PREC_FP32, "tf32": K.PREC_TF32, "bf16": K.PREC_BF16, "fp32tc": K.PREC_FP32_TC}
# weights are U(-a, a): the benchmark configurations' scale, the usual one in front of a ReLU, the reference's own
INIT = {"fan_in": lambda f: f ** -0.5, "he": lambda f: (6.0 / f) ** 0.5, "reference": lambda f: 0.1}
_FP = C.POINTER(C.c_float)


def _train(name, widths, batch, precision, iters, kind="train", **kw):
    case = {"name": name, "kind": kind, "widths": ",".join(map(str, widths)), "batch": batch, "precision": precision,
            "iters": iters, "mode": "baseline", "init": "he", "lr": 1e-4, "graph": False, "grad_bf16": False}
    case.update(kw)
    return case


def listed():
    return [
        # smallest call: one blocking step of a small network on a batch of 32, in the default precision
        _train("online_small_fp32", [128, 256, 128, 64], 32, "fp32", 1, kind="online", lr=0.01),
        # 5 x 1024^2, batch 1024, the configuration's 10 iterations in exact fp32 (the default precision)
        _train("c1_fp32", [1024] * 6, 1024, "fp32", 10, init="fan_in", lr=0.01),
        # the same network as a latency-bound bf16 job: one CUDA graph per step
        _train("c1_bf16_graph", [1024] * 6, 1024, "bf16", 256, init="fan_in", graph=True),
        # the same network fed from the host, fp32-class results on the tensor cores
        _train("c1_fp32tc_stream", [1024] * 6, 1024, "fp32tc", 32, kind="stream", init="fan_in"),
        # deep and narrow: 20 x 512^2, batch 2048 (at 1/sqrt(fan_in) the signal fades over 20 ReLU layers
        # and the weights stop moving, so it is drawn at the scale that keeps it, like the other networks)
        _train("c3_bf16", [512] * 21, 2048, "bf16", 64),
        # wide: 8 x 4096^2, batch 8192 (the benchmark's default workload)
        _train("c4_bf16", [4096] * 9, 8192, "bf16", 64, init="fan_in", lr=0.01),
        # the same fed from the host: inputs and targets of every step cross the host link
        _train("c4_bf16_stream", [4096] * 9, 8192, "bf16", 32, kind="stream", init="fan_in", lr=0.01),
        # the wide network's tf32 option at the rows one of eight GPUs holds
        _train("c4_shard_tf32", [4096] * 9, 1024, "tf32", 96, init="fan_in", lr=0.001),
        # widest layers (8192^2) at one GPU's rows out of eight, bf16 gradients
        _train("c5_shard_bf16", [8192] * 3, 2048, "bf16", 96, grad_bf16=True),
        # the reference's own topology and arithmetic: seven layers of 1024 ending in one unit
        _train("reference_bf16", [1024] * 7 + [1], 1024, "bf16", 128, mode="ref", init="reference", lr=1e-10),
        # a small classifier with ragged widths (rows that are not multiples of 16 bytes, a 10-wide output)
        _train("ragged_bf16", [784, 500, 300, 10], 1000, "bf16", 64),
        # one GEMM of the caller's own, rectangular
        {"name": "sgemm_tf32", "kind": "sgemm", "m": 1000, "n": 2048, "k": 768, "transa": False, "transb": True,
         "precision": "tf32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "stream", "online", "sgemm"])
    if kind == "sgemm":
        precision = rng.choice(["tf32", "fp32"])
        top = 4096 if precision == "tf32" else 2048
        dims = [_log_int(rng, 64, top) for _ in range(3)]
        if precision == "tf32":  # rows of whole 16-byte pieces
            dims = [max(16, d // 4 * 4) for d in dims]
        return {"kind": "sgemm", "m": dims[0], "n": dims[1], "k": dims[2], "transa": rng.random() < 0.3,
                "transb": rng.random() < 0.5, "precision": precision}
    precision = rng.choice(["bf16", "bf16", "tf32", "fp32tc", "fp32"])
    ragged = rng.random() < 0.25
    if kind == "online":
        layers, top, batch = rng.randint(1, 4), 512, _log_int(rng, 8, 256)
    else:
        layers = rng.randint(2, 12)
        top = 1024 if ragged or precision == "fp32" else 4096
        batch = _log_int(rng, 128, 2048 if ragged or precision == "fp32" else 8192)
    if rng.random() < 0.5:
        widths = [_log_int(rng, 64, top)] * (layers + 1)
    else:
        widths = [_log_int(rng, 64, top) for _ in range(layers + 1)]
    if not ragged:
        widths = [max(64, w // 32 * 32) for w in widths]
        batch = max(8, batch // 8 * 8)
    elif rng.random() < 0.5:
        widths[-1] = rng.randint(1, 40)
    case = _train("", widths, batch, precision, 1, kind=kind)
    del case["name"]
    if kind != "online":
        # as many steps as keep a pass between a few milliseconds and a few hundred
        rate = 4e12 if precision == "fp32" or ragged else 150e12 if precision == "fp32tc" else 400e12
        case["iters"] = max(2, min(64, int(0.15 * rate / _step_flops(widths, batch))))
        case["graph"] = kind == "train" and rng.random() < 0.3
        case["grad_bf16"] = precision == "bf16" and rng.random() < 0.3
        if rng.random() < 0.2:
            case["mode"], case["init"], case["lr"] = "ref", "fan_in", 1e-10
    return case


def _widths(case):
    return [int(w) for w in case["widths"].split(",")]


def _step_flops(widths, batch):
    return sum(6.0 * batch * a * b for a, b in zip(widths, widths[1:]))


def _matrix(g, rows, cols, what, a=1.0):
    t = torch.empty(rows, cols, device="cuda")
    if what == "normal":
        return t.normal_(generator=g)
    if what == "sign":
        return t.uniform_(-1.0, 1.0, generator=g).sign_()
    return t.uniform_(-a, a, generator=g)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["kind"] == "sgemm":
        m, n, k = case["m"], case["n"], case["k"]
        ta, tb = case["transa"], case["transb"]
        a = _matrix(g, k if ta else m, m if ta else k, "uniform")
        b = _matrix(g, n if tb else k, k if tb else n, "uniform")
        return {"case": case, "mlp": MLP([16, 16], 16), "a": a, "b": b, "c": torch.zeros(m, n, device="cuda")}
    nf, batch = _widths(case), case["batch"]
    mode = K.MODE_REF if case["mode"] == "ref" else K.MODE_BASELINE
    mlp = MLP(nf, batch, mode=mode, precision=PREC[case["precision"]], lr=case["lr"], use_graph=case["graph"],
              grad_bf16=case["grad_bf16"])
    for l in range(len(nf) - 1):
        mlp.upload_weights(l, _matrix(g, nf[l + 1], nf[l], "uniform", INIT[case["init"]](nf[l])).cpu().numpy())
    state = {"case": case, "mlp": mlp, "nf": nf}
    x = lambda: _matrix(g, batch, nf[0], "normal").cpu()  # noqa: E731
    t = lambda: _matrix(g, batch, nf[-1], "sign").cpu()  # noqa: E731
    if case["kind"] == "train":
        mlp.upload_input(x().numpy())
        mlp.upload_target(t().numpy())
    else:  # three batches in page-locked memory, as a data loader keeps them
        pairs = [(x().pin_memory(), t().pin_memory()) for _ in range(1 if case["kind"] == "online" else 3)]
        state["batches"] = pairs
        state["ptrs"] = [(C.cast(p.data_ptr(), _FP), C.cast(q.data_ptr(), _FP)) for p, q in pairs]
    return state


def _weights(state):
    return [state["mlp"].weights(l) for l in range(len(state["nf"]) - 1)]


def run(state):
    case, mlp = state["case"], state["mlp"]
    if case["kind"] == "sgemm":
        a, b, c = state["a"], state["b"], state["c"]
        rc = mlp.lib.b2_sgemm(mlp._h, PREC[case["precision"]], int(case["transa"]), int(case["transb"]), case["m"],
                              case["n"], case["k"], 1.0, a.data_ptr(), a.shape[1], b.data_ptr(), b.shape[1], 0.0,
                              c.data_ptr(), c.shape[1])
        if rc != K.OK:
            raise K.B2Error(rc, mlp.lib.b2_last_error(mlp._h).decode())
        return c
    if case["kind"] == "train":
        mlp.step(case["iters"])
        return [mlp.loss()] + _weights(state)
    ldx, ldt = state["nf"][0], state["nf"][-1]
    if case["kind"] == "online":
        xp, tp = state["ptrs"][0]
        return [mlp.train_step_host(xp, ldx, tp, ldt)] + _weights(state)
    losses = []
    for i in range(case["iters"]):
        xp, tp = state["ptrs"][i % len(state["ptrs"])]
        mlp.train_step_host_async(xp, ldx, tp, ldt)
        if i:
            losses.append(mlp.wait_loss())
    losses.append(mlp.wait_loss())
    return [np.array(losses)] + _weights(state)


def work(case):
    if case["kind"] == "sgemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4.0 * (m * k + k * n + m * n), "flops": 2.0 * m * n * k}
    nf, batch, iters = _widths(case), case["batch"], case["iters"]
    params = sum(a * b for a, b in zip(nf, nf[1:]))
    # every step reads its batch and reads and writes the fp32 weights; the weights are read back once
    per_step = 4.0 * (batch * (nf[0] + nf[-1]) + 2 * params)
    return {"bytes": iters * per_step + 4.0 * params, "flops": iters * _step_flops(nf, batch)}


# Relative 2-norm distance of the outputs, four times the largest seen over two passes between the step
# with its GEMM sums in 64 bits and the same step with them in 32 bits, or as the device adds them
# (operands rounded at the same points). What the sums' order changes is which ReLU masks flip and
# which stores round the other way, and training carries that on: it grows with the size of the
# updates, hence the split by weight scale, and far less than this shows after a single step.
_REL = {
    "fan_in": {"fp32": 3e-4, "fp32tc": 1e-6, "tf32": 4e-5, "bf16": 2.5e-4},
    "he": {"fp32": 3e-4, "fp32tc": 5e-4, "tf32": 1e-3, "bf16": 3e-3},
    "reference": {"bf16": 2e-3},
}


def tolerance(case):
    if case["kind"] == "sgemm":  # a single sum: fp32 rounding, or the tensor core's truncating adds
        return {"rel": 3e-5, "max": 1e-4} if case["precision"] == "tf32" else {"rel": 3e-6, "max": 3e-5}
    rel = _REL[case["init"]][case["precision"]]
    return {"rel": rel / 16 if case["kind"] == "online" else rel}
