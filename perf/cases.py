"""The work that users of this package have it do, as measurable cases.

A case is a dict of plain values:

``op``              ``"scan"`` (:func:`scan_cu` for bf16, :func:`scan_cu_single` for fp32) or ``"gated"`` (:func:`scan_gated`)
``dtype``           ``"bf16"`` or ``"f32"``, the storage type; the state is fp32 in both
``batch, seq, width``  the tensors' shape ``[B, T, D]``
``gates``           the distribution of alpha (``workloads.make_inputs``); ``"gated"`` cases draw the raw gate activations
``grad``            a training step (forward, then the gradients of every input) or a forward alone under ``no_grad``
``state``           start from a given state ``h0`` and return the state after the last row (chunked prefill, decoding, truncated
                    back-propagation)
``reverse``         scan from the last row to the first (the second half of a bidirectional layer)
``mode``            ``backward_mode`` of the training step
``parts``           the tensors are one of ``parts`` slices of the channels of tensors that are this many times as wide (one
                    device's share of a layer that is split by channels); 1: tensors of their own
"""
import math

import torch

from fast_sequential_scan_b200 import scan_cu, scan_cu_single, scan_gated
from fast_sequential_scan_b200.workloads import Workload, make_gate_inputs, make_inputs


def _case(op="scan", dtype="bf16", gates="sigmoid", grad=True, state=False, reverse=False, mode="saved", parts=1, *, batch, seq, width,
          **more):
    return dict(more, op=op, dtype=dtype, gates=gates, grad=grad, state=state, reverse=reverse, mode=mode, parts=parts, batch=batch,
                seq=seq, width=width)


def listed():
    return [
        # one token for every sequence of a serving batch, the state carried from call to call: nothing but latency
        _case(name="decode", batch=16, seq=1, width=2560, gates="hawk", grad=False, state=True),
        # the smallest training step of the benchmark configurations
        _case(name="train_small", batch=2, seq=1024, width=768),
        # the headline training step
        _case(name="train", batch=8, seq=2048, width=1024),
        # a training step whose sequence length fits no tile
        _case(name="train_ragged", batch=4, seq=3000, width=2048, gates="uniform_0.5"),
        # a width that rows of 16 bytes do not divide: every row starts at another alignment
        _case(name="train_odd_width", batch=4, seq=1000, width=1001, gates="uniform_0.5"),
        # the backward-in-time half of a bidirectional layer
        _case(name="train_reverse", batch=4, seq=4096, width=2048, gates="uniform_0.5", reverse=True),
        # fp32 training at the size of a recurrent language model's layer
        _case(name="train_f32", batch=16, seq=4096, width=2560, gates="hawk", dtype="f32"),
        # long context: one device's 65,536 rows
        _case(name="train_long", batch=1, seq=65536, width=4096, gates="uniform_0.9"),
        # chunked prefill: a chunk of the prompt continues the state of the one before it
        _case(name="prefill", batch=4, seq=4096, width=2048, gates="uniform_0.5", grad=False, state=True),
        # prefill and training of a gated recurrent layer from its raw gate activations
        _case(name="gated_prefill", op="gated", batch=4, seq=1000, width=2048, gates="hawk", grad=False),
        _case(name="gated_train", op="gated", batch=16, seq=4096, width=2560, gates="hawk"),
        _case(name="gated_train_f32", op="gated", batch=4, seq=2048, width=2560, gates="hawk", dtype="f32"),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    dtype = rng.choice(["bf16", "bf16", "f32"])
    kind = rng.choice(["train", "train", "train", "odd", "reverse", "state", "prefill", "decode", "gated", "gated_prefill"])
    gates = rng.choice(["sigmoid", "uniform_0.5", "uniform_0.9", "hawk"])
    if kind == "decode":
        return _case(batch=_log_uniform(rng, 1, 128), seq=rng.choice([1, 1, 2, 4]), width=8 * _log_uniform(rng, 64, 640), gates="hawk",
                     dtype=dtype, grad=False, state=True, reverse=False)
    # elements of one tensor: from the small training step's to half of the largest case's
    elements = _log_uniform(rng, 1 << 20, 1 << 26)
    width = 8 * _log_uniform(rng, 16, 512)
    batch = max(1, min(_log_uniform(rng, 1, 32), elements // (64 * width)))
    seq = max(64, min(65536, elements // (batch * width)))
    if kind == "odd":
        return _case(batch=batch, seq=seq, width=width + rng.choice([1, 2, 3, 4, 5, 7]), gates=gates, dtype=dtype)
    if kind in ("gated", "gated_prefill"):
        return _case(op="gated", batch=batch, seq=seq, width=width, gates="hawk", dtype=dtype, grad=kind == "gated")
    if kind == "train":
        return _case(batch=batch, seq=seq, width=width, gates=gates, dtype=dtype, mode=rng.choice(["saved", "saved", "inplace", "recompute"]),
                     parts=rng.choice([1, 1, 2, 4]))
    return _case(batch=batch, seq=seq, width=width, gates=gates, dtype=dtype, grad=kind != "prefill",
                 state=kind != "reverse", reverse=kind == "reverse")


def _share(t, parts):
    """Slice number ``parts - 1`` of the channels of ``t``, as a view."""
    width = t.shape[2] // parts
    return t[:, :, (parts - 1) * width:]


def prepare(case, seed):
    shape = (case["batch"], case["seq"], case["width"] * case["parts"])
    w = Workload("case", *shape, case["gates"], case["dtype"])
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    if case["op"] == "gated":
        r, i, x, lam = make_gate_inputs(w, "cuda", seed)
        inputs = {"r": r, "i": i, "x": x, "lam": lam}
        grad = torch.randn(shape, generator=gen, device="cuda").to(w.torch_dtype) if case["grad"] else None
    else:
        a, b, grad = (_share(t, case["parts"]) for t in make_inputs(w, "cuda", seed))
        inputs = {"alpha": a, "beta": b}
        if case["state"]:
            inputs["h0"] = torch.randn((shape[0], shape[2]), generator=gen, device="cuda")
    last = torch.randn((shape[0], shape[2]), generator=gen, device="cuda") if case["state"] and case["grad"] else None
    if case["grad"]:
        inputs = {k: t.requires_grad_() for k, t in inputs.items()}
    return {"case": case, "inputs": inputs, "grad": grad if case["grad"] else None, "grad_last": last}


def _forward(case, inputs):
    if case["op"] == "gated":
        return scan_gated(inputs["r"], inputs["i"], inputs["x"], inputs["lam"])
    scan = scan_cu if case["dtype"] == "bf16" else scan_cu_single
    if case["state"]:
        return scan(inputs["alpha"], inputs["beta"], h0=inputs["h0"], return_final_state=True, reverse=case["reverse"])
    if case["reverse"]:
        return scan(inputs["alpha"], inputs["beta"], reverse=True)
    if case["mode"] != "saved":
        return scan(inputs["alpha"], inputs["beta"], backward_mode=case["mode"])
    return scan(inputs["alpha"], inputs["beta"])


def run(state):
    case, inputs = state["case"], state["inputs"]
    if not case["grad"]:
        with torch.no_grad():
            return _forward(case, inputs)
    out = _forward(case, inputs)
    outs, grads = (list(out), [state["grad"], state["grad_last"]]) if case["state"] else ([out], [state["grad"]])
    gradients = list(torch.autograd.grad(outs, list(inputs.values()), grads))
    # "inplace" writes the gradient of beta over h, which must not be read after the backward
    return gradients if case["mode"] == "inplace" else outs + gradients


def work(case):
    n = case["batch"] * case["seq"] * case["width"]
    size = 2 if case["dtype"] == "bf16" else 4
    # tensors: the scan reads alpha, beta and writes h, its backward reads alpha, h, the gradient of h and writes two gradients;
    # the gated scan reads r, i, x and writes h, its backward reads those, h and the gradient of h and writes three gradients
    forward, backward = (4, 8) if case["op"] == "gated" else (3, 5)
    vectors = 2 if case["state"] else 0
    flops = 2.0
    if case["op"] == "gated":
        flops += 12.0
    if case["grad"]:
        flops += 26.0 if case["op"] == "gated" else 3.0
        vectors *= 2
    tensors = forward + (backward if case["grad"] else 0)
    return {"bytes": float(tensors * n * size + 4 * vectors * case["batch"] * case["width"]), "flops": flops * n}


def tolerance(case):
    # About four times what the outputs of this package differ from the same formulas in 64 bits, measured over 257 and 2,048 rows of
    # every distribution: bf16 2.4e-3 (7.5e-3 at most for one value) for the scan, 4.9e-3 (4.4e-2) for the gated scan, whose gates are
    # rounded to bf16 before they are scanned; fp32 1.3e-7 (1.2e-6) and 6.0e-7 (9.3e-6).
    if case["dtype"] == "bf16":
        return {"rel": 2e-2, "max": 0.18} if case["op"] == "gated" else {"rel": 1e-2, "max": 0.03}
    return {"rel": 2.5e-6, "max": 4e-5} if case["op"] == "gated" else {"rel": 5e-7, "max": 5e-6}
