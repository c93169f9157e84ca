"""The work a user of this framework has it do, as cases that can be timed.

Five kinds of case:

* ``loop``    a training step's two calls on a GPU replica: push the local change, pull the shared values;
* ``table``   the same two calls on a table of named tensors (one shared arena, a dict of tensors on the caller's side);
* ``scales``  the per-tensor magnitudes of such a table;
* ``rounds``  sync rounds: every replica of a group adds an update and rounds carry the updates through rings in device
              memory, all replicas on one GPU, launched in the order in which frames travel (a kernel never waits for
              another);
* ``live``    two replicas with their engine threads running: an update, until it has arrived and nothing is on its way.
"""
from __future__ import annotations

import math
import socket

import numpy as np
import torch

import sharedtensor
from sharedtensor_b200 import _native
from sharedtensor_b200.parallel.local_wiring import connect_local, connect_mesh

EXAMPLE = 240                # the reference's 4 x 5 x 6 x 2 example tensor
CHAR_RNN = 3_320_385         # trainable parameters of the 2-layer, 512-wide char-RNN
HEADLINE = 100_000_000       # the headline benchmark's tensor
GPT2 = 124_439_808           # GPT-2 small
GPT2_SHAPE = {"vocab": 50257, "ctx": 1024, "width": 768, "layers": 12}


def listed() -> list[dict]:
    return [
        # the smallest tensor anybody shares: every microsecond is call and launch
        {"name": "loop_example", "kind": "loop", "n": EXAMPLE, "dtype": "float32", "push": "update", "offset": 0},
        # a small model in fp32, its size odd: addFromTensor of a delta, copyToTensor
        {"name": "loop_char_rnn", "kind": "loop", "n": CHAR_RNN, "dtype": "float32", "push": "delta", "offset": 0},
        # the headline tensor through the README's loop: pushUpdate(new, current), copyToTensor
        {"name": "loop_headline", "kind": "loop", "n": HEADLINE, "dtype": "float32", "push": "update", "offset": 0},
        # bf16 training over fp32 masters: addScaledBF16 of the gradient, copyToTensorBF16
        {"name": "loop_gpt2_bf16", "kind": "loop", "n": GPT2, "dtype": "bfloat16", "push": "delta", "offset": 0},
        # the same model handled as a dict of 148 tensors
        {"name": "table_gpt2", "kind": "table", **GPT2_SHAPE},
        # its per-tensor magnitudes, as a monitor reads them
        {"name": "scales_gpt2", "kind": "scales", **GPT2_SHAPE},
        # one tree edge, the smallest tensor of the size sweep: launch latency of a hop
        {"name": "pair_1ki", "kind": "rounds", "topology": "pair", "members": 2, "n": 1024, "bits": 8, "block": 32},
        # one tree edge in the reference's format, one sign bit per element, scales shared by larger blocks
        {"name": "pair_char_rnn_sign", "kind": "rounds", "topology": "pair", "members": 2, "n": CHAR_RNN, "bits": 1, "block": 256},
        # one tree edge of the headline tensor
        {"name": "pair_headline", "kind": "rounds", "topology": "pair", "members": 2, "n": HEADLINE, "bits": 8, "block": 32},
        # an inner node of the tree with all its three edges: what arrives on one is passed on over the others
        {"name": "hub_16m", "kind": "rounds", "topology": "star", "members": 4, "n": 16_000_003, "bits": 4, "block": 64},
        # the eight-GPU mesh group of the headline benchmark: seven rings in, seven rings out
        {"name": "mesh8_4mi", "kind": "rounds", "topology": "mesh", "members": 8, "n": 4 * 1024 * 1024, "bits": 8, "block": 32},
        # the default, free-running engine: how long one update takes until both ends are quiet again
        {"name": "live_1mi", "kind": "live", "n": 1024 * 1024, "bits": 8, "block": 32},
    ]


def _log_between(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["loop", "loop", "rounds", "rounds", "rounds", "table", "scales", "live"])
    if kind == "loop":
        dtype, push = rng.choice([("float32", "update"), ("float32", "delta"), ("bfloat16", "delta")])
        return {"kind": kind, "n": _log_between(rng, EXAMPLE, GPT2), "dtype": dtype, "push": push, "offset": rng.choice([0, 0, 0, 1])}  # 1: a slice at an odd element
    if kind in ("table", "scales"):
        return {"kind": kind, "vocab": _log_between(rng, 65, 50257), "ctx": _log_between(rng, 50, 1024),
                "width": _log_between(rng, 33, 768), "layers": rng.randint(1, 12)}
    if kind == "live":
        return {"kind": kind, "n": _log_between(rng, 1024, 16 * 1024 * 1024), "bits": rng.choice([1, 8, 8]), "block": 32}
    topology = rng.choice(["pair", "pair", "star", "mesh"])
    members = {"pair": 2, "star": rng.randint(3, 4), "mesh": rng.randint(3, 8)}[topology]
    most = {"pair": HEADLINE, "star": 32_000_000, "mesh": 32_000_000 // members}[topology]
    return {"kind": kind, "topology": topology, "members": members, "n": _log_between(rng, 1024, most),
            "bits": rng.choice([1, 2, 4, 8, 8, 8]), "block": rng.choice([32, 32, 32, 64, 256, 1024, 4096])}


# ---------------------------------------------------------------------------------------------
# what a user's program holds before the call
# ---------------------------------------------------------------------------------------------
def _port() -> int:
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _table_shapes(case: dict) -> dict[str, torch.Size]:
    d = case["width"]
    layer = {"ln1.w": (d,), "ln1.b": (d,), "qkv.w": (3 * d, d), "qkv.b": (3 * d,), "proj.w": (d, d), "proj.b": (d,),
             "ln2.w": (d,), "ln2.b": (d,), "fc.w": (4 * d, d), "fc.b": (4 * d,), "out.w": (d, 4 * d), "out.b": (d,)}
    shapes = {"tok": (case["vocab"], d), "pos": (case["ctx"], d)}
    for i in range(case["layers"]):
        shapes.update({f"h{i}.{k}": v for k, v in layer.items()})
    shapes.update({"lnf.w": (d,), "lnf.b": (d,)})
    return {k: torch.Size(v) for k, v in shapes.items()}


def _normal(n: int, std: float, gen: torch.Generator, dtype=torch.float32, offset: int = 0) -> torch.Tensor:
    """n samples of N(0, std); `offset`: the tensor starts that many elements into its storage."""
    t = torch.empty(n + offset, device="cuda", dtype=torch.float32).normal_(0.0, std, generator=gen).to(dtype)
    return t[offset:]


def _named(flat: torch.Tensor, shapes: dict[str, torch.Size]) -> dict[str, torch.Tensor]:
    """Tensors of the given shapes in one buffer of the caller's, last one first (the order gradient buckets have)."""
    out, off = {}, 0
    for k in reversed(list(shapes)):
        out[k] = flat[off: off + shapes[k].numel()].view(shapes[k])
        off += shapes[k].numel()
    return {k: out[k] for k in shapes}


class _Values:
    """The values of a replica as a tensor on its memory."""

    def __init__(self, rep, n: int):
        self.rep = rep
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (rep.values_ptr(), False), "version": 3}


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "loop":
        n, dtype, off = case["n"], getattr(torch, case["dtype"]), case["offset"]
        st = sharedtensor.createOrFetch("127.0.0.1", _port(), _normal(n, 1.0, gen))
        s = {"kind": kind, "st": st, "push": case["push"], "bf16": dtype == torch.bfloat16,
             "cur": torch.empty(n + off, device="cuda", dtype=dtype)[off:],
             "delta": _normal(n, 0.1 if dtype == torch.bfloat16 else 1e-3, gen, dtype, off)}  # bf16: a gradient, scaled by -lr
        if case["push"] == "update" and not s["bf16"]:
            s["old"] = _normal(n, 1.0, gen, offset=off)
            s["new"] = (torch.empty(n + off, device="cuda")[off:]).copy_(s["old"] + s["delta"])
        return s
    if kind in ("table", "scales"):
        shapes = _table_shapes(case)
        n = sum(v.numel() for v in shapes.values())
        init = _named(_normal(n, 1.0, gen), shapes)
        for i, t in enumerate(init.values()):  # tensors of different magnitudes, as a model's are
            t.mul_(2.0 ** -(i % 9))
        tab = sharedtensor.createOrFetchTable("127.0.0.1", _port(), init)
        if kind == "scales":
            return {"kind": kind, "tab": tab, "flat": tab.copyToFlat(tab.new_flat())}
        params, grads = torch.empty(n, device="cuda"), _normal(n, 1e-3, gen)
        return {"kind": kind, "tab": tab, "params": params, "out": _named(params, shapes), "deltas": _named(grads, shapes)}
    n = case["n"]
    if kind == "live":
        opts = {"bits": case["bits"], "scale_mode": f"block{case['block']}", "rejoin": False}
        port = _port()
        init = _normal(n, 1.0, gen)
        parent = sharedtensor.createOrFetch("127.0.0.1", port, init, **opts)
        child = sharedtensor.createOrFetch("127.0.0.1", port, torch.zeros_like(init), **opts)
        return {"kind": kind, "child": child, "parent": parent, "delta": _normal(n, 1e-3, gen), "cur": torch.empty(n, device="cuda")}
    cu = _native.cuda()
    cfg = cu.GpuConfig()
    cfg.bits, cfg.block = case["bits"], case["block"]
    m = case["members"]
    reps = [cu.GpuReplica(torch.cuda.current_device(), n, cfg) for _ in range(m)]
    if case["topology"] == "mesh":
        connect_mesh(reps)
        order = [[i] for i in range(m)] * 2                             # every member speaks, then every member hears the rest
    elif case["topology"] == "star":
        for leaf in reps[1:]:
            connect_local(reps[0], leaf)
        order = [list(range(1, m)), [0], list(range(1, m))]             # leaves to hub, hub to leaves, leaves
    else:
        connect_local(reps[0], reps[1])
        order = [[0], [1], [0]]
    init = _normal(n, 1.0, gen)
    here = torch.cuda.current_stream().cuda_stream
    for r in reps:  # all replicas hold the initial state and every edge knows it
        r.load_values(init.data_ptr(), here)
        for link in range(r.n_links()):
            r.copy_mirror_from_values(link)
    torch.cuda.synchronize()
    return {"kind": kind, "reps": reps, "order": order, "deltas": [_normal(n, 1e-3, gen) for _ in reps],
            "streams": [torch.cuda.ExternalStream(r.comm_stream()) for r in reps], "events": [torch.cuda.Event() for _ in reps],
            "values": [torch.as_tensor(_Values(r, n), device="cuda") for r in reps]}


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _run_rounds(s: dict) -> list:
    reps, streams, events = s["reps"], s["streams"], s["events"]
    for r, d in zip(reps, s["deltas"]):
        r.add(d.data_ptr(), r.comm_stream())
    before = s["order"][-1]
    for phase in s["order"]:
        for i in before:
            events[i].record(streams[i])
        for j in phase:
            for i in before:
                if i != j:
                    streams[j].wait_event(events[i])
            reps[j].round()
        before = phase
    return s["values"]


def run(s: dict):
    kind = s["kind"]
    if kind == "rounds":
        return _run_rounds(s)
    if kind == "loop":
        st = s["st"]
        if s["bf16"]:
            st.addScaledBF16(s["delta"], -0.3)
            return st.copyToTensorBF16(s["cur"])
        if s["push"] == "update":
            st.pushUpdate(s["new"], s["old"])
        else:
            st.addFromTensor(s["delta"])
        return st.copyToTensor(s["cur"])
    if kind == "table":
        s["tab"].addFromTensors(s["deltas"])
        s["tab"].copyToTensors(s["out"])
        return s["params"]
    if kind == "scales":
        got = s["tab"].scales(s["flat"])
        return {"sumsq": np.array([v["sumsq"] for v in got.values()]), "rms_exp": np.array([v["rms_exp"] for v in got.values()])}
    s["parent"].addFromTensor(s["delta"])
    quiet = s["parent"].flush() and s["child"].flush()
    return [s["child"].copyToTensor(s["cur"]), quiet]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# ---------------------------------------------------------------------------------------------
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "loop":
        if case["dtype"] == "bfloat16":
            per = 10 + 6               # add: bf16 in, values in and out; pull: values in, bf16 out
        else:
            per = (16 if case["push"] == "update" else 12) + 8
        return {"bytes": per * case["n"], "flops": 2 * case["n"]}
    if kind in ("table", "scales"):
        n = sum(v.numel() for v in _table_shapes(case).values())
        return {"bytes": (20 if kind == "table" else 4) * n, "flops": 2 * n}
    n, frame = case["n"], case["bits"] / 8 + 1 / case["block"]
    if kind == "live":                 # add; frame made (values, mirror) and taken (values, mirror); pull
        return {"bytes": (12 + 12 + 16 + 8 + 2 * frame) * n, "flops": 10 * n}
    m = case["members"]
    # a visit of a replica: values read, and written where something arrived; every mirror read and written; frames
    if case["topology"] == "mesh":     # a pass that speaks (and hears), a pass that hears the rest
        per = m * (12 + 2 * 16 + 2 * (m - 1) * frame)
    elif case["topology"] == "star":   # leaves speak, the hub hears and passes on, the leaves hear
        k = m - 1
        per = m * 12 + k * (12 + frame) + (8 + k * 8 + 2 * k * frame) + k * (16 + frame)
    else:                              # one speaks, the other hears and speaks, the first hears
        per = 2 * 12 + (12 + frame) + (16 + 2 * frame) + (16 + frame)
    return {"bytes": per * n, "flops": 10 * per / 4 * n}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "scales":
        return {"rel": 1e-9, "differ": 0.01}   # fp64 sums; an exponent may tie
    if kind == "loop" and case["dtype"] == "bfloat16":
        return {"rel": 2e-3}                   # fp32 values rounded to bf16: a last-bit difference of a few elements
    return {"rel": 1e-5}                       # fp32 sums
