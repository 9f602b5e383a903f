"""The work a user of this framework has it do, as timed cases.

One mixture-of-experts FFN layer on quantized GGUF blocks is the unit of everything here (`CudaBackend.moe_ffn`).
A program runs it in three ways, and a case is one of them:

  op     one un-recorded call on rows that are in device memory: `moe_ffn(op)`.  A prompt chunk, or a decode step of
         a host that launches every op itself.
  stack  the MoE sub-layers of one decode step, norm and residual add inside (`MoeStack`), recorded once and replayed.
  host   decode steps of a host whose rows start and end in its own memory: a host-paced plan (recorded once, launched
         once per run of steps, each step released by a ticket).

Shapes are those of the benchmark's configurations and tests: hidden 2048 with 128 experts of 768 or 256 of 512
(+ shared expert), hidden 7168 with 256 experts of 2048 in groups; the drawn cases add plain sizes around them.  Values
follow the same configurations: random blocks with f16 scales of U[1e-4, 1e-3], router N(0, 0.02), activations N(0, 1),
and for prompt chunks the Zipf(1.1) expert popularity of the prefill configuration.
"""
import dataclasses
import math

import torch

from moe4all_b200 import CudaBackend, DType, MoeFfn
from moe4all_b200.devgen import BLOCKS, DeviceLayer
from moe4all_b200.stack import MoeStack

FORMATS = {"q4k": 12, "q5k": 13, "q6k": 14, "q8_0": 8, "q4_0": 2, "iq4_xs": 23, "mxfp4": 39}

# (hidden, experts, used, expert width, shared-expert width, sigmoid-gated shared expert, gating, groups, groups used)
SMALL = dict(ne=2048, n_expert=128, n_used=8, n_ff=768, sh_ff=0, gated=False, gating=0, groups=0, groups_used=0)
WIDE = dict(ne=2048, n_expert=256, n_used=8, n_ff=512, sh_ff=512, gated=True, gating=0, groups=0, groups_used=0)
BIG = dict(ne=7168, n_expert=256, n_used=8, n_ff=2048, sh_ff=2048, gated=False, gating=1, groups=8, groups_used=4)

# A sub-layer's norm weight: small, so that the sub-layer adds a fraction of the residual stream to it, as in a trained
# model, and not hundreds of times its size; the routers of a stack are scaled up by as much.
NORM_SCALE = 0.04


def case(kind, shape, rows, layers=1, steps=1, zipf=0.0, norm=False, banks="q4k,q4k,q6k", name=None):
    c = dict(kind=kind, rows=rows, layers=layers, steps=steps, zipf=zipf, norm=norm, banks=banks, **shape)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One token through one layer, launched op by op: the smallest call there is.
        case("op", SMALL, 1, name="op_1row"),
        # Single-stream decode, the headline: a replayed step through 8 layers, whose 4 GB of weights are cold in L2.
        case("stack", WIDE, 1, layers=8, name="stack_1stream"),
        # A few concurrent streams.
        case("stack", WIDE, 4, layers=8, name="stack_4streams"),
        # A full decode batch: every expert of a layer is hit by some row.
        case("stack", WIDE, 32, layers=8, name="stack_32streams"),
        # Chat with the sampling loop on the host: a token's rows come from host memory and its result returns there.
        case("host", WIDE, 1, layers=4, steps=16, name="host_16steps"),
        # An odd batch (a speculative window, a ragged tail) on the other kind of layer of a Q4_K_M file: Q4_K down banks.
        case("op", WIDE, 13, banks="q4k,q4k,q4k", name="op_13rows_q4k"),
        # A layer of experts of 28 MB at a decode batch of 64, experts chosen within groups.
        case("op", BIG, 64, name="big_64rows"),
        # The ragged last chunk of a prompt, with the norm and the residual add inside the call.
        case("op", WIDE, 777, zipf=1.1, norm=True, name="prompt_777"),
        # The prefill configuration: a 4096-token chunk with skewed expert popularity.
        case("op", WIDE, 4096, zipf=1.1, name="prompt_4096"),
        # The largest: 8192 tokens through the layer of 28 MB experts.
        case("op", BIG, 8192, name="big_prompt_8192"),
        # A Q5_K_M file: Q5_K gate and up with Q6_K down, two streams of decode ...
        case("stack", WIDE, 2, layers=4, banks="q5k,q5k,q6k", name="stack_2streams_q5k"),
        # ... and a prompt chunk of the Q8_0 file of the same model.
        case("op", WIDE, 1024, zipf=1.1, banks="q8_0,q8_0,q8_0", name="prompt_1024_q8"),
    ]


def _expert_bytes(c):
    g, u, d = (FORMATS[b] for b in c["banks"].split(","))
    per = lambda dt, n: n // BLOCKS[dt][0] * BLOCKS[dt][1]
    return c["n_ff"] * (per(g, c["ne"]) + per(u, c["ne"])) + c["ne"] * per(d, c["n_ff"])


def draw(rng):
    rows_to = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    most = work(case("op", BIG, 8192))
    while True:
        if rng.random() < 0.5:
            shape = dict(rng.choice([SMALL, WIDE, WIDE, BIG]))
        else:
            n_expert = rng.choice([32, 64, 96, 128, 160, 256])
            n_ff = 256 * rng.choice([1, 2, 3, 4, 6])
            shape = dict(ne=256 * rng.choice([4, 6, 8, 10, 12, 16]), n_expert=n_expert, n_used=rng.choice([2, 4, 6, 8]), n_ff=n_ff,
                         sh_ff=rng.choice([0, n_ff]), gated=rng.random() < 0.5, gating=rng.choice([0, 0, 1]), groups=0, groups_used=0)
        banks = rng.choice(["q4k,q4k,q6k"] * 6 + ["q4k,q4k,q4k"] * 3 + ["q5k,q5k,q6k", "q8_0,q8_0,q8_0", rng.choice(["q4_0,q4_0,q4_0", "iq4_xs,iq4_xs,q6k", "mxfp4,mxfp4,mxfp4"])])
        kind = rng.choice(["op", "op", "op", "stack", "stack", "host"])
        if kind == "op":
            rows = rows_to(1, 8192)
            c = case(kind, shape, rows, zipf=1.1 if rows >= 256 and not shape["groups"] else 0.0, norm=rng.random() < 0.5, banks=banks)
        elif kind == "stack":
            c = case(kind, shape, rows_to(1, 64), layers=rows_to(2, 8), banks=banks)
        else:
            c = case(kind, shape, rows_to(1, 8), layers=rng.choice([2, 4]), steps=rows_to(4, 32), banks=banks)
        w = work(c)
        held = c["layers"] * c["n_expert"] * _expert_bytes(c)
        if held <= 8e9 and w["bytes"] <= most["bytes"] and w["flops"] <= most["flops"]:
            return c


_backend = []


def backend():
    """The program's one backend: device, stream and scratch."""
    if not _backend:
        _backend.append(CudaBackend(0))
    return _backend[0]


def _layer(be, c, seed):
    """One layer's weights, and its selection bias where experts are chosen within groups."""
    d = DeviceLayer(be, seed, c["ne"], c["n_expert"], c["n_ff"], sh_ff=c["sh_ff"], gated_shared=c["gated"],
                    router_std=0.02 / NORM_SCALE if c["kind"] == "stack" else 0.02, dtypes=tuple(FORMATS[b] for b in c["banks"].split(",")))
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    if c["zipf"]:
        # popularity in the router's last column, for rows whose last element is 1
        order = torch.randperm(c["n_expert"], generator=gen, device="cuda")
        d.t["router"][:-16].view(torch.float32).view(c["n_expert"], c["ne"])[:, -1] = -c["zipf"] * torch.log((order + 1).float())
    if c["groups"]:
        d.bias = torch.randn(c["n_expert"], generator=gen, device="cuda") * 0.05
    return d


def _route_kw(be, c, d):
    g, u, dn = (DType(FORMATS[b]) for b in c["banks"].split(","))
    kw = dict(gating=c["gating"], gate_dtype=g, up_dtype=u, down_dtype=dn)
    if c["groups"]:
        kw.update(scale=2.5, n_expert_groups=c["groups"], n_expert_groups_used=c["groups_used"], exp_probs_b=be.wrap_tensor(d.bias))
    return kw


def _op(be, c, d, x, dst, **kw):
    b = d.b
    return MoeFfn(x=x, router=b["router"], gate_exps=b["gate"], up_exps=b["up"], down_exps=b["down"], dst=dst, rows=c["rows"], ne=c["ne"],
                  n_expert=c["n_expert"], n_used=c["n_used"], n_ff_exp=c["n_ff"], sh_gate=b.get("sh_gate"), sh_up=b.get("sh_up"),
                  sh_down=b.get("sh_down"), sh_gate_inp=b.get("sh_gate_inp"), sh_ff=c["sh_ff"], **_route_kw(be, c, d), **kw)


def prepare(c, seed):
    be = backend()
    rows, ne, k = c["rows"], c["ne"], c["n_used"]
    gen = torch.Generator(device="cuda").manual_seed(seed * 1009 + 7)
    layers = [_layer(be, c, seed * 1009 + 16 * i + 11) for i in range(c["layers"])]
    s = {"c": c, "be": be, "layers": layers}
    if c["kind"] == "host":
        _prepare_host(s, gen)
        return s
    s["x"] = torch.randn(rows, ne, generator=gen, device="cuda")
    if c["zipf"]:
        s["x"][:, -1] = 1.0
    x = be.wrap_tensor(s["x"])
    if c["kind"] == "op":
        s["out"] = {"dst": torch.zeros(rows, ne, device="cuda"), "ids": torch.zeros(rows, k, dtype=torch.int32, device="cuda"),
                    "wts": torch.zeros(rows, k, device="cuda")}
        o = {name: be.wrap_tensor(t) for name, t in s["out"].items()}
        kw = {}
        if c["norm"]:
            s["norm"] = 1.0 + 0.1 * torch.randn(ne, generator=gen, device="cuda")
            kw = dict(norm_weight=be.wrap_tensor(s["norm"]), residual=x)
        torch.cuda.synchronize()
        s["op"] = _op(be, c, layers[0], x, o["dst"], ids_out=o["ids"], wts_out=o["wts"], **kw)
        return s
    norms = [NORM_SCALE * (1.0 + 0.1 * torch.randn(ne, generator=gen, device="cuda")) for _ in layers]
    torch.cuda.synchronize()
    st = MoeStack(be, layers, norms, rows, ne, c["n_expert"], k, c["n_ff"], sh_ff=c["sh_ff"])
    for i, d in enumerate(layers):
        st.ops[i] = dataclasses.replace(st.ops[i], **_route_kw(be, c, d))
    # the first layer reads the step's rows where the caller has them; the others work on the stack's own rows
    st.ops[0] = dataclasses.replace(st.ops[0], x=x, residual=x)
    st.record()
    be.sync()
    s["stack"] = st
    return s


def _prepare_host(s, gen):
    """Steps that rotate over the layers' weights, each from pinned rows to pinned results, recorded as one plan."""
    c, be = s["c"], s["be"]
    rows, ne, steps = c["rows"], c["ne"], c["steps"]
    nbytes = rows * ne * 4
    s["rows"] = torch.randn(steps, rows, ne, generator=gen, device="cuda").cpu()
    s["stage"], s["last"] = torch.empty(rows, ne).pin_memory(), torch.empty(rows, ne).pin_memory()
    s["out"] = torch.zeros(steps, rows, ne)
    torch.cuda.synchronize()
    x_in, dst = be.alloc(nbytes), be.wrap(s["last"].data_ptr(), nbytes)  # the last kernel of a step writes host memory itself
    ops = [_op(be, c, d, x_in, dst) for d in s["layers"]]
    be.moe_ffn(ops[0])
    be.sync()
    be.graph_begin()
    for i in range(steps):
        be.upload_ptr_gated(x_in, s["stage"].data_ptr(), nbytes, i + 1)
        be.moe_ffn(ops[i % len(ops)])
        be.host_signal(i + 1)
    s["plan"] = be.graph_end()
    s["keep"] = (x_in, dst, ops)
    s["in_ptrs"] = [s["rows"][i].data_ptr() for i in range(steps)]
    s["out_ptrs"] = [s["out"][i].data_ptr() for i in range(steps)]


def run(s):
    c, be = s["c"], s["be"]
    if c["kind"] == "op":
        be.moe_ffn(s["op"])
        return s["out"]
    if c["kind"] == "stack":
        s["stack"].replay()
        return s["stack"].hidden
    nbytes = c["rows"] * c["ne"] * 4
    be.host_reset()
    be.execute(s["plan"])
    be.host_steps(1, s["stage"].data_ptr(), s["in_ptrs"], nbytes, s["last"].data_ptr(), s["out_ptrs"], nbytes)
    return s["out"]


def work(c):
    """The distinct experts' blocks, the router and the rows, each once; a call of many rows hits nearly every expert."""
    rows, ne, E, k, ff = c["rows"], c["ne"], c["n_expert"], c["n_used"], c["n_ff"]
    distinct = E * (1.0 - (1.0 - k / E) ** rows)
    shared = c["sh_ff"] / ff
    nbytes = (distinct + shared) * _expert_bytes(c) + E * ne * 4 + 2 * rows * ne * 4
    flops = 6 * rows * ne * (k * ff + c["sh_ff"]) + 2 * rows * E * ne
    n = c["steps"] if c["kind"] == "host" else c["layers"]
    return {"bytes": n * nbytes, "flops": n * flops}


def tolerance(c):
    # Expert ids are whole numbers and have to agree.  The operands of the expert products are 16-bit (fixed-point or
    # f16 activations, f16 weights on the tensor cores): a few 1e-4 of a layer's result.
    if c["kind"] != "stack":
        return {"rel": 1e-3, "max": 2e-2, "differ": 0.0}
    # In a chain of layers that difference can change which of two nearly equal experts a row takes one layer later.
    return {"rel": 1e-2, "max": 0.5, "differ": 0.0}
