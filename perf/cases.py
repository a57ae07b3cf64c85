"""Workloads by which the speed of this framework is judged, through its public entry points.

A case is a dict of plain values:

  kind     decode          one token for every sequence, recurrent_gdn2 with the state updated in place
           first_token     one token with no state yet (the closed form), recurrent_gdn2
           short           a few tokens that follow a state (a speculative draft, a short turn), recurrent_gdn2
           prefill         chunk_gdn2 without gradients
           packed_prefill  prompts of several lengths packed along time, chunk_gdn2_varlen without gradients
           train           chunk_gdn2 and the gradients of every input
           packed_train    the same for packed sequences, chunk_gdn2_varlen
  batch, time, heads       sizes (head dimension 128 everywhere); packed kinds have lengths ("12,300,77") instead
  dtype    type of q, k, v, beta, w and the output: bf16 or fp16
  g        type of the log-decay: fp32, or "same" as the others
  raw      True: q, k are raw projections and beta, w, g pre-activations, the operator applies the layer's
           input prologue (L2 normalisation, sigmoid, -softplus) itself
  state    True: an initial state is given, and for training the final state has a cotangent too

Inputs follow the distributions of the benchmark: q, k normalised N(0, 1), v N(0, 1), beta and w
sigmoid(N(0, 1)), g = -clamp(softplus(N(-2, 1)), 5), states 0.02 N(0, 1).
"""

import math

import torch

from gdn2_sm120_b200 import chunk_gdn2, recurrent_gdn2
from gdn2_sm120_b200.varlen import chunk_gdn2_varlen

DIM = 128
STATE = DIM * DIM
TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# largest number of (batch, token, head) rows of a case that goes through whole sequences
MAX_ROWS = 4 * 8192 * 32


def _case(name, kind, heads, *, batch=1, time=1, lengths="", dtype="bf16", g="fp32", raw=False, state=True):
    case = {"kind": kind, "heads": heads, "dtype": dtype, "g": g, "raw": raw, "state": state}
    if lengths:
        case["lengths"] = lengths
    else:
        case["batch"], case["time"] = batch, time
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # one user's interactive decoding: nothing but latency
        _case("decode_b1_h16", "decode", 16, batch=1),
        # a serving step of a full batch, the decode configuration of the benchmark
        _case("decode_b64_h32", "decode", 32, batch=64),
        # the first token of 256 new sequences, the benchmark's zero-state configuration
        _case("first_token_b256_h32", "first_token", 32, batch=256, state=False),
        # a short turn on running sequences whose layer hands over raw projections
        _case("short_b4_t32_h16_raw", "short", 16, batch=4, time=32, raw=True),
        # the prefill configuration of the benchmark: continued prompts, final states kept
        _case("prefill_b8_t4096_h16", "prefill", 16, batch=8, time=4096),
        # one long document, the longest single sequence of the benchmark grid, raw projections
        _case("prefill_b1_t32768_h16_raw", "prefill", 16, batch=1, time=32768, raw=True, state=False),
        # a serving engine's prefill step: prompts of mixed lengths, many of them short
        _case("packed_prefill_n16_h16", "packed_prefill", 16, state=False,
              lengths="1371,87,412,2048,33,725,166,940,64,517,1203,290,7,655,1818,256"),
        # training on short texts: below the length of one tensor-core chunk
        _case("train_b16_t48_h16", "train", 16, batch=16, time=48, state=False),
        # one sequence per GPU, a common fine-tuning step
        _case("train_b1_t2048_h16", "train", 16, batch=1, time=2048, state=False),
        # a length that is no multiple of anything, fp16, the layer's prologue in the operator
        _case("train_b2_t4133_h16_fp16_raw", "train", 16, batch=2, time=4133, dtype="fp16", raw=True, state=False),
        # documents packed into one row of 8192 tokens
        _case("packed_train_n8_h16", "packed_train", 16, state=False, lengths="911,2300,150,1640,77,1202,514,1398"),
        # the training configuration of the benchmark, state in and out: the largest
        _case("train_b4_t8192_h32", "train", 32, batch=4, time=8192),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("decode", "first_token", "short", "prefill", "packed_prefill", "train", "train", "packed_train"))
    heads = rng.choice((2, 4, 6, 8, 12, 16, 20, 24, 32))
    options = {
        "dtype": rng.choice(("bf16", "bf16", "bf16", "fp16")),
        "g": rng.choice(("fp32", "fp32", "fp32", "same")),
        "raw": rng.random() < 0.35,
        "state": rng.random() < 0.5,
    }
    if kind in ("decode", "first_token", "short"):
        options["state"] = kind != "first_token"
        batch = _log_int(rng, 1, 256 if kind != "short" else 32)
        return _case("", kind, heads, batch=batch, time=_log_int(rng, 2, 63) if kind == "short" else 1, **options)
    if kind in ("packed_prefill", "packed_train"):
        sequences = _log_int(rng, 2, 32)
        longest = _log_int(rng, 64, 4096)
        lengths, room = [], min(16384, MAX_ROWS // heads)
        for _ in range(sequences):
            length = min(room, rng.randint(1, longest))
            if length:
                lengths.append(length)
            room -= length
        return _case("", kind, heads, lengths=",".join(str(x) for x in lengths), **options)
    time = _log_int(rng, 64, 32768) if kind == "prefill" else _log_int(rng, 8, 16384)
    batch = _log_int(rng, 1, max(1, min(16, MAX_ROWS // (heads * time))))
    return _case("", kind, heads, batch=batch, time=time, **options)


def _lengths(case):
    return [int(x) for x in case["lengths"].split(",")] if "lengths" in case else [case["time"]] * case["batch"]


def prepare(case, seed):
    dtype = TYPES[case["dtype"]]
    g_dtype = torch.float32 if case["g"] == "fp32" else dtype
    lengths, heads = _lengths(case), case["heads"]
    packed = "lengths" in case
    batch, time = (1, sum(lengths)) if packed else (case["batch"], case["time"])
    generator = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, device="cuda", generator=generator)

    shape = (batch, time, heads, DIM)
    q, k, v = normal(*shape), normal(*shape), normal(*shape)
    beta, w, g = normal(*shape), normal(*shape), normal(*shape) - 2.0
    if not case["raw"]:
        q, k = torch.nn.functional.normalize(q, dim=-1), torch.nn.functional.normalize(k, dim=-1)
        beta, w = torch.sigmoid(beta), torch.sigmoid(w)
        g = -torch.nn.functional.softplus(g).clamp(max=5.0)
    inputs = [q.to(dtype), k.to(dtype), v.to(dtype), g.to(g_dtype), beta.to(dtype), w.to(dtype)]
    made = {"kind": case["kind"], "inputs": inputs, "initial": None}
    states = len(lengths) if packed else batch
    if case["state"]:
        made["initial"] = 0.02 * normal(states, heads, DIM, DIM)
    if packed:
        ends = [0]
        for length in lengths:
            ends.append(ends[-1] + length)
        made["cu_seqlens"] = torch.tensor(ends, dtype=torch.int32)  # read on the host by the operator
    if case["kind"] in ("train", "packed_train"):
        for x in inputs:
            x.requires_grad_(True)
        made["d_out"] = normal(*shape).to(dtype)
        if case["state"]:
            made["initial"].requires_grad_(True)
            made["d_final"] = normal(states, heads, DIM, DIM)
    made["flags"] = {"use_qk_l2norm_in_kernel": case["raw"], "use_gate_in_kernel": case["raw"]}
    return made


def run(state):
    kind, inputs, initial, flags = state["kind"], state["inputs"], state["initial"], state["flags"]
    if kind == "decode":
        return recurrent_gdn2(*inputs, initial, inplace_final_state=True, **flags)
    if kind in ("first_token", "short"):
        return recurrent_gdn2(*inputs, initial, **flags)
    if kind == "prefill":
        return chunk_gdn2(*inputs, initial, output_final_state=True, **flags)
    if kind == "packed_prefill":
        return chunk_gdn2_varlen(*inputs, state["cu_seqlens"], initial, output_final_state=True, **flags)
    with_state = initial is not None
    if kind == "train":
        out, final = chunk_gdn2(*inputs, initial, output_final_state=with_state, **flags)
    else:
        out, final = chunk_gdn2_varlen(*inputs, state["cu_seqlens"], initial, output_final_state=with_state, **flags)
    if with_state:
        return [out, final, *torch.autograd.grad([out, final], [*inputs, initial], [state["d_out"], state["d_final"]])]
    return [out, *torch.autograd.grad(out, inputs, state["d_out"])]


def work(case):
    lengths, heads = _lengths(case), case["heads"]
    rows = sum(lengths) * heads
    units = len(lengths) * heads
    train = case["kind"] in ("train", "packed_train")
    g_bytes = DIM * (4 if case["g"] == "fp32" else 2)
    if case["kind"] == "first_token":  # neither the gate of an empty state nor its decay matters
        return {"bytes": rows * 5 * 2 * DIM + units * 4 * STATE, "flops": units * 2 * STATE}
    inputs = 5 * 2 * DIM + g_bytes
    moved = rows * (inputs + 2 * DIM)                      # forward: inputs and the output
    if train:
        moved += rows * (inputs + 2 * DIM + inputs)        # backward: inputs, output cotangent, six gradients
        if case["state"]:
            moved += units * 4 * STATE * 4                 # initial and final state, and their cotangents
    else:
        moved += units * 4 * STATE * (2 if case["state"] else 1)
    # decay, erase, write and read of the state: 3 multiply-adds of 128 x 128 per token and direction
    return {"bytes": moved, "flops": rows * 6 * STATE * (3 if train else 1)}


def tolerance(case):
    longest = max(_lengths(case))
    if longest < 64:
        # exact fp32 recurrence: what is left is a 16-bit result that rounds to the neighbouring value
        return {"rel": 2e-3, "max": 2e-2}
    # tensor-core products of tf32 operands, 16-bit outputs and gradients
    return {"rel": 6e-3}
