"""GPU tests of calls at the edge of what the entry points accept: buffers of the smallest documented alignment,
non-finite values, strong decays, flags that are no booleans, threads beside a blocked launch."""

from __future__ import annotations

import threading
import time

import numpy as np
import pytest
import torch

import gdn2_oracle as oracle
from gdn2_sm120_b200 import _lib, chunk_gdn2, chunk_kernels, recurrent_gdn2
from gdn2_sm120_b200.varlen import chunk_gdn2_varlen

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _at_offset(size, offset):
    """`size` bytes that start `offset` bytes past a 256-byte boundary."""

    base = torch.empty(size + 512, dtype=torch.uint8, device=DEV)
    skip = -base.data_ptr() % 256 + offset
    return base[skip:skip + size]


# (batch, time, heads): two launches; at 37 heads and 21 chunks prep and scan share one
@pytest.mark.parametrize("batch,time,heads", [(1, 130, 2), (1, 21 * 64, 37)])
@pytest.mark.parametrize("training", [False, True])
def test_chunk_forward_takes_buffers_aligned_to_16_bytes(batch, time, heads, training):
    q, k, v, g, beta, w, s0 = [t.to(DEV) for t in oracle.make_inputs(batch, time, heads, seed=time)]
    full = chunk_kernels.supported_tokens(time)
    sizes = (chunk_kernels.workspace_bytes(batch, full, heads, training),
             chunk_kernels.scratch_bytes(batch, full, heads, False, training=training))
    results = []
    for offset in (0, 16, 48):
        workspace, scratch = (_at_offset(size, offset) for size in sizes)
        assert workspace.data_ptr() % 32 == scratch.data_ptr() % 32 == offset % 32
        out, fin = torch.empty_like(v), torch.empty_like(s0)
        bnd = torch.empty(batch, full // 64 + 1, heads, 128, 128, device=DEV) if training else None
        _lib.call("gdn2_chunk_forward", q.device, *(t.data_ptr() for t in (q, k, v, g, beta, w, s0, out, fin)),
                  _lib.ptr(bnd), workspace.data_ptr(), scratch.data_ptr(), batch, time, heads, full, int(training),
                  _lib.dtype_code(q.dtype), _lib.dtype_code(g.dtype), 128 ** -0.5, _lib.stream_ptr(q.device))
        results.append((out, fin) if bnd is None else (out, fin, bnd))
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))


# Every term of dg_t holds exp(g_t): a product of at most 16 exponentials of 2 units in the last place each is
# right to 4e-6, the 16 x 16 solve and the sums over channels as much again: 1e-5 for each token.  "mixed": a
# third of the decays strong and the others weak; "zeroed": some decays are exactly zero, and so is their dg.
@pytest.mark.parametrize("decay", [-1.0, -5.0, -10.0, -15.0, -25.0, "mixed", "zeroed"])
@pytest.mark.parametrize("time", [1, 16, 17, 47])
def test_log_decay_gradients_of_short_sequences_at_any_decay(time, decay):
    batch, heads = 2, 2
    cpu = list(oracle.make_inputs(batch, time, heads, seed=time))
    gen = torch.Generator().manual_seed(time + 1)
    u, third = torch.rand(cpu[3].shape, generator=gen), torch.rand(cpu[3].shape, generator=gen) < 0.33
    if decay == "mixed":
        cpu[3] = torch.where(third, -20.0 * u, -0.05 * u)
    elif decay == "zeroed":
        cpu[3] = torch.where(third, torch.full_like(u, -float("inf")), -0.5 * u)
    else:
        cpu[3] = decay * (0.5 + u)
    d_out = torch.randn(cpu[2].shape, generator=gen).to(cpu[2].dtype)
    d_fin = torch.randn((batch, heads, 128, 128), generator=gen)
    _, _, ref = oracle.recurrence_grads(*cpu, d_out, d_fin)
    leaves = [t.to(DEV).requires_grad_(True) for t in cpu]
    out, fin = chunk_gdn2(*leaves[:6], leaves[6], output_final_state=True)
    dg = torch.autograd.grad([out, fin], leaves, [d_out.to(DEV), d_fin.to(DEV)])[3]
    if decay == "zeroed":
        assert (dg.cpu()[third] == 0).all()
    for t in range(time):
        err = oracle.rel_l2(dg[:, t], ref[3][:, t])
        assert err < 1e-5, f"token {t}: rel-L2 {err:.3e}"


RAW = {"use_qk_l2norm_in_kernel": True, "use_gate_in_kernel": True}


# -inf and the type's lowest value close a gate completely (sigmoid = 0): nothing is written, the state stays zero
@pytest.mark.parametrize("closed", [-float("inf"), torch.finfo(torch.bfloat16).min])
@pytest.mark.parametrize("time", [1, 5, 40, 64, 101])
def test_closed_gates_of_the_fused_prologue_write_nothing(time, closed):
    cpu = oracle.make_raw_inputs(1, time, 2, seed=time)
    q, k, v, g, beta, w = [t.to(DEV) for t in cpu[:6]]
    w[:, :, 1] = closed
    with torch.no_grad():
        out, fin = chunk_gdn2(q, k, v, g, beta, w, output_final_state=True, **RAW)
    assert (out[:, :, 1] == 0).all() and (fin[:, 1] == 0).all()
    assert (out[:, :, 0] != 0).any() and torch.isfinite(out).all()


# the first sequence ends inside a pair of tokens whose second one is the next sequence's
@pytest.mark.parametrize("first", [100, 101])
def test_a_nan_behind_the_end_of_a_packed_sequence_stays_there(first):
    cpu = oracle.make_raw_inputs(1, 200, 2, seed=first)
    seq = [t.to(DEV) for t in cpu[:6]]
    with torch.no_grad():
        expected, _ = chunk_gdn2_varlen(*seq, [0, first, 200], **RAW)
        for t in seq:
            t[0, first] = float("nan")
        out, _ = chunk_gdn2_varlen(*seq, [0, first, 200], **RAW)
    assert torch.equal(out[:, :first], expected[:, :first])


# spans of 16 tokens: in the middle of the only one, in the second, at the first token of one
@pytest.mark.parametrize("time,at", [(12, 5), (40, 20), (33, 16), (16, 15)])
@pytest.mark.parametrize("name,value", [("q", "nan"), ("k", "nan"), ("v", "inf"), ("g", "nan"), ("beta", "nan"), ("w", "nan")])
def test_outputs_do_not_depend_on_later_tokens(time, at, name, value):
    seq = dict(zip(("q", "k", "v", "g", "beta", "w"), [t.to(DEV) for t in oracle.make_inputs(2, time, 2, seed=time)]))
    with torch.no_grad():
        expected, _ = chunk_gdn2(*seq.values())
        seq[name][:, at, 1, 7] = float(value)
        out, _ = chunk_gdn2(*seq.values())
    assert torch.equal(out[:, :at], expected[:, :at]) and torch.equal(out[:, :, 0], expected[:, :, 0])
    assert not torch.isfinite(out[:, at, 1]).all()


@pytest.mark.parametrize("time", [1, 5, 64, 100])
def test_final_state_out_that_is_the_initial_state_is_refused(time):
    tensors = [t.to(DEV) for t in oracle.make_inputs(2, time, 2, seed=time)]
    before = tensors[6].clone()
    with pytest.raises(ValueError, match="final_state_out must not overlap"):
        recurrent_gdn2(*tensors, final_state_out=tensors[6])
    assert torch.equal(tensors[6], before)


@pytest.mark.parametrize("flag", [1, np.True_])
@pytest.mark.parametrize("time", [1, 5, 64])
def test_inplace_update_with_a_flag_that_is_no_bool(time, flag):
    tensors = [t.to(DEV) for t in oracle.make_inputs(2, time, 2, seed=time)]
    expected = recurrent_gdn2(*tensors)
    out, state = recurrent_gdn2(*tensors, inplace_final_state=flag)
    assert state is tensors[6] and torch.equal(state, expected[1]) and torch.equal(out, expected[0])


@pytest.mark.parametrize("budget", [1e10, 10 ** 20])
def test_a_scratch_budget_that_is_no_64_bit_int(monkeypatch, budget):
    tensors = [t.to(DEV) for t in oracle.make_inputs(2, 130, 2, seed=3)]
    leaves = [t.clone().requires_grad_(True) for t in tensors]
    expected = chunk_gdn2(*tensors, output_final_state=True)
    monkeypatch.setattr(chunk_kernels, "SCRATCH_BUDGET_BYTES", budget)
    for got in (chunk_gdn2(*tensors, output_final_state=True), chunk_gdn2(*leaves, output_final_state=True),
                recurrent_gdn2(*tensors)):
        assert torch.equal(got[0], expected[0]) and torch.equal(got[1], expected[1])


def test_other_python_threads_run_while_a_launch_waits():
    """Launches behind a kernel of a second fill the launch queue, and one waits until it is over: a thread that
    only looks at the clock must go on meanwhile."""

    tensors = [t.to(DEV) for t in oracle.make_inputs(1, 1, 2, seed=1)]
    recurrent_gdn2(*tensors, inplace_final_state=True)
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), []

    def watch():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    watcher = threading.Thread(target=watch)
    watcher.start()
    longest = 0.0
    torch.cuda._sleep(2_000_000_000)
    for _ in range(20000):
        begin = time.perf_counter()
        recurrent_gdn2(*tensors, inplace_final_state=True)
        longest = max(longest, time.perf_counter() - begin)
        if longest > 0.1:
            break
    stop.set()
    watcher.join()
    torch.cuda.synchronize()
    assert longest > 0.1, "no launch waited"
    assert max(gaps) < 0.5 * longest


def test_packed_backward_checks_the_free_memory(monkeypatch):
    leaves = [t.to(DEV).requires_grad_(True) for t in oracle.make_inputs(1, 300, 2, seed=5)[:6]]
    out, _ = chunk_gdn2_varlen(*leaves, [0, 100, 300])
    monkeypatch.setattr(chunk_kernels, "CHECK_MEMORY_MIN_BYTES", 0)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (0, 0))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device: 0)
    # 2 + 4 chunks of 2 heads: dZ of 36 KiB each, and cotangents of 64 KiB at 6 + 2 checkpoints
    needed = 12 * 36 * 1024 + 16 * 65536
    with pytest.raises(ValueError, match=f"packed backward needs {needed} bytes"):
        torch.autograd.grad(out.float().sum(), leaves)
