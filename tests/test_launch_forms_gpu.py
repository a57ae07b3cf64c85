"""GPU tests of what a dispatch rule chooses between: the joint launch of prep and scan, packed batches that
take several launches, the token spans' loads of unaligned tensors, and calls from threads that have made no
CUDA call yet.  The forms run the same arithmetic in the same order, so results are compared bit for bit; one
unit of each case is held against the oracle with the tolerances of test_autograd_gpu.py."""

from __future__ import annotations

import threading

import pytest
import torch

import gdn2_oracle as oracle
from gdn2_sm120_b200 import _lib, chunk_gdn2, chunk_kernels
from gdn2_sm120_b200.chunk import chunk_forward
from gdn2_sm120_b200.varlen import chunk_gdn2_varlen
from test_autograd_gpu import _check_unit_alone_and_against_oracle, _device_inputs, _step

pytestmark = pytest.mark.gpu
DEV = "cuda"


# (at most SMs / 4 sequences x heads, and enough chunks: the smallest that qualify at 37, 32 and 16 heads, one
# chunk less, and ragged ends of 1 and 63 tokens)
@pytest.mark.parametrize("batch,heads,time,kernels", [(1, 37, 21 * 64, 1), (2, 16, 26 * 64, 1), (2, 16, 25 * 64, 2),
                                                      (2, 16, 26 * 64 + 1, 1), (1, 16, 70 * 64 + 63, 1)])
def test_joint_launch_equals_a_unit_alone_and_the_oracle(batch, heads, time, kernels):
    tensors, d_out, d_fin = _device_inputs(batch, time, heads, seed=time)
    full = _step(tensors, d_out, d_fin)
    assert _lib.lib().gdn2_chunk_forward_kernels() == kernels
    _check_unit_alone_and_against_oracle(tensors, d_out, d_fin, batch - 1, heads - 1, full)


# One head has its scans' value rows split over two CTAs forward and four back, 37, 38 and 74 heads over two (or four
# and two) and 75 over none: one chunk, a partial one of a token, and several with a ragged end
@pytest.mark.parametrize("time", [64, 65, 200])
@pytest.mark.parametrize("heads", [37, 38, 74, 75])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_scans_of_split_value_rows_equal_whole_ones(heads, time, dtype):
    tensors, d_out, d_fin = _device_inputs(2, time, 75, seed=time)
    tensors, d_out = [t.to(dtype) if t.dtype == torch.bfloat16 else t for t in tensors], d_out.to(dtype)
    out, fin, grads = _step(tensors, d_out, d_fin)  # 150 sequences x heads: never split
    h = slice(75 - heads, 75)
    part = [t[1:2, :, h].contiguous() for t in tensors[:6]] + [tensors[6][1:2, h].contiguous()]
    for single in (part, [t[:, :, :1].contiguous() for t in part[:6]] + [part[6][:, :1].contiguous()]):
        n = single[6].shape[1]
        at = slice(75 - heads, 75 - heads + n)
        o, f, gr = _step(single, d_out[1:2, :, at].contiguous(), d_fin[1:2, at].contiguous())
        assert torch.equal(o, out[1:2, :, at]) and torch.equal(f, fin[1:2, at])
        for a, b in zip(gr[:6], grads[:6]):
            assert torch.equal(a, b[1:2, :, at])
        assert torch.equal(gr[6], grads[6][1:2, at])


# Scans of value rows are split while the longest sequence stays the longest part of the call: equal lengths up to half
# (a quarter) of the SMs whatever their length, packed ones by their chunks and the cost of a CTA.  (The rule only: no
# launch.)
@pytest.mark.parametrize("lengths,heads,most,parts", [
    ([64], 74, 2, 2), ([64], 75, 2, 1), ([4096], 74, 4, 2), ([4096], 37, 4, 4), ([4096], 38, 4, 2), ([64], 1, 2, 2),
    ([100, 200, 300], 32, 2, 1), ([100, 200, 300], 24, 2, 2), ([64, 128, 192, 256], 24, 2, 1),
    ([300, 300, 600], 32, 2, 1), ([300, 300, 600], 24, 2, 2), ([1400, 700, 350, 175], 32, 2, 2),
    ([911, 2300, 150, 1640, 77, 1202, 514, 1398], 16, 4, 2), ([2600, 64, 70, 700], 16, 4, 4)])
def test_rule_that_splits_value_rows(lengths, heads, most, parts):
    chunks = [-(-n // 64) for n in lengths]
    assert _lib.lib().gdn2_chunk_value_parts(sum(chunks) * heads, len(chunks) * heads, max(chunks), 148, most) == parts


# four sequences of which one is long: split at 16 heads (2 * 56 units a head <= 41 * 148), not in the sequences alone
def test_packed_scans_of_split_value_rows_equal_single_sequences():
    lengths, heads = [2600, 64, 70, 700], 16
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    tensors, d_out, _ = _device_inputs(1, cu[-1], heads, seed=5)
    torch.manual_seed(5)
    states = 0.02 * torch.randn(len(lengths), heads, 128, 128, device=DEV)
    d_fin = 0.01 * torch.randn_like(states)
    leaves = [t.requires_grad_(True) for t in (*tensors[:6], states)]
    out, fin = chunk_gdn2_varlen(*leaves[:6], cu, leaves[6], output_final_state=True)
    grads = torch.autograd.grad((out.float() * d_out.float()).sum() + (fin * d_fin).sum(), leaves)
    for i, (lo, hi) in enumerate(zip(cu, cu[1:])):
        single = [t[:, lo:hi].detach().clone() for t in leaves[:6]] + [states[i:i + 1].detach().clone()]
        o, f, gr = _step(single, d_out[:, lo:hi], d_fin[i:i + 1])
        assert torch.equal(o, out[:, lo:hi]) and torch.equal(f, fin[i:i + 1])
        for a, b in zip(gr[:6], grads[:6]):
            assert torch.equal(a, b[:, lo:hi])
        assert torch.equal(gr[6], grads[6][i:i + 1])


@pytest.mark.parametrize("dtype,g_dtype", [(torch.bfloat16, torch.float32), (torch.float16, torch.float16)])
@pytest.mark.parametrize("raw", [False, True])
def test_joint_launch_equals_two_launches(dtype, g_dtype, raw):
    tensors, _, _ = _device_inputs(2, 40 * 64 + 17, 16, seed=7)
    q, k, v, g, beta, w = [t.to(g_dtype if i == 3 else dtype) for i, t in enumerate(tensors[:6])]
    flags = {"use_qk_l2norm_in_kernel": True, "use_gate_in_kernel": True} if raw else {}
    with torch.no_grad():
        launched = _lib.LAUNCHES[0]
        joint = chunk_gdn2(q, k, v, g, beta, w, tensors[6], output_final_state=True, **flags)
        assert _lib.lib().gdn2_chunk_forward_kernels() == _lib.LAUNCHES[0] - launched == 1
        _lib.profile_enable(True)  # times the kernels one by one: never joint
        try:
            apart = chunk_gdn2(q, k, v, g, beta, w, tensors[6], output_final_state=True, **flags)
            assert _lib.lib().gdn2_chunk_forward_kernels() == 2
        finally:
            _lib.profile_enable(False)
    assert torch.equal(joint[0], apart[0]) and torch.equal(joint[1], apart[1])


# scanning CTAs that prepare none, some and nearly all of the units that the others could not have ready in time
@pytest.mark.parametrize("heads,time", [(16, 30 * 64), (24, 48 * 64), (28, 33 * 64 + 9), (37, 21 * 64), (37, 64 * 64)])
@pytest.mark.parametrize("raw", [False, True])
def test_joint_launches_whose_scans_prepare_first_equal_two_launches(heads, time, raw):
    tensors, _, _ = _device_inputs(1, time, heads, seed=heads + time)
    flags = {"use_qk_l2norm_in_kernel": True, "use_gate_in_kernel": True} if raw else {}
    with torch.no_grad():
        joint = chunk_gdn2(*tensors, output_final_state=True, **flags)
        assert _lib.lib().gdn2_chunk_forward_kernels() == 1
        _lib.profile_enable(True)  # times the kernels one by one: never joint
        try:
            apart = chunk_gdn2(*tensors, output_final_state=True, **flags)
        finally:
            _lib.profile_enable(False)
    assert torch.equal(joint[0], apart[0]) and torch.equal(joint[1], apart[1])


# (four scans at least, a quarter of the SMs at most, 32 chunks: the smallest and widest grids, one chunk less, and
# ragged ends of 1 and 63 tokens)
@pytest.mark.parametrize("batch,heads,time,kernels", [(1, 4, 32 * 64, 1), (1, 3, 32 * 64, 2), (2, 16, 31 * 64, 2),
                                                      (2, 16, 32 * 64 + 1, 1), (1, 37, 32 * 64 + 63, 1)])
@pytest.mark.parametrize("dtype,g_dtype", [(torch.bfloat16, torch.float32), (torch.float16, torch.float16)])
def test_joint_backward_equals_two_launches_and_the_oracle(batch, heads, time, kernels, dtype, g_dtype):
    tensors, d_out, d_fin = _device_inputs(batch, time, heads, seed=time)
    tensors = [t.to(g_dtype if i == 3 else dtype) for i, t in enumerate(tensors[:6])] + [tensors[6]]
    d_out = d_out.to(dtype)
    launched = _lib.LAUNCHES[0]
    full = _step(tensors, d_out, d_fin)
    assert _lib.LAUNCHES[0] - launched == _lib.lib().gdn2_chunk_forward_kernels() + kernels
    again = _step(tensors, d_out, d_fin)  # (a second call finds other memory, or the first one's marks)
    _lib.profile_enable(True)  # times the kernels one by one: never joint
    try:
        apart = _step(tensors, d_out, d_fin)
    finally:
        _lib.profile_enable(False)
    for other in (again, apart):
        assert torch.equal(full[0], other[0]) and torch.equal(full[1], other[1])
        assert all(torch.equal(a, b) for a, b in zip(full[2], other[2]))
    if dtype == torch.bfloat16:
        _check_unit_alone_and_against_oracle(tensors, d_out, d_fin, batch - 1, heads - 1, full)


# The scans' maps of v, w, the output and its cotangent differ from those of the other kernels in the width of the box
# alone where value rows are split (halves, quarters), and are the same where they are not
@pytest.mark.parametrize("batch,heads,time", [(1, 16, 2048), (1, 2, 192), (2, 38, 130)])
def test_a_repeated_training_step_encodes_no_tensor_map(batch, heads, time):
    tensors, d_out, _ = _device_inputs(batch, time, heads, seed=2)
    leaves = [t.requires_grad_(True) for t in tensors]

    def step():
        out, _ = chunk_gdn2(*leaves)
        torch.autograd.grad(out, leaves, d_out)

    for _ in range(4):  # until the allocator hands out the same blocks
        step()
    before = _lib.lib().gdn2_tensor_maps_encoded()
    for _ in range(3):
        step()
    assert _lib.lib().gdn2_tensor_maps_encoded() == before > 0


# a unit whose mark is seen before its cotangent rows or its dZ tile are in memory reads what lay there before: NaN
# here, in the fewest and the most scans and with a partial chunk
@pytest.mark.parametrize("batch,heads,time", [(1, 4, 40 * 64), (1, 37, 32 * 64 + 5)])
def test_joint_backward_never_reads_ahead_of_a_mark(batch, heads, time):
    (q, k, v, g, beta, w, s0), d_out, d_fin = _device_inputs(batch, time, heads, seed=time)
    scale, full = 128 ** -0.5, -(-time // 64) * 64
    _, _, aux = chunk_forward(q, k, v, g, beta, w, s0, scale=scale, return_aux=True)
    slots = torch.empty((batch, full // 64 + 1, heads, 128, 128), device=DEV)
    scratch = torch.empty(chunk_kernels.scratch_bytes(batch, full, heads, True) // 4, device=DEV)
    first = None
    for _ in range(25):
        slots.fill_(float("nan"))
        scratch.fill_(float("nan"))
        grads = [torch.full_like(x, float("nan")) for x in (q, k, v, g, beta, w, s0)]
        _lib.call("gdn2_chunk_backward", q.device, *[x.data_ptr() for x in (q, k, v, g, beta, w, d_out, d_fin)],
                  aux.chunk_boundaries.data_ptr(), slots.data_ptr(), aux.workspace[0].data_ptr(), scratch.data_ptr(),
                  *[x.data_ptr() for x in grads], batch, time, heads, full, _lib.dtype_code(q.dtype),
                  _lib.dtype_code(g.dtype), scale, _lib.stream_ptr(q.device))
        assert _lib.lib().gdn2_chunk_backward_kernels() == 1
        if first is None:
            first = grads
            assert all(torch.isfinite(x.float()).all() for x in grads)
        assert all(torch.equal(a, b) for a, b in zip(grads, first))


# a unit whose mark is seen before one of its tiles is in memory gives a scan what lay there before: NaN here, where the
# scans wait for the preparing CTAs alone (8 and 16 heads) and where they prepare units themselves first
@pytest.mark.parametrize("heads,time", [(8, 50 * 64), (16, 40 * 64 + 17), (37, 21 * 64)])
@pytest.mark.parametrize("training,prologue", [(False, 0), (False, 3), (True, 0)])
def test_joint_forward_never_reads_ahead_of_a_mark(heads, time, training, prologue):
    tensors, _, _ = _device_inputs(1, time, heads, seed=time)
    full = -(-time // 64) * 64
    workspace = torch.empty(chunk_kernels.workspace_bytes(1, full, heads, training) // 4, device=DEV)
    scratch = torch.empty(0 if training else chunk_kernels.scratch_bytes(1, full, heads) // 4, device=DEV)
    slots = torch.empty((1, full // 64 + 1, heads, 128, 128), device=DEV) if training else None
    out, fin = torch.empty_like(tensors[2]), torch.empty_like(tensors[6])
    codes = _lib.dtype_code(tensors[0].dtype), _lib.dtype_code(tensors[3].dtype)

    def call():
        workspace.fill_(float("nan"))
        scratch.fill_(float("nan"))
        common = [x.data_ptr() for x in (*tensors, out, fin)]
        buffers = [workspace.data_ptr(), scratch.data_ptr() or None]
        sizes, last = (1, time, heads, full), (128 ** -0.5,)
        if prologue:
            _lib.call("gdn2_chunk_forward_fused", out.device, *common, *buffers, *sizes, *codes, *last, prologue,
                      _lib.stream_ptr(out.device))
        else:
            _lib.call("gdn2_chunk_forward", out.device, *common, slots.data_ptr() if training else None, *buffers, *sizes,
                      int(training), *codes, *last, _lib.stream_ptr(out.device))

    _lib.profile_enable(True)  # times the kernels one by one: never joint
    try:
        call()
        assert _lib.lib().gdn2_chunk_forward_kernels() == 2
    finally:
        _lib.profile_enable(False)
    wanted = out.clone(), fin.clone()
    assert all(torch.isfinite(x.float()).all() for x in wanted)
    for _ in range(20):
        call()
        assert _lib.lib().gdn2_chunk_forward_kernels() == 1
        assert torch.equal(out, wanted[0]) and torch.equal(fin, wanted[1])


# 255 .. 257 and 513: around one and two launch tables of 256 sequences
@pytest.mark.parametrize("count", [255, 256, 257, 513])
def test_packed_batches_around_the_table_size(count):
    lengths = [(7 * i) % 40 if i % 50 else 64 + i % 70 for i in range(count)]
    heads, total = 1, sum(lengths)
    tensors, d_out, _ = _device_inputs(1, total, heads, seed=count)
    torch.manual_seed(count)
    states = 0.02 * torch.randn(count, heads, 128, 128, device=DEV)
    d_fin = 0.01 * torch.randn_like(states)
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    leaves = [t.requires_grad_(True) for t in (*tensors[:6], states)]
    out, fin = chunk_gdn2_varlen(*leaves[:6], cu, leaves[6], output_final_state=True)
    grads = torch.autograd.grad((out.float() * d_out.float()).sum() + (fin * d_fin).sum(), leaves)
    for i in {0, 1, 50, 51, count // 2, count - 2, count - 1}:
        lo, hi = cu[i], cu[i + 1]
        if lo == hi:
            assert torch.equal(fin[i], states[i]) and torch.equal(grads[6][i], d_fin[i])
            continue
        single = [t[:, lo:hi].detach().clone() for t in leaves[:6]] + [states[i:i + 1].detach().clone()]
        o, f, gr = _step(single, d_out[:, lo:hi], d_fin[i:i + 1])
        assert torch.equal(o, out[:, lo:hi]) and torch.equal(f, fin[i:i + 1])
        for a, b in zip(gr[:6], grads[:6]):
            assert torch.equal(a, b[:, lo:hi])
        assert torch.equal(gr[6], grads[6][i:i + 1])


# spans of one token, a whole span, one token more, and several spans
@pytest.mark.parametrize("time", [2, 16, 17, 48])
def test_token_spans_of_unaligned_tensors(time):
    cpu = oracle.make_inputs(2, time, 3, seed=time)

    def shifted(t):  # the same values one element past an aligned address
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
        view = flat[1:].view(t.shape)
        view.copy_(t)
        return view

    with torch.no_grad():
        expected = chunk_gdn2(*[t.to(DEV) for t in cpu], output_final_state=True)
        got = chunk_gdn2(*[shifted(t) for t in cpu[:6]], cpu[6].to(DEV), output_final_state=True)
    assert torch.equal(got[0], expected[0]) and torch.equal(got[1], expected[1])


def test_training_in_a_thread_without_a_context():
    tensors, d_out, d_fin = _device_inputs(1, 130, 2, seed=3)
    expected = _step(tensors, d_out, d_fin)
    results = []
    worker = threading.Thread(target=lambda: results.append(_step(tensors, d_out, d_fin)))
    worker.start()
    worker.join()
    assert results and torch.equal(results[0][0], expected[0]) and torch.equal(results[0][1], expected[1])
    for a, b in zip(results[0][2], expected[2]):
        assert torch.equal(a, b)


# 1 to 4 spans, whole and partial; 74 pairs x 2 tiles fill the SMs once, 75 do not
@pytest.mark.parametrize("time", [16, 17, 33, 63])
@pytest.mark.parametrize("batch,heads", [(2, 37), (3, 25)])
def test_token_spans_at_the_grid_where_the_form_changes(batch, heads, time):
    tensors, d_out, d_fin = _device_inputs(batch, time, heads, seed=time)
    full = _step(tensors, d_out, d_fin)
    _check_unit_alone_and_against_oracle(tensors, d_out, d_fin, batch - 1, heads - 1, full)


# token by token up to 9 tokens (inputs of 4 read at once; raw inputs up to 8), spans from there on
@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("time", [2, 4, 5, 8, 9, 10])
def test_few_tokens_with_and_without_the_prologue(time, raw):
    make = oracle.make_raw_inputs if raw else oracle.make_inputs
    cpu = make(3, time, 2, seed=time)
    state = 0.05 * torch.randn(3, 2, 128, 128, generator=torch.Generator().manual_seed(time))
    flags = {"use_qk_l2norm_in_kernel": True, "use_gate_in_kernel": True} if raw else {}
    with torch.no_grad():
        out, fin = chunk_gdn2(*[t.to(DEV) for t in cpu[:6]], state.to(DEV), output_final_state=True, **flags)
    plain = cpu[:6]
    if raw:
        q, k, v, g, beta, w = [t.double() for t in cpu[:6]]
        norm = lambda x: x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        plain = (norm(q), norm(k), v, -torch.nn.functional.softplus(g), torch.sigmoid(beta), torch.sigmoid(w))
    ref_out, ref_state = oracle.recurrence(*plain, state)
    # exact fp32, one rounding to bf16 of at most 2^-9 = 1.95e-3 of a value: each token by itself, so that a wrong row
    # cannot hide among the others
    for t in range(time):
        assert oracle.rel_l2(out[:, t], ref_out[:, t]) < 2.2e-3, t
    assert oracle.rel_l2(fin, ref_state) < 1e-5


def test_joint_launch_replays_from_a_cuda_graph():
    tensors, _, _ = _device_inputs(1, 80 * 64, 16, seed=11)
    with torch.no_grad():
        expected = chunk_gdn2(*tensors, output_final_state=True)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            chunk_gdn2(*tensors, output_final_state=True)
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = chunk_gdn2(*tensors, output_final_state=True)
        assert _lib.lib().gdn2_chunk_forward_kernels() == 1
        for _ in range(2):
            got[0].zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(got[0], expected[0]) and torch.equal(got[1], expected[1])


# the longest sequences that go token by token and one token more: alone, in a grid and packed, the same bits
@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("time", [8, 9, 10])
def test_a_few_tokens_alone_in_a_batch_and_packed(time, raw):
    tensors, _, _ = _device_inputs(24, time, 4, seed=time)
    flags = {"use_qk_l2norm_in_kernel": True, "use_gate_in_kernel": True} if raw else {}
    with torch.no_grad():
        out, fin = chunk_gdn2(*tensors, output_final_state=True, **flags)
        alone = chunk_gdn2(*[t[3:4] for t in tensors], output_final_state=True, **flags)
        rows = [t.reshape(1, 24 * time, 4, 128) for t in tensors[:6]]
        launched = _lib.LAUNCHES[0]
        packed = chunk_gdn2_varlen(*rows, [time * i for i in range(25)], tensors[6], output_final_state=True, **flags)
    assert _lib.LAUNCHES[0] == launched + 1
    assert torch.equal(alone[0], out[3:4]) and torch.equal(alone[1], fin[3:4])
    assert torch.equal(packed[0].view_as(out), out) and torch.equal(packed[1], fin)


# whole chunks only (short sequences beside them do not count), and one sequence that ends in a partial chunk
@pytest.mark.parametrize("lengths", [(64, 192, 128, 640), (128, 40, 64, 0, 256), (64, 192, 129)])
def test_packed_gradients_with_and_without_a_partial_chunk(lengths):
    heads, total = 3, sum(lengths)
    tensors, d_out, _ = _device_inputs(1, total, heads, seed=total)
    states = 0.02 * torch.randn(len(lengths), heads, 128, 128, device=DEV)
    d_fin = 0.01 * torch.randn_like(states)
    leaves = [t.requires_grad_(True) for t in (*tensors[:6], states)]
    cu = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    out, fin = chunk_gdn2_varlen(*leaves[:6], cu, leaves[6], output_final_state=True)
    grads = torch.autograd.grad((out.float() * d_out.float()).sum() + (fin * d_fin).sum(), leaves)
    for i, (lo, hi) in enumerate(zip(cu, cu[1:])):
        if lo < hi:
            single = [t[:, lo:hi].detach() for t in leaves[:6]] + [states[i:i + 1].detach()]
            o, f, gr = _step(single, d_out[:, lo:hi], d_fin[i:i + 1])
            assert torch.equal(o, out[:, lo:hi]) and torch.equal(f, fin[i:i + 1])
            assert all(torch.equal(a, b[:, lo:hi]) for a, b in zip(gr[:6], grads[:6]))
            assert torch.equal(gr[6], grads[6][i:i + 1])


# The queue of units and the marks lie in scratch that a replay finds as the one before left it: a replay
# that did not clear them would find every unit taken, or finished before it is.  (The leaves are made on the capturing
# stream: the autograd engine runs a leaf's last step where the leaf was made.)
@pytest.mark.parametrize("batch,heads,time", [(1, 16, 40 * 64), (2, 16, 33 * 64 + 7)])
def test_joint_training_step_replays_from_a_cuda_graph(batch, heads, time):
    tensors, d_out, _ = _device_inputs(batch, time, heads, seed=12)
    others, other_d_out, _ = _device_inputs(batch, time, heads, seed=13)
    expected = []
    for values, cotangent in ((tensors, d_out), (others, other_d_out)):
        leaves = [t.clone().requires_grad_(True) for t in values]
        out, _ = chunk_gdn2(*leaves)
        expected.append([out.detach(), *torch.autograd.grad(out, leaves, cotangent)])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        leaves = [t.clone().requires_grad_(True) for t in tensors]
        cotangent = d_out.clone()

        def step():
            out, _ = chunk_gdn2(*leaves)
            return [out, *torch.autograd.grad(out, leaves, cotangent)]

        step()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            launched = _lib.LAUNCHES[0]
            got = step()
            assert _lib.lib().gdn2_chunk_forward_kernels() == 1 and _lib.LAUNCHES[0] - launched == 2
        for turn in (0, 1, 1, 0):
            with torch.no_grad():
                for leaf, value in zip(leaves, (tensors, others)[turn]):
                    leaf.copy_(value)
                cotangent.copy_((d_out, other_d_out)[turn])
                for t in got:
                    t.fill_(float("nan"))
            graph.replay()
            stream.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, expected[turn]))


# the fewest scans and units that a joint forward has (4 scans, with the prologue 8, and 400 units), with its smallest
# number of preparing CTAs; fewer scans take two launches
@pytest.mark.parametrize("heads,time,raw,kernels", [(4, 100 * 64, False, 1), (7, 58 * 64, False, 1), (8, 50 * 64, True, 1),
                                                    (4, 99 * 64 + 1, False, 1), (4, 99 * 64, False, 2),
                                                    (3, 134 * 64 + 1, False, 2), (7, 58 * 64, True, 2),
                                                    (1, 400 * 64, False, 2)])
def test_joint_forward_of_few_scans_equals_two_launches(heads, time, raw, kernels):
    tensors, _, _ = _device_inputs(1, time, heads, seed=heads)
    flags = {"use_qk_l2norm_in_kernel": True, "use_gate_in_kernel": True} if raw else {}
    with torch.no_grad():
        joint = chunk_gdn2(*tensors, output_final_state=True, **flags)
        assert _lib.lib().gdn2_chunk_forward_kernels() == kernels
        _lib.profile_enable(True)  # times the kernels one by one: never joint
        try:
            apart = chunk_gdn2(*tensors, output_final_state=True, **flags)
            assert _lib.lib().gdn2_chunk_forward_kernels() == 2
        finally:
            _lib.profile_enable(False)
    assert torch.equal(joint[0], apart[0]) and torch.equal(joint[1], apart[1])
