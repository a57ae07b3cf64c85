"""GPU tests of packed variable-length sequences (``chunk_gdn2_varlen``) and grouped value heads
(``expand_grouped_heads``): every packed sequence must give exactly what a separate call gives."""

from __future__ import annotations

import pytest
import torch

import gdn2_oracle as oracle
from gdn2_sm120_b200 import chunk_gdn2
from gdn2_sm120_b200.varlen import chunk_gdn2_varlen, expand_grouped_heads

DEV = "cuda"


def _packed_case(lengths, heads, seed):
    cases = [oracle.make_inputs(1, n, heads, seed=seed + i) for i, n in enumerate(lengths)]
    packed = [torch.cat([c[j] for c in cases], dim=1) for j in range(6)]
    states = torch.cat([c[6] for c in cases], dim=0)
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    return cases, packed, states, cu


@pytest.mark.gpu
def test_packed_sequences_equal_separate_calls_forward_and_backward():
    lengths = [70, 5, 0, 200, 64]
    cases, packed, states, cu = _packed_case(lengths, 2, seed=900)
    gen = torch.Generator().manual_seed(1)
    d_out = (torch.randn(packed[2].shape, generator=gen) * 0.1).bfloat16().to(DEV)
    d_fin = (torch.randn(states.shape, generator=gen) * 0.01).to(DEV)

    leaves = [t.to(DEV).requires_grad_(True) for t in packed]
    s0 = states.to(DEV).requires_grad_(True)
    out, fin = chunk_gdn2_varlen(*leaves, torch.tensor(cu, dtype=torch.int32), s0, output_final_state=True)
    assert out.shape == packed[2].shape and fin.shape == states.shape
    grads = torch.autograd.grad((out.float() * d_out.float()).sum() + (fin * d_fin).sum(), (*leaves, s0))

    for i, n in enumerate(lengths):
        lo, hi = cu[i], cu[i + 1]
        if n == 0:
            assert torch.equal(fin[i], s0[i]) and torch.equal(grads[6][i], d_fin[i])
            continue
        single = [t[:, lo:hi].detach().clone().requires_grad_(True) for t in leaves]
        s_single = s0[i:i + 1].detach().clone().requires_grad_(True)
        o, f = chunk_gdn2(*single, s_single, output_final_state=True)
        gr = torch.autograd.grad((o.float() * d_out[:, lo:hi].float()).sum() + (f * d_fin[i:i + 1]).sum(),
                                 (*single, s_single))
        assert torch.equal(o, out[:, lo:hi]) and torch.equal(f, fin[i:i + 1])
        for a, b in zip(gr[:6], grads[:6]):
            assert torch.equal(a, b[:, lo:hi])
        assert torch.equal(gr[6], grads[6][i:i + 1])
    # one sequence against the oracle as well
    ref_out, ref_state = oracle.recurrence(*cases[3])
    torch.testing.assert_close(out[:, cu[3]:cu[4]].float().cpu(), ref_out.float(), rtol=2e-2, atol=1e-2)
    assert oracle.rel_l2(fin[3:4], ref_state) < 1e-3


@pytest.mark.gpu
def test_packed_inference_without_states_and_with_fused_flags():
    lengths = [33, 130]
    raws = [oracle.make_raw_inputs(1, n, 2, seed=50 + i) for i, n in enumerate(lengths)]
    packed = [torch.cat([c[j] for c in raws], dim=1).to(DEV) for j in range(6)]
    with torch.no_grad():
        out, fin = chunk_gdn2_varlen(*packed, [0, 33, 163], use_qk_l2norm_in_kernel=True,
                                     use_gate_in_kernel=True, output_final_state=True)
        for i, (lo, hi) in enumerate(((0, 33), (33, 163))):
            o, f = chunk_gdn2(*(t[:, lo:hi] for t in packed), use_qk_l2norm_in_kernel=True,
                              use_gate_in_kernel=True, output_final_state=True)
            assert torch.equal(o, out[:, lo:hi]) and torch.equal(f, fin[i:i + 1])
        assert chunk_gdn2_varlen(*packed, [0, 33, 163])[1] is None


def test_cu_seqlens_and_group_validation():
    q = torch.zeros(1, 10, 2, 128)
    with pytest.raises(ValueError, match="start at 0 and end"):
        chunk_gdn2_varlen(q, q, q, q, q, q, [0, 4, 9])
    with pytest.raises(ValueError, match="non-decreasing"):
        chunk_gdn2_varlen(q, q, q, q, q, q, [0, 7, 4, 10])
    with pytest.raises(TypeError, match="int32 or int64"):
        chunk_gdn2_varlen(q, q, q, q, q, q, torch.tensor([0.0, 10.0]))
    with pytest.raises(ValueError, match=r"\[1, total, H, 128\]"):
        chunk_gdn2_varlen(torch.zeros(2, 5, 2, 128), q, q, q, q, q, [0, 5])
    with pytest.raises(ValueError, match="multiple"):
        expand_grouped_heads(q, q, q, q, 3)
    a = torch.arange(2 * 3 * 2 * 4, dtype=torch.float32).view(2, 3, 2, 4).requires_grad_(True)
    wide = expand_grouped_heads(a, a, a, a, 6)[0]
    assert wide.shape == (2, 3, 6, 4) and wide.is_contiguous()
    assert torch.equal(wide[:, :, 0], a[:, :, 0]) and torch.equal(wide[:, :, 2], a[:, :, 0])
    assert torch.equal(wide[:, :, 3], a[:, :, 1])
    (grad,) = torch.autograd.grad(wide.sum(), a)
    assert torch.equal(grad, torch.full_like(a, 3.0))


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [(200, 33, 7, 130, 3), (64, 9, 10, 1), (700, 48), (65, 2, 4)])
def test_short_sequences_beside_the_scans(lengths):
    """The token kernels of a packed forward run beside the chunk scans: what follows on the stream sees every output
    and state, eagerly and in a replayed graph, bit for bit as from separate calls."""
    heads, total = 5, sum(lengths)
    cpu = oracle.make_inputs(1, total, heads, seed=61)
    args = [t.cuda() for t in cpu[:6]]
    state = (torch.randn(len(lengths), heads, 128, 128, generator=torch.Generator().manual_seed(62)) * 0.02).cuda()
    bounds = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    wanted_out, wanted_state = [], []
    for i, (a, b) in enumerate(zip(bounds, bounds[1:])):
        out, fin = chunk_gdn2(*(x[:, a:b].contiguous() for x in args), state[i:i + 1], output_final_state=True)
        wanted_out.append(out)
        wanted_state.append(fin)
    wanted_out, wanted_state = torch.cat(wanted_out, 1), torch.cat(wanted_state, 0)

    def call():
        out, fin = chunk_gdn2_varlen(*args, bounds, state, output_final_state=True)
        return out.clone(), fin.clone()  # right behind on the stream

    with torch.no_grad():
        for _ in range(20):
            out, fin = call()
            assert torch.equal(out, wanted_out) and torch.equal(fin, wanted_state)
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            call()
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = call()
    for _ in range(5):
        for x in captured:
            x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(captured[0], wanted_out) and torch.equal(captured[1], wanted_state)


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [(200, 33, 7, 130, 3), (64, 9, 10, 1), (700, 63)])
def test_short_sequences_beside_the_backward_of_the_others(lengths):
    """The reverse scans run beside the short sequences' reverse kernel and their VJP beside the other one: gradients
    read right behind on the stream, eagerly and from a replayed graph, are those of separate calls bit for bit."""
    heads, total = 5, sum(lengths)
    cpu = oracle.make_inputs(1, total, heads, seed=71)
    leaves = [t.cuda().requires_grad_(True) for t in cpu[:6]]
    gen = torch.Generator().manual_seed(72)
    state = (torch.randn(len(lengths), heads, 128, 128, generator=gen) * 0.02).cuda().requires_grad_(True)
    d_out = torch.randn(leaves[2].shape, generator=gen).to(leaves[2].dtype).cuda()
    d_fin = torch.randn(state.shape, generator=gen).cuda()
    bounds = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    wanted = [[] for _ in range(7)]
    for i, (a, b) in enumerate(zip(bounds, bounds[1:])):
        parts = [x.detach()[:, a:b].contiguous().requires_grad_(True) for x in leaves]
        start = state.detach()[i:i + 1].clone().requires_grad_(True)
        out, fin = chunk_gdn2(*parts, start, output_final_state=True)
        grads = torch.autograd.grad([out, fin], [*parts, start], [d_out[:, a:b].contiguous(), d_fin[i:i + 1]])
        for w, g in zip(wanted, grads):
            w.append(g)
    wanted = [torch.cat(w, 1) for w in wanted[:6]] + [torch.cat(wanted[6], 0)]

    def step():
        out, fin = chunk_gdn2_varlen(*leaves, bounds, state, output_final_state=True)
        return [g.clone() for g in torch.autograd.grad([out, fin], [*leaves, state], [d_out, d_fin])]

    for _ in range(10):
        assert all(torch.equal(g, w) for g, w in zip(step(), wanted))
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(5):
        for x in captured:
            x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(captured, wanted))


# several waves of CTAs in every kernel that runs beside another one: 12 sequences of spans, 14 of a few tokens
@pytest.mark.gpu
@pytest.mark.parametrize("raw", [False, True])
@pytest.mark.parametrize("dtype,g_dtype", [(torch.bfloat16, torch.float32), (torch.float16, torch.float32),
                                           (torch.float16, torch.float16), (torch.bfloat16, torch.bfloat16)])
def test_many_short_sequences_beside_two_long_ones(dtype, g_dtype, raw):
    lengths, heads = [37, 5] * 6 + [300] + [3, 8, 1, 6] * 2 + [130] + [20, 63] * 3, 16
    make = oracle.make_raw_inputs if raw else oracle.make_inputs
    cpu = make(1, sum(lengths), heads, seed=81, dtype=dtype, g_dtype=g_dtype)
    leaves = [x.to(DEV).requires_grad_(True) for x in cpu[:6]]
    gen = torch.Generator().manual_seed(82)
    state = (torch.randn(len(lengths), heads, 128, 128, generator=gen) * 0.02).to(DEV).requires_grad_(True)
    d_out = torch.randn(leaves[2].shape, generator=gen).to(DEV, dtype)
    d_fin = torch.randn(state.shape, generator=gen).to(DEV)
    flags = {"use_qk_l2norm_in_kernel": raw, "use_gate_in_kernel": raw}
    bounds = [sum(lengths[:i]) for i in range(len(lengths) + 1)]

    def step(*inputs, call, d):
        results = call(*inputs)
        return [*results, *torch.autograd.grad(results, inputs, d)]

    wanted, wanted_plain = [], []
    for i, (a, b) in enumerate(zip(bounds, bounds[1:])):
        parts = [x.detach()[:, a:b].contiguous().requires_grad_(True) for x in leaves]
        parts.append(state.detach()[i:i + 1].clone().requires_grad_(True))
        single = lambda *x: chunk_gdn2(*x[:6], x[6], output_final_state=True, **flags)  # noqa: E731
        wanted.append(step(*parts, call=single, d=[d_out[:, a:b].contiguous(), d_fin[i:i + 1]]))
        with torch.no_grad():
            wanted_plain.append(single(*parts))
    join = lambda rows, i: torch.cat([r[i] for r in rows], 0 if i in (1, 8) else 1)  # noqa: E731

    packed = lambda *x: chunk_gdn2_varlen(*x[:6], bounds, x[6], output_final_state=True, **flags)  # noqa: E731
    for _ in range(5):
        got = [x.clone() for x in step(*leaves, state, call=packed, d=[d_out, d_fin])]  # right behind on the stream
        for i, x in enumerate(got):
            assert torch.equal(x, join(wanted, i)), i
        with torch.no_grad():
            plain = [x.clone() for x in packed(*leaves, state)]
        for i, x in enumerate(plain):
            assert torch.equal(x, join(wanted_plain, i)), i
