"""GPU parity tests of forward + backward through the public autograd API.

Ground truth: the float64 recurrence of the oracle and torch.autograd through it, on the
identical (already 16-bit-rounded) inputs.  Tolerances written once here:

  outputs (16-bit)            |x - ref| <= 1e-2 + 2e-2 |ref|       (specification)
  fp32 tensors S_T, dS0, dg   relative L2 <= 1e-3                  (specification)
  16-bit gradients            relative L2 <= 4e-3 -- their final cast alone costs
                              ~2e-3 -- and max-abs error <= 5e-3   (reference contract);
                              on top of that the error IN EXCESS of the cast floor (the
                              distance of the correctly rounded reference from the
                              reference) must stay <= 1e-3, and the fp32 values before
                              the cast are held to 1e-3 directly where the test entry
                              point gdn2_chunk_backward_f32grads applies
"""

from __future__ import annotations

import pytest
import torch

import gdn2_oracle as oracle
from conftest import load_golden
from gdn2_sm120_b200 import chunk_backward, chunk_gdn2

pytestmark = pytest.mark.gpu
DEV = "cuda"
FP32_REL = 1e-3
LOWP_REL = 4e-3


def excess_over_cast_floor(got, ref):
    """Relative L2 error of a 16-bit tensor beyond what rounding the exact values to its dtype costs.

    The rounding error of the final cast and the arithmetic error before it are independent, so
    their squares add: excess^2 = err^2 - floor^2 (clamped at zero)."""

    err = oracle.rel_l2(got, ref)
    floor = oracle.rel_l2(ref.to(got.dtype), ref)
    return max(err * err - floor * floor, 0.0) ** 0.5


def check_gradient(name, got, ref):
    limit = FP32_REL if got.dtype == torch.float32 else LOWP_REL
    err = oracle.rel_l2(got, ref)
    assert err < limit, f"{name}: rel-L2 {err:.3e} >= {limit}"
    if got.dtype != torch.float32 and got.numel() >= 4096:
        excess = excess_over_cast_floor(got, ref)
        assert excess < FP32_REL, f"{name}: rel-L2 beyond the cast floor {excess:.3e} >= {FP32_REL}"


def run_case(batch, time, heads, *, seed, dtype=torch.bfloat16, g_dtype=torch.float32,
             with_state=True, with_final_grad=True, scale=None):
    cpu = oracle.make_inputs(batch, time, heads, seed=seed, dtype=dtype, g_dtype=g_dtype,
                             with_state=with_state)
    gen = torch.Generator().manual_seed(seed + 1)
    d_out = (torch.randn(cpu[2].shape, generator=gen) * 0.1).to(dtype)
    d_fin = torch.randn((batch, heads, 128, 128), generator=gen) * 0.01 if with_final_grad else None
    ref_out, ref_state, ref_grads = oracle.recurrence_grads(*cpu, d_out, d_fin, scale=scale)

    leaves = [t.to(DEV).requires_grad_(True) for t in cpu[:6]]
    s0 = cpu[6].to(DEV).requires_grad_(True) if with_state else None
    out, fin = chunk_gdn2(*leaves, s0, scale=scale, output_final_state=with_final_grad)
    objective = (out.float() * d_out.to(DEV).float()).sum()
    if with_final_grad:
        objective = objective + (fin * d_fin.to(DEV)).sum()
    wanted = leaves + ([s0] if with_state else [])
    grads = torch.autograd.grad(objective, wanted)

    torch.testing.assert_close(out.float().cpu(), ref_out.float(), rtol=2e-2, atol=1e-2)
    if with_final_grad:
        assert oracle.rel_l2(fin, ref_state) < FP32_REL
    names = ("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0")
    for name, got, ref in zip(names, grads, ref_grads):
        assert got.dtype == (cpu[names.index(name)].dtype if name != "dS0" else torch.float32)
        check_gradient(name, got, ref)
        assert oracle.max_abs(got, ref) < 5e-3 * max(1.0, ref.abs().max().item()), name
    return grads


@pytest.mark.parametrize("time", [1, 3, 16, 19, 47, 63])
def test_short_sequence_gradients(time):
    run_case(2, time, 3, seed=2_605_000 + time)


@pytest.mark.parametrize("time", [64, 128, 129, 143])
@pytest.mark.parametrize("with_state", [True, False])
@pytest.mark.parametrize("with_final_grad", [True, False])
def test_long_sequence_gradients(time, with_state, with_final_grad):
    run_case(1, time, 2, seed=2_605_100 + time, with_state=with_state, with_final_grad=with_final_grad)


@pytest.mark.parametrize("dtype,g_dtype", [(torch.float16, torch.float32), (torch.float16, torch.float16),
                                           (torch.bfloat16, torch.bfloat16)])
def test_gradient_dtypes(dtype, g_dtype):
    grads = run_case(1, 24, 2, seed=99, dtype=dtype, g_dtype=g_dtype, scale=0.125)
    assert grads[3].dtype == g_dtype


def test_benchmark_config0_against_reference_golden_gradients():
    """B=1, T=64, H=2, loss = mean(o^2) + mean(S_T^2): compare with what the reference's own
    PyTorch path produced (fixture generated by tests/golden/make_golden.py)."""

    rec = load_golden("config0_b1_t64_h2")
    leaves = [rec[n].to(DEV).requires_grad_(True) for n in ("q", "k", "v", "g", "beta", "w")]
    s0 = rec["initial_state"].to(DEV).requires_grad_(True)
    out, fin = chunk_gdn2(*leaves, s0, output_final_state=True)
    loss = out.float().square().mean() + fin.square().mean()
    grads = torch.autograd.grad(loss, leaves + [s0])
    assert abs(loss.item() - float(rec["loss"])) < 1e-3 * abs(float(rec["loss"]))
    torch.testing.assert_close(out.float().cpu(), rec["out"].float(), rtol=2e-2, atol=1e-2)
    assert oracle.rel_l2(fin, rec["final_state"]) < FP32_REL
    # The loss cotangent 2*o/n is formed from each side's own 16-bit output, so the two
    # cotangents already differ by output rounding (~3e-3); every gradient inherits that.
    for name, got in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), grads):
        assert oracle.rel_l2(got, rec[name].double()) < 8e-3, name


def test_chunk_backward_direct_api():
    cpu = oracle.make_inputs(2, 21, 2, seed=321)
    gen = torch.Generator().manual_seed(5)
    d_out = (torch.randn(cpu[2].shape, generator=gen) * 0.1).bfloat16()
    d_fin = torch.randn((2, 2, 128, 128), generator=gen) * 0.01
    _, ref_state, ref = oracle.recurrence_grads(*cpu, d_out, d_fin, scale=0.125)
    q, k, v, g, beta, w, s0 = (t.to(DEV) for t in cpu)
    grads = chunk_backward(q, k, v, g, beta, w, ref_state.float().to(DEV), d_out.to(DEV), d_fin.to(DEV),
                           0.125, initial_state=s0)
    assert len(grads) == 7
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), grads, ref):
        check_gradient(name, got, want)


def test_zero_sequence_known_answer():
    """All sequence inputs zero: the state never changes, so dq = scale S_0 dO,
    dg_t = sum_v dS_T * S_0 for every token, every other sequence gradient vanishes and
    dS_0 = dS_T exactly (same known answer as reference tests/test_backward.py:283-327)."""

    b, t, h = 1, 5, 2
    gen = torch.Generator().manual_seed(12)
    zeros = torch.zeros((b, t, h, 128), dtype=torch.bfloat16)
    g = torch.zeros((b, t, h, 128))
    s0 = torch.randn((b, h, 128, 128), generator=gen) * 0.1
    d_out = (torch.randn((b, t, h, 128), generator=gen) * 0.1).bfloat16()
    d_fin = torch.randn((b, h, 128, 128), generator=gen) * 0.01
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        grads = chunk_backward(*(x.to(DEV) for x in (zeros, zeros, zeros, g, zeros, zeros)), s0.to(DEV),
                               d_out.to(DEV), d_fin.to(DEV), 0.25, initial_state=s0.to(DEV))
    side.synchronize()
    dq, dk, dv, dg, dbeta, dw, ds0 = (x.cpu() for x in grads)
    want_dq = 0.25 * torch.einsum("bhkv,bthv->bthk", s0, d_out.float())
    torch.testing.assert_close(dq.float(), want_dq, rtol=2e-2, atol=2e-3)
    # with q = 0 the state cotangent is constant: dg_t = sum_v dS_T * S_0 for every token
    want_dg = (d_fin * s0).sum(-1).unsqueeze(1).expand(b, t, h, 128)
    torch.testing.assert_close(dg, want_dg, rtol=1e-4, atol=2e-5)
    torch.testing.assert_close(ds0, d_fin, rtol=0, atol=0)
    assert torch.count_nonzero(dbeta) == 0 and torch.count_nonzero(dw) == 0 and torch.count_nonzero(dv) == 0
    want_dk = torch.zeros_like(dk)  # dk = dS' u + beta*de with u = 0, beta = 0
    torch.testing.assert_close(dk, want_dk, rtol=0, atol=0)


def test_empty_sequence_autograd_edge():
    shape = (1, 0, 1, 128)
    inputs = [torch.empty(shape, device=DEV, dtype=torch.float32 if i == 3 else torch.bfloat16,
                          requires_grad=True) for i in range(6)]
    s0 = torch.randn((1, 1, 128, 128), device=DEV, requires_grad=True)
    out, fin = chunk_gdn2(*inputs, s0, output_final_state=True)
    assert out.shape == shape
    torch.testing.assert_close(fin, s0, rtol=0, atol=0)
    grads = torch.autograd.grad(out.float().sum() + fin.sum(), (*inputs, s0))
    assert all(gr.shape == shape for gr in grads[:-1])
    torch.testing.assert_close(grads[-1], torch.ones_like(s0), rtol=0, atol=0)


def test_gradients_without_initial_state_and_non_contiguous_cotangent():
    cpu = oracle.make_inputs(1, 10, 2, seed=808, with_state=False)
    leaves = [t.to(DEV).requires_grad_(True) for t in cpu[:6]]
    out, fin = chunk_gdn2(*leaves, output_final_state=True)
    gen = torch.Generator().manual_seed(9)
    wide = (torch.randn((1, 10, 2, 256), generator=gen) * 0.1).bfloat16()
    d_out = wide[..., ::2]  # non-contiguous upstream gradient
    assert not d_out.is_contiguous()
    grads = torch.autograd.grad((out.float() * d_out.to(DEV).float()).sum(), leaves)
    _, _, ref = oracle.recurrence_grads(*cpu, d_out.contiguous(), None)
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw"), grads, ref):
        check_gradient(name, got, want)


def test_ragged_tail_t8200_single_head_against_oracle():
    """T = 8200 = 128 full chunks + an 8-token tail: forward runs chunk kernels then token kernels,
    backward the token kernels first (reference order, backward_parallel.py:1493-1522)."""

    run_case(1, 8200, 1, seed=8200)


def test_training_configuration_shard_independence():
    """Benchmark training shape per head: B=4, T=8192 is too large for the CPU oracle in full, so
    check one (batch, head) unit of a B=2, H=4 problem against the oracle and against the same unit
    run alone (results must not depend on the rest of the grid)."""

    cpu = oracle.make_inputs(2, 8192, 4, seed=0)
    gen = torch.Generator().manual_seed(1)
    d_out = (torch.randn(cpu[2].shape, generator=gen) * 0.1).bfloat16()
    d_fin = torch.randn((2, 4, 128, 128), generator=gen) * 0.01

    def grads_of(tensors, do, df):
        leaves = [t.to(DEV).requires_grad_(True) for t in tensors]
        out, fin = chunk_gdn2(*leaves[:6], leaves[6], output_final_state=True)
        obj = (out.float() * do.to(DEV).float()).sum() + (fin * df.to(DEV)).sum()
        return out, fin, torch.autograd.grad(obj, leaves)

    out, fin, grads = grads_of(cpu, d_out, d_fin)
    sub = tuple(t[1:2, :, 2:3].contiguous() for t in cpu[:6]) + (cpu[6][1:2, 2:3].contiguous(),)
    sub_do, sub_df = d_out[1:2, :, 2:3].contiguous(), d_fin[1:2, 2:3].contiguous()
    out_s, fin_s, grads_s = grads_of(sub, sub_do, sub_df)
    assert torch.equal(out_s, out[1:2, :, 2:3]) and torch.equal(fin_s, fin[1:2, 2:3])
    for a, b in zip(grads_s[:6], grads[:6]):
        assert torch.equal(a, b[1:2, :, 2:3])
    assert torch.equal(grads_s[6], grads[6][1:2, 2:3])
    ref_out, ref_state, ref = oracle.recurrence_grads(*sub, sub_do, sub_df)
    torch.testing.assert_close(out_s.float().cpu(), ref_out.float(), rtol=2e-2, atol=1e-2)
    assert oracle.rel_l2(fin_s, ref_state) < FP32_REL
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), grads_s, ref):
        check_gradient(name, got, want)


@pytest.mark.parametrize("dtype,g_dtype", [(torch.float16, torch.float32), (torch.float16, torch.float16),
                                           (torch.bfloat16, torch.bfloat16)])
def test_chunk_path_gradient_dtypes(dtype, g_dtype):
    """The tensor-core chunk path (3 full chunks + a 7-token tail) for every sequence / gate dtype
    pair the kernels are instantiated for."""

    grads = run_case(1, 199, 2, seed=4242, dtype=dtype, g_dtype=g_dtype)
    assert grads[3].dtype == g_dtype


@pytest.mark.parametrize("dtype,g_dtype", [(torch.float16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_more_chunk_heads_than_sms(dtype, g_dtype):
    """160 chunk-heads: the persistent VJP kernel gives some CTAs a second chunk-head whose tiles were
    fetched during the first one's final phase.  One (batch, head) unit is checked against the oracle
    and, bit for bit, against the same unit run alone."""

    cpu = oracle.make_inputs(2, 1024, 5, seed=77, dtype=dtype, g_dtype=g_dtype)
    gen = torch.Generator().manual_seed(78)
    d_out = (torch.randn(cpu[2].shape, generator=gen) * 0.1).to(dtype)
    d_fin = torch.randn((2, 5, 128, 128), generator=gen) * 0.01

    def grads_of(tensors, do, df):
        leaves = [t.to(DEV).requires_grad_(True) for t in tensors]
        out, fin = chunk_gdn2(*leaves[:6], leaves[6], output_final_state=True)
        obj = (out.float() * do.to(DEV).float()).sum() + (fin * df.to(DEV)).sum()
        return out, fin, torch.autograd.grad(obj, leaves)

    out, fin, grads = grads_of(cpu, d_out, d_fin)
    sub = tuple(t[1:2, :, 3:4].contiguous() for t in cpu[:6]) + (cpu[6][1:2, 3:4].contiguous(),)
    sub_do, sub_df = d_out[1:2, :, 3:4].contiguous(), d_fin[1:2, 3:4].contiguous()
    out_s, fin_s, grads_s = grads_of(sub, sub_do, sub_df)
    assert torch.equal(out_s, out[1:2, :, 3:4]) and torch.equal(fin_s, fin[1:2, 3:4])
    for a, b in zip(grads_s[:6], grads[:6]):
        assert torch.equal(a, b[1:2, :, 3:4])
    assert torch.equal(grads_s[6], grads[6][1:2, 3:4])
    ref_out, ref_state, ref = oracle.recurrence_grads(*sub, sub_do, sub_df)
    torch.testing.assert_close(out_s.float().cpu(), ref_out.float(), rtol=2e-2, atol=1e-2)
    assert oracle.rel_l2(fin_s, ref_state) < FP32_REL
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), grads_s, ref):
        check_gradient(name, got, want)


def test_benchmark_shape_is_deterministic():
    """Two runs of the same training step at a benchmark-sized grid (2048 chunk-heads, 14 chunk-heads
    per persistent CTA) give bit-identical outputs and gradients: no result depends on warp or CTA
    timing."""

    torch.manual_seed(5)
    batch, time, heads = 2, 4096, 16
    q = torch.nn.functional.normalize(torch.randn(batch, time, heads, 128, device=DEV), dim=-1).bfloat16()
    k = torch.nn.functional.normalize(torch.randn(batch, time, heads, 128, device=DEV), dim=-1).bfloat16()
    v = torch.randn(batch, time, heads, 128, device=DEV).bfloat16()
    g = -torch.nn.functional.softplus(torch.randn(batch, time, heads, 128, device=DEV) - 2.0).clamp(max=5.0)
    beta = torch.sigmoid(torch.randn(batch, time, heads, 128, device=DEV)).bfloat16()
    w = torch.sigmoid(torch.randn(batch, time, heads, 128, device=DEV)).bfloat16()
    s0 = 0.02 * torch.randn(batch, heads, 128, 128, device=DEV)
    d_out = (0.1 * torch.randn(batch, time, heads, 128, device=DEV)).bfloat16()

    def run():
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v, g, beta, w, s0)]
        out, fin = chunk_gdn2(*leaves[:6], leaves[6], output_final_state=True)
        grads = torch.autograd.grad((out.float() * d_out.float()).sum() + fin.square().sum(), leaves)
        return (out, fin, *grads)

    first = run()
    second = run()
    for a, b in zip(first, second):
        assert torch.equal(a, b)
    assert all(torch.isfinite(t.float()).all() for t in first)


def test_full_training_configuration_far_corner():
    """The benchmark's training configuration in full (B=4, T=8192, H=32: 16 384 chunk-heads, 4.3 GB of
    state checkpoints and as much again for their cotangents, so offsets pass 2^32): the last
    (batch, head) unit, whose data sits at the far end of every buffer, must equal the same unit run
    alone bit for bit (the unit-sized problem is checked against the oracle by the tests above)."""

    torch.manual_seed(11)
    batch, time, heads = 4, 8192, 32
    shape = (batch, time, heads, 128)
    q = torch.nn.functional.normalize(torch.randn(shape, device=DEV), dim=-1).bfloat16()
    k = torch.nn.functional.normalize(torch.randn(shape, device=DEV), dim=-1).bfloat16()
    v = torch.randn(shape, device=DEV).bfloat16()
    g = -torch.nn.functional.softplus(torch.randn(shape, device=DEV) - 2.0).clamp(max=5.0)
    beta = torch.sigmoid(torch.randn(shape, device=DEV)).bfloat16()
    w = torch.sigmoid(torch.randn(shape, device=DEV)).bfloat16()
    s0 = 0.02 * torch.randn(batch, heads, 128, 128, device=DEV)
    d_out = (0.1 * torch.randn(shape, device=DEV)).bfloat16()
    d_fin = 0.01 * torch.randn(batch, heads, 128, 128, device=DEV)

    def run(tensors, do, df):
        leaves = [t.clone().requires_grad_(True) for t in tensors]
        out, fin = chunk_gdn2(*leaves[:6], leaves[6], output_final_state=True)
        grads = torch.autograd.grad((out.float() * do.float()).sum() + (fin * df).sum(), leaves)
        return out, fin, grads

    out, fin, grads = run((q, k, v, g, beta, w, s0), d_out, d_fin)
    b, h = batch - 1, heads - 1
    sub = tuple(t[b:b + 1, :, h:h + 1].contiguous() for t in (q, k, v, g, beta, w)) + (s0[b:b + 1, h:h + 1].contiguous(),)
    out_s, fin_s, grads_s = run(sub, d_out[b:b + 1, :, h:h + 1].contiguous(), d_fin[b:b + 1, h:h + 1].contiguous())
    assert torch.equal(out_s, out[b:b + 1, :, h:h + 1]) and torch.equal(fin_s, fin[b:b + 1, h:h + 1])
    for a, full in zip(grads_s[:6], grads[:6]):
        assert torch.equal(a, full[b:b + 1, :, h:h + 1])
    assert torch.equal(grads_s[6], grads[6][b:b + 1, h:h + 1])
    assert all(torch.isfinite(t.float()).all() for t in grads)


# ---- untested-before configurations ---------------------------------------------------------------
def _device_inputs(batch, time, heads, seed):
    torch.manual_seed(seed)
    shape = (batch, time, heads, 128)
    q = torch.nn.functional.normalize(torch.randn(shape, device=DEV), dim=-1).bfloat16()
    k = torch.nn.functional.normalize(torch.randn(shape, device=DEV), dim=-1).bfloat16()
    v = torch.randn(shape, device=DEV).bfloat16()
    g = -torch.nn.functional.softplus(torch.randn(shape, device=DEV) - 2.0).clamp(max=5.0)
    beta = torch.sigmoid(torch.randn(shape, device=DEV)).bfloat16()
    w = torch.sigmoid(torch.randn(shape, device=DEV)).bfloat16()
    s0 = 0.02 * torch.randn(batch, heads, 128, 128, device=DEV)
    d_out = (0.1 * torch.randn(shape, device=DEV)).bfloat16()
    d_fin = 0.01 * torch.randn(batch, heads, 128, 128, device=DEV)
    return (q, k, v, g, beta, w, s0), d_out, d_fin


def _step(tensors, d_out, d_fin):
    leaves = [t.clone().requires_grad_(True) for t in tensors]
    out, fin = chunk_gdn2(*leaves[:6], leaves[6], output_final_state=True)
    grads = torch.autograd.grad((out.float() * d_out.float()).sum() + (fin * d_fin).sum(), leaves)
    return out, fin, grads


def _unit(tensors, d_out, d_fin, b, h):
    sub = tuple(t[b:b + 1, :, h:h + 1].contiguous() for t in tensors[:6]) + (tensors[6][b:b + 1, h:h + 1].contiguous(),)
    return sub, d_out[b:b + 1, :, h:h + 1].contiguous(), d_fin[b:b + 1, h:h + 1].contiguous()


def _check_unit_alone_and_against_oracle(tensors, d_out, d_fin, b, h, full):
    out, fin, grads = full
    sub, sub_do, sub_df = _unit(tensors, d_out, d_fin, b, h)
    out_s, fin_s, grads_s = _step(sub, sub_do, sub_df)
    assert torch.equal(out_s, out[b:b + 1, :, h:h + 1]) and torch.equal(fin_s, fin[b:b + 1, h:h + 1])
    for a, whole in zip(grads_s[:6], grads[:6]):
        assert torch.equal(a, whole[b:b + 1, :, h:h + 1])
    assert torch.equal(grads_s[6], grads[6][b:b + 1, h:h + 1])
    cpu = [t.cpu() for t in sub]
    ref_out, ref_state, ref = oracle.recurrence_grads(*cpu, sub_do.cpu(), sub_df.cpu())
    torch.testing.assert_close(out_s.float().cpu(), ref_out.float(), rtol=2e-2, atol=1e-2)
    check_gradient("out", out_s, ref_out)  # (relative: the outputs are of the order of atol above)
    assert oracle.rel_l2(fin_s, ref_state) < FP32_REL
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), grads_s, ref):
        check_gradient(name, got, want)


@pytest.mark.slow
def test_sequence_length_16384_unit_against_oracle_and_inside_a_grid():
    """T = 16384 (the sequence length of the 8-GPU configuration; 256 chunks per head): one
    (batch, head) unit of a B=2, H=4 grid equals the unit run alone bit for bit, and the unit agrees
    with the float64 recurrence."""

    tensors, d_out, d_fin = _device_inputs(2, 16384, 4, seed=16384)
    full = _step(tensors, d_out, d_fin)
    _check_unit_alone_and_against_oracle(tensors, d_out, d_fin, 1, 2, full)


@pytest.mark.slow
def test_ragged_tail_t8200_full_training_grid():
    """B=4, T=8200, H=32: the 8-token tail runs on the token kernels for all 128 heads at once (before
    the chunks in backward, after them in forward).  The far-corner unit equals the unit run alone bit
    for bit and agrees with the float64 recurrence."""

    tensors, d_out, d_fin = _device_inputs(4, 8200, 32, seed=8201)
    full = _step(tensors, d_out, d_fin)
    assert all(torch.isfinite(t.float()).all() for t in full[2])
    _check_unit_alone_and_against_oracle(tensors, d_out, d_fin, 3, 31, full)


# ---- fp32 values of the 16-bit gradients (before their final cast) --------------------------------
@pytest.mark.parametrize("time,heads", [(256, 2), (1024, 1)])
def test_chunk_backward_fp32_gradients_meet_the_fp32_tolerance(time, heads):
    """gdn2_chunk_backward_f32grads writes dq, dk, dv, dbeta, dw as fp32: every gradient of the chunk
    path is then within 1e-3 relative L2 of the float64 recurrence, the tolerance the 16-bit tensors
    cannot show because their own rounding costs ~2e-3."""

    from gdn2_sm120_b200 import chunk_kernels
    from gdn2_sm120_b200.chunk import chunk_forward

    cpu = oracle.make_inputs(1, time, heads, seed=5150 + time)
    gen = torch.Generator().manual_seed(5151)
    d_out = (torch.randn(cpu[2].shape, generator=gen) * 0.1).bfloat16()
    d_fin = torch.randn(cpu[6].shape, generator=gen) * 0.01
    _, _, ref = oracle.recurrence_grads(*cpu, d_out, d_fin)
    q, k, v, g, beta, w, s0 = (t.to(DEV) for t in cpu)
    scale = 128 ** -0.5
    _, _, aux = chunk_forward(q, k, v, g, beta, w, s0, scale=scale, return_aux=True)
    grads = tuple(torch.empty(x.shape, device=DEV, dtype=torch.float32) for x in (q, k, v, g, beta, w))
    d_s0 = torch.empty_like(s0)
    chunk_kernels.backward(q, k, v, g, beta, w, aux.workspace, aux.chunk_boundaries, d_out.to(DEV),
                           d_fin.to(DEV), grads, d_s0, 1, time, heads, time, scale, f32_grads=True)
    assert chunk_kernels.read_status(aux.workspace, 1, time, heads) == 0
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), (*grads, d_s0), ref):
        err = oracle.rel_l2(got, want)
        assert err < FP32_REL, f"{name}: rel-L2 {err:.3e}"


# ---- stage level: what the kernels leave in their buffers ------------------------------------------
def _unblock(raw, rows, cols, rs, cs):
    """Read a blocked fp32 tile X[r][c] (8-row x 16-byte core matrices, byte strides rs / cs) out of
    a uint8 buffer."""

    r = torch.arange(rows, device=raw.device).view(-1, 1)
    c = torch.arange(cols, device=raw.device).view(1, -1)
    offset = (r // 8) * rs + (c // 4) * cs + (r % 8) * 16 + (c % 4) * 4
    return raw.view(torch.float32)[(offset // 4).reshape(-1)].view(rows, cols)


def test_stage_level_residual_dz_and_boundary_cotangent_against_stage_oracle():
    """One chunk-head (the inputs of the stage fixture generated from the reference's proofs): the
    residual R the forward scan saves, dZ = T^T dR that the reverse scan hands to the VJP kernel and
    the cotangent at the chunk start, against oracle.chunk_wy_forward / chunk_wy_vjp and the fixture."""

    from gdn2_sm120_b200 import chunk_kernels
    from gdn2_sm120_b200.chunk import chunk_forward

    rec = load_golden("stage_chunk64")
    q, k, v, g, beta, w = (rec[n].to(DEV) for n in ("q", "k", "v", "g", "beta", "w"))
    s0, d_out, d_s1 = rec["initial_state"].to(DEV), rec["d_out"].to(DEV), rec["d_s1"].to(DEV)
    scale = rec["scale"]
    out, fin, aux = chunk_forward(q, k, v, g, beta, w, s0, scale=scale, return_aux=True)
    grads = tuple(torch.empty_like(x) for x in (q, k, v, g, beta, w))
    d_s0 = torch.empty_like(s0)
    d_bnd, scratch = chunk_kernels.backward(q, k, v, g, beta, w, aux.workspace, aux.chunk_boundaries, d_out,
                                            d_s1, grads, d_s0, 1, 64, 1, 64, scale, keep_d_boundaries=True)
    torch.cuda.synchronize()
    seq = tuple(rec[n][0, :, 0] for n in ("q", "k", "v", "g", "beta", "w"))
    f = oracle.chunk_wy_forward(*seq, rec["initial_state"][0, 0], scale=scale)
    # training workspace of one chunk-head: D (512 B), status block (256 B), the residual R [64][128],
    # then the other row-major tiles both scans read:
    # Q [64][128], Kn [64][128], Yt [128][64] (32 KiB each), At [64][64], Tt [64][64] (16 KiB each)
    ws0 = aux.workspace[0]
    off_rn = 512 + 256
    assert ws0.numel() == off_rn + 4 * 32768 + 2 * 16384
    resid = ws0[off_rn:off_rn + 32768].view(torch.float32).view(64, 128)
    assert oracle.rel_l2(resid, f["R"]) < FP32_REL
    tiles = ws0[off_rn + 32768:].view(torch.float32)
    tile_q, tile_kn = tiles[:8192].view(64, 128), tiles[8192:16384].view(64, 128)
    tile_yt, tile_at = tiles[16384:24576].view(128, 64), tiles[24576:28672].view(64, 64)
    tile_tt = tiles[28672:32768].view(64, 64)
    # both are zero where j > i; the quadrant j >= 32, i < 32 is neither written nor read
    tile_at, tile_tt = tile_at.clone(), tile_tt.clone()
    tile_at[32:, :32] = 0
    tile_tt[32:, :32] = 0
    # tf32 operands: 2^-11 relative per element
    assert oracle.rel_l2(tile_q, f["Qg"]) < FP32_REL and oracle.rel_l2(tile_kn, f["Kt"]) < FP32_REL
    assert oracle.rel_l2(tile_yt, f["Y"].T) < FP32_REL and oracle.rel_l2(tile_at, f["A"].T) < FP32_REL
    assert oracle.rel_l2(tile_tt, f["T"].T) < FP32_REL
    d_r = f["A"].T @ rec["d_out"][0, :, 0].double() + f["Kt"] @ rec["d_s1"][0, 0].double()
    d_z = f["T"].T @ d_r
    got_dz = _unblock(scratch[:36864], 64, 128, 4608, 144)   # padded strides of the VJP kernel's tile
    assert oracle.rel_l2(got_dz, d_z) < FP32_REL
    # boundary cotangents: slot 1 is dS1 as given, slot 0 the cotangent at the chunk start
    assert torch.equal(d_bnd[0, 1, 0], d_s1[0, 0])
    assert oracle.rel_l2(d_bnd[0, 0, 0], rec["d_s0"][0, 0]) < FP32_REL
    assert torch.equal(d_bnd[0, 0, 0], d_s0[0, 0])
    assert torch.equal(aux.chunk_boundaries[0, 0, 0], s0[0, 0]) and torch.equal(aux.chunk_boundaries[0, 1, 0], fin[0, 0])
    assert oracle.rel_l2(fin[0, 0], rec["final_state"][0, 0]) < FP32_REL
    for name, got in zip(("dq", "dk", "dv", "dg", "dbeta", "dw"), grads):
        check_gradient(name, got[0, :, 0], rec["stage_" + name][0, :, 0].double())


# ---- batch waves -------------------------------------------------------------------------------------
@pytest.mark.parametrize("time", [320, 330])
def test_batch_waves_give_the_single_wave_result(monkeypatch, time):
    """With a scratch budget that admits one batch row per wave the forward and backward run as three
    waves sharing one scratch buffer: outputs and gradients equal the single-wave run bit for bit
    (320 tokens = 5 whole chunks; 330 = 6 chunks, the last one with 10 of its 64 tokens)."""

    from gdn2_sm120_b200 import chunk_kernels

    tokens = chunk_kernels.supported_tokens(time)
    tensors, d_out, d_fin = _device_inputs(3, time, 2, seed=77)
    single = _step(tensors, d_out, d_fin)
    assert len(chunk_kernels.plan_waves(3, tokens, 2, training=True)) == 1
    monkeypatch.setattr(chunk_kernels, "SCRATCH_BUDGET_BYTES", chunk_kernels._backward_wave_bytes(1, tokens, 2))
    assert chunk_kernels.plan_waves(3, tokens, 2, training=True) == [(0, 1), (1, 2), (2, 3)]
    waved = _step(tensors, d_out, d_fin)
    assert torch.equal(single[0], waved[0]) and torch.equal(single[1], waved[1])
    for a, b in zip(single[2], waved[2]):
        assert torch.equal(a, b)


def test_memory_check_names_the_bytes():
    from gdn2_sm120_b200 import chunk_kernels

    with pytest.raises(ValueError, match=r"needs 1000000000000000 bytes .* of device memory"):
        chunk_kernels.check_memory(10 ** 15, torch.device(DEV, torch.cuda.current_device()), "chunk forward")


# ---- the direct backward API ---------------------------------------------------------------------------
def test_chunk_backward_rejects_a_final_state_it_cannot_reproduce():
    """A forward that started from a non-zero state, differentiated without `initial_state`: the
    reference accepts this up to 128 tokens (it inverts the recurrence from `final_state`,
    backward.py:1286-1298); here the forward is re-run from zero, arrives elsewhere and the call raises
    instead of returning the gradients of a different forward."""

    cpu = oracle.make_inputs(1, 12, 2, seed=90)
    _, ref_state = oracle.recurrence(*cpu, scale=0.125)
    q, k, v, g, beta, w, s0 = (t.to(DEV) for t in cpu)
    d_out = torch.zeros_like(v)
    d_fin = torch.ones_like(s0)
    with pytest.raises(ValueError, match="initial_state"):
        chunk_backward(q, k, v, g, beta, w, ref_state.float().to(DEV), d_out, d_fin, 0.125)
    grads = chunk_backward(q, k, v, g, beta, w, ref_state.float().to(DEV), d_out, d_fin, 0.125, initial_state=s0)
    assert len(grads) == 7


def test_chunk_backward_direct_api_uses_the_chunk_kernels_from_64_tokens():
    from gdn2_sm120_b200 import _lib

    cpu = oracle.make_inputs(1, 256, 2, seed=256)
    gen = torch.Generator().manual_seed(6)
    d_out = (torch.randn(cpu[2].shape, generator=gen) * 0.1).bfloat16()
    d_fin = torch.randn((1, 2, 128, 128), generator=gen) * 0.01
    _, ref_state, ref = oracle.recurrence_grads(*cpu, d_out, d_fin)
    q, k, v, g, beta, w, s0 = (t.to(DEV) for t in cpu)
    _lib.KERNEL_EVENTS = {}
    try:
        grads = chunk_backward(q, k, v, g, beta, w, ref_state.float().to(DEV), d_out.to(DEV), d_fin.to(DEV),
                               initial_state=s0)
        called = set(_lib.KERNEL_EVENTS)
    finally:
        _lib.KERNEL_EVENTS = None
    assert called == {"gdn2_chunk_forward", "gdn2_chunk_backward"}
    for name, got, want in zip(("dq", "dk", "dv", "dg", "dbeta", "dw", "dS0"), grads, ref):
        check_gradient(name, got, want)
