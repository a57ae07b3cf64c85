"""GPU tests of calls at the edge of what the entry points accept: buffers of the smallest documented alignment,
non-finite values, strong decays, flags that are no booleans, threads beside a blocked launch."""

from __future__ import annotations

import pytest
import torch

import gdn2_oracle as oracle
from gdn2_sm120_b200 import _lib, chunk_kernels

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
