"""The FP16 panel conversion where its vectors can go wrong (GPU): rows that start
on any element, fewer samples than a vector, the longest row held in registers
and longer ones, and source rows that do not start where the destination's do.
Bit for bit the NumPy rule (``scaled_f16``), weights included."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 2, 3, 4, 5, 7, 127, 501, 1501, 2048, 2049, 2051, 2055, 5001])
@pytest.mark.parametrize("offset,pad", [(0, 0), (1, 0), (3, 0), (0, 1), (2, 6)])
def test_f16_panel_rows(ns, offset, pad, cuda_kernel_factory):
    import torch
    from pstm_b200.base import KernelConfig, TraceBlock
    from pstm_b200.cuda_kernel import scaled_f16
    n = 19
    rng = np.random.default_rng(ns)
    a = (rng.standard_normal((n, ns)) * 10.0 ** rng.uniform(-6, 6, (n, 1))).astype(np.float32)
    a[3] = 0.0
    a[5, -1] = 1e7   # the largest sample is the last
    a[6, 0] = -1e7   # or the first
    buf = torch.zeros(offset + n * (ns + pad), dtype=torch.float32, device="cuda")
    view = buf[offset:].view(n, ns + pad)[:, :ns]
    view.copy_(torch.as_tensor(a))
    z = torch.zeros(n, dtype=torch.float64, device="cuda")
    tb = TraceBlock(amplitudes=view, source_x=z, source_y=z, receiver_x=z, receiver_y=z, offset=z, midpoint_x=z,
                    midpoint_y=z, weights=None, sample_rate_ms=2.0)
    got = cuda_kernel_factory(KernelConfig()).to_f16_panel(tb)
    want, inv = scaled_f16(a)
    np.testing.assert_array_equal(got.amplitudes.cpu().numpy().view(np.uint16), want.view(np.uint16))
    np.testing.assert_array_equal(got.weights.cpu().numpy(), inv)
