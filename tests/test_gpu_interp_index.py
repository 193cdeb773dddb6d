"""The interpolators at chosen sample indices (GPU).

One trace with its source and receiver on the pillar and all weights off: the
image at t is the trace at t, so the times choose the index.  The index is formed
in FP64 to about 2^-44 of itself (2^-38 samples here), on the fast path too, and
decides in FP64 which sample is nearest.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _at(trace, s, method, precision, factory):
    """The interpolated trace at the sample indices s."""
    from pstm_b200.base import KernelConfig, OutputTile, VelocitySlice, create_trace_block
    z = np.zeros(1)
    cfg = KernelConfig(max_aperture_m=1000.0, min_aperture_m=500.0, apply_spreading=False, apply_obliquity=False,
                       aa_enabled=False, interpolation_method=method)
    out = OutputTile(image=np.zeros((1, 1, len(s))), fold=np.zeros((1, 1, len(s)), np.int32), x_axis=z, y_axis=z,
                     t_axis_ms=4.0 * np.asarray(s))
    tb = create_trace_block(np.asarray(trace, np.float32)[None], z, z, z, z, sample_rate_ms=4.0)
    k = factory(cfg, precision=precision)
    k.migrate_tile(tb, out, VelocitySlice(vrms=np.full(len(s), 2000.0), is_1d=True))
    return out.image[0, 0]


def _trace(n=64):
    return np.random.default_rng(9).uniform(-1.0, 1.0, n).astype(np.float32)


@pytest.mark.parametrize("precision", ["exact", "fast", "fp32"])
@pytest.mark.parametrize("method", ["nearest", "sinc4", "sinc8", "sinc16"])
def test_nearest_sample_is_decided_in_fp64(method, precision, cuda_kernel_factory):
    """Fractions 2^-26 to 2^-31 below and above one half: an FP32 fraction has them
    all at one half.  Sums of at most 16 FP32 products of weights whose magnitudes
    add up to less than 3: 16 x 3 x 2^-24 = 2.9e-6 of the largest sample."""
    tr = _trace()
    i = 12 + np.arange(40)
    s = i + 0.5 + np.where(np.arange(40) % 2, 1.0, -1.0) * 2.0 ** -(26.0 + np.arange(40) % 6)
    got = _at(tr, s, method, precision, cuda_kernel_factory)
    ref = np.array([oracle.interp(tr, x, method) for x in s])
    assert np.abs(got - ref).max() <= (1e-10 if precision == "exact" else 3e-6)


@pytest.mark.parametrize("precision", ["exact", "fast"])
@pytest.mark.parametrize("method", ["lanczos3", "lanczos5", "sinc8"])
def test_fractions_beside_a_sample(method, precision, cuda_kernel_factory):
    """Fractions 2^-6 to 2^-31 away from a sample, on either side."""
    tr = _trace()
    i = 12 + np.arange(40)
    eps = 2.0 ** -(6.0 + (np.arange(40) // 2) * 1.3)
    s = i + np.where(np.arange(40) % 2, eps, 1.0 - eps)
    got = _at(tr, s, method, precision, cuda_kernel_factory)
    ref = np.array([oracle.interp(tr, x, method) for x in s])
    assert np.abs(got - ref).max() <= (1e-10 if precision == "exact" else 3e-6)


@pytest.mark.parametrize("precision", ["exact", "fast", "fp32"])
@pytest.mark.parametrize("method", ["nearest", "sinc4", "sinc8", "sinc16", "lanczos3", "lanczos5"])
def test_on_a_sample_the_others_do_not_count(method, precision, cuda_kernel_factory):
    """Within 1e-10 of a sample nearest and the wide methods return it, even beside samples that
    are not finite (the taps' weights there are 0, and 0 x NaN is NaN)."""
    tr = _trace()
    tr[[20, 30, 40]] = np.nan, np.inf, -np.inf
    s = np.array([22.0, 23.0, 28.0, 32.0, 38.0, 42.0])
    got = _at(tr, s, method, precision, cuda_kernel_factory)
    assert np.abs(got - tr[s.astype(int)]).max() <= 1e-9
