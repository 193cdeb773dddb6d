"""The weights' FP32 arithmetic on the exact path (GPU): rounding and range."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import rel_l2
from oracle import oracle

pytestmark = pytest.mark.gpu

METHOD = {"straight_ray": "migrate_tile", "curved_ray": "migrate_tile_curved_ray",
          "anisotropic_vti": "migrate_tile_vti", "curved_vti": "migrate_tile_curved_vti"}


def _case(kind, amps, k0=0.5):
    from pstm_b200.base import KernelConfig, OutputTile, VelocitySlice, create_trace_block
    rng = np.random.default_rng(31)
    n = len(amps)
    mid, half = rng.uniform(-900.0, 1100.0, (n, 2)), rng.uniform(-500.0, 500.0, (n, 2))
    s, r = mid - half, mid + half
    tb = create_trace_block(amps, s[:, 0], s[:, 1], r[:, 0], r[:, 1], sample_rate_ms=4.0)
    cfg = KernelConfig(max_aperture_m=1e5, min_aperture_m=1e5, taper_fraction=0.0, aa_enabled=False, kernel_type=kind,
                       vti_eta_constant=0.1, curved_ray_k=k0)
    nt = 128
    out = lambda: OutputTile(image=np.zeros((2, 4, nt)), fold=np.zeros((2, 4, nt), np.int32),   # noqa: E731
                             x_axis=20.0 * np.arange(2), y_axis=20.0 * np.arange(4),
                             t_axis_ms=800.0 + 11.0 * np.arange(nt))
    return tb, VelocitySlice(vrms=2000.0 + 3.0 * np.arange(nt), is_1d=True), cfg, out


@pytest.mark.parametrize("kind,k0", [("anisotropic_vti", 0.5), ("curved_ray", 0.5), ("curved_ray", 0.0),
                                     ("curved_vti", 0.5), ("curved_vti", 0.0)])
def test_traveltime_of_the_weights_is_rounded(kind, k0, cuda_kernel_factory):
    """Traces of ones leave nothing but the weights.  A traveltime rounded to FP32
    leaves them without a bias; one cut to 24 bits is short by half a unit in the
    last place, 2^-25 to 2^-24 of it, and the weight K / T^2 long by twice that,
    8.6e-8 on average.  The other roundings are of either sign: three per pair, and
    one of K per point, 3e-8 / sqrt(1024 points).  Bound: a third of the cut's."""
    tb, vel, cfg, out = _case(kind, np.ones((2000, 1500), np.float32), k0)
    got, ref = out(), out()
    getattr(cuda_kernel_factory(cfg), METHOD[kind])(tb, got, vel)
    oracle.migrate(tb, ref, vel, cfg, kind=kind)
    assert np.all(ref.image > 0)
    assert abs(np.mean(got.image / ref.image - 1.0)) <= 3e-8


@pytest.mark.parametrize("scale", [2.0 ** -116, 2.0 ** 100])
@pytest.mark.parametrize("kind,k0", [("straight_ray", 0.5), ("anisotropic_vti", 0.5), ("curved_ray", 0.5),
                                     ("curved_ray", 0.0), ("curved_vti", 0.5), ("curved_vti", 0.0)])
def test_amplitudes_near_the_ends_of_fp32(kind, k0, scale, cuda_kernel_factory):
    """Weights of about 2^-12 leave an amplitude of 2^-116 a normal FP32 number; the
    steps on the way to the product must not lose what the product keeps."""
    amps = np.random.default_rng(3).standard_normal((300, 900)).astype(np.float32)
    tb, vel, cfg, out = _case(kind, amps, k0)
    tiny = dataclasses.replace(tb, amplitudes=(np.asarray(tb.amplitudes, np.float64) * scale).astype(np.float32))
    got, ref = out(), out()
    getattr(cuda_kernel_factory(cfg), METHOD[kind])(tiny, got, vel)
    oracle.migrate(tiny, ref, vel, cfg, kind=kind)
    assert rel_l2(got.image / scale, ref.image / scale) <= 1e-5
