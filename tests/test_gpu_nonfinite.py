"""Geometry that is not finite (GPU): such a trace adds nothing to the image.

A traveltime that is infinite or not a number has no sample index, so no pair of
the trace is inside its record; the fold asks the midpoint alone.  Expected is the
FP64 oracle on the panel with the trace's weight 0 in finite geometry (and, where
the midpoint is not finite, far away: it is in no aperture).  Tolerances as in
tests/test_gpu_parity.py.
"""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import rel_l2
from oracle import oracle

pytestmark = pytest.mark.gpu

METHOD = {"straight_ray": "migrate_tile", "curved_ray": "migrate_tile_curved_ray",
          "anisotropic_vti": "migrate_tile_vti", "curved_vti": "migrate_tile_curved_vti"}
ARRAYS = ["source_x", "source_y", "receiver_x", "receiver_y", "midpoint_x", "midpoint_y"]


@pytest.mark.parametrize("k0", [0.5, 0.0])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e200])
@pytest.mark.parametrize("precision", ["exact", "fast", "fp32"])
@pytest.mark.parametrize("kind", list(METHOD))
def test_trace_with_a_coordinate_that_is_not_finite(kind, precision, value, k0, cuda_kernel_factory):
    from pstm_b200.base import KernelConfig, OutputTile, VelocitySlice, create_trace_block
    rng = np.random.default_rng(5)
    n, nt = 60, 70
    mid, half = rng.uniform(-200.0, 300.0, (n, 2)), rng.uniform(-300.0, 300.0, (n, 2))
    s, r = mid - half, mid + half
    amps = 1.0 + 0.1 * rng.standard_normal((n, 250)).astype(np.float32)   # every sample counts
    tb = create_trace_block(amps, s[:, 0], s[:, 1], r[:, 0], r[:, 1], sample_rate_ms=4.0, weights=np.ones(n))
    bad = dataclasses.replace(tb, **{a: np.array(getattr(tb, a)) for a in ARRAYS})
    good = dataclasses.replace(tb, **{a: np.array(getattr(tb, a)) for a in ARRAYS}, weights=np.ones(n))
    for i, a in enumerate(ARRAYS):
        getattr(bad, a)[3 + 7 * i] = value
        good.weights[3 + 7 * i] = 0.0
        if a.startswith("mid"):
            getattr(good, a)[3 + 7 * i] = 1e7
    cfg = KernelConfig(max_aperture_m=900.0, min_aperture_m=300.0, kernel_type=kind, grid_dx=20.0, grid_dy=20.0,
                       vti_eta_constant=0.1, curved_ray_k=k0)
    vel = VelocitySlice(vrms=np.full(nt, 2000.0), is_1d=True)

    def out():
        return OutputTile(image=np.zeros((3, 5, nt)), fold=np.zeros((3, 5, nt), np.int32),
                          x_axis=20.0 * np.arange(3), y_axis=20.0 * np.arange(5), t_axis_ms=40.0 + 4.0 * np.arange(nt))
    k = cuda_kernel_factory(cfg, precision=precision)
    got, ref = out(), out()
    getattr(k, METHOD[kind])(bad, got, vel)
    oracle.migrate(good, ref, vel, cfg, kind=kind)
    np.testing.assert_array_equal(got.fold, ref.fold)
    assert rel_l2(got.image, ref.image) <= (1e-5 if precision == "exact" else 1e-4)
