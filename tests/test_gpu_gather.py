"""The gather kernel at the sizes where its tiling can go wrong (GPU).

A CTA takes 8 pillars and 64 output times, traces in chunks of 32 shared over
up to 8 CTAs of a cluster, and a window of every trace row, copied from the
16-byte boundary below it.  Sizes here sit one below, on and above those; the
panel's rows are packed (no padding), so they start on any element; and the
windows are made not to fit (a velocity that jumps), to cover the whole row
(eta below the bounds' range) and to hang over either end of the trace.

Against the FP64 oracle: fold bit-exact, image relative L2 <= 1e-5 with the
FP64 sample index and <= 1e-4 with FP32 traveltime, the tolerances of
tests/test_gpu_parity.py for FP32 traces.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2
from oracle import oracle

pytestmark = pytest.mark.gpu

METHOD = {"straight_ray": "migrate_tile", "curved_ray": "migrate_tile_curved_ray",
          "anisotropic_vti": "migrate_tile_vti", "curved_vti": "migrate_tile_curved_vti"}
BASE = dict(nx=5, ny=6, nt=70, n=90, ns=120, t0=0.0, dt_out=4.0, kind="straight_ray", precision="exact", eta=0.1,
            jump=1.0, aperture=900.0, taper=0.1, aa=True, weights=False, k=0.5, spread=1500.0)
CASES = {
    "one_of_everything": dict(nx=1, ny=1, nt=1, n=1, ns=2, t0=0.0),
    "below_a_block": dict(nx=1, ny=7, nt=63, n=31, ns=101),
    "a_block": dict(nx=2, ny=4, nt=64, n=32, ns=104),
    "above_a_block": dict(nx=3, ny=9, nt=65, n=33, ns=103),
    "every_split_used": dict(nx=2, ny=4, nt=64, n=8 * 32 + 1),
    "odd_rows_weights": dict(ns=117, n=300, weights=True),
    "late_record": dict(t0=100.0, ns=61),
    "short_record": dict(ns=40),
    "hard_cut": dict(taper=0.0),
    "coarse_times": dict(dt_out=32.0, nt=130, ns=1100),
    "window_too_long": dict(jump=40.0, nt=100, dt_out=40.0, ns=3000, spread=8000.0, aperture=4000.0),
    "vti_unbounded_eta": dict(kind="anisotropic_vti", eta=-0.2),
    "vti_negative_eta": dict(kind="anisotropic_vti", eta=-0.1),
    "vti": dict(kind="anisotropic_vti", nt=129),
    "curved": dict(kind="curved_ray", nt=129),
    "curved_falling": dict(kind="curved_ray", k=-0.3),
    "curved_straight": dict(kind="curved_ray", k=0.0),
    "curved_vti": dict(kind="curved_vti", nt=129),
    "curved_vti_negative_eta": dict(kind="curved_vti", eta=-0.1),
    "fast_trace_ends": dict(precision="fast", ns=70),
    "fp32_trace_ends": dict(precision="fp32", ns=70, weights=True),
    "fp32_curved_vti": dict(precision="fp32", kind="curved_vti", n=300),
}


@pytest.mark.parametrize("trace_dtype", ["f32", "bf16"])
@pytest.mark.parametrize("name", list(CASES))
def test_edges_of_the_tiling(name, trace_dtype, cuda_kernel_factory):
    from pstm_b200.base import KernelConfig, OutputTile, VelocitySlice, create_trace_block
    from pstm_b200.cuda_kernel import bf16_bits_to_float32, float32_to_bf16_bits
    c = {**BASE, **CASES[name]}
    rng = np.random.default_rng(17)
    s, r = rng.uniform(0, c["spread"], (c["n"], 2)), rng.uniform(0, c["spread"], (c["n"], 2))
    amps = rng.standard_normal((c["n"], c["ns"])).astype(np.float32)
    amps = np.cumsum(amps, axis=1) - 0.8 * np.roll(np.cumsum(amps, axis=1), 3, axis=1)   # band-limited
    amps = bf16_bits_to_float32(float32_to_bf16_bits(amps.astype(np.float32)))
    w = rng.uniform(0.5, 2.0, c["n"]) if c["weights"] else None
    tb = create_trace_block(amps, s[:, 0], s[:, 1], r[:, 0], r[:, 1], sample_rate_ms=4.0, start_time_ms=c["t0"],
                            weights=w)
    t = np.arange(c["nt"]) * c["dt_out"]
    v = 1600.0 + 400.0 * np.arange(c["nt"]) / c["nt"]
    v[c["nt"] // 2:] *= c["jump"]   # in the middle of a block
    vel = VelocitySlice(vrms=v, is_1d=True)
    cfg = KernelConfig(max_aperture_m=c["aperture"], min_aperture_m=300.0, taper_fraction=c["taper"],
                       aa_enabled=c["aa"], grid_dx=20.0, grid_dy=20.0, kernel_type=c["kind"], curved_ray_v0=1500.0,
                       curved_ray_k=c["k"], vti_eta_constant=c["eta"])
    shape = (c["nx"], c["ny"], c["nt"])

    def out():
        return OutputTile(image=np.zeros(shape), fold=np.zeros(shape, np.int32),
                          x_axis=600.0 + 20.0 * np.arange(c["nx"]), y_axis=650.0 + 20.0 * np.arange(c["ny"]),
                          t_axis_ms=t)
    k = cuda_kernel_factory(cfg, trace_dtype=trace_dtype, precision=c["precision"])
    got, ref = out(), out()
    getattr(k, METHOD[c["kind"]])(tb, got, vel)
    oracle.migrate(tb, ref, vel, cfg, kind=c["kind"])
    np.testing.assert_array_equal(got.fold, ref.fold)
    assert rel_l2(got.image, ref.image) <= (1e-5 if c["precision"] == "exact" else 1e-4)
