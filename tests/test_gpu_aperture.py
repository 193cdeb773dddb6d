"""Apertures at their limits (GPU): a maximum below the minimum, and none at all.

The reference drops a trace beyond the maximum aperture before it looks at the
time-varying one (numba_cpu_optimized.py:168-175), and raises the time-varying
one to the minimum without another look at the maximum, so a maximum below the
minimum cuts image and fold alike.

Against the FP64 oracle: fold bit-exact, image relative L2 <= 1e-5 with the
FP64 sample index and <= 1e-4 with FP32 traveltime, the tolerances of
tests/test_gpu_parity.py for FP32 traces.
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


def _case(kind="straight_ray", nt=140, n=400, **kw):
    from pstm_b200.base import KernelConfig, VelocitySlice, create_trace_block
    rng = np.random.default_rng(23)
    mid, half = rng.uniform(-500.0, 800.0, (n, 2)), rng.uniform(-400.0, 400.0, (n, 2))
    s, r = mid - half, mid + half
    amps = rng.standard_normal((n, 300)).astype(np.float32)
    tb = create_trace_block(amps, s[:, 0], s[:, 1], r[:, 0], r[:, 1], sample_rate_ms=4.0)
    cfg = KernelConfig(kernel_type=kind, grid_dx=20.0, grid_dy=20.0, vti_eta_constant=0.1, **kw)
    return tb, VelocitySlice(vrms=1600.0 + 5.0 * np.arange(nt), is_1d=True), cfg


def _out(nt=140, t0=20.0, nx=5, ny=6):
    from pstm_b200.base import OutputTile
    return OutputTile(image=np.zeros((nx, ny, nt)), fold=np.zeros((nx, ny, nt), np.int32),
                      x_axis=20.0 * np.arange(nx), y_axis=20.0 * np.arange(ny), t_axis_ms=t0 + 6.0 * np.arange(nt))


def _device(tb, vel, out):
    import torch
    from pstm_b200.base import VelocitySlice
    dev = lambda a: a if a is None else torch.as_tensor(np.ascontiguousarray(a)).cuda()
    names = ("amplitudes", "source_x", "source_y", "receiver_x", "receiver_y", "offset", "midpoint_x", "midpoint_y",
             "weights")
    return (dataclasses.replace(tb, **{k: dev(getattr(tb, k)) for k in names}),
            VelocitySlice(vrms=dev(vel.vrms), is_1d=True),
            lambda: dataclasses.replace(out, **{k: dev(getattr(out, k))
                                                for k in ("image", "fold", "x_axis", "y_axis", "t_axis_ms")}))


def _check(tb, vel, cfg, kind, precision, got, ref):
    oracle.migrate(tb, ref, vel, cfg, kind=kind)
    assert np.abs(ref.image).max() > 0 and 0 < ref.fold.max() < tb.n_traces
    np.testing.assert_array_equal(got.fold, ref.fold)
    assert rel_l2(got.image, ref.image) <= (1e-5 if precision == "exact" else 1e-4)


@pytest.mark.parametrize("taper", [0.1, 0.0])
@pytest.mark.parametrize("precision", ["exact", "fast", "fp32"])
@pytest.mark.parametrize("kind", list(METHOD))
def test_maximum_below_the_minimum(kind, precision, taper, cuda_kernel_factory):
    tb, vel, cfg = _case(kind, max_aperture_m=300.0, min_aperture_m=500.0, taper_fraction=taper)
    k = cuda_kernel_factory(cfg, precision=precision)
    got, ref = _out(t0=0.0), _out(t0=0.0)
    getattr(k, METHOD[kind])(tb, got, vel)
    _check(tb, vel, cfg, kind, precision, got, ref)


@pytest.mark.parametrize("form", ["runs", "bins", "scatter", "executor", "tile"])
def test_every_form_cuts_at_the_maximum(form, cuda_kernel_factory):
    """Forms that select traces by the maximum aperture and forms that do not agree."""
    import torch
    from pstm_b200.cuda_kernel import Bin
    from pstm_b200.executor import TiledExecutor
    tb, vel, cfg = _case(max_aperture_m=300.0, min_aperture_m=500.0)
    k = cuda_kernel_factory(cfg)
    ref = _out()
    dtb, dvel, fresh = _device(tb, vel, ref)
    got = fresh()
    if form == "runs":
        k.migrate_tile_runs(dtb, [[0, 150], [150, 151], [151, 400]], got, dvel, cfg)
    elif form == "bins":
        k.migrate_bins(dtb, [Bin(0, 400, got.image, got.fold)], got, dvel, cfg)
    elif form == "scatter":
        k.migrate_scatter(dtb, got, dvel, cfg, segment_traces=32)
    elif form == "executor":
        ex = TiledExecutor(k, dtb, ref.x_axis, ref.y_axis, ref.t_axis_ms, lambda *a: dvel, cfg, tile=4, spatial=True)
        ex.run(got.image, got.fold)
    else:
        k.migrate_tile(dtb, got, dvel, cfg)
    k.synchronize()
    got = dataclasses.replace(got, image=got.image.cpu().numpy(), fold=got.fold.cpu().numpy())
    torch.cuda.synchronize()
    _check(tb, vel, cfg, "straight_ray", "exact", got, ref)


@pytest.mark.parametrize("precision", ["exact", "fast"])
@pytest.mark.parametrize("method", ["nearest", "cubic", "sinc8", "lanczos3"])
def test_interpolators_cut_at_the_maximum(method, precision, cuda_kernel_factory):
    tb, vel, cfg = _case(max_aperture_m=300.0, min_aperture_m=500.0, interpolation_method=method)
    k = cuda_kernel_factory(cfg, precision=precision)
    got, ref = _out(), _out()
    k.migrate_tile(tb, got, vel)
    _check(tb, vel, cfg, "straight_ray", precision, got, ref)


def test_learned_form_cuts_at_the_maximum(cuda_kernel_factory):
    """eta = 0 and a network that answers 0: the learned traveltime is the straight one."""
    import torch
    from pstm_b200 import surrogate as S
    tb, vel, cfg = _case("anisotropic_vti", max_aperture_m=300.0, min_aperture_m=500.0)
    cfg = dataclasses.replace(cfg, vti_eta_constant=0.0)
    k = cuda_kernel_factory(cfg)
    ref = _out()
    dtb, dvel, fresh = _device(tb, vel, ref)
    got = fresh()
    zero = S.Net(torch.zeros(S.N_PARAMS, dtype=torch.float32, device="cuda"),
                 S.survey_domain("anisotropic_vti", h_max_m=3200.0), out_scale=0.5)
    _, rep = k.migrate_tile_learned(dtb, got, dvel, zero, cfg, max_residual_ms=-1.0)
    torch.cuda.synchronize()
    assert rep["used_surrogate"]
    got = dataclasses.replace(got, image=got.image.cpu().numpy(), fold=got.fold.cpu().numpy())
    _check(tb, vel, cfg, "anisotropic_vti", "fp32", got, ref)


@pytest.mark.parametrize("taper", [0.1, 1.0, 0.0])
@pytest.mark.parametrize("precision", ["exact", "fast", "fp32"])
@pytest.mark.parametrize("kind,k", [("straight_ray", 0.5), ("curved_ray", 0.0), ("anisotropic_vti", 0.5)])
def test_no_aperture_at_time_zero(kind, k, precision, taper, cuda_kernel_factory):
    """Without a minimum the aperture of t = 0 is 0 m: only a midpoint on the pillar
    lies inside it, at full weight, whatever the other times of its block take."""
    from pstm_b200.base import create_trace_block
    tb, vel, cfg = _case(kind, max_aperture_m=800.0, min_aperture_m=0.0, taper_fraction=taper, apply_obliquity=False,
                         curved_ray_k=k)
    sx, sy, rx, ry = (np.array(a) for a in (tb.source_x, tb.source_y, tb.receiver_x, tb.receiver_y))
    sx[7], sy[7], rx[7], ry[7] = 20.0 - 60.0, 40.0, 20.0 + 60.0, 40.0   # midpoint on pillar (1, 2)
    tb = create_trace_block(np.asarray(tb.amplitudes), sx, sy, rx, ry, sample_rate_ms=4.0)
    ker = cuda_kernel_factory(cfg, precision=precision)
    got, ref = _out(t0=0.0), _out(t0=0.0)
    getattr(ker, METHOD[kind])(tb, got, vel)
    _check(tb, vel, cfg, kind, precision, got, ref)
    assert np.count_nonzero(ref.image[:, :, 0]) == 1
    tol = 1e-5 if precision == "exact" else 1e-4
    assert np.abs(got.image[:, :, 0] - ref.image[:, :, 0]).max() <= tol * np.abs(ref.image[1, 2, 0])
