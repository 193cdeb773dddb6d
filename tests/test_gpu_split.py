"""The traces of one output shared by the CTAs of a cluster (GPU).

A tile too small to fill the device has its traces divided, in whole chunks of
32, among 2, 4 or 8 CTAs, whose FP64 sums rank 0 adds in rank order; runs cross
the boundaries of the shares; bins of unequal size in one launch have unequal
numbers of shares in clusters of one size, and the ranks without a share leave.

Against the FP64 oracle: fold bit-exact, image relative L2 <= 1e-5 with the FP64
sample index and <= 1e-4 with FP32 traveltime, the tolerances of
tests/test_gpu_parity.py for FP32 traces.  A bin is summed in the order of the
same traces as a tile of their own: bit-equal.
"""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from conftest import rel_l2
from oracle import oracle

pytestmark = pytest.mark.gpu

METHOD = {"straight_ray": "migrate_tile", "curved_vti": "migrate_tile_curved_vti"}
FORMS = [("straight_ray", "exact"), ("curved_vti", "exact"), ("straight_ray", "fast")]


def shares(items, n):
    """The rule of csrc/plan.h (split_traces)."""
    best, least = 1, np.inf
    for s in (1, 2, 4, 8):
        cost = -(-items * s // 296) * (4 + -(-n // (32 * s)))
        if cost < 0.85 * least:
            least, best = cost, s
    return best


def _case(n, kind, nt=64):
    import torch
    from pstm_b200.base import KernelConfig, OutputTile, VelocitySlice, create_trace_block
    rng = np.random.default_rng(n)
    mid, half = rng.uniform(-300.0, 400.0, (n, 2)), rng.uniform(-300.0, 300.0, (n, 2))
    s, r = mid - half, mid + half
    tb = create_trace_block(rng.standard_normal((n, 203)).astype(np.float32), s[:, 0], s[:, 1], r[:, 0], r[:, 1],
                            sample_rate_ms=4.0, weights=rng.uniform(0.5, 1.5, n))
    cfg = KernelConfig(max_aperture_m=600.0, min_aperture_m=200.0, kernel_type=kind, grid_dx=20.0, grid_dy=20.0,
                       vti_eta_constant=0.1)
    vel = VelocitySlice(vrms=1600.0 + 6.0 * np.arange(nt), is_1d=True)
    ref = OutputTile(image=np.zeros((2, 4, nt)), fold=np.zeros((2, 4, nt), np.int32), x_axis=20.0 * np.arange(2),
                     y_axis=20.0 * np.arange(4), t_axis_ms=12.0 * np.arange(nt))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()   # noqa: E731
    names = ("amplitudes", "source_x", "source_y", "receiver_x", "receiver_y", "offset", "midpoint_x", "midpoint_y",
             "weights")
    dtb = dataclasses.replace(tb, **{k: dev(getattr(tb, k)) for k in names})
    fresh = lambda: dataclasses.replace(ref, **{   # noqa: E731
        k: dev(getattr(ref, k)) for k in ("image", "fold", "x_axis", "y_axis", "t_axis_ms")})
    return tb, vel, ref, cfg, dtb, VelocitySlice(vrms=dev(vel.vrms), is_1d=True), fresh


def _rows(tb, idx):
    names = ("amplitudes", "source_x", "source_y", "receiver_x", "receiver_y", "offset", "midpoint_x", "midpoint_y",
             "weights")
    return dataclasses.replace(tb, **{k: getattr(tb, k)[idx] for k in names})


def _check(got, tb, vel, ref, cfg, kind, precision):
    ref = dataclasses.replace(ref, image=np.zeros_like(ref.image), fold=np.zeros_like(ref.fold))
    oracle.migrate(tb, ref, vel, cfg, kind=kind)
    assert np.abs(ref.image).max() > 0
    np.testing.assert_array_equal(got.fold.cpu().numpy(), ref.fold)
    assert rel_l2(got.image.cpu().numpy(), ref.image) <= (1e-5 if precision == "exact" else 1e-4)


@pytest.mark.parametrize("n,n_shares", [(32, 1), (33, 2), (64, 2), (128, 4), (129, 8), (1000, 8)])
@pytest.mark.parametrize("kind,precision", FORMS)
def test_every_number_of_shares(kind, precision, n, n_shares, cuda_kernel_factory):
    assert shares(1, n) == n_shares
    tb, vel, ref, cfg, dtb, dvel, fresh = _case(n, kind)
    k = cuda_kernel_factory(cfg, precision=precision)
    got = fresh()
    getattr(k, METHOD[kind])(dtb, got, dvel, cfg)
    k.synchronize()
    _check(got, tb, vel, ref, cfg, kind, precision)


@pytest.mark.parametrize("runs", [[[0, 1], [2, 700], [701, 702], [720, 1000]],
                                  [[3 * i, 3 * i + 2] for i in range(333)],
                                  [[0, 128], [128, 256], [256, 384], [900, 1000]]])
@pytest.mark.parametrize("kind,precision", FORMS)
def test_runs_across_the_shares(kind, precision, runs, cuda_kernel_factory):
    rows = np.concatenate([np.arange(a, b) for a, b in runs])
    assert shares(1, len(rows)) == 8
    tb, vel, ref, cfg, dtb, dvel, fresh = _case(1000, kind)
    k = cuda_kernel_factory(cfg, precision=precision)
    got = fresh()
    k.migrate_tile_runs(dtb, runs, got, dvel, cfg, kernel_type=kind)
    k.synchronize()
    _check(got, _rows(tb, rows), vel, ref, cfg, kind, precision)


@pytest.mark.parametrize("kind,precision", FORMS)
def test_bins_of_unequal_shares(kind, precision, cuda_kernel_factory):
    from pstm_b200.cuda_kernel import Bin
    counts = [32, 1000, 64, 0, 128, 1, 256]
    assert [shares(1, n) for n in counts if n] == [1, 8, 2, 4, 1, 8]
    tb, vel, ref, cfg, dtb, dvel, fresh = _case(sum(counts), kind)
    k = cuda_kernel_factory(cfg, precision=precision)
    outs, begin = [fresh() for _ in counts], np.cumsum(counts) - counts
    k.migrate_bins(dtb, [Bin(int(b), n, o.image, o.fold) for b, n, o in zip(begin, counts, outs)], outs[0], dvel, cfg,
                   kernel_type=kind)
    k.synchronize()
    for b, n, got in zip(begin, counts, outs):
        rows = slice(int(b), int(b) + n)
        if n == 0:
            assert not got.image.any() and not got.fold.any()
            continue
        _check(got, _rows(tb, rows), vel, ref, cfg, kind, precision)
        alone = fresh()
        getattr(k, METHOD[kind])(_rows(dtb, rows), alone, dvel, cfg)
        k.synchronize()
        np.testing.assert_array_equal(got.image.cpu().numpy(), alone.image.cpu().numpy())
