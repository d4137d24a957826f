"""The phase sum as a nonuniform Fourier transform (msp_nufft.cu) against the
direct per-sample sum, at the edges of its tiles, grids and work items.

A time grid whose last sample is moved by 1e-9 of itself is not uniform, so
it takes the direct kernel (FP64 phases, sincos per sample and pair), which
other tests pin to the oracle; all other samples must agree.

Tolerances: FP64 phases w t reach 2 pi x 600 MHz x 20 us = 8e4 rad, rounded to
9e-12 at worst in either form, on amplitudes that sum to 0.5: 1e-11.  Mixed:
the library's 1e-6 (both forms start from FP32 eigenvectors)."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels, workloads
from muspinsim_gb300 import quaternion as Q
from muspinsim_gb300.orientations import orientation_rows_to_quats, zcw_gen
from tests.helpers import oracle_powder, random_hermitian

pytestmark = pytest.mark.gpu


def _curves(dim, orient, times, slots, mode, prec, scale=1.0):
    rng = np.random.default_rng(dim + len(times))
    wl = workloads.random_system_workload(rng, dim, zcw_gen(orient), times, (0.0, 0.0, 0.02))
    sy = wl.system()
    qs, _ = orientation_rows_to_quats(wl.orientations)
    B = Q.rotate(qs, wl.fields[0])
    p = Q.rotate(qs, wl.polarization)
    slot = np.sort(np.arange(orient) % slots).astype(np.int32)
    Hs, Z = sy.hamiltonian_matrix(), sy.zeeman_operators()
    temp = 3.0 if mode == _lib.MODE_EVOLVE else None
    out, status = kernels.powder_run(
        dim, Hs, Z, B, p, np.full(orient, scale / orient), slot, slots, times, mode=mode,
        precision=prec, dims=list(sy.dimension), mu_index=0, gammas=sy.gammas, temperature=temp)
    assert int(status.max().item()) == 0
    return out.cpu().numpy(), wl


# 777: a ragged grid; 4096 / 4097: one and two time tiles; 8193: three; 64:
# the smallest grid; slots: one and several rows, items of unequal length
@pytest.mark.parametrize("prec,dim,orient,nt,slots", [
    (_lib.PREC_FP64, 24, 500, 64, 1),
    (_lib.PREC_FP64, 8, 700, 777, 3),
    (_lib.PREC_FP64, 12, 101, 4096, 1),
    (_lib.PREC_FP64, 12, 101, 4097, 2),
    (_lib.PREC_FP64, 4, 333, 8193, 1),
    (_lib.PREC_MIXED, 24, 4100, 1001, 1),
    (_lib.PREC_MIXED, 24, 1400, 4097, 2),
])
@pytest.mark.parametrize("mode", [_lib.MODE_FAST, _lib.MODE_EVOLVE])
@pytest.mark.parametrize("t0", [0.0, 0.3])
def test_matches_direct_sum(prec, dim, orient, nt, slots, mode, t0):
    times = np.linspace(t0, t0 + 19.0, nt)
    moved = times.copy()
    moved[-1] *= 1.0 + 1e-9
    assert kernels.uniform_grid(times)[0] and not kernels.uniform_grid(moved)[0]
    a, _ = _curves(dim, orient, times, slots, mode, prec)
    b, _ = _curves(dim, orient, moved, slots, mode, prec)
    tol = 1e-11 if prec == _lib.PREC_FP64 else 1e-6
    assert np.abs(a[:, :-1] - b[:, :-1]).max() <= tol


def test_matches_oracle():
    times = np.linspace(0.0, 20.0, 1500)
    a, wl = _curves(12, 200, times, 1, _lib.MODE_FAST, _lib.PREC_FP64)
    assert np.abs(a[0] - oracle_powder(wl)).max() <= 1e-10


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_amplitude_range(scale):
    """The fixed-point scale follows the weights."""
    times = np.linspace(0.0, 19.0, 777)
    a, _ = _curves(8, 700, times, 1, _lib.MODE_FAST, _lib.PREC_FP64)
    b, _ = _curves(8, 700, times, 1, _lib.MODE_FAST, _lib.PREC_FP64, scale)
    assert np.abs(b / scale - a).max() <= 1e-11


def test_non_finite_inputs_stay_non_finite():
    times = np.linspace(0.0, 19.0, 777)
    a, _ = _curves(8, 700, times, 2, _lib.MODE_FAST, _lib.PREC_FP64, np.nan)
    assert np.isnan(a).all()


# the adjoint's transform against the direct sums (a grid that is not uniform,
# its moved last sample without weight); the gradients are sums over 1e5 terms
# with phases rounded to 1e-11: 1e-9 of their norm
@pytest.mark.parametrize("dim,orient,nt,slots,t0", [(8, 300, 777, 1, 0.0), (8, 300, 777, 3, 0.4),
                                                    (4, 2000, 64, 1, 0.0), (24, 40, 4097, 2, -1.0)])
def test_adjoint_matches_direct_sum(dim, orient, nt, slots, t0):
    times = np.linspace(t0, t0 + 12.0, nt)
    moved = times.copy()
    moved[-1] *= 1.0 + 1e-9
    assert kernels.uniform_grid(times)[0] and not kernels.uniform_grid(moved)[0]
    rng = np.random.default_rng(nt)
    wl = workloads.random_system_workload(rng, dim, zcw_gen(orient), times, (0.0, 0.0, 0.02))
    sy = wl.system()
    qs, _ = orientation_rows_to_quats(wl.orientations)
    B, p = Q.rotate(qs, wl.fields[0]), Q.rotate(qs, wl.polarization)
    slot = np.sort(np.arange(orient) % slots).astype(np.int32)
    g = rng.normal(size=(slots, nt))
    g[:, -1] = 0.0
    got = [kernels.adjoint_fast(dim, sy.hamiltonian_matrix(), sy.zeeman_operators(), B, p,
                                np.full(orient, 1 / orient), slot, slots, t, g)
           for t in (times, moved)]
    for a, b in zip(got[0][:2], got[1][:2]):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)


# a frequency that is not finite: its row is not either, the others are untouched
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_field(prec, bad):
    rng = np.random.default_rng(3)
    n, S = 24, 3000 if prec == _lib.PREC_MIXED else 300
    H, Z = random_hermitian(rng, n), np.array([random_hermitian(rng, n) for _ in range(3)])
    B, p = 0.1 * rng.normal(size=(S, 3)), np.tile([0.0, 0.0, 1.0], (S, 1))
    slot = (np.arange(S) * 3 // S).astype(np.int32)
    times = np.linspace(0.0, 3.0, 2000)
    good = kernels.powder_run(n, H, Z, B, p, np.full(S, 1 / S), slot, 3, times, precision=prec)[0]
    B[S // 2] = bad
    got = kernels.powder_run(n, H, Z, B, p, np.full(S, 1 / S), slot, 3, times, precision=prec)[0]
    got, good = got.cpu().numpy(), good.cpu().numpy()
    assert not np.isfinite(got[1]).any()
    assert np.abs(got[[0, 2]] - good[[0, 2]]).max() <= 1e-11
