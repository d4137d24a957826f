"""The n > 64 snapshots (msp_large_solve.cu, msp_large_refine.cu) at the sizes
where their stages change form (registers per thread, shared or global memory
for the reduction and the back-transformation, partial tiles), on spectra that
take the cluster branches and the FP64 solver, and in more snapshots than fit
at once.

Reference: P(t) = sum_jk |M_jk|^2 cos 2 pi (l_j - l_k) t / 2n from numpy's
eigenpairs.  Levels are backward stable to 16 n eps |H| (|H| < 60 here, n <=
226), so 2 pi t |dl| stays below 4e-10 at t <= 1 in FP64; MIXED carries FP32
amplitudes (1e-6, as for the other MIXED kernels)."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu

TIMES = np.linspace(0.0, 1.0, 33)
TOL = {_lib.PREC_FP64: 1e-9, _lib.PREC_MIXED: 1e-6}
PAULI = np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]])


def _herm(rng, n):
    return 0.02 * random_hermitian(rng, n)


def _pairs(H, p):
    n = len(H)
    lam, U = np.linalg.eigh(H)
    s = np.kron(np.tensordot(p, PAULI, 1), np.eye(n // 2))
    return lam, np.abs(U.conj().T @ s @ U) ** 2 / (2 * n)


def _signal(H, p, times=TIMES):
    lam, A = _pairs(H, p)
    return np.array([(np.exp(2j * np.pi * lam * t) @ A @ np.exp(-2j * np.pi * lam * t)).real
                     for t in times])


def _unit(rng, size):
    p = rng.normal(size=(size, 3))
    return p / np.linalg.norm(p, axis=1)[:, None]


def _run(Hsys, Z, B, p, times=TIMES, prec=_lib.PREC_FP64, mode=_lib.MODE_FAST, **kw):
    S = len(B)
    out, st = kernels.powder_run(len(Hsys), Hsys, Z, B, p, np.ones(S), np.arange(S, dtype=np.int32),
                                 S, times, mode=mode, precision=prec, **kw)
    assert int(st.max().item()) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n", [66, 96, 98, 128, 130, 192, 194, 222, 226])
def test_random(n, prec):
    rng = np.random.default_rng(n)
    Hsys = _herm(rng, n)
    Z = np.array([_herm(rng, n) for _ in range(3)])
    B, p = 0.3 * rng.normal(size=(3, 3)), _unit(rng, 3)
    got = _run(Hsys, Z, B, p, prec=prec)
    for k in range(3):
        ref = _signal(Hsys + np.tensordot(B[k], Z, 1), p[k])
        assert np.abs(got[k] - ref).max() <= TOL[prec]


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n", [72, 200])
def test_degenerate_and_clustered(n, prec):
    rng = np.random.default_rng(n)
    Z = np.zeros((3, n, n), dtype=complex)
    spectra = [np.zeros((n, n), dtype=complex), 3.0 * np.eye(n, dtype=complex),
               np.diag(rng.normal(size=n)).astype(complex),
               np.kron(np.eye(2), _herm(rng, n // 2)),
               np.kron(_herm(rng, n // 4), np.eye(4))]
    for gap in (1e-13, 1e-10, 1e-7, 1e-4):
        w = np.repeat(rng.normal(0, 10, n // 4), 4) * (1 + gap * rng.normal(size=n))
        q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
        H = (q * w) @ q.conj().T
        spectra.append(0.5 * (H + H.conj().T))
    p = _unit(rng, 1)
    for H in spectra:
        got = _run(H, Z, np.zeros((1, 3)), p, prec=prec)
        assert np.abs(got[0] - _signal(H, p[0])).max() <= TOL[prec]


# outside the range of the FP32 stages: the FP64 solver
@pytest.mark.parametrize("scale", [1e-20, 1e20])
def test_fp64_scales(scale):
    rng = np.random.default_rng(7)
    H, p = _herm(rng, 70), _unit(rng, 1)
    Z = np.zeros((3, 70, 70), dtype=complex)
    got = _run(scale * H, Z, np.zeros((1, 3)), p, times=TIMES / scale)
    assert np.abs(got[0] - _signal(H, p[0])).max() <= TOL[_lib.PREC_FP64]


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
def test_more_snapshots_than_slots(prec):
    rng = np.random.default_rng(11)
    n, S = 66, 900
    Hsys = _herm(rng, n)
    Z = np.array([_herm(rng, n) for _ in range(3)])
    B, p = 0.3 * rng.normal(size=(S, 3)), _unit(rng, S)
    got = _run(Hsys, Z, B, p, times=TIMES[:5], prec=prec)
    for k in (0, 151, 607, 608, 759, 760, 899):
        ref = _signal(Hsys + np.tensordot(B[k], Z, 1), p[k], TIMES[:5])
        assert np.abs(got[k] - ref).max() <= TOL[prec]


@pytest.mark.parametrize("dims", [(2, 5, 7), (2, 9, 9), (2, 4, 7, 4)])
def test_general_path(dims):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    Hsys = _herm(rng, n)
    Z = np.array([_herm(rng, n) for _ in range(3)])
    B, p = 0.3 * rng.normal(size=(2, 3)), _unit(rng, 2)
    kw = dict(dims=list(dims), mu_index=0, gammas=np.ones(len(dims)))
    got = _run(Hsys, Z, B, p, mode=_lib.MODE_EVOLVE, **kw)
    tau = 0.4
    mean = _run(Hsys, Z, B, p, mode=_lib.MODE_INTEGRAL, tau=tau, **kw)
    for k in range(2):
        H = Hsys + np.tensordot(B[k], Z, 1)
        lam, A = _pairs(H, p[k])
        assert np.abs(got[k] - _signal(H, p[k])).max() <= TOL[_lib.PREC_FP64]
        w = 2 * np.pi * (lam[:, None] - lam)
        assert abs(mean[k].item() - (A / (1 + (w * tau) ** 2)).sum()) <= TOL[_lib.PREC_FP64]


# a Hamiltonian that is not a number: reported or carried through, and the next
# snapshot is not touched
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n", [24, 32, 66, 96])
def test_nan_field(n, prec):
    rng = np.random.default_rng(n)
    Hsys = _herm(rng, n)
    Z = np.array([_herm(rng, n) for _ in range(3)])
    B, p = 0.3 * rng.normal(size=(3, 3)), _unit(rng, 3)
    B[1] = np.nan
    out, _ = kernels.powder_run(n, Hsys, Z, B, p, np.ones(3), np.arange(3, dtype=np.int32), 3, TIMES,
                                precision=prec)
    got = out.cpu().numpy()
    for k in (0, 2):
        ref = _signal(Hsys + np.tensordot(B[k], Z, 1), p[k])
        assert np.abs(got[k] - ref).max() <= TOL[prec]
