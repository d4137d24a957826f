"""The Householder + QL first stage (msp_ql_warp.cu) at the sizes where its
kernels change form (lanes per matrix, matrices per CTA, registers per lane) and
with a ragged last CTA, and on spectra without reflectors or with clusters.  The
batches are large enough for the dispatch to take it.

Reference: P(t) = sum_jk |M_jk|^2 cos 2 pi (l_j - l_k) t / 2n from numpy's
eigenpairs; 1e-6 as for the other MIXED results, 1e-9 in FP64 (levels backward
stable to 16 n eps |H|, |H| < 30, t <= 1: 2 pi t |dl| < 2e-11)."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu

TIMES = np.linspace(0.0, 1.0, 9)
TOL = {_lib.PREC_FP64: 1e-9, _lib.PREC_MIXED: 1e-6}
PAULI = np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]])


def _herm(rng, n):
    return 0.02 * random_hermitian(rng, n)


def _signal(H, p):
    n = len(H)
    lam, U = np.linalg.eigh(H)
    s = np.kron(np.tensordot(p, PAULI, 1), np.eye(n // 2))
    A = np.abs(U.conj().T @ s @ U) ** 2 / (2 * n)
    return np.array([(np.exp(2j * np.pi * lam * t) @ A @ np.exp(-2j * np.pi * lam * t)).real
                     for t in TIMES])


def _check(Hsys, Z, B, prec, rng, which):
    S = len(B)
    p = rng.normal(size=(S, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    out, st = kernels.powder_run(len(Hsys), Hsys, Z, B, p, np.ones(S), np.arange(S, dtype=np.int32),
                                 S, TIMES, precision=prec)
    assert int(st.max().item()) == 0
    got = out.cpu().numpy()
    for k in which:
        ref = _signal(Hsys + np.tensordot(B[k], Z, 1), p[k])
        assert np.abs(got[k] - ref).max() <= TOL[prec]


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n,S", [(6, 4099), (8, 4097), (10, 3300), (16, 2049), (18, 1821),
                                 (24, 1366), (26, 1300), (30, 1100), (32, 1025)])
def test_sizes(n, S, prec):
    rng = np.random.default_rng(n)
    Z = np.array([_herm(rng, n) for _ in range(3)])
    _check(_herm(rng, n), Z, 0.3 * rng.normal(size=(S, 3)), prec, rng,
           [0, 1, 31, 32, S // 2, S - 17, S - 2, S - 1])


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n", [8, 24, 32])
def test_spectra(n, prec):
    rng = np.random.default_rng(n)
    S = 4100
    Z = np.zeros((3, n, n), dtype=complex)
    near = np.repeat(rng.normal(0, 5, n // 4), 4) * (1 + 1e-7 * rng.normal(size=n))
    q, _ = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
    H = (q * near) @ q.conj().T
    tri = np.diag(rng.normal(size=n)) + np.diag(np.ones(n - 1) * 1j, 1) + np.diag(-1j * np.ones(n - 1), -1)
    for Hs in (np.zeros((n, n), dtype=complex), 3.0 * np.eye(n, dtype=complex),
               np.diag(rng.normal(size=n)).astype(complex), tri,
               np.kron(np.eye(2), _herm(rng, n // 2)), 0.5 * (H + H.conj().T)):
        _check(Hs, Z, np.zeros((S, 3)), prec, rng, [0, 1, S - 1])


# both sides of the batch size from which the dispatch takes QL: 608 snapshots (a warp
# per scheduler of 152 SMs) times 8 - n / 4, at least one
@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n,edge", [(10, 3648), (12, 3040), (16, 2432), (20, 1824), (22, 1824),
                                    (24, 1216), (28, 608), (32, 608)])
@pytest.mark.parametrize("over", [0, 1])
def test_dispatch_edges(n, edge, over, prec):
    rng = np.random.default_rng(100 + n)
    S = edge + over
    Z = np.array([_herm(rng, n) for _ in range(3)])
    _check(_herm(rng, n), Z, 0.3 * rng.normal(size=(S, 3)), prec, rng, [0, 33, S // 2, S - 2, S - 1])
