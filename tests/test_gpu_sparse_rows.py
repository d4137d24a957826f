"""H X of the refinement where H is sparse: rows of one entry, around the
filling from which a Hamiltonian counts as dense (n / 2 entries in the fullest
row), one full row among short ones, rows of uneven length, and sparse and dense
snapshots in one launch.

Reference: P(t) = sum_jk |M_jk|^2 cos 2 pi (l_j - l_k) t / 2n from numpy's
eigenpairs, with the bounds of tests/test_gpu_large.py (|H| < 60 here too; MIXED
carries FP32 amplitudes)."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu

TIMES = np.linspace(0.0, 1.0, 33)
TOL = {_lib.PREC_FP64: 1e-9, _lib.PREC_MIXED: 1e-6}
PAULI = np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]])


def _signal(H, p):
    n = len(H)
    lam, U = np.linalg.eigh(H)
    A = np.abs(U.conj().T @ np.kron(np.tensordot(p, PAULI, 1), np.eye(n // 2)) @ U) ** 2 / (2 * n)
    return np.array([(np.exp(2j * np.pi * lam * t) @ A @ np.exp(-2j * np.pi * lam * t)).real
                     for t in TIMES])


def _patterns(n):
    """Name and mask of the nonzero entries, Hermitian."""
    i = np.arange(n)
    away = np.abs(i[:, None] - i)
    ring = np.minimum(away, n - away)  # 2 b + 1 entries per row at ring <= b
    half = (n // 2 - 1) // 2
    yield ring == 0
    yield ring <= half
    yield ring <= half + 1
    yield (ring == 0) | (i == 0) | (i[:, None] == 0)  # one full row
    yield (i * i[:, None]) % 5 == 1  # empty rows
    yield (i ^ i[:, None]) & (n - 1 - (i ^ i[:, None])) == 0  # uneven rows


@pytest.mark.parametrize("prec", [_lib.PREC_FP64, _lib.PREC_MIXED])
@pytest.mark.parametrize("n", [2, 6, 12, 18, 24, 30, 32, 48, 64, 66, 98, 192, 514])
def test_patterns(n, prec):
    rng = np.random.default_rng(n)
    full = 0.02 * random_hermitian(rng, n)
    Z = np.array([0.02 * random_hermitian(rng, n) for _ in range(3)])
    p = rng.normal(size=(2, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    B = np.array([[0.0, 0.0, 0.0], [0.1, -0.2, 0.05]])  # the second one is dense
    for mask in _patterns(n):
        assert (mask == mask.T).all()
        Hsys = np.where(mask, full, 0.0)
        out, st = kernels.powder_run(n, Hsys, Z, B, p, np.ones(2), np.arange(2, dtype=np.int32), 2,
                                     TIMES, precision=prec)
        assert int(st.max().item()) == 0
        got = out.cpu().numpy()
        for k in range(2):
            ref = _signal(Hsys + np.tensordot(B[k], Z, 1), p[k])
            assert np.abs(got[k] - ref).max() <= TOL[prec]
