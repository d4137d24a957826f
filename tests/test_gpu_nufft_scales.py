"""The FP64 phase sum's fixed-point amplitudes at the ends of their range: one pair
that is nearly the whole sum of its work item, of either sign of its offset, and
weights near the ends of FP64.

Reference: the weights' sum times one snapshot's P(t) from numpy.  Phases are
good to 1e-12 at |l| t < 100, amplitudes and window to 1e-14 of the sum."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian
from tests.test_gpu_sparse_rows import PAULI

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, -1.0, 1e-290, 1e290])
@pytest.mark.parametrize("rest", [0.0, 1e-40, 1e-3])
@pytest.mark.parametrize("n", [2, 6])
def test_one_large_amplitude(n, rest, scale):
    S, times = 6000, np.linspace(0.0, 2.0, 1501)
    H = 0.02 * random_hermitian(np.random.default_rng(n), n)
    p = np.array([0.48, -0.6, 0.64])
    w = np.full(S, rest)
    w[S // 3] = 1.0
    out, st = kernels.powder_run(n, H, np.zeros((3, n, n), dtype=complex), np.zeros((S, 3)),
                                 np.tile(p, (S, 1)), scale * w, np.zeros(S, dtype=np.int32), 1, times,
                                 precision=_lib.PREC_FP64)
    assert int(st.max().item()) == 0
    lam, U = np.linalg.eigh(H)
    A = np.abs(U.conj().T @ np.kron(np.tensordot(p, PAULI, 1), np.eye(n // 2)) @ U) ** 2 / (2 * n)
    ref = np.array([(np.exp(2j * np.pi * lam * t) @ A @ np.exp(-2j * np.pi * lam * t)).real
                    for t in times])
    got = out.cpu().numpy()[0] / scale
    assert np.abs(got - w.sum() * ref).max() <= 2e-12 * w.sum()
