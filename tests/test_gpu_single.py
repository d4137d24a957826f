"""Building blocks of the single-Hamiltonian API at the edges of their blocks:
the expectation series (times per CTA, rows per block, column slabs, the n =
256 switch) and the changes of basis (columns per CTA), against numpy.

Tolerances: sums of n^2 terms bounded by one with phases 2 pi l t up to 2e4
rad: the reference's own phase rounding, 4e-12 per term, on coefficients of
2-norm 1; basis changes: n eps of the norms."""

import numpy as np
import pytest

from muspinsim_gb300 import kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 24, 64, 65, 256, 257])
@pytest.mark.parametrize("nt,nops", [(1, 1), (16, 3), (37, 2)])
def test_expectation_series(n, nt, nops):
    rng = np.random.default_rng(n + nt)
    lam = rng.normal(0, 100, n)
    rho = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    ops = rng.normal(size=(nops, n, n)) + 1j * rng.normal(size=(nops, n, n))
    times = rng.uniform(-2.0, 15.0, nt)
    C = rho[None] * ops.transpose(0, 2, 1)
    scale = np.linalg.norm(C, axis=(1, 2))
    got = kernels.evolve_expect(lam, rho, ops, times).cpu().numpy()
    ph = np.exp(2j * np.pi * lam[:, None] * times[None, :])
    ref = np.einsum("it,oij,jt->to", ph.conj(), C, ph)
    assert got.shape == (nt, nops)
    assert (np.abs(got - ref) / scale).max() <= 1e-11 * np.sqrt(n)


# up to n = 4, 128 times per CTA
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("nt", [127, 128, 129, 300])
def test_expectation_series_of_few_levels(n, nt):
    test_expectation_series(n, nt, 2)


@pytest.mark.parametrize("n", [1, 2, 4, 5, 24, 63, 64])
@pytest.mark.parametrize("batch", [1, 3])
@pytest.mark.parametrize("shared", ["none", "u", "m"])
@pytest.mark.parametrize("adjoint", [False, True])
def test_basis_change(n, batch, shared, adjoint):
    rng = np.random.default_rng(n)
    U = np.array([np.linalg.eigh(random_hermitian(rng, n))[1] for _ in range(batch)])
    M = rng.normal(size=(batch, n, n)) + 1j * rng.normal(size=(batch, n, n))
    if shared == "u":
        U = U[:1]
    elif shared == "m":
        M = M[:1]
    got = kernels.basis_change(U, M, adjoint).cpu().numpy()
    Uh = U.conj().transpose(0, 2, 1)
    ref = U @ M @ Uh if adjoint else Uh @ M @ U
    assert np.abs(got - ref).max() <= 16 * n * np.finfo(float).eps * np.abs(M).max() * n
