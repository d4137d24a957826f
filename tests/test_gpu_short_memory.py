"""Runs on a card that has no room for the scratch the fastest form wants: they
take the forms with the smaller scratch instead, with the same results.  The
limit is the allocator's own (a fraction of the card for this process).

Tolerance: both forms hold the library's 1e-10 against the oracle."""

import contextlib
import ctypes

import numpy as np
import pytest
import torch

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def _room(nbytes):
    """At most nbytes more than what is held now."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + nbytes) / total)
    try:
        yield
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def _system(n, S, seed):
    rng = np.random.default_rng(seed)
    H = 0.5 * random_hermitian(rng, n)
    Z = np.array([random_hermitian(rng, n) for _ in range(3)])
    p = rng.normal(size=(S, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    return [torch.as_tensor(x).cuda() for x in (H, Z, 0.1 * rng.normal(size=(S, 3)), p,
                                                np.full(S, 1.0 / S))]


# FP64 integrals of 60,000 snapshots of n = 32 (eigenvector scratch), 1,500 rows of
# 4,096 samples (Fourier form), 152 snapshots of n = 96 in flight
@pytest.mark.parametrize("n,S,rows,nt,mode", [(32, 60000, 1, 1, _lib.MODE_INTEGRAL),
                                              (48, 1500, 1500, 4096, _lib.MODE_FAST),
                                              (96, 152, 1, 64, _lib.MODE_FAST)])
def test_powder(n, S, rows, nt, mode):
    H, Z, F, p, w = _system(n, S, n)
    slot = torch.as_tensor(np.arange(S) * rows // S, dtype=torch.int32).cuda()
    times = np.linspace(0.0, 2.0, nt)
    kw = dict(mode=mode, tau=0.5)
    if mode != _lib.MODE_FAST:
        kw.update(dims=[2, 2, n // 4], mu_index=0, gammas=[135.5, 40.0, 40.0])

    def run():
        plan = kernels.PowderPlan(n, H, Z, F, p, w, slot, rows, times, **kw)
        return plan.workspace_bytes, plan.run().clone()

    full, ref = run()
    least = ctypes.c_size_t(0)
    plan = kernels.PowderPlan(n, H, Z, F, p, w, slot, rows, times, **kw)
    _lib.call("msp_powder_min_workspace", ctypes.byref(plan.args), ctypes.byref(least))
    del plan
    assert full > least.value + 16 * MB
    out = 3 * 8 * rows * nt + 8 * MB
    with _room((full + least.value) // 2 + out):
        used, got = run()
    assert least.value <= used < full
    assert np.abs((got - ref).cpu().numpy()).max() <= 1e-10


def test_adjoint():
    n, S, rows, nt = 24, 600, 300, 8192
    H, Z, F, p, w = _system(n, S, 1)
    times = torch.as_tensor(np.linspace(0.0, 4.0, nt)).cuda()
    slot = (torch.arange(S, dtype=torch.int32) // 2).cuda()
    g = torch.as_tensor(np.random.default_rng(2).normal(size=(rows, nt))).cuda()

    def run():
        return kernels.adjoint_fast(n, H, Z, F, p, w, slot, rows, times, g)

    ref = run()
    with _room(128 * MB):  # the transform's tables take 320 MB
        got = run()
    for a, b in zip(got[:2], ref[:2]):
        a, b = a.cpu().numpy(), b.cpu().numpy()
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)


def test_celio():
    rng = np.random.default_rng(3)
    S, D = 8000, 4
    q = torch.linalg.qr(torch.as_tensor(rng.normal(size=(S, 2, D, D)) + 0j).cuda())[0]
    mats = q.reshape(S, -1).contiguous()
    ph = torch.as_tensor(rng.random((S, 1, 4))).cuda()
    sig = np.tile(np.array([[1, 0], [0, -1]], complex), (S, 1, 1))
    mu = np.tile(np.array([1, 0], complex), (S, 1))
    mu, sig = torch.as_tensor(mu).cuda(), torch.as_tensor(sig).cuda()

    def run():
        return kernels.celio_run(_lib.CELIO_PURE, [2, 2, 2], [(0, 1), (0, 2)], [0, D * D], mats, True,
                                 S, 1, 2, 6, mu_psi=mu, sigma=sig, phases=ph)[0].clone()

    ref = run()
    with _room(48 * MB):  # the digit fragments take 98 MB
        got = run()
    assert np.abs((got - ref).cpu().numpy()).max() <= 1e-12


def test_batch():
    rng = np.random.default_rng(4)
    systems, per, n, nt = 1500, 1, 48, 4096
    H = [0.5 * random_hermitian(rng, n) for _ in range(4)]
    Z = [np.array([random_hermitian(rng, n) for _ in range(3)]) for _ in range(4)]
    pick = np.arange(systems) % 4
    p = rng.normal(size=(systems * per, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    args = ([H[k] for k in pick], [Z[k] for k in pick], 0.1 * rng.normal(size=(systems * per, 3)), p,
            np.ones(systems * per), np.arange(0, systems * per + 1, per, dtype=np.int32),
            np.linspace(0.0, 2.0, nt))

    def run():
        plan = kernels.MultiPlan(*args, precision=_lib.PREC_FP64)
        out, nbytes = plan.run().clone(), plan.workspace_bytes
        plan.close()
        return nbytes, out

    full, ref = run()
    inputs = 4 * 16 * n * n * systems
    with _room(2 * inputs + 2 * 8 * systems * nt):  # the copies that are joined, then freed
        used, got = run()
    assert used < full
    assert np.abs((got - ref).cpu().numpy()).max() <= 1e-10
