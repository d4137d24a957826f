"""The transform as the phase sum of a heterogeneous batch (msp_multi.cu) against
the direct sum of the same plan (which a tuned item size asks for): several rows
per bucket of uneven length, an empty system, chunks, an offset grid, a graph.

Tolerances: the two sums of sum |a| = 1 per row differ by the transform's window
(FP64 1e-14, MIXED 1e-8) and by the direct sums' own rounding (FP64 phases 1e-12,
MIXED FP32 phases and running sums 1e-6)."""

import numpy as np
import pytest

from muspinsim_gb300 import _lib, kernels
from tests.helpers import random_hermitian

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("t0", [0.0, 0.7])
@pytest.mark.parametrize("prec,dims,counts,T,tol", [
    (_lib.PREC_FP64, [8, 12, 12, 8, 12], [90, 150, 0, 33, 201], 1500, 2e-12),
    (_lib.PREC_MIXED, [24, 8, 24], [700, 60, 411], 4500, 2e-6)])
@pytest.mark.parametrize("chunk", [0, 7000])
def test_matches_direct(prec, dims, counts, T, tol, t0, graph, chunk):
    rng = np.random.default_rng(T)
    H = [0.02 * random_hermitian(rng, n) for n in dims]
    Z = [np.array([0.02 * random_hermitian(rng, n) for _ in range(3)]) for n in dims]
    first = np.concatenate([[0], np.cumsum(counts)])
    S = first[-1]
    B = 0.3 * rng.normal(size=(S, 3))
    p = rng.normal(size=(S, 3))
    p /= np.linalg.norm(p, axis=1)[:, None]
    w = np.concatenate([np.full(c, 1.0 / max(c, 1)) for c in counts])
    times = t0 + np.linspace(0.0, 2.0, T)
    if chunk and prec == _lib.PREC_MIXED:
        chunk *= 15
    out = []
    for tuning in (None, [{"n": n, "snaps_per_item": 4} for n in sorted(set(dims))]):
        plan = kernels.MultiPlan(H, Z, B, p, w, first, times, precision=prec, tuning=tuning,
                                 max_pairs_per_chunk=chunk)
        plan.run(graph=graph)
        out.append(plan.run(graph=graph).cpu().numpy())
        assert int(plan.status.max().item()) == 0
        plan.close()
    assert np.abs(out[0] - out[1]).max() <= tol
    assert (out[0][[k for k, c in enumerate(counts) if c == 0]] == 0).all()
