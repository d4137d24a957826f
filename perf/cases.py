"""Cases that time this framework: what its users have it compute, through its
public entry points, with the 64-bit answer each result is held against.

A case is a plain dict; ``kind`` names the entry point:

* ``powder``  -- ``powder_average``: one system, an orientation grid given as
  host rows, P(t) on a uniform grid.
* ``scan``    -- ``powder_scan``: decaying integrals of an ALC field scan on a
  device-generated ZCW grid.
* ``thermal`` -- ``ExperimentRunner.run`` at a finite temperature (the general
  evolution path), one output row per field, uniform or log-spaced times.
* ``lindblad`` -- ``ExperimentRunner.run`` with dissipation terms.
* ``celio``   -- ``ExperimentRunner.run`` with Celio's Trotter method and
  averaged random initial states.
* ``batch``   -- ``MultiSystemBatch.result``: many systems of uneven size in
  one CUDA-graph launch.
* ``fit``     -- ``GradientFitter.loss_and_grad``: forward curve and adjoint.
* ``single``  -- ``Hamiltonian.evolve`` and ``.integrate_decaying`` of one
  Hamiltonian, as a program that drives its own loop calls them.

``fp64`` is the framework's default precision and is compared as float64.
``mixed`` computes in single precision (it promises max |dP| <= 1e-6, not
double-precision results), so a program that asks for it keeps the curves in
float32, the precision they have; so does ``run``.
"""

import math

import numpy as np
import torch

from muspinsim_gb300 import simconfig
from muspinsim_gb300.adjoint import GradientFitter, TorchSpinHamiltonian
from muspinsim_gb300.experiment import ExperimentRunner
from muspinsim_gb300.hamiltonian import Hamiltonian
from muspinsim_gb300.multi import MultiSystemBatch
from muspinsim_gb300.powder import OrientationGrid, powder_average, powder_scan
from muspinsim_gb300.spinop import DensityOperator
from muspinsim_gb300.spinsys import MuonSpinSystem

# spin, gyromagnetic ratio (MHz/T), quadrupole moment (millibarn)
SPINS = {
    "e": (0.5, -28024.9514242, 0.0),
    "mu": (0.5, 28024.9514242 / 206.7669883, 0.0),
    "H": (0.5, 42.577478518, 0.0),
    "F": (0.5, 40.0776, 0.0),
    "N": (1.0, 3.077706, 20.44),
    "V": (3.5, 11.2133, -52.0),
}
MU_TAU = 2.19703  # us
MU_0 = 1.25663706127e-06
PLANCK = 6.62607015e-34
BOLTZMANN = 1.380649e-23
EFG_TO_MHZ = 9.7173624424e21 * 1.602176634e-19 * 1e-37 / PLANCK

# The systems of the benchmark's heterogeneous batch, by dimension.
BY_DIM = {4: "mu H", 8: "mu e H", 12: "mu e N", 24: "mu e H N", 48: "mu e H H N",
          96: "mu e H H H N", 192: "mu e H H H H N"}


def listed():
    return [
        # One muonium radical, one orientation: a user's first script and the
        # inner call of any hand-written loop.  Latency and launches.
        {"name": "mu_e_one_orientation", "kind": "powder", "spins": "mu e", "orient": 1,
         "times": 1000, "t_max": 10.0, "field": 0.01, "precision": "fp64"},
        # The benchmark's powder: 24-dimensional radical, full grid, in both
        # precisions; fp64 is what a user gets by default.
        {"name": "radical24_powder_mixed", "kind": "powder", "spins": "mu e H N",
         "orient": 10000, "times": 4096, "t_max": 20.0, "field": 0.01, "precision": "mixed"},
        {"name": "radical24_powder_fp64", "kind": "powder", "spins": "mu e H N",
         "orient": 10000, "times": 4096, "t_max": 20.0, "field": 0.01, "precision": "fp64"},
        # A larger molecule on a coarse grid, above the dimension up to which
        # one CTA holds a Hamiltonian in shared memory; ragged sizes.
        {"name": "radical96_powder_fp64", "kind": "powder", "spins": "mu e H H H N",
         "orient": 49, "times": 1501, "t_max": 15.0, "field": 0.02, "precision": "fp64"},
        # Avoided-level-crossing scans, the other observable of the method.
        {"name": "radical32_alc_mixed", "kind": "scan", "spins": "mu e H H H", "fields": 201,
         "b_max": 1.0, "orient": 1000, "precision": "mixed"},
        {"name": "radical12_alc_fp64", "kind": "scan", "spins": "mu e N", "fields": 101,
         "b_max": 2.0, "orient": 144, "precision": "fp64"},
        # A temperature- and field-dependent run from an input file: every
        # field is its own output curve, thermal nuclei and electron.
        {"name": "radical12_thermal_fp64", "kind": "thermal", "spins": "mu e N", "fields": 5,
         "orient": 233, "times": 777, "t_max": 8.0, "temperature": 4.0, "spacing": "uniform",
         "precision": "fp64"},
        # Comparing candidate sites and isotopologues: many systems at once.
        {"name": "uneven_batch_mixed", "kind": "batch", "systems": 21, "dims": "4 8 12 24 48 96 192",
         "orient": 64, "times": 2048, "t_max": 20.0, "field": 0.01, "precision": "mixed"},
        # One step of a least-squares fit of an F-mu-F geometry.
        {"name": "fmuf_fit_step_fp64", "kind": "fit", "spins": "mu F F", "orient": 2000,
         "times": 1000, "t_max": 20.0, "field": 0.001, "precision": "fp64"},
        # Spin-lattice relaxation: the Lindblad form of a powder run.
        {"name": "radical8_lindblad_fp64", "kind": "lindblad", "spins": "mu e H", "orient": 200,
         "times": 1000, "t_max": 10.0, "temperature": 20.0, "field": 0.003, "precision": "fp64"},
        # The site geometry of the reference's Trotter example, three of its
        # four vanadium neighbours.
        {"name": "v3_celio_fp64", "kind": "celio", "spins": "mu V V V", "orient": 8,
         "averages": 19, "k": 10, "times": 50, "t_max": 10.0, "precision": "fp64"},
        # A program that drives single Hamiltonians itself.
        {"name": "radical24_hamiltonian_fp64", "kind": "single", "spins": "mu e H N",
         "times": 2000, "t_max": 10.0, "field": 0.1},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(spins):
    return int(np.prod([int(2 * SPINS[s][0] + 1) for s in spins.split()]))


def _cost(c):
    """Roughly proportional to a case's time, to keep drawn ones bounded."""
    if c["kind"] not in ("powder", "scan", "thermal"):
        return 0.0
    n = _dim(c["spins"])
    per = n * n * c.get("times", 1) + 50.0 * n**3
    return per * c["orient"] * c.get("fields", 1) * (50 if c["precision"] == "fp64" else 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["powder"] * 4 + ["scan"] * 2 + ["thermal"] * 2
                          + ["batch", "fit", "lindblad", "celio", "single"])
        c = {"kind": kind}
        precision = rng.choice(["fp64", "mixed"])
        if kind == "powder":
            spins = rng.choice(["mu e", "mu F F", "mu e N", "mu e H N", "mu e H H H",
                                "mu e H H N", "mu e H H H N"])
            c.update(spins=spins, orient=_log(rng, 1, 10000), times=_log(rng, 100, 4096),
                     t_max=round(rng.uniform(5.0, 20.0), 3), field=round(rng.uniform(0, 0.1), 5),
                     precision=precision)
        elif kind == "scan":
            c.update(spins=rng.choice(["mu e H", "mu e N", "mu e H N", "mu e H H H"]),
                     fields=_log(rng, 10, 400), b_max=round(rng.uniform(0.5, 3.0), 3),
                     orient=_log(rng, 30, 1000), precision=precision)
        elif kind == "thermal":
            c.update(spins=rng.choice(["mu e", "mu e H", "mu e N", "mu e H N"]),
                     fields=rng.randint(1, 8), orient=_log(rng, 20, 500),
                     times=_log(rng, 100, 2000), t_max=round(rng.uniform(4.0, 16.0), 3),
                     temperature=round(rng.uniform(1.0, 50.0), 2),
                     spacing=rng.choice(["uniform", "uniform", "uniform", "log"]),
                     precision=precision)
        elif kind == "batch":
            c.update(systems=rng.randint(5, 21), dims="4 8 12 24 48 96 192"[:rng.choice(
                     [6, 9, 12, 15, 19])].rstrip(), orient=_log(rng, 8, 64),
                     times=_log(rng, 200, 2048), t_max=round(rng.uniform(5.0, 20.0), 3),
                     field=round(rng.uniform(0, 0.1), 5), precision="mixed")
        elif kind == "fit":
            c.update(spins="mu F F", orient=_log(rng, 100, 2000), times=_log(rng, 100, 1000),
                     t_max=round(rng.uniform(5.0, 20.0), 3),
                     field=round(rng.uniform(0.0002, 0.01), 5), precision="fp64")
        elif kind == "lindblad":
            c.update(spins=rng.choice(["mu e", "mu e H"]), orient=_log(rng, 20, 200),
                     times=_log(rng, 100, 1000), t_max=round(rng.uniform(4.0, 10.0), 3),
                     temperature=round(rng.uniform(2.0, 50.0), 2),
                     field=round(rng.uniform(0.0005, 0.02), 5), precision=precision)
        elif kind == "celio":
            c.update(spins=rng.choice(["mu V V", "mu V V V"]), orient=rng.randint(1, 8),
                     averages=rng.randint(4, 19), k=rng.randint(4, 10), times=_log(rng, 20, 50),
                     t_max=round(rng.uniform(4.0, 10.0), 3), precision=precision)
        else:
            c.update(spins=rng.choice(["mu e", "mu F F", "mu e N", "mu e H N", "mu e H H N"]),
                     times=_log(rng, 100, 2000), t_max=round(rng.uniform(5.0, 20.0), 3),
                     field=round(rng.uniform(0.001, 1.0), 4))
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------ inputs


def _haar(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    return q * np.sign(np.diag(r))


def _vector(rng, lo, hi):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v) * rng.uniform(lo, hi)


def _efg(rng, lo, hi):
    v = rng.normal(size=(3, 3))
    v = 0.5 * (v + v.T)
    v -= np.trace(v) / 3.0 * np.eye(3)
    return v * (rng.uniform(lo, hi) / np.abs(np.linalg.eigvalsh(v)).max())


def _couplings(spins, rng, trotter=False):
    """(kind, first spin, second spin or None, value) with the benchmark
    workloads' distributions: anisotropic hyperfine tensors with eigenvalues
    ~ N(0, 50) MHz, dipoles at 1-3 A (1.0-1.4 A to fluorine, 1.6-2.0 A to
    vanadium), random traceless field gradients."""
    out = []
    for i, s in enumerate(spins):
        if "e" in spins and s != "e":
            q = _haar(rng)
            out.append(("hyperfine", i, spins.index("e"),
                        q @ np.diag(rng.normal(0.0, 50.0, 3)) @ q.T))
        if i and s != "e":
            lo, hi = {"F": (1.0, 1.4), "V": (1.6, 2.0)}.get(s, (1.0, 3.0))
            out.append(("dipolar", 0, i, _vector(rng, lo, hi)))
        if SPINS[s][0] > 0.5:
            lo, hi = (0.02, 0.06) if trotter else (0.1, 1.0)
            out.append(("quadrupolar", i, None, _efg(rng, lo, hi)))
    return out


def _system(spins, couplings):
    system = MuonSpinSystem(list(spins))
    for kind, i, j, value in couplings:
        if kind == "hyperfine":
            system.add_hyperfine_term(i, value, j)
        elif kind == "dipolar":
            system.add_dipolar_term(i, j, value)
        else:
            system.add_quadrupolar_term(i, value)
    return system


def _rows(n, rng):
    """(theta, phi) rows spread evenly over the sphere, turned at random."""
    j = np.arange(n)
    theta = np.arccos(1.0 - (2.0 * j + 1.0) / n)
    phi = (rng.uniform(0, 2 * np.pi) + j * np.pi * (3.0 - 5.0**0.5)) % (2 * np.pi)
    return np.stack([theta, phi], axis=1)


def _times(c):
    if c.get("spacing") == "log":
        return np.concatenate([[0.0], np.geomspace(1e-3, c["t_max"], c["times"] - 1)])
    return np.linspace(0.0, c["t_max"], c["times"])


def _inputs(c, seed):
    """The plain numbers behind a case, from the seed alone: what prepare()
    hands to the framework and exact() works from."""
    rng = np.random.default_rng(seed)
    kind = c["kind"]
    d = {"rng": rng, "pol": np.array([0.0, 0.0, 1.0])}
    if kind == "batch":
        dims = [int(x) for x in c["dims"].split()]
        d["many"] = []
        for k in range(c["systems"]):
            spins = BY_DIM[dims[k % len(dims)]].split()
            d["many"].append((spins, _couplings(spins, rng)))
    else:
        d["spins"] = c["spins"].split()
        d["couplings"] = _couplings(d["spins"], rng, trotter=kind == "celio")
    if kind == "scan":
        d["rows"] = _zcw(c["orient"])
        d["fields"] = np.linspace(0.0, c["b_max"] * rng.uniform(0.95, 1.0), c["fields"])
        return d
    d["rows"] = _rows(c.get("orient", 1), rng)
    d["times"] = _times(c)
    if kind == "thermal":
        d["fields"] = np.linspace(0.002, 0.05, c["fields"]) if c["fields"] > 1 \
            else np.array([0.01])
        d["fields"] = d["fields"] * rng.uniform(0.9, 1.1)
    elif kind == "fit":
        curve = 0.5 * np.cos(np.linspace(0, 3, c["times"]))
        d["data"] = curve + rng.normal(0, 0.01, c["times"])
    elif kind == "single":
        b = rng.normal(size=3)
        d["b"] = c["field"] * b / np.linalg.norm(b)
    elif kind == "celio":
        d["draws"] = int(rng.integers(2**31))
    return d


def _zcw(n):
    """The framework's ZCW grid of n points over the sphere."""
    g0 = max(1, int(round(n / ((1.0 + 5**0.5) / 2.0) ** 2)))
    g = next(g for delta in range(n + 1) for g in (g0 + delta, g0 - delta)
             if 1 <= g < max(n, 2) and math.gcd(g, n) == 1)
    j = np.arange(n, dtype=np.int64)
    return np.stack([np.arccos(np.clip(2.0 * (j / n) - 1.0, -1.0, 1.0)),
                     2.0 * np.pi * (((j * g) % n) / n)], axis=1)


def _runner(c, d, **more):
    terms = [(kind, {"i": i + 1} if j is None else {"i": i + 1, "j": j + 1}, value)
             for kind, i, j, value in d["couplings"]]
    terms += more.pop("terms", [])
    params = simconfig.make_params(d["spins"], terms, d["times"], d["rows"],
                                   polarization=[d["pol"]], **more)
    return ExperimentRunner(simconfig.ParamsInput(params), precision=c["precision"])


#: dissipation rates (MHz) by spin
RATES = {"e": 2.0, "H": 0.3}


def prepare(case, seed):
    c, d = case, _inputs(case, seed)
    kind = c["kind"]
    s = {"case": c}
    if kind == "powder":
        s.update(system=_system(d["spins"], d["couplings"]), rows=d["rows"], times=d["times"],
                 pol=d["pol"])
    elif kind == "scan":
        s.update(system=_system(d["spins"], d["couplings"]),
                 grid=OrientationGrid("zcw", c["orient"]), fields=d["fields"], pol=d["pol"])
    elif kind == "thermal":
        s["runner"] = _runner(c, d, field=[[b] for b in d["fields"]],
                              temperature=[c["temperature"]])
    elif kind == "lindblad":
        terms = [("dissipation", {"i": i + 1}, [RATES[x]]) for i, x in enumerate(d["spins"])
                 if x in RATES]
        s["runner"] = _runner(c, d, field=[[c["field"]]], temperature=[c["temperature"]],
                              terms=terms)
    elif kind == "celio":
        s["runner"] = _runner(c, d, celio=(c["k"], c["averages"]))
        s["draws"] = d["draws"]
    elif kind == "batch":
        s["batch"] = MultiSystemBatch([_system(*m) for m in d["many"]], d["rows"], c["field"],
                                      d["pol"], d["times"], precision=c["precision"])
    elif kind == "fit":
        th = TorchSpinHamiltonian(d["spins"])
        r = [value for _, _, _, value in d["couplings"]]
        unit = [torch.as_tensor(v / np.linalg.norm(v), device=th.device) for v in r]

        def model(p):
            return (th.dipolar(0, 1, p[0] * unit[0]) + th.dipolar(0, 2, p[1] * unit[1]), p[2])

        s["fitter"] = GradientFitter(model, th.Z, d["rows"], d["times"], d["data"], d["pol"],
                                     precision=c["precision"])
        s["x"] = [torch.tensor(x, dtype=torch.float64, device=th.device, requires_grad=True)
                  for x in (np.linalg.norm(r[0]), np.linalg.norm(r[1]), [0.0, 0.0, c["field"]])]
    else:
        system = _system(d["spins"], d["couplings"])
        H = system.hamiltonian_matrix() + np.einsum("a,aij->ij", d["b"],
                                                    system.zeeman_operators())
        n = H.shape[0]
        mu = np.diag([1.0, 0.0]).astype(complex)
        rho = DensityOperator(np.kron(mu, np.eye(n // 2)) * (2.0 / n), list(system.dimension))
        s.update(matrix=H, dim=list(system.dimension), rho=rho, times=d["times"],
                 ops=[system.muon_operator([0.0, 0.0, 1.0]), system.muon_operator([1.0, 0.0, 0.0])])
    return s


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "powder":
        y = powder_average(s["system"], s["rows"], c["field"], s["pol"], s["times"],
                           precision=c["precision"])
    elif kind == "scan":
        y = powder_scan(s["system"], s["grid"], s["fields"], s["pol"], y_axis="integral",
                        precision=c["precision"])
    elif kind in ("thermal", "lindblad"):
        y = s["runner"].run()
    elif kind == "celio":
        np.random.seed(s["draws"])
        y = s["runner"].run()
    elif kind == "batch":
        y = s["batch"].result(graph=True)
    elif kind == "fit":
        loss, grads = s["fitter"].loss_and_grad(s["x"])
        return {"loss": loss.detach(), "grads": list(grads)}
    else:
        H = Hamiltonian(s["matrix"], s["dim"])
        return {"evolved": H.evolve(s["rho"], s["times"], s["ops"]),
                "integral": H.integrate_decaying(s["rho"], MU_TAU, s["ops"])}
    return y.astype(np.float32) if c["precision"] == "mixed" else y


# ------------------------------------------------------------------ least work


def work(case):
    """Bytes: rows, fields, times and coupling matrices in, curves out.
    Flops: per snapshot an n x n complex Hermitian eigendecomposition with
    vectors (about 36 n^3 real operations) and two eigenbasis products
    (16 n^3); per eigenvalue pair a constant (20) and per output sample the
    share of a fast transform (5 log2 T), which is all that the sum over
    pairs needs on a uniform grid."""
    c = case
    kind = c["kind"]
    times = c.get("times", 1)
    rows = c.get("fields", 1) if kind != "batch" else c["systems"]
    size = 8 if c.get("precision", "fp64") == "fp64" else 4
    if kind == "batch":
        dims = [int(x) for x in c["dims"].split()]
        ns = [dims[k % len(dims)] for k in range(c["systems"])]
        snapshots = [(n, c["orient"]) for n in ns]
        mats = sum(4 * 16 * n * n for n in ns)
    else:
        n = _dim(c["spins"])
        snapshots = [(n, c.get("orient", 1) * c.get("fields", 1))]
        mats = 4 * 16 * n * n
    size_in = 16 * c.get("orient", 1) + 8 * times + mats
    size_out = size * rows * times
    if kind == "celio":
        dims = [int(2 * SPINS[s][0] + 1) for s in c["spins"].split()]
        v = int(np.prod(dims))
        per_pass = sum(8 * v * (2 * d + d) for d in dims[1:])
        states = c["orient"] * c["averages"]
        return {"bytes": size_in + 4 * v * states + size_out,
                "flops": states * c["k"] * (times - 1) * per_pass}
    if kind == "lindblad":
        n = snapshots[0][0]
        return {"bytes": size_in + size_out,
                "flops": c["orient"] * (25 * 8 * n**6 + 8 * n**4 * times)}
    flops = sum(s * (52 * n**3 + (20 * n * n / 2 if times > 1 else 10 * n * n))
                for n, s in snapshots)
    if times > 1:
        flops += rows * times * 5 * max(1.0, math.log2(times))
    if kind == "fit":
        flops *= 3
    return {"bytes": size_in + size_out, "flops": flops}


# ------------------------------------------------------------------ the 64-bit answers


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _spin(I):
    m = np.arange(I, -I - 1, -1)
    up = np.diag(np.sqrt(I * (I + 1) - m[1:] * (m[1:] + 1)), 1).astype(complex)
    return np.array([(up + up.T) / 2, (up - up.T) / 2j, np.diag(m)])


def _embed(spins):
    """Every spin's three operators on the whole space, the first slowest."""
    dims = [int(2 * SPINS[s][0] + 1) for s in spins]
    out = []
    for i, s in enumerate(spins):
        left, right = int(np.prod(dims[:i])), int(np.prod(dims[i + 1:]))
        out.append([np.kron(np.kron(np.eye(left), op), np.eye(right))
                    for op in _spin(SPINS[s][0])])
    return np.array(out)


def _tensor(spins, coupling):
    """(i, j, 3 x 3 tensor in MHz) of one coupling."""
    kind, i, j, value = coupling
    if kind == "hyperfine":
        return i, j, value
    if kind == "dipolar":
        r = np.linalg.norm(value)
        k = -MU_0 * PLANCK / (2 * np.pi) * SPINS[spins[i]][1] * SPINS[spins[j]][1] * 1e6
        return i, j, k / (2 * (r * 1e-10) ** 3) * (3 * np.outer(value, value) / r**2 - np.eye(3))
    I, _, q = SPINS[spins[i]]
    return i, i, EFG_TO_MHZ * q / (2 * I * (2 * I - 1)) * value


def _matrices(spins, couplings):
    S = _embed(spins)
    H = np.zeros(S.shape[2:], dtype=complex)
    for c in couplings:
        i, j, T = _tensor(spins, c)
        for a in range(3):
            for b in range(3):
                H += T[a, b] * (S[i, a] @ S[j, b])
    Z = sum(SPINS[s][1] * S[i] for i, s in enumerate(spins))
    return H, Z, S


def _turns(rows):
    """Rotation matrices taking lab vectors into each row's crystal frame."""
    theta, phi = rows[:, 0], rows[:, 1]
    one, zero = np.ones_like(theta), np.zeros_like(theta)

    def about_z(x):
        return np.array([[np.cos(x), -np.sin(x), zero], [np.sin(x), np.cos(x), zero],
                         [zero, zero, one]]).transpose(2, 0, 1)

    y = np.array([[np.cos(theta), zero, -np.sin(theta)], [zero, one, zero],
                  [np.sin(theta), zero, np.cos(theta)]]).transpose(2, 0, 1)
    return about_z(-phi) @ y @ about_z(-phi)


def _thermal(spins, p, B, T):
    """Muon along p, every other spin thermal in its own Zeeman field."""
    rho = np.ones((1, 1))
    for s in spins:
        I, g, _ = SPINS[s]
        S = _spin(I)
        if s == "mu":
            one = 0.5 * np.eye(2) + np.einsum("a,aij->ij", p, S)
        else:
            e, v = np.linalg.eigh(np.einsum("a,aij->ij", B, S))
            x = -PLANCK * 1e6 * g * e / (BOLTZMANN * T)
            w = np.exp(x - x.max())
            one = (v * (w / w.sum())) @ v.conj().T
        rho = np.kron(rho, one)
    return rho


def _up(a, kind=torch.complex128):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=kind, device=_device())


def _curve(spins, couplings, fields, pols, weights, times, temperature=None, tau=None):
    """sum_s w_s Tr(O_s rho_s(t)) over snapshots of one system, or the
    integral against exp(-t / tau) over tau."""
    H, Z, S = _matrices(spins, couplings)
    n = H.shape[0]
    H, Z = _up(H), _up(Z)
    mu = _up(S[0])
    t = None if times is None else _up(times, torch.float64)
    out = 0.0 if times is None else torch.zeros(len(times), dtype=torch.float64, device=H.device)
    j, k = np.tril_indices(n, -1)
    j, k = torch.as_tensor(j, device=H.device), torch.as_tensor(k, device=H.device)
    chunk = max(1, min(len(fields), (1 << 22) // (n * n)))
    for s0 in range(0, len(fields), chunk):
        at = slice(s0, s0 + chunk)
        e, U = torch.linalg.eigh(H + torch.einsum("sa,aij->sij", _up(fields[at]), Z))
        O = torch.einsum("sa,aij->sij", _up(pols[at]), mu)
        if temperature is None:
            rho = (O + 0.5 * torch.eye(n, dtype=O.dtype, device=O.device)) * (2.0 / n)
        else:
            rho = _up(np.array([_thermal(spins, p, b, temperature)
                                for p, b in zip(pols[at], fields[at])]))
        Uh = U.conj().transpose(1, 2)
        C = (Uh @ rho @ U) * (Uh @ O @ U).transpose(1, 2) * _up(weights[at])[:, None, None]
        w = 2 * np.pi * (e[:, :, None] - e[:, None, :])
        if times is None:
            # int exp(-i w t) exp(-t / tau) dt / tau = 1 / (1 + i w tau)
            out += float((C / (1.0 + 1j * w * tau)).real.sum())
            continue
        out += C.diagonal(dim1=1, dim2=2).real.sum()
        cr, ci = 2 * C[:, j, k].real.reshape(-1), 2 * C[:, j, k].imag.reshape(-1)
        w = w[:, j, k].reshape(-1)
        step = max(1, (1 << 24) // len(times))
        for b in range(0, len(w), step):
            ph = w[b:b + step, None] * t[None, :]
            out += cr[b:b + step] @ torch.cos(ph)
            if temperature is not None:
                out += ci[b:b + step] @ torch.sin(ph)
    return out if times is None else out.cpu().numpy()


def _exact_fit(c, d):
    """Loss and gradient from the derivative of exp(-2 pi i H t) in H's
    eigenbasis: divided differences, safe where levels meet."""
    spins, n = d["spins"], 8
    r = [value for _, _, _, value in d["couplings"]]
    _, Z, S = _matrices(spins, [])
    parts, dparts = [], []
    for k in range(2):
        one = ("dipolar", 0, k + 1, r[k])
        parts.append(_matrices(spins, [one])[0])
        dparts.append(-3.0 / np.linalg.norm(r[k]) * parts[k])
    R = _turns(d["rows"])
    N = len(R)
    pol = _up(R @ d["pol"])
    t = _up(d["times"], torch.float64)
    B = _up(R @ np.array([0.0, 0.0, c["field"]]))
    Zt, mu = _up(Z), _up(S[0])
    # derivatives of H_s: two distances (the same for all s), three field axes
    dB = torch.einsum("sab,aij->sbij", _up(R), Zt)
    dH = torch.cat([_up(np.array(dparts))[None].expand(N, 2, n, n), dB], dim=1)
    P = torch.zeros(len(t), dtype=torch.float64, device=t.device)
    G = torch.zeros(5, len(t), dtype=torch.float64, device=t.device)
    for s0 in range(0, N, 50):
        at = slice(s0, s0 + 50)
        e, U = torch.linalg.eigh(_up(parts[0] + parts[1])
                                 + torch.einsum("sa,aij->sij", B[at], Zt))
        Uh = U.conj().transpose(1, 2)
        O = Uh @ torch.einsum("sa,aij->sij", pol[at], mu) @ U
        D = Uh[:, None] @ dH[at] @ U[:, None]
        x = 2 * np.pi * e[:, None, :] * t[None, :, None]  # (s, T, n)
        ph = torch.exp(-1j * x)
        # V = exp(-i H t) and dV_jk = D_jk (-2 pi i t) exp(-i mean) sinc(half gap)
        half = 0.5 * (x[..., :, None] - x[..., None, :])
        F = torch.exp(-0.5j * (x[..., :, None] + x[..., None, :])) \
            * torch.sinc(half / np.pi) * (-2j * np.pi * t)[None, :, None, None]
        # P = (2 / n) Tr(O V O V^dag); M = V^dag-side factor O V^dag O
        M = torch.einsum("sij,stj,sjk->stik", O, ph.conj(), O)
        P += (2.0 / n / N) * torch.einsum("stii,sti->t", M, ph).real
        FM = F * M.transpose(2, 3)
        G += (4.0 / n / N) * torch.einsum("stjk,spjk->pt", FM, D).real
    res = P - _up(d["data"], torch.float64)
    g = (2 * res[None, :] * G).sum(dim=1).cpu().numpy()
    return {"loss": torch.as_tensor(float((res * res).sum()), dtype=torch.float64),
            "grads": [g[0], g[1], g[2:]]}


def _exact_lindblad(c, d):
    H0, Z, S = _matrices(d["spins"], d["couplings"])
    n = H0.shape[0]
    eye, R = np.eye(n), _turns(d["rows"])
    out = np.zeros(len(d["times"]))
    for turn in R:
        B, p = turn @ np.array([0.0, 0.0, c["field"]]), turn @ d["pol"]
        H = H0 + np.einsum("a,aij->ij", B, Z)
        L = -1j * (np.kron(H, eye) - np.kron(eye, H.T))
        z = B / np.linalg.norm(B)
        x = np.cross([0.0, 0.0, 1.0], z) if abs(z[2]) < 0.9 else np.cross([1.0, 0.0, 0.0], z)
        x /= np.linalg.norm(x)
        y = np.cross(z, x)
        for i, s in enumerate(d["spins"]):
            if s not in RATES:
                continue
            up = np.einsum("a,aij->ij", x + 1j * y, S[i])
            f = math.exp(-PLANCK * SPINS[s][1] * c["field"] * 1e6 / (BOLTZMANN * c["temperature"]))
            for A, rate in ((up, f), (up.conj().T, 1.0)):
                M = A.conj().T @ A
                L = L + RATES[s] / np.pi * rate / (1 + f) * (
                    np.kron(A, A.conj()) - 0.5 * (np.kron(M, eye) + np.kron(eye, M.T)))
        rho = _thermal(d["spins"], p, B, c["temperature"]).reshape(-1)
        O = np.einsum("a,aij->ij", p, S[0])
        lam, V = np.linalg.eig(L)
        amp = (O.T.reshape(-1) @ V) * np.linalg.solve(V, rho)
        out += (np.exp(2 * np.pi * d["times"][:, None] * lam[None, :]) @ amp).real / len(R)
    return out


def _exact_celio(c, d):
    spins = d["spins"]
    dims = [int(2 * SPINS[s][0] + 1) for s in spins]
    half = int(np.prod(dims)) // 2
    S, A, T = c["orient"], c["averages"], c["times"]
    dt = d["times"][1] - d["times"][0]
    factors = []
    for first in range(len(spins)):
        for coupling in d["couplings"]:
            i, j, M = _tensor(spins, coupling)
            if i != first:
                continue
            a, b = _spin(SPINS[spins[i]][0]), _spin(SPINS[spins[j]][0])
            h = sum(M[x, y] * (a[x] @ b[y] if i == j else np.kron(a[x], b[y]))
                    for x in range(3) for y in range(3))
            e, v = np.linalg.eigh(h)
            u = (v * np.exp(-2j * np.pi * e * dt / c["k"])) @ v.conj().T
            factors.append((i, j, _up(u)))
    draws = np.random.RandomState(d["draws"]).random_sample(S * A * half).reshape(S, A, half)
    pols = _turns(d["rows"]) @ d["pol"]
    sig = 2 * np.einsum("sa,aij->sij", pols, _spin(0.5))
    mu = np.array([np.linalg.eigh(m)[1][:, 1] for m in sig])
    psi = np.einsum("si,sah->saih", mu, np.exp(2j * np.pi * draws) / math.sqrt(half))
    psi, sig = _up(psi).reshape([S * A] + dims), _up(np.repeat(sig, A, axis=0))
    out = np.zeros(T)
    for k in range(T):
        x = psi.reshape(S * A, 2, half)
        out[k] = 0.5 / (S * A) * float(torch.einsum("xih,xij,xjh->", x.conj(), sig, x).real)
        for _ in range(c["k"] if k < T - 1 else 0):
            for i, j, u in factors:
                if i == j:
                    moved = torch.tensordot(u, psi, dims=([1], [i + 1]))
                    psi = moved.movedim(0, i + 1)
                else:
                    u4 = u.reshape(dims[i], dims[j], dims[i], dims[j])
                    moved = torch.tensordot(u4, psi, dims=([2, 3], [i + 1, j + 1]))
                    psi = moved.movedim((0, 1), (i + 1, j + 1))
    return out


def _exact_single(c, d):
    H, Z, S = _matrices(d["spins"], d["couplings"])
    n = H.shape[0]
    e, U = np.linalg.eigh(H + np.einsum("a,aij->ij", d["b"], Z))
    rho = U.conj().T @ np.kron(np.diag([1.0, 0.0]), np.eye(n // 2)) @ U * (2.0 / n)
    w = 2 * np.pi * (e[:, None] - e[None, :]).reshape(-1)
    C = np.array([(rho * (U.conj().T @ S[0, a] @ U).T).reshape(-1) for a in (2, 0)])
    ph = np.exp(-1j * d["times"][:, None] * w[None, :])
    return {"evolved": ph @ C.T, "integral": (C / (1.0 / MU_TAU + 1j * w)).sum(axis=1)}


def exact(case, seed):
    c, d = case, _inputs(case, seed)
    kind = c["kind"]
    if kind == "fit":
        return _exact_fit(c, d)
    if kind == "lindblad":
        return _exact_lindblad(c, d)
    if kind == "celio":
        return _exact_celio(c, d)
    if kind == "single":
        return _exact_single(c, d)
    R = _turns(d["rows"])
    N = len(R)
    pols, w = R @ d["pol"], np.full(N, 1.0 / N)

    def fields(b):
        return R @ np.array([0.0, 0.0, b])

    if kind == "powder":
        return _curve(d["spins"], d["couplings"], fields(c["field"]), pols, w, d["times"])
    if kind == "batch":
        return np.array([_curve(spins, cs, fields(c["field"]), pols, w, d["times"])
                         for spins, cs in d["many"]])
    if kind == "scan":
        return np.array([_curve(d["spins"], d["couplings"], fields(b), pols, w, None, tau=MU_TAU)
                         for b in d["fields"]])
    y = np.array([_curve(d["spins"], d["couplings"], fields(b), pols, w, d["times"],
                         c["temperature"]) for b in d["fields"]])
    return y if len(y) > 1 else y[0]
