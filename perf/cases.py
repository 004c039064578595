"""Performance cases of the B200 libhalf, through the calls that a program makes.

The cells are the package's synthetic ones (``halfb200.synth``): the 2-atom Si
cell (725 plane waves, 16 bands, LDA), the 12-atom HfO2 cell (3,400 plane
waves, 64 bands, PBE, s/p/d channels), the 64-atom Si cell (11,000 plane
waves, 160 bands) and the 216-atom Si cell with vacancies (38,000 plane waves,
480 bands).  The seed displaces every atom (0.02 A per component, as in a
relaxation or an MD run), which moves the density and the operator and lifts
the symmetry degeneracies; the pseudopotentials stay.

Kinds of case:

* ``solve``    ``Context.solve``: operator preparation and the all-band acc
               eigensolver for one k point; ``solve_kpoints`` for several;
* ``relax``    ``Context.set_positions`` and the solve at the new positions:
               one step of a relaxation;
* ``apply``    ``Context.apply_hs``: H psi and S psi of host band blocks;
* ``force``    ``Context.nonlocal_forces`` of given states (the backward of
               the band energy);
* ``density``  ``Context.output_density`` of given states and
               ``Context.ionic_forces`` of that density;
* ``gemm``     ``halfb200.tc_cgemm`` on device operands: the mixed mode's
               tensor-core product.

Solves return the eigenvalues alone (the call without a vector buffer):
eigenvectors are defined up to a phase, and within 1e-9 only where levels are
well apart.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "deepaw-half_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import halfb200  # noqa: E402
from halfb200 import synth  # noqa: E402


def listed():
    return [
        # one band through the operator of the smallest cell: what a call costs before any work
        {"name": "apply_si2_1", "kind": "apply", "cell": "si2", "bands": 1, "k": "0.125,0.25,0.375"},
        # a band block of a small cell at a general k point, an odd count (a host eigensolver's H psi)
        {"name": "apply_hfo2_37", "kind": "apply", "cell": "hfo2", "bands": 37, "k": "0.25,-0.125,0.5"},
        # all bands of the 64-atom cell
        {"name": "apply_si64_160", "kind": "apply", "cell": "si64", "bands": 160, "k": "0.25,0.25,0"},
        # smallest solve, the default precision (the plain FP64 iteration)
        {"name": "solve_si2_fp64", "kind": "solve", "cell": "si2", "bands": 16, "k": "0.125,0.25,0.375",
         "nk": 1, "precision": "fp64", "tol": 1e-6},
        # small cell, mixed precision
        {"name": "solve_hfo2_mixed", "kind": "solve", "cell": "hfo2", "bands": 64, "k": "0,0,0", "nk": 1,
         "precision": "mixed", "tol": 1e-6},
        # a relaxation step in FP64 with guard bands, an odd band count, a general k point
        {"name": "relax_hfo2_guarded", "kind": "relax", "cell": "hfo2", "bands": 51, "k": "0.25,0.25,0.25",
         "nk": 1, "precision": "fp64_guarded", "tol": 1e-6},
        # four k points of the 64-atom cell's mesh in one batch
        {"name": "kmesh_si64_mixed", "kind": "solve", "cell": "si64", "bands": 160, "k": "0.25,0,0", "nk": 4,
         "precision": "mixed", "tol": 2e-5},
        # the largest: one k point of the 216-atom cell
        {"name": "solve_si216v_mixed", "kind": "solve", "cell": "si216v", "bands": 480, "k": "0.5,0,0", "nk": 1,
         "precision": "mixed", "tol": 2e-5},
        # backward: the force of the 64-atom cell's bands
        {"name": "force_si64_160", "kind": "force", "cell": "si64", "bands": 160, "k": "0.25,0.25,0.25"},
        # output density and the ion-position forces on it, two k points
        {"name": "density_hfo2", "kind": "density", "cell": "hfo2", "bands": 44, "k": "0,0.25,0", "nk": 2},
        # inner product X^H Y of a 216-atom block (bands + guard bands squared, K = plane waves)
        {"name": "gemm_inner", "kind": "gemm", "op": "C", "m": 600, "n": 600, "kk": 38089},
        # rotation X Y of a 64-atom block with some bands locked: odd sizes
        {"name": "gemm_rotate_odd", "kind": "gemm", "op": "N", "m": 11023, "n": 187, "kk": 193},
    ]


_BANDS = {"si2": (4, 24), "hfo2": (24, 72), "si64": (96, 176)}


def draw(rng):
    kind = rng.choice(["apply", "apply", "solve", "solve", "relax", "force", "density", "gemm", "gemm"])
    if kind == "gemm":
        if rng.random() < 0.5:
            mn = [int(round(math.exp(rng.uniform(math.log(9), math.log(600))))) for _ in range(2)]
            return {"kind": "gemm", "op": "C", "m": mn[0], "n": mn[1],
                    "kk": int(round(math.exp(rng.uniform(math.log(700), math.log(38232)))))}
        return {"kind": "gemm", "op": "N", "m": int(round(math.exp(rng.uniform(math.log(700), math.log(38232))))),
                "n": rng.randint(9, 400), "kk": rng.randint(9, 600)}
    cell = rng.choice(["si2", "hfo2", "si64"])
    lo, hi = _BANDS[cell]
    k = ",".join("%.4f" % rng.uniform(-0.5, 0.5) for _ in range(3))
    if kind == "apply":
        top = {"si2": 64, "hfo2": 160, "si64": 200}[cell]
        return {"kind": "apply", "cell": cell, "bands": int(round(math.exp(rng.uniform(0, math.log(top))))), "k": k}
    if kind == "force":
        return {"kind": "force", "cell": cell, "bands": rng.randint(lo, hi), "k": k}
    if kind == "density":
        cell = rng.choice(["si2", "hfo2"])
        lo, hi = _BANDS[cell]
        return {"kind": "density", "cell": cell, "bands": rng.randint(lo, hi), "k": k, "nk": rng.randint(1, 3)}
    c = {"kind": kind, "cell": cell, "bands": rng.randint(lo, hi), "k": k, "nk": 1,
         "precision": rng.choice(["mixed", "fp64_guarded"]), "tol": 2e-5 if cell == "si64" else 1e-6}
    if kind == "solve" and rng.random() < 0.4:
        c["nk"] = rng.randint(2, 5)
    return c


def _k(case):
    return np.array([float(x) for x in case["k"].split(",")])


def _mesh(case):
    """nk k points: the case's and its neighbours along the three axes."""
    k0 = _k(case)
    steps = [(0, 0, 0), (0, 0.25, 0), (0, 0, 0.25), (0.25, 0.25, 0), (0, 0.25, 0.25)]
    return np.array([k0 + np.array(s) for s in steps[:case.get("nk", 1)]])


def _cell(name, rng):
    """The named synthetic cell with displaced atoms."""
    w = synth.workload(name)
    shift = rng.normal(0.0, 0.02, size=w.positions.shape) @ np.linalg.inv(w.lattice)
    w.positions = np.mod(w.positions + shift, 1.0)
    return w


def _density(w):
    """Atom-centred Gaussians (0.8 A) and a background, rho * Omega in file
    order, summed in reciprocal space."""
    n = w.grid
    rec = 2 * np.pi * np.linalg.inv(w.lattice)
    m = [np.fft.fftfreq(x, 1.0 / x) for x in n]
    ph = [np.exp(-2j * np.pi * np.outer(m[i], w.positions[:, i])) for i in range(3)]
    s = ((ph[0][:, None, :] * ph[1][None, :, :]).reshape(n[0] * n[1], -1) @ ph[2].T).reshape(n)
    g2 = 0
    for a in range(3):
        g = rec[a, 0] * m[0][:, None, None] + rec[a, 1] * m[1][None, :, None] + rec[a, 2] * m[2][None, None, :]
        g2 = g2 + g * g
    rho = np.fft.ifftn(s * np.exp(-0.5 * 0.8 ** 2 * g2)).real
    rho = w.nelect * (0.75 * rho / rho.mean() + 0.25)
    return rho.transpose(2, 1, 0).ravel()


def _write(w, folder):
    """CHGCAR and POTCAR of a cell."""
    pot = os.path.join(folder, "POTCAR")
    rng = np.random.default_rng(w.seed + 1000)
    with open(pot, "w") as f:
        for spec in w.species:
            f.write(synth.potcar_text(synth.species_dataset(spec, rng)))
    v = _density(w)
    chg = os.path.join(folder, "CHGCAR")
    with open(chg, "w") as f:
        f.write("synthetic\n 1.0\n")
        for a in w.lattice:
            f.write(" %.16f %.16f %.16f\n" % tuple(a))
        f.write(" ".join(s.element for s in w.species) + "\n" + " ".join(str(c) for c in w.counts) + "\nDirect\n")
        for p in w.positions:
            f.write(" %.16f %.16f %.16f\n" % tuple(p))
        f.write("\n %d %d %d\n" % tuple(w.grid))
        full = len(v) // 5 * 5
        f.write((" %.16E %.16E %.16E %.16E %.16E\n" * (full // 5)) % tuple(v[:full]))
        f.write(" ".join("%.16E" % x for x in v[full:]) + "\n")
    return chg, pot


def _states(rng, nb, n):
    """nb band vectors of norm 1; (n, nb), each band contiguous."""
    x = rng.normal(size=(nb, n)) + 1j * rng.normal(size=(nb, n))
    x /= np.linalg.norm(x, axis=1)[:, None]
    return x.T


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "gemm":
        g = torch.Generator(device="cuda").manual_seed(seed)
        m, n, kk = case["m"], case["n"], case["kk"]
        # column-major operands: a (rows, cols) matrix is held as a (cols, rows) tensor
        a = torch.randn((m, kk) if case["op"] == "C" else (kk, m), dtype=torch.complex64, device="cuda", generator=g)
        b = torch.randn((n, kk), dtype=torch.complex64, device="cuda", generator=g)
        if case["op"] == "C":   # a projection: Y = H X lies in the span of X up to a residual
            b = 0.1 * b + torch.randn((n, m), dtype=torch.complex64, device="cuda", generator=g) @ a / math.sqrt(m)
        return {"case": case, "a": a, "b": b, "c": torch.zeros((n, m), dtype=torch.complex64, device="cuda")}
    w = _cell(case["cell"], rng)
    with tempfile.TemporaryDirectory() as d:
        chg, pot = _write(w, d)
        ctx = halfb200.Context(chg, pot, w.encut, xc=w.xc, solver="acc")
    s = {"case": case, "ctx": ctx, "k": _k(case)}
    nb = case["bands"]
    if case["kind"] in ("solve", "relax"):
        ctx.set_acc(tol=case["tol"], max_iterations=1000, precision=case["precision"])
        s["mesh"] = _mesh(case)
        if case["kind"] == "relax":
            step = rng.normal(0.0, 0.01, size=w.positions.shape) @ np.linalg.inv(w.lattice)
            s["positions"] = w.positions + step
    elif case["kind"] == "density":
        s["mesh"] = _mesh(case)
        s["weights"] = np.full(len(s["mesh"]), 1.0 / len(s["mesh"]))
        s["psi"] = [_states(rng, nb, ctx.npw(k)) for k in s["mesh"]]
        s["occ"] = rng.uniform(0.0, 2.0, size=(len(s["mesh"]), nb))
    else:
        s["psi"] = _states(rng, nb, ctx.npw(s["k"]))
        if case["kind"] == "force":
            s["eps"] = np.sort(rng.uniform(-5.0, 5.0, size=nb))
            s["occ"] = rng.uniform(0.0, 2.0, size=nb)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gemm":
        m, n, kk = case["m"], case["n"], case["kk"]
        halfb200.tc_cgemm(case["op"], "N", m, n, kk, 1.0 + 0j, state["a"].data_ptr(), kk if case["op"] == "C" else m,
                          state["b"].data_ptr(), kk, 0j, state["c"].data_ptr(), m)
        return state["c"]
    ctx = state["ctx"]
    if kind == "apply":
        return list(ctx.apply_hs(state["k"], state["psi"]))
    if kind == "force":
        return ctx.nonlocal_forces(state["k"], state["psi"], state["eps"], state["occ"], 0.25)
    if kind == "density":
        rho, charge = ctx.output_density(state["mesh"], state["weights"], state["psi"], state["occ"])
        return {"rho": rho, "charge": charge, "forces": ctx.ionic_forces(rho)}
    if kind == "relax":
        ctx.set_positions(state["positions"])
    if len(state["mesh"]) == 1:
        return ctx.solve(state["mesh"][0], case["bands"])[0]
    return ctx.solve_kpoints(state["mesh"], case["bands"])


#: Block iterations that a solve to the tolerance takes at the least, from unit vectors.
_ITERATIONS = 10


def work(case):
    if case["kind"] == "gemm":
        m, n, kk = case["m"], case["n"], case["kk"]
        return {"bytes": 8 * (m * kk + n * kk + m * n), "flops": 8 * m * n * kk}
    w = synth.workload(case["cell"])
    vol, nr = abs(np.linalg.det(w.lattice)), float(np.prod(w.grid))
    npw = vol * (w.encut / 3.80998) ** 1.5 / (6 * np.pi ** 2)
    npr = float(sum(c * sum(2 * l + 1 for l in s.lps) for s, c in zip(w.species, w.counts)))
    m, nk = case["bands"], case.get("nk", 1)
    local = 2 * 5 * nr * math.log2(nr)                  # two box transforms of a band
    sweep = m * (local + 3 * 8 * npw * npr)             # H psi and S psi of m bands
    if case["kind"] == "apply":
        return {"bytes": 16 * 3 * npw * m + 8 * nr, "flops": sweep}
    if case["kind"] == "force":
        return {"bytes": 16 * npw * m, "flops": 4 * 8 * npw * npr * m}
    if case["kind"] == "density":
        return {"bytes": nk * 16 * npw * m + 16 * nr,
                "flops": nk * m * (local / 2 + 8 * npw * npr) + nr * w.nions * 16}
    # solve: per iteration one sweep and the projections, the S-orthogonalisation
    # and the rotations of the block
    return {"bytes": nk * (16 * npw * (m + npr) + 8 * nr),
            "flops": nk * _ITERATIONS * (sweep + 20 * 8 * npw * m * m)}


def exact(case, seed):
    """The product in 64 bits.  The other kinds have no value in plain torch
    or numpy: their operator comes out of the pseudopotential, exchange-
    correlation and augmentation set-up that is most of the library itself.
    Their results are FP64 (the solves' eigenvalues converge to it in every
    mode) and are held to that type's bound."""
    if case["kind"] != "gemm":
        return None
    s = prepare(case, seed)
    a, b = s["a"].to(torch.complex128), s["b"].to(torch.complex128)
    return b @ a.conj().T if case["op"] == "C" else b @ a
