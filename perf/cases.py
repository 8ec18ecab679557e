"""The work that users of this package have it do, as cases that can be timed and checked.

``listed()`` gives the cases by name and ``draw(rng)`` further ones of the same ranges; ``prepare``
makes what a program holds before the call (inputs from the seed, and the operator, plan or step that
such a program keeps), ``run`` is one pass through the public entry points and returns its outputs,
``work`` counts the bytes and operations a pass cannot do without, and ``exact`` gives the outputs as
plain torch computes them in 64 bits, where they have such a value.

Kinds of case (``case["kind"]``):

- ``apply``: ``CuspFactoredHamiltonian.apply``, the Rayleigh--Ritz and Lanczos apply;
- ``filter``: ``chebyshev_filter`` of one system, the Chebyshev step of a single solve;
- ``ensemble_filter``: ``BatchedHamiltonian.filter``, the same for many systems in one launch;
- ``adjoint``: ``adjoint.CuspApply`` forward and backward (gradients to the orbitals and potential);
- ``poisson``: ``CoulombCutoffPoisson.solve_batch``;
- ``xc``: ``functional_by_name(...).evaluate``, spin-restricted or spin-polarised;
- ``potentials``: ``KohnShamStep.potentials`` (one system) or ``BatchedKohnShamStep.potentials``;
- ``ritz``: ``batch.batched_rayleigh_ritz``;
- ``geometry``: ``build_cusp_geometry``;
- ``scf``: ``solve_self_consistent``, a whole plain float64 solve.

The operator cases take the cusp factor's own face weights exp(-2u), u = sum_a Z_a |r - R_a|, with the
pointwise mass weight, so that their outputs have a value in closed form; the others build the real
geometry.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

DEVICE = "cuda:0"
F64 = torch.float64

#: staggered first-derivative weights at the distances 1/2, 3/2, ... of the face, by order
TAPS = {2: (1.0,), 4: (9.0 / 8.0, -1.0 / 24.0), 6: (75.0 / 64.0, -25.0 / 384.0, 3.0 / 640.0),
        8: (1225.0 / 1024.0, -245.0 / 3072.0, 49.0 / 5120.0, -5.0 / 7168.0)}

#: nuclei (charges, positions along z in bohr) and electrons of the systems the repository solves
SYSTEMS = {"h": ((1.0,), (0.0,), 1.0), "he": ((2.0,), (0.0,), 2.0), "h2": ((1.0, 1.0), (-0.7, 0.7), 2.0),
           "h2plus": ((1.0, 1.0), (-1.0, 1.0), 1.0)}


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: the bare H atom's block (one state and four extra) on its 33^3 grid, applied
        # once in every Rayleigh--Ritz step and Lanczos step
        dict(name="apply-h-33", kind="apply", system="h", nx=33, ny=33, nz=33, h=0.25, order=8, orbitals=5,
             dtype="float64"),
        # the plain float64 He solve: one Chebyshev filter call, about 150 of them per solve
        dict(name="filter-he-65", kind="filter", system="he", nx=65, ny=65, nz=65, h=0.25, order=8, orbitals=5,
             degree=20, dtype="float64"),
        # the mixed-precision ensemble: the float filter of many He systems in one launch
        dict(name="filter-ens-65", kind="ensemble_filter", system="he", nx=65, ny=65, nz=65, h=0.25, orbitals=5,
             batch=64, degree=20, dtype="float32"),
        # the adjoint pass at h = 0.16: forward and vector-Jacobian product of the apply
        dict(name="adjoint-he-101", kind="adjoint", system="he", nx=101, ny=101, nz=101, h=0.16, orbitals=5),
        # the Hartree solves of a batch of H2 systems on their ragged grid
        dict(name="poisson-h2-batch", kind="poisson", nx=81, ny=81, nz=91, h=0.2, pad=2.5, batch=8),
        # the GGA of the H2 system on its whole grid
        dict(name="xc-pbe-h2", kind="xc", functional="pbe", n_spin=1, points=81 * 81 * 91),
        # a spin-polarised functional on the He grid's points
        dict(name="xc-blyp-spin", kind="xc", functional="blyp", n_spin=2, points=65 * 65 * 65),
        # one SCF iteration's potentials of one system: what the drop-in computes twice per iteration
        dict(name="potentials-he-65", kind="potentials", system="he", functional="lda_vwn", nx=65, ny=65, nz=65,
             h=0.25, batch=1),
        # the same for an ensemble
        dict(name="potentials-ens-65", kind="potentials", system="he", functional="lda_vwn", nx=65, ny=65, nz=65,
             h=0.25, batch=32),
        # the ensemble's Rayleigh--Ritz step in float64
        dict(name="ritz-ens-65", kind="ritz", system="he", nx=65, ny=65, nz=65, h=0.25, orbitals=5, batch=32),
        # one member of the bond scan: its geometry, built before every solve and six times per nucleus
        # in a nuclear gradient
        dict(name="geometry-h2plus", kind="geometry", system="h2plus", nx=49, ny=49, nz=57, h=0.25),
        # a whole plain float64 solve on a small grid, as the quick runs and tests do
        dict(name="scf-he-33", kind="scf", system="he", functional="lda_vwn", nx=33, ny=33, nz=33, h=0.5),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _grid(rng, low, high):
    """Three edges between low and high, each at most a quarter off a common size, odd and even."""
    size = math.exp(rng.uniform(math.log(low), math.log(high)))
    return [max(low, min(high, int(round(size * rng.uniform(0.8, 1.25))))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["apply", "filter", "ensemble_filter", "adjoint", "poisson", "xc", "potentials", "ritz", "geometry",
                       "scf"])
    h = round(rng.uniform(0.16, 0.35), 3)
    if kind in ("apply", "filter"):
        nx, ny, nz = _grid(rng, 17, 101)
        case = dict(kind=kind, system=rng.choice(["h", "he", "h2"]), nx=nx, ny=ny, nz=nz, h=h, order=8,
                    orbitals=rng.randint(1, 8), dtype=rng.choice(["float64", "float32"]))
        if rng.random() < 0.15:
            case.update(order=rng.choice([2, 4, 6]), dtype="float64")
        if kind == "filter":
            case["degree"] = rng.randint(8, 20)
        return case
    if kind == "ensemble_filter":
        nx, ny, nz = _grid(rng, 25, 81)
        dtype = rng.choice(["float64", "float32", "float32"])
        orbitals = rng.randint(2, 6)
        most = 64 * 5 * 65 ** 3 / (nx * ny * nz * orbitals) / (3 if dtype == "float64" else 1.2)
        return dict(kind=kind, system=rng.choice(["h", "he", "h2"]), nx=nx, ny=ny, nz=nz, h=h, orbitals=orbitals,
                    batch=_log_int(rng, 2, max(2, min(96, most))), degree=rng.randint(8, 20), dtype=dtype)
    if kind == "adjoint":
        nx, ny, nz = _grid(rng, 33, 101)
        return dict(kind=kind, system=rng.choice(["h", "he", "h2"]), nx=nx, ny=ny, nz=nz, h=h, orbitals=rng.randint(1, 6))
    if kind == "poisson":
        nx, ny, nz = _grid(rng, 25, 101)
        most = 8 * 91 ** 3 / (nx * ny * nz)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, h=h, pad=rng.choice([2.0, 2.5, 2.5]),
                    batch=_log_int(rng, 1, max(1, min(32, most))))
    if kind == "xc":
        return dict(kind=kind, functional=rng.choice(["lda_vwn", "lda_pw92", "lda_pz81", "pbe", "blyp"]),
                    n_spin=rng.choice([1, 1, 2]), points=_log_int(rng, 20000, 900000))
    if kind == "potentials":
        nx, ny, nz = _grid(rng, 33, 73)
        most = 32 * 65 ** 3 / (nx * ny * nz)
        functional = rng.choice(["lda_vwn", "lda_vwn", "pbe", "blyp"])
        if functional != "lda_vwn":
            most /= 4
        batch = 1 if rng.random() < 0.4 else _log_int(rng, 2, max(2, min(48, most)))
        return dict(kind=kind, system=rng.choice(["he", "h2"]), functional=functional, nx=nx, ny=ny, nz=nz, h=h,
                    batch=batch)
    if kind == "ritz":
        nx, ny, nz = _grid(rng, 25, 81)
        orbitals = rng.randint(2, 10)
        most = 32 * 5 * 65 ** 3 / (nx * ny * nz * orbitals)
        return dict(kind=kind, system=rng.choice(["h", "he", "h2"]), nx=nx, ny=ny, nz=nz, h=h, orbitals=orbitals,
                    batch=_log_int(rng, 1, max(1, min(64, most))))
    if kind == "geometry":
        nx, ny, nz = _grid(rng, 33, 65)
        return dict(kind=kind, system=rng.choice(["h", "he", "h2", "h2plus"]), nx=nx, ny=ny, nz=nz, h=h)
    nx, ny, nz = _grid(rng, 25, 37)
    return dict(kind="scf", system=rng.choice(["he", "h2"]), functional="lda_vwn", nx=nx, ny=ny, nz=nz,
                h=round(rng.uniform(0.35, 0.5), 3))


# ----------------------------------------------------------------------------------------- inputs
def _package():
    return __graft_entry__.package()


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _randn(shape, gen, dtype=F64):
    return torch.randn(shape, generator=gen, device=DEVICE, dtype=dtype)


def _uniform(low, high, shape, gen):
    return low + (high - low) * torch.rand(shape, generator=gen, device=DEVICE, dtype=F64)


def _nuclei(case):
    charges, zs, electrons = SYSTEMS[case["system"]]
    return charges, [(0.0, 0.0, z) for z in zs], electrons


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _origin(case):
    """The coordinate origin is the lattice point in the middle of the box."""
    return tuple(-case["h"] * (n // 2) for n in _shape(case))


def _axes(case, shift=(0.0, 0.0, 0.0), extra=(0, 0, 0)):
    return [o + case["h"] * (s + torch.arange(n + e, device=DEVICE, dtype=F64))
            for o, n, s, e in zip(_origin(case), _shape(case), shift, extra)]


def _distance(axes, position):
    x, y, z = (a - p for a, p in zip(axes, position))
    return torch.sqrt(x[:, None, None] ** 2 + y[None, :, None] ** 2 + z[None, None, :] ** 2)


def _weight(case, axes):
    """exp(-2 u) with u = sum_a Z_a |r - R_a|."""
    charges, positions, _ = _nuclei(case)
    return torch.exp(-2.0 * sum(q * _distance(axes, r) for q, r in zip(charges, positions)))


def _faces(case):
    """The weight at the staggered faces of each axis: order more faces than nodes along it."""
    order = case.get("order", 8)
    out = []
    for d in range(3):
        shift, extra = [0.0, 0.0, 0.0], [0, 0, 0]
        shift[d], extra[d] = 0.5 - order / 2, order
        out.append(_weight(case, _axes(case, shift, extra)))
    return out


def _smooth(case, gen, count, depth):
    """``(count, N)`` smooth wells: five Gaussians each, of amplitudes N(0, depth)."""
    axes = _axes(case)
    half = [0.35 * case["h"] * n for n in _shape(case)]
    out = torch.zeros((count, *_shape(case)), device=DEVICE, dtype=F64)
    for k in range(5):
        a = depth * _randn((count,), gen)
        w = _uniform(0.7, 2.0, (count,), gen)
        c = [_uniform(-s, s, (count,), gen) for s in half]
        g = [torch.exp(-((x[None, :] - ci[:, None]) ** 2) / (2.0 * w[:, None] ** 2)) for x, ci in zip(axes, c)]
        out += a[:, None, None, None] * g[0][:, :, None, None] * g[1][:, None, :, None] * g[2][:, None, None, :]
    return out.reshape(count, -1)


def _operator_fields(case, seed):
    """What an operator is made of, in float64: faces, 1/weight, one potential per system, the measure
    and the orbital block. Every call with the same seed gives the same values."""
    gen = _generator(seed)
    batch = case.get("batch", 1)
    charges, positions, _ = _nuclei(case)
    weight = _weight(case, _axes(case)).reshape(-1)
    # the transformed potential of the cusp factor is smooth at the nuclei: -Z^2/2 there, -Z/r outside
    base = sum(-q / torch.sqrt(_distance(_axes(case), r) ** 2 + (2.0 / q) ** 2) for q, r in zip(charges, positions))
    potential = base.reshape(1, -1) + _smooth(case, gen, batch, 0.3)
    block = _randn((batch, case["orbitals"], weight.numel()), gen)
    return dict(faces=_faces(case), weight=weight, potential=potential, block=block, gen=gen)


def _interval(case):
    """Filter interval (lower, upper, spectrum_min): the top of the spectrum of the uniform operator
    with a margin for the varying weights, as a Lanczos enclosure would give it."""
    taps = 2.0 * sum(abs(t) for t in TAPS[case.get("order", 8)]) / case["h"]
    return 2.0, 1.5 * taps * taps * 1.6 + 10.0, -8.0


class _Factor:
    """The cusp factor as the operator reads it."""

    def __init__(self, faces, weight):
        self._faces = tuple(faces)
        self.weight = weight

    def face_weights(self, accuracy):
        return self._faces


class _Quadrature:
    """The bare operator terms as the operator reads them."""

    def __init__(self, potential, inverse_weight, measure):
        self._terms = (potential, inverse_weight, measure)

    def bare_operator_terms(self):
        return self._terms


def _operator_parts(case, fields):
    pkg = _package()
    grid = pkg.UniformGrid(_shape(case), case["h"], _origin(case), device=DEVICE, fd_order=case.get("order", 8))
    factor = _Factor(fields["faces"], fields["weight"])
    measure = pkg.Measure(grid, fields["weight"] * case["h"] ** 3)
    quadrature = _Quadrature(torch.zeros_like(fields["weight"]), 1.0 / fields["weight"], measure)
    return pkg, grid, factor, quadrature


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else F64


def _geometry(case):
    pkg = _package()
    charges, positions, electrons = _nuclei(case)
    grid = pkg.UniformGrid(_shape(case), case["h"], _origin(case), device=DEVICE)
    return pkg, pkg.build_cusp_geometry(grid, charges, positions), electrons


def _densities(case, seed, count):
    """``(count, N)`` electron densities: screened 1s densities of the nuclei with seeded exponents."""
    gen = _generator(seed)
    charges, positions, electrons = _nuclei(case)
    total = torch.zeros((count, *_shape(case)), device=DEVICE, dtype=F64)
    for q, r in zip(charges, positions):
        d = _distance(_axes(case), r)
        zeta = q * _uniform(0.75, 1.0, (count,), gen)
        share = electrons / len(charges)
        total += share * (zeta ** 3 / math.pi)[:, None, None, None] * torch.exp(-2.0 * zeta[:, None, None, None] * d[None])
    return total.reshape(count, -1)


def _xc_inputs(case, seed):
    """Densities and sigmas as a molecule's grid has them: exponential tails down to about 1e-9, with the
    gradient of such a tail times a seeded factor; the two spins differ by up to a factor of three."""
    gen = _generator(seed)
    p, s = case["points"], case["n_spin"]
    r = 8.0 * torch.rand(p, generator=gen, device=DEVICE, dtype=F64) ** (1.0 / 3.0)
    zeta = _uniform(1.1, 1.3, (p,), gen)
    total = 2.0 * zeta ** 3 / math.pi * torch.exp(-2.0 * zeta * r)
    if s == 1:
        density = total[None]
    else:
        part = _uniform(0.25, 0.75, (p,), gen)
        density = torch.stack([total * part, total * (1.0 - part)])
    if case["functional"].startswith("lda"):
        return density, None
    grad = 2.0 * zeta[None] * density * _uniform(0.5, 1.2, (s, p), gen)
    if s == 1:
        return density, grad ** 2
    cosine = _uniform(-0.2, 1.0, (p,), gen)
    return density, torch.stack([grad[0] ** 2, grad[0] * grad[1] * cosine, grad[1] ** 2])


# -------------------------------------------------------------------------------------- prepare, run
def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("apply", "filter", "adjoint"):
        fields = _operator_fields(case, seed)
        pkg, grid, factor, quadrature = _operator_parts(case, fields)
        dtype = _dtype(case)
        state["hamiltonian"] = pkg.CuspFactoredHamiltonian(grid, factor, extra_potential=fields["potential"][0],
                                                           quadrature=quadrature, dtype=dtype)
        state["block"] = fields["block"][0].to(dtype)
        if kind == "adjoint":
            state["block"].requires_grad_(True)
            state["potential"] = fields["potential"][0].clone().requires_grad_(True)
            state["seed_grad"] = _randn(fields["block"][0].shape, fields["gen"])
    elif kind == "ensemble_filter":
        fields = _operator_fields(case, seed)
        pkg, grid, factor, quadrature = _operator_parts(case, fields)
        state["hamiltonian"] = pkg.batch.BatchedHamiltonian(grid, factor, quadrature, fields["potential"],
                                                            dtype=_dtype(case))
        state["block"] = fields["block"].to(_dtype(case))
        lower, upper, low = _interval(case)
        rows = [pkg.chebyshev_coefficients(case["degree"], lower + 0.01 * b, upper, low) for b in range(case["batch"])]
        state["table"] = torch.tensor(rows, dtype=F64, device=DEVICE)
    elif kind == "ritz":
        fields = _operator_fields(case, seed)
        pkg, grid, factor, quadrature = _operator_parts(case, fields)
        state["hamiltonian"] = pkg.batch.BatchedHamiltonian(grid, factor, quadrature, fields["potential"])
        state["block"] = fields["block"]
    elif kind == "poisson":
        pkg = _package()
        grid = pkg.UniformGrid(_shape(case), case["h"], _origin(case), device=DEVICE)
        state["solver"] = pkg.CoulombCutoffPoisson(grid, pad_factor=case["pad"], max_batch=case["batch"])
        state["density"] = _poisson_density(case, seed)
    elif kind == "xc":
        state["functional"] = _package().functional_by_name(case["functional"])
        state["density"], state["sigma"] = _xc_inputs(case, seed)
    elif kind == "potentials":
        pkg, geometry, electrons = _geometry(case)
        density = _densities(case, seed, case["batch"])
        if case["batch"] == 1:
            state["step"] = pkg.KohnShamStep(geometry, case["functional"], electrons)
        else:
            state["step"] = pkg.batch.BatchedKohnShamStep(geometry, case["functional"], electrons, case["batch"])
        state["density"] = density
    elif kind == "geometry":
        # the scan's bond, displaced a little: other nuclei of the same system on the same grid
        rng = np.random.default_rng(seed)
        charges, positions, _ = _nuclei(case)
        state["charges"] = charges
        state["positions"] = [tuple(float(c) for c in np.asarray(r) + rng.uniform(-0.05, 0.05, 3)) for r in positions]
        pkg = _package()
        state["grid"] = pkg.UniformGrid(_shape(case), case["h"], _origin(case), device=DEVICE)
    else:
        pkg, geometry, electrons = _geometry(case)
        perturbation = _smooth(case, _generator(seed), 1, 0.02)[0]
        state["step"] = pkg.KohnShamStep(geometry, case["functional"], electrons, seed=int(seed) % 1000,
                                         external_potential=perturbation)
        state["mixing"] = pkg.MixingConfig(scheme="linear", alpha=0.3)
    return state


def _poisson_density(case, seed):
    gen = _generator(seed)
    n = case["nx"] * case["ny"] * case["nz"]
    return _smooth(case, gen, case["batch"], 0.5) + 0.05 * _randn((case["batch"], n), gen)


def run(state):
    case = state["case"]
    kind = case["kind"]
    pkg = _package()
    if kind == "apply":
        return state["hamiltonian"].apply(state["block"])
    if kind == "filter":
        return pkg.chebyshev_filter(state["hamiltonian"], state["block"], case["degree"], *_interval(case))
    if kind == "ensemble_filter":
        return state["hamiltonian"].filter(state["block"], state["table"], case["degree"])
    if kind == "adjoint":
        out = pkg.adjoint.CuspApply.apply(state["block"], state["potential"], state["hamiltonian"])
        grads = torch.autograd.grad(out, (state["block"], state["potential"]), state["seed_grad"])
        return {"out": out.detach(), "block_grad": grads[0], "potential_grad": grads[1]}
    if kind == "ritz":
        evals, vectors, norms, orth, info = pkg.batch.batched_rayleigh_ritz(state["hamiltonian"], state["block"],
                                                                            check_orthonormality=False)
        return {"values": evals, "vectors": vectors, "residuals": norms, "info": info}
    if kind == "poisson":
        return state["solver"].solve_batch(state["density"])
    if kind == "xc":
        out = state["functional"].evaluate(state["density"], state["sigma"])
        got = {"e": out.e_xc, "v": out.v_xc}
        if out.v_sigma is not None:
            got["v_sigma"] = out.v_sigma
        return got
    if kind == "potentials":
        p = state["step"].potentials(state["density"])
        return {"effective": p.effective, "v_hartree": p.v_hartree, "hartree": p.hartree_energy, "xc": p.xc_energy,
                "double_counting": p.xc_double_counting}
    if kind == "geometry":
        g = pkg.build_cusp_geometry(state["grid"], state["charges"], state["positions"])
        potential, inverse_weight, measure = g.quadrature.bare_operator_terms()
        faces = g.factor.face_weights(8)
        # the fields on the grid (the number of quadrature nodes goes with the nuclei's places)
        return {"weight": g.factor.weight, "faces": list(faces), "mass": g.quadrature.mass_weights,
                "far": g.quadrature.far_weights, "potential": potential, "inverse": inverse_weight,
                "measure": measure.quadrature, "hartree": g.step.v1s_grid}
    out = pkg.solve_self_consistent(state["step"], state["mixing"])
    names = sorted(out.energies)
    return {"density": out.density, "energies": torch.tensor([out.energies[k] for k in names], dtype=F64),
            "values": torch.tensor(out.eigenvalues, dtype=F64), "iterations": out.scf_iterations}


# -------------------------------------------------------------------------------------------- work
def _apply_flops(order):
    """Per point and orbital: in each direction a face (order/2 differences and multiply-adds, and its
    weight) and the sum over the point's faces; then the mass weight and the potential."""
    return 3 * (1.5 * order + 1 + 2 * order) + 4


def work(case):
    kind = case["kind"]
    if kind == "xc":
        s, gga = case["n_spin"], not case["functional"].startswith("lda")
        sig = (1 if s == 1 else 3) if gga else 0
        return {"bytes": 8.0 * case["points"] * (2 * s + 2 * sig + 1), "flops": case["points"] * (400.0 if gga else 150.0)}
    n = float(case["nx"] * case["ny"] * case["nz"])
    size = 4 if case.get("dtype") == "float32" else 8
    batch = case.get("batch", 1)
    if kind in ("apply", "filter", "ensemble_filter", "adjoint", "ritz"):
        m = case["orbitals"] * batch
        geometry = size * n * (4 + batch)
        per = _apply_flops(case.get("order", 8))
        if kind == "apply":
            return {"bytes": size * n * 2 * m + geometry, "flops": n * m * per}
        if kind == "adjoint":
            return {"bytes": size * n * 4 * m + geometry + size * n, "flops": n * m * (2 * per + 6)}
        if kind == "ritz":
            k = case["orbitals"]
            return {"bytes": size * n * 2 * m + geometry + size * n, "flops": n * m * (per + 10 * k + 6)}
        return {"bytes": size * n * 2 * m + geometry, "flops": n * m * (per + 4) * case["degree"]}
    if kind == "poisson":
        pad = case["pad"] ** 3 * n
        return {"bytes": 8.0 * (2 * n * batch + pad / 2), "flops": batch * 2.5 * pad * math.log2(pad) * 0.5}
    if kind == "potentials":
        pad = 2.5 ** 3 * n
        return {"bytes": 8.0 * (batch * 3 * n + 6 * n + pad / 2), "flops": batch * (1.25 * pad * math.log2(pad) + 300 * n)}
    if kind == "geometry":
        return {"bytes": 8.0 * 16 * n, "flops": 2000.0 * n}
    # a solve: about 25 iterations of four filter calls of degree 20 on five orbitals
    return {"bytes": 8.0 * 20 * n, "flops": 25 * 4 * 20 * 5 * n * _apply_flops(8)}


# ------------------------------------------------------------------------------------------- exact
def _divergence(x, faces, order, h):
    """sum_d D_d^T [w_d D_d x] of ``(..., nx, ny, nz)`` float64 boxes, zero outside the box."""
    half = order // 2
    c = [-t for t in reversed(TAPS[order])] + list(TAPS[order])
    c = [v / h for v in c]
    out = torch.zeros_like(x)
    for axis in range(3):
        dim = x.dim() - 3 + axis
        n = x.shape[dim]
        shape = list(x.shape)
        shape[dim] = order - 1
        pad = torch.zeros(shape, device=x.device, dtype=x.dtype)
        wide = torch.cat([pad, x, pad], dim=dim)  # node i at index i + order - 1
        face = sum(c[j] * wide.narrow(dim, j, n + order - 1) for j in range(order))  # the faces between, in order
        face = face * faces[axis].narrow(axis, 0, n + order - 1)
        out += sum(c[order - 1 - k] * face.narrow(dim, k, n) for k in range(order))
    return out


def _apply_exact(case, fields, potential, x):
    box = x.reshape(*x.shape[:-1], *_shape(case))
    div = _divergence(box, fields["faces"], case.get("order", 8), case["h"]).reshape(x.shape)
    return 0.5 * div / fields["weight"] + potential * x


def _filter_exact(case, fields, potential, x, lower, upper, low):
    """The scaled Chebyshev recurrence; ``lower`` may be one value per system."""
    e, c = 0.5 * (upper - lower), 0.5 * (upper + lower)
    sigma = first = e / (low - c)
    y = (_apply_exact(case, fields, potential, x) - c * x) * (first / e)
    previous = x
    for _ in range(2, case["degree"] + 1):
        new = 1.0 / (2.0 / first - sigma)
        y, previous = (_apply_exact(case, fields, potential, y) - c * y) * (2.0 * new / e) - (sigma * new) * previous, y
        sigma = new
    return y


def _poisson_exact(case, seed):
    shape, h = _shape(case), case["h"]

    def friendly(n):
        while True:
            r = n
            for p in (2, 3, 5):
                while r % p == 0:
                    r //= p
            if r == 1:
                return n
            n += 1

    pad = [friendly(int(math.ceil(case["pad"] * n))) for n in shape]
    radius = 0.5 * min(n * h for n in pad)
    f = [torch.fft.fftfreq(n, d=h, device=DEVICE, dtype=F64) for n in pad[:2]]
    f.append(torch.fft.rfftfreq(pad[2], d=h, device=DEVICE, dtype=F64))
    kx, ky, kz = (2.0 * math.pi * v for v in f)
    g2 = kx[:, None, None] ** 2 + ky[None, :, None] ** 2 + kz[None, None, :] ** 2
    kernel = 4.0 * math.pi * (1.0 - torch.cos(torch.sqrt(g2) * radius)) / g2
    kernel[0, 0, 0] = 2.0 * math.pi * radius ** 2
    density = _poisson_density(case, seed).reshape(-1, *shape)
    out = []
    for rho in density:
        v = torch.fft.irfftn(torch.fft.rfftn(rho, s=pad, dim=(0, 1, 2)) * kernel, s=pad, dim=(0, 1, 2))
        out.append(v[:shape[0], :shape[1], :shape[2]].reshape(-1))
    return torch.stack(out)


def _ritz_exact(case, fields):
    """Ritz values and residual norms; the vectors' signs are free, so they have no value."""
    x = fields["block"]
    q = fields["weight"] * case["h"] ** 3
    gram = torch.einsum("bip,p,bjp->bij", x, q, x)
    lower = torch.linalg.cholesky(gram)
    basis = torch.linalg.solve_triangular(lower, x, upper=False)
    applied = _apply_exact(case, fields, fields["potential"][:, None], basis)
    sub = torch.einsum("bip,p,bjp->bij", basis, q, applied)
    values, rotation = torch.linalg.eigh(0.5 * (sub + sub.transpose(1, 2)))
    vectors = rotation.transpose(1, 2) @ basis
    residual = rotation.transpose(1, 2) @ applied - values[..., None] * vectors
    norms = torch.einsum("bip,p,bip->bi", residual, q, residual).sqrt()
    return {"values": values, "vectors": None, "residuals": norms, "info": None}


# the functionals' energy densities per volume, as their papers give them
def _rs(n):
    return (3.0 / (4.0 * math.pi * n)) ** (1.0 / 3.0)


def _f_zeta(z):
    return ((1 + z) ** (4 / 3) + (1 - z) ** (4 / 3) - 2) / (2 ** (4 / 3) - 2)


FPP0 = 4.0 / (9.0 * (2 ** (1 / 3) - 1))


def _slater(u, d):
    return -2 ** (1 / 3) * 0.75 * (3 / math.pi) ** (1 / 3) * (u ** (4 / 3) + d ** (4 / 3))


def _vwn(u, d):
    def aux(x, a, x0, b, c):
        bx, b0, q = x * x + b * x + c, x0 * x0 + b * x0 + c, math.sqrt(4 * c - b * b)
        at = torch.atan(q / (2 * x + b))
        return a * (torch.log(x * x / bx) + 2 * b / q * at
                    - b * x0 / b0 * (torch.log((x - x0) ** 2 / bx) + 2 * (b + 2 * x0) / q * at))

    n, z = u + d, (u - d) / (u + d)
    x = torch.sqrt(_rs(n))
    para = aux(x, 0.0310907, -0.10498, 3.72744, 12.9352)
    ferro = aux(x, 0.01554535, -0.32500, 7.06042, 18.0578)
    stiff = aux(x, -1 / (6 * math.pi ** 2), -0.0047584, 1.13107, 13.0045)
    return n * (para + stiff * _f_zeta(z) * (1 - z ** 4) / FPP0 + (ferro - para) * _f_zeta(z) * z ** 4)


def _pw92_eps(rs, z, modified):
    def g(a, a1, b1, b2, b3, b4):
        s = torch.sqrt(rs)
        return -2 * a * (1 + a1 * rs) * torch.log1p(1 / (2 * a * (b1 * s + b2 * rs + b3 * rs * s + b4 * rs * rs)))

    a = (0.0310907, 0.01554535, 0.0168869) if modified else (0.031091, 0.015545, 0.016887)
    para = g(a[0], 0.21370, 7.5957, 3.5876, 1.6382, 0.49294)
    ferro = g(a[1], 0.20548, 14.1189, 6.1977, 3.3662, 0.62517)
    stiff = -g(a[2], 0.11125, 10.357, 3.6231, 0.88026, 0.49671)
    return para + stiff * _f_zeta(z) * (1 - z ** 4) / (FPP0 if modified else 1.709921) + (ferro - para) * _f_zeta(z) * z ** 4


def _pz81(u, d):
    def eps(rs, gamma, b1, b2, a, b, c, e):
        low = a * torch.log(rs) + b + c * rs * torch.log(rs) + e * rs
        return torch.where(rs >= 1, gamma / (1 + b1 * torch.sqrt(rs) + b2 * rs), low)

    n, z = u + d, (u - d) / (u + d)
    rs = _rs(n)
    para = eps(rs, -0.1423, 1.0529, 0.3334, 0.0311, -0.048, 0.0020, -0.0116)
    ferro = eps(rs, -0.0843, 1.3981, 0.2611, 0.01555, -0.0269, 0.0007, -0.0048)
    return n * (para + _f_zeta(z) * (ferro - para))


def _pbe(u, d, uu, ud, dd):
    kappa, mu, beta = 0.804, 0.2195149727645171, 0.06672455060314922
    gamma = (1 - math.log(2)) / math.pi ** 2
    kf = (3 * math.pi ** 2) ** (1 / 3)
    e = 0.0
    for n, s in ((u, uu), (d, dd)):
        s2 = 4 * s / (4 * kf ** 2 * (2 * n) ** (8 / 3))
        e = e + 0.5 * (-0.75 * (3 / math.pi) ** (1 / 3) * (2 * n) ** (4 / 3)) * (1 + kappa - kappa / (1 + mu * s2 / kappa))
    n, z = u + d, (u - d) / (u + d)
    eps = _pw92_eps(_rs(n), z, True)
    phi = 0.5 * ((1 + z) ** (2 / 3) + (1 - z) ** (2 / 3))
    t2 = (uu + 2 * ud + dd) / (4 * phi ** 2 * (4 * kf * n ** (1 / 3) / math.pi) * n * n)
    a = beta / gamma / (torch.exp(-eps / (gamma * phi ** 3)) - 1)
    return e + n * (eps + gamma * phi ** 3 * torch.log1p(beta / gamma * t2 * (1 + a * t2) / (1 + a * t2 + (a * t2) ** 2)))


def _blyp(u, d, uu, ud, dd):
    e, beta = 0.0, 0.0042
    for n, s in ((u, uu), (d, dd)):
        x = torch.sqrt(s) / n ** (4 / 3)
        e = e - n ** (4 / 3) * (1.5 * (3 / (4 * math.pi)) ** (1 / 3) + beta * x * x / (1 + 6 * beta * x * torch.asinh(x)))
    a, b, c, dl = 0.04918, 0.132, 0.2533, 0.349
    n, m13 = u + d, (u + d) ** (-1 / 3)
    den = 1 + dl * m13
    omega = torch.exp(-c * m13) / den * n ** (-11 / 3)
    delta = c * m13 + dl * m13 / den
    sigma = uu + 2 * ud + dd
    inner = u * d * (2 ** (11 / 3) * 0.3 * (3 * math.pi ** 2) ** (2 / 3) * (u ** (8 / 3) + d ** (8 / 3))
                     + (47 / 18 - 7 * delta / 18) * sigma - (2.5 - delta / 18) * (uu + dd)
                     - (delta - 11) / 9 * (u / n * uu + d / n * dd))
    inner = inner - 2 / 3 * n * n * sigma + (2 / 3 * n * n - u * u) * dd + (2 / 3 * n * n - d * d) * uu
    return e - 4 * a / den * u * d / n - a * b * omega * inner


def _xc_exact(case, seed):
    density, sigma = _xc_inputs(case, seed)
    name = case["functional"]
    density = density.clone().requires_grad_(True)
    u, d = (0.5 * density[0], 0.5 * density[0]) if case["n_spin"] == 1 else (density[0], density[1])
    if sigma is None:
        e = _slater(u, d) + (_vwn(u, d) if name == "lda_vwn" else
                             _pz81(u, d) if name == "lda_pz81" else
                             (u + d) * _pw92_eps(_rs(u + d), (u - d) / (u + d), False))
        return {"e": e.detach(), "v": torch.autograd.grad(e.sum(), density)[0]}
    sigma = sigma.clone().requires_grad_(True)
    s = [0.25 * sigma[0]] * 3 if case["n_spin"] == 1 else [sigma[0], sigma[1], sigma[2]]
    e = (_pbe if name == "pbe" else _blyp)(u, d, *s)
    v, vs = torch.autograd.grad(e.sum(), (density, sigma))
    return {"e": e.detach(), "v": v, "v_sigma": vs}


def exact(case, seed):
    kind = case["kind"]
    if kind == "xc":
        return _xc_exact(case, seed)
    if kind == "poisson":
        return _poisson_exact(case, seed)
    if kind == "ritz":
        return _ritz_exact(case, _operator_fields(case, seed))
    if kind in ("apply", "filter", "ensemble_filter", "adjoint"):
        fields = _operator_fields(case, seed)
        # the inputs as run() has them: a float32 block is one of float32 values
        block = fields["block"].to(_dtype(case)).to(F64)
        potential = fields["potential"][:, None]
        if kind == "apply":
            return _apply_exact(case, fields, potential[0], block[0])
        if kind == "filter":
            return _filter_exact(case, fields, potential[0], block[0], *_interval(case))
        if kind == "ensemble_filter":
            lower, upper, low = _interval(case)
            return torch.stack([_filter_exact(case, fields, potential[b], block[b], lower + 0.01 * b, upper, low)
                                for b in range(case["batch"])])
        bar = _randn(fields["block"][0].shape, fields["gen"])
        box = (bar / fields["weight"]).reshape(-1, *_shape(case))
        div = _divergence(box, fields["faces"], 8, case["h"]).reshape(bar.shape)
        return {"out": _apply_exact(case, fields, potential[0], block[0]), "block_grad": 0.5 * div + potential[0] * bar,
                "potential_grad": (bar * block[0]).sum(dim=0)}
    return None
