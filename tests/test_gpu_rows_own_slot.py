"""A slot is no partner of itself in the FP64 row kernels' angular sums: what
the g and q splines are at cos = 1, which no two neighbours of an atom may
reach, must not enter the objective, the residuals or the gradient.

Clusters in cells of 30 A, so that no image is near: dimers (rows of one slot,
no triplet at all), and bent chains of three atoms (one triplet each, at
cos = -0.17) whose angular splines get c (x - x_k)^3 beyond their next to last
knot x_k -- exactly representable, zero at every sampled cosine, c h^3 at 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STYLES = [("meam/spline", 1), ("meam/spline", 2), ("gmeam/spline", 2), ("jmeam/spline", 1), ("jmeam2/spline", 2)]


def _angular(spec):
    return [g for i, g in enumerate(spec.groups) if i in (4, 6, 8)]


def _cells(shapes, ntypes, seed, types=None):
    from meamzilla_b200 import synth
    rng = np.random.default_rng(seed)
    cells = []
    for k, shape in enumerate(shapes):
        pos = np.asarray(shape) + rng.normal(0.0, 0.02, np.shape(shape))
        n = len(pos)
        ty = rng.integers(0, ntypes, n) if types is None else np.asarray(types[k])
        cells.append(synth.Cell(lattice=np.eye(3) * 30.0, types=ty, pos=pos + 12.0, force0=rng.normal(0, 0.3, (n, 3)),
                                energy0=-1.0, stress0=rng.normal(0, 1e-3, 6)))
    return cells


def _spec(style, ntypes, rcut=3.0, ng=15):
    from meamzilla_b200 import synth
    spec = synth.in_range_variant(synth.teacher_potential(style, ntypes, rcut, seed=11))
    for group in _angular(spec):
        for s in group:
            x = np.linspace(-1.0, 1.0, ng)
            s.y = np.interp(x, np.linspace(-1.0, 1.0, s.nknots), s.y)
    return spec


def _evaluator(spec, cells, n=1):
    from meamzilla_b200.potential import Database, Evaluator, PotentialFile
    pot = PotentialFile.from_spec(spec)
    db = Database.from_cells(cells, pot)
    return pot, db, Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=n)


def _coefficients(spec, groups):
    """Indices of the coefficients of the given function groups (splines wholly free or wholly fixed)."""
    at, out = 0, []
    for i, group in enumerate(spec.groups):
        for s in group:
            n = s.nknots + 2 if s.fixed is None else 0
            if i in groups:
                out += list(range(at, at + n))
            at += n
    return np.array(out)


DIMER = [[0.0, 0.0, 0.0], [2.4, 0.3, 0.1]]
# A and C see B only (f, rho and phi end at 3.0; A-C is 3.7 apart): cos(A-B-C) = -0.17
CHAIN = [[2.4, 0.0, 0.0], [0.0, 0.0, 0.0], [-0.41, 2.36, 0.0]]


@pytest.mark.parametrize("style,ntypes", STYLES)
def test_no_triplets_no_influence(style, ntypes):
    """Dimers: residuals and objective do not depend on g and q, bit for bit,
    and their gradient is zero."""
    from meamzilla_b200.potential import MZ_FP64
    spec = _spec(style, ntypes, ng=8)
    pot, db, ev = _evaluator(spec, _cells([DIMER] * 7, ntypes, seed=3), n=2)
    assert db.stats()["max_row"] == 1
    ang = _coefficients(spec, (4, 6, 8))
    assert ang.size and pot.ncoeff == _coefficients(spec, range(9)).size
    x = np.repeat(pot.coeffs()[None], 2, 0)
    x[1, ang] += 1e6 * np.random.default_rng(4).normal(size=ang.size)
    out = ev.objective(x, MZ_FP64, errvec=True)
    assert np.array_equal(out["errvec"][0], out["errvec"][1]) and out["obj"][0] == out["obj"][1]
    dens = [ev.densities(x[0]), ev.densities(x[1])]
    assert np.array_equal(*dens)
    obj, grad = ev.objective_grad(x, MZ_FP64)
    assert np.array_equal(obj, out["obj"])
    assert np.all(grad[:, ang] == 0.0) and np.any(grad != 0.0)


@pytest.mark.parametrize("big", [0.0, 1e6, 1e9])
@pytest.mark.parametrize("style,ntypes", STYLES)
def test_value_at_one_does_not_matter(style, ntypes, big):
    """Chains, angular splines `big` times their size at cos = 1.  The second
    derivatives' solve leaves eps 0.27^7 = 1e-4 eps of the value at 1 (seven
    knots from the next to last one to the sampled interval) in the sampled
    one, in FP64 on either side: eight of those beside the parity tests' 1e-12
    (energy per atom) and, with slopes of up to 100 / A, 1e-10 (forces)."""
    import oracle
    from meamzilla_b200.potential import MZ_FP64
    spec = _spec(style, ntypes)
    most = 0.0
    for group in _angular(spec):
        for s in group:
            h = 2.0 / (s.nknots - 1)
            top = big * np.max(np.abs(s.y))
            most = max(most, top)
            s.y = s.y.copy()
            s.y[-1] += top
            s.grad = s.grad + np.array([0.0, 3.0 * top / h])
    pot, db, ev = _evaluator(spec, _cells([CHAIN] * 9, ntypes, seed=5))
    assert db.stats()["max_row"] == 2
    x = pot.coeffs()
    out = ev.objective(x[None], MZ_FP64, forces=True, energy=True)
    ref = oracle.CRestatement.for_evaluator(ev).objective(x, full=True)
    noise = 8 * 1e-4 * 2.2e-16 * most
    assert np.max(np.abs(out["energy"][0] - ref["energy"])) <= 1e-12 + noise
    assert np.max(np.abs(out["forces"][0] - ref["forces"])) <= 1e-10 + 100 * noise


def test_gmeam_without_a_triplet_species():
    """One B in cells of A: no A atom has two B neighbours, so g of A-B-B has no
    influence -- zero gradient, residuals bit-identical, and Powell's method
    says so instead of normalising a column of rounding."""
    from meamzilla_b200 import synth
    from meamzilla_b200.optimize import powell_fit
    from meamzilla_b200.potential import MZ_FP64
    spec = _spec("gmeam/spline", 2, rcut=4.0, ng=8)
    for group in (0, 3):  # no B-B pair either: phi and f of it are not fitted
        s = spec.groups[group][2]
        s.fixed, s.bc = np.ones(s.nknots, dtype=int), (1, 1)
    rng = np.random.default_rng(8)
    cells = []
    for _ in range(6):
        grid = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
        pos = ((grid + np.array([[0, 0, 0], [.5, .5, .5]])) / 3).reshape(-1, 3) * 9.6 + rng.normal(0, 0.05, (54, 3))
        types = np.zeros(54, dtype=int)
        types[rng.integers(54)] = 1
        cells.append(synth.Cell(lattice=np.eye(3) * 9.6, types=types, pos=pos, force0=rng.normal(0, 0.3, (54, 3)),
                                energy0=-1.0, stress0=rng.normal(0, 1e-3, 6)))
    pot, db, ev = _evaluator(spec, cells, n=_coefficients(spec, range(5)).size)
    x = pot.coeffs()
    first = _coefficients(spec, (4,))[0]
    per = spec.groups[4][0].nknots + 2
    # g of centre A (type 0): splines A-AA, A-AB, A-BB
    abb = np.arange(first + 2 * per, first + 3 * per)
    two = np.stack([x, x])
    two[1, abb] += rng.normal(size=per)
    out = ev.objective(two, MZ_FP64, errvec=True)
    assert np.array_equal(out["errvec"][0], out["errvec"][1]) and out["obj"][0] == out["obj"][1]
    assert np.all(ev.objective_grad(x[None], MZ_FP64)[1][0, abb] == 0.0)
    said = []
    powell_fit(ev, x, max_steps=1, precision=MZ_FP64, log=said.append)
    assert "does not depend on coefficient %d," % abb[0] in said[-1], said

