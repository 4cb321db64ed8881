"""The FP64 row kernels (a warp for a few atoms) where their dispatch and
their tiles can go wrong: rows just inside and beyond the 32, 64 and 128 slots
that pick the lanes per atom (beyond 128: the block kernel), angular knots
that cover [-1, 1] and that do not, one, two and three species, an atom count
that is no multiple of a warp's atoms, isolated atoms, and batches large
enough for several candidates per CTA.  Against the C restatement of the
reference: objective 1e-12 relative, forces 1e-10 eV/A (the FP64 bars of the
parity tests); gradient against its tangent-linear form, 1e-10 of the
component plus 1e-13 of the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(style, ntypes, rcut, seed, ncells=3, gspan=(-1.0, 1.0), rows=None, isolated=1):
    """Database whose longest row is in (rows[0], rows[1]]: cells of one shape
    at a density that grows until it is."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import Database, PotentialFile
    spec = synth.teacher_potential(style, ntypes, rcut, seed)
    if style != "pair/spline":
        spec = synth.in_range_variant(spec)
    for group in (spec.groups[4:5] + spec.groups[6:7] + spec.groups[8:9] if len(spec.groups) > 4 else []):
        for s in group:
            s.left, s.right = gspan
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(seed)
    for a in np.arange(6.2, 3.2, -0.05):
        cells = []
        for c in range(ncells):
            m = 2
            grid = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
            frac = ((grid + np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])) / m).reshape(-1, 3)
            n = len(frac) - c % 3  # 32, 31, 30 atoms
            L = np.eye(3) * a * m
            pos = frac[:n] @ L + rng.uniform(-0.05, 0.05, (n, 3))
            cells.append(synth.Cell(lattice=L, types=rng.integers(0, ntypes, n), pos=pos,
                                    force0=rng.normal(0, 0.3, (n, 3)), energy0=-1.0, stress0=rng.normal(0, 1e-3, 6)))
        # isolated atoms: empty rows
        for k in range(isolated):
            cells.insert(len(cells) - 2 * k, synth.Cell(
                lattice=np.eye(3) * 30.0, types=np.zeros(1, dtype=int), pos=np.zeros((1, 3)), force0=np.zeros((1, 3))))
        db = Database.from_cells(cells, pot)
        if rows is None or db.stats()["max_row"] > rows[0]:
            break
    if rows is not None:
        assert rows[0] < db.stats()["max_row"] <= rows[1], db.stats()
    return pot, db


def _oracle(ev):
    import oracle
    return oracle.CRestatement.for_evaluator(ev)


CASES = [("eam/spline", 1, 4.0, (8, 32)), ("eam/spline", 2, 5.5, (32, 64)), ("eam/spline", 3, 7.0, (64, 128)),
         ("meam/spline", 1, 4.0, (8, 32)), ("meam/spline", 2, 5.5, (32, 64)), ("meam/spline", 1, 7.0, (64, 128)),
         ("meam/spline", 2, 8.0, (128, 256)), ("gmeam/spline", 2, 4.0, (8, 32)), ("gmeam/spline", 3, 5.5, (32, 64)),
         ("jmeam/spline", 1, 5.5, (32, 64)), ("jmeam2/spline", 2, 4.0, (8, 32)), ("pair/spline", 2, 5.5, (8, 64))]


@pytest.mark.parametrize("gspan", [(-1.0, 1.0), (-0.7, 0.6)])
@pytest.mark.parametrize("style,ntypes,rcut,rows", CASES)
def test_rows_match_oracle(style, ntypes, rcut, rows, gspan):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    if gspan[0] != -1.0 and style in ("eam/spline", "pair/spline"):
        pytest.skip("no angular functions")
    pot, db = _setup(style, ntypes, rcut, seed=31, gspan=gspan, rows=rows)
    ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=3)
    X = synth.perturbed(pot.coeffs(), 3, 0.01, seed=5)
    out = ev.objective(X, MZ_FP64, errvec=True, forces=True, energy=True, stress=True)
    refused = style == "gmeam/spline" and ntypes == 3  # the FP64 adjoint's tables do not fit
    if not refused:
        obj, grad = ev.objective_grad(X, MZ_FP64)
    orc = _oracle(ev)
    for c in range(3):
        ref = orc.objective(X[c], full=True)
        assert abs(out["obj"][c] - ref["obj"]) <= 1e-12 * abs(ref["obj"])
        assert np.max(np.abs(out["forces"][c] - ref["forces"])) <= 1e-10
        assert np.max(np.abs(out["energy"][c] - ref["energy"])) <= 1e-10
        assert np.max(np.abs(out["stress"][c] - ref["stress"])) <= 1e-10
    if refused:
        return
    assert np.array_equal(obj, out["obj"])
    t = orc.gradient(X[0])
    assert np.all(np.abs(grad[0] - t) <= 1e-10 * np.abs(t) + 1e-13 * np.max(np.abs(t)))


@pytest.mark.parametrize("style", ["eam/spline", "meam/spline", "jmeam/spline"])
def test_candidates_of_a_batch_do_not_depend_on_it(style):
    """A candidate's FP64 values are bit-identical alone and in a batch large
    enough for several candidates per CTA."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    pot, db = _setup(style, 1, 5.5, seed=7, ncells=70, rows=(8, 64))
    n = 131
    X = synth.perturbed(pot.coeffs(), n, 0.01, seed=6)
    one = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=1)
    many = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=n)
    a = many.objective(X, MZ_FP64, errvec=True)
    for c in (0, 1, 2, 63, 129, 130):
        b = one.objective(X[c:c + 1], MZ_FP64, errvec=True)
        assert a["obj"][c] == b["obj"][0]
        assert np.array_equal(a["errvec"][c], b["errvec"][0])


def test_gradient_with_several_segments_per_cta():
    """1.4 M slots: more segments of the radial sums than CTAs, so that some
    CTAs take two and some none.  The gradient along five directions against
    the tangent-linear oracle: rounding of sums over 4e4 atoms, 1e-11 of
    |gradient| |direction|."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    pot, db = _setup("eam/spline", 1, 5.5, seed=3, ncells=1200, rows=(40, 64))
    assert db.stats()["npairs"] > 1.25e6
    ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=1)
    x = synth.perturbed(pot.coeffs(), 1, 0.01, seed=5)
    orc = _oracle(ev)
    g = [ev.objective_grad(x, MZ_FP64)[1][0] for _ in range(3)]
    assert np.array_equal(g[0], g[1]) and np.array_equal(g[0], g[2])
    rng = np.random.default_rng(2)
    for _ in range(5):
        d = rng.normal(size=x.size)
        t = orc.tangent(x[0], d)[1]
        assert abs(g[0] @ d - t) <= 1e-11 * np.linalg.norm(g[0]) * np.linalg.norm(d)


@pytest.mark.parametrize("style,rcut,rows", [("meam/spline", 7.0, (64, 128)), ("meam/spline", 4.0, (8, 32)),
                                             ("gmeam/spline", 7.0, (64, 128))])
def test_empty_rows_between_others(style, rcut, rows):
    """Empty rows that a warp takes after others, whose staged slots they must
    not read: 90 cells of 30 to 32 atoms and 40 isolated atoms.  The gradient
    along three directions against the tangent-linear oracle: rounding of sums
    over 3e3 atoms, 1e-11 of |gradient| |direction|."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    pot, db = _setup(style, 1, rcut, seed=3, ncells=90, rows=rows, isolated=40)
    ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=1)
    x = synth.perturbed(pot.coeffs(), 1, 0.01, seed=5)
    orc = _oracle(ev)
    obj, g = ev.objective_grad(x, MZ_FP64)
    assert np.array_equal(obj, ev.objective(x, MZ_FP64))
    rng = np.random.default_rng(2)
    for _ in range(3):
        d = rng.normal(size=x.size)
        t = orc.tangent(x[0], d)[1]
        assert abs(g[0] @ d - t) <= 1e-11 * np.linalg.norm(g[0]) * np.linalg.norm(d)
