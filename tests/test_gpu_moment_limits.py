"""Mixed-precision meam where the moment path's tables are at and beyond the
device's shared memory (U of 64 knots, two species; 224 to 242 KB of 227):
the calls run, on the row kernels where they do not fit, within the mixed
precision bars of the parity tests (objective 1e-6, forces 1e-5 of the largest
one or of 1 eV/A)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nr", [(64, 9), (64, 10), (64, 11), (64, 12), (64, 13), (60, 14)])
def test_mixed_calls_near_the_limit(nu, nr):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED, Database, Evaluator, PotentialFile
    spec = synth.in_range_variant(synth.teacher_potential("meam/spline", 2, 4.3, seed=2))
    for i, group in enumerate(spec.groups):
        for s in group:
            n = {0: nr, 1: nr, 2: nu, 3: nr, 4: 8}[i]
            s.y = np.interp(np.linspace(s.left, s.right, n), np.linspace(s.left, s.right, s.nknots), s.y)
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    cells = synth.make_cells(30, lambda r: 60, rng, ntypes=2)
    for c in cells:
        c.force0 = rng.normal(0, 0.3, c.force0.shape)
    ev = Evaluator(Database.from_cells(cells, pot), pot, 1.0, 1.0, 0, max_candidates=64)
    X = synth.perturbed(pot.coeffs(), 64, 0.01, seed=5)
    a, b = ev.objective(X, MZ_FP64, forces=True), ev.objective(X, MZ_MIXED, forces=True)
    assert np.all(np.abs(a["obj"] - b["obj"]) <= 1e-6 * a["obj"])
    assert np.max(np.abs(a["forces"] - b["forces"])) <= 1e-5 * max(1.0, np.max(np.abs(a["forces"])))
    ev.objective_grad(X[:2], MZ_MIXED)


def test_mixed_calls_without_pairs():
    """Isolated atoms alone: nothing to contract, the row kernels serve."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED, Database, Evaluator, PotentialFile
    rng = np.random.default_rng(3)
    cells = [synth.Cell(lattice=np.eye(3) * 30.0, types=np.zeros(1, dtype=int), pos=np.zeros((1, 3)),
                        force0=rng.normal(0, 0.3, (1, 3)), energy0=-1.0, stress0=rng.normal(0, 1e-3, 6)) for _ in range(5)]
    pot = PotentialFile.from_spec(synth.in_range_variant(synth.teacher_potential("meam/spline", 1, 4.3, seed=2)))
    db = Database.from_cells(cells, pot)
    assert db.stats()["npairs"] == 0
    ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=3)
    X = synth.perturbed(pot.coeffs(), 3, 0.01, seed=5)
    a, b = ev.objective_grad(X, MZ_FP64), ev.objective_grad(X, MZ_MIXED)
    assert np.all(np.abs(a[0] - b[0]) <= 1e-6 * a[0])
    assert np.max(np.abs(a[1] - b[1])) <= 1e-4 * np.max(np.abs(a[1]))
    assert np.all(np.abs(ev.objective(X, MZ_MIXED) - a[0]) <= 1e-6 * a[0])


# knots of f and g: (f + 2) (g + 2) species features.  Up to 256 run in
# integers; the contraction on the CUDA cores takes the rest (and all with
# MZ_FM8ADJ=0), in blocks of up to 512 threads from 257 features on; 480 do not
# fit its shared memory.
@pytest.mark.parametrize("ntypes,nf,ng,adj8", [(1, 20, 12, "1"), (1, 14, 14, "0"), (1, 14, 14, "1"), (2, 8, 10, "0"),
                                               (2, 12, 10, "1"), (2, 12, 13, "1"), (2, 14, 13, "1")])
def test_gradient_of_many_features(ntypes, nf, ng, adj8, monkeypatch):
    """The moment path's gradient within the mixed precision bar, 1e-4 of its
    largest component, of the FP64 one, for every candidate of a group of 64
    and of a group of 8."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED, Database, Evaluator, PotentialFile
    monkeypatch.setenv("MZ_FM", "2")
    monkeypatch.setenv("MZ_FM8ADJ", adj8)
    spec = synth.in_range_variant(synth.teacher_potential("meam/spline", ntypes, 4.3, seed=2))
    for group, n in ((3, nf), (4, ng)):
        for s in spec.groups[group]:
            s.y = np.interp(np.linspace(s.left, s.right, n), np.linspace(s.left, s.right, s.nknots), s.y)
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    cells = synth.make_cells(6, lambda r: 40, rng, ntypes=ntypes)
    for c in cells:
        c.force0 = rng.normal(0, 0.3, c.force0.shape)
    db = Database.from_cells(cells, pot)
    for n in (64, 8):
        ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=n)
        X = synth.perturbed(pot.coeffs(), n, 0.01, seed=5)
        a, b = ev.objective_grad(X, MZ_FP64)[1], ev.objective_grad(X, MZ_MIXED)[1]
        assert (ev.moment_path(MZ_MIXED, True) > 0) == ((nf + 2) * (ng + 2) * ntypes < 480)
        assert np.all(np.max(np.abs(a - b), axis=1) <= 1e-4 * np.max(np.abs(a), axis=1))
