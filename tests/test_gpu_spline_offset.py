"""A constant added to a spline's knot values does not spoil its slopes: y''
depends on differences of the values only, and the tables are formed from
those.  Forces of potentials whose phi and U are shifted by 1e6 against the C
restatement of the reference's tridiagonal solve, 1e-10 eV/A (the FP64 bar of
the parity tests; the shift drops out of every force)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("style", ["eam/spline", "meam/spline"])
def test_forces_of_shifted_splines(style):
    import oracle
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Database, Evaluator, PotentialFile
    spec = synth.in_range_variant(synth.teacher_potential(style, 1, 4.5, seed=2))
    for group in (0, 2):
        spec.groups[group][0].y = spec.groups[group][0].y + 1e6
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    grid = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    frac = ((grid + np.array([[0, 0, 0], [.5, .5, .5]])) / 3).reshape(-1, 3)
    cells = [synth.Cell(lattice=np.eye(3) * 9.6, types=np.zeros(54, dtype=int), pos=frac * 9.6 + rng.normal(0, 0.08, (54, 3)),
                        force0=np.zeros((54, 3)), energy0=0.0, stress0=np.zeros(6)) for _ in range(4)]
    ev = Evaluator(Database.from_cells(cells, pot), pot, 1.0, 1.0, 0, max_candidates=1)
    x = pot.coeffs()
    f = ev.objective(x[None], MZ_FP64, forces=True)["forces"][0]
    ref = oracle.CRestatement.for_evaluator(ev).objective(x, full=True)["forces"]
    assert np.max(np.abs(f - ref)) <= 1e-10
