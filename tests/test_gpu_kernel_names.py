"""Profiling names the kernels that ran: the FP64 row kernels by their own
names, the block kernels where those serve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("style,rcut,ran,not_ran", [
    ("meam/spline", 4.3, {"k_rows", "k_rows_adj", "k_rows_radial", "k_rows_grad_final"}, {"k_atoms", "k_adj", "k_grad_final"}),
    ("jmeam/spline", 4.3, {"k_rows", "k_adj", "k_grad_final"}, {"k_atoms", "k_rows_adj", "k_rows_grad_final"}),
    ("eam/spline", 9.0, {"k_atoms", "k_adj", "k_grad_final"}, {"k_rows", "k_rows_adj", "k_rows_grad_final"})])
def test_kernel_names(style, rcut, ran, not_ran):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Database, Evaluator, PotentialFile
    pot = PotentialFile.from_spec(synth.in_range_variant(synth.teacher_potential(style, 1, rcut, seed=2)))
    db = Database.from_cells(synth.make_cells(3, lambda r: 40, np.random.default_rng(6)), pot)
    assert (db.stats()["max_row"] > 128) == (rcut > 8)
    ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=1)
    x = synth.perturbed(pot.coeffs(), 1, 0.01, seed=5)
    ev.objective_grad(x, MZ_FP64)
    ev.profile(True)
    ev.kernel_times()
    ev.objective_grad(x, MZ_FP64)
    names = set(ev.kernel_times())
    assert ran <= names and not (not_ran & names), names
