"""What the launch tuner times, and what it hands on: nothing that a call does
not run, and to a context without room for the moment path a row variant that
was timed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(style, ntypes, rcut, ncells, seed):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import Database, PotentialFile
    spec = synth.in_range_variant(synth.teacher_potential(style, ntypes, rcut, seed=2))
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(seed)
    cells = synth.make_cells(ncells, lambda r: int(np.exp(r.uniform(np.log(16), np.log(300)))), rng, ntypes=ntypes)
    for c in cells:
        c.force0 = rng.normal(0, 0.3, c.force0.shape)
    return pot, Database.from_cells(cells, pot)


def test_fp64_rows_have_no_forward_variant():
    """jmeam gradients run k_rows forward and k_adj backward: the forward's block
    size is not a choice (timing it picked one of three by noise)."""
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    for k in range(8):
        pot, db = _workload("jmeam/spline", 1, 4.5, 3 + k, seed=k)
        ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=1)
        ev.objective_grad(synth.perturbed(pot.coeffs(), 1, 0.01, seed=5), MZ_FP64)
        t = ev.tuning(MZ_FP64, True)
        assert t["forward_block_slots"] == 256 and t["adjoint_block_slots"] == 256


def test_row_variant_where_the_moment_path_does_not_fit():
    """The first context finds the moment path far ahead and times no row
    variant; a context of the same shape on 600 MB, which cannot hold that
    path, times its own.  Two candidates per CTA are 1.16 to 1.2 times as fast
    there."""
    import torch
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import MZ_MIXED, Evaluator
    pot, db = _workload("meam/spline", 2, 5.5, 60, seed=6)
    X = synth.perturbed(pot.coeffs(), 64, 0.01, seed=5)
    first = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=64)
    obj = first.objective(X, MZ_MIXED)
    assert first.moment_path(MZ_MIXED, False)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (600 << 20), dtype=torch.uint8, device="cuda")
    try:
        second = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=64)
        got = second.objective(X[:8], MZ_MIXED)
        on, tuning = second.moment_path(MZ_MIXED, False), second.tuning(MZ_MIXED, False)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert on == 0
    assert np.all(np.abs(got - obj[:8]) <= 1e-6 * np.abs(got))
    assert tuning["forward_candidates_per_cta"] == 2
