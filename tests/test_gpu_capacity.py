"""How many candidates a launch holds when device memory binds: what the
packed pair forces (24 bytes a slot and candidate) allow, not the 32-byte
records' three quarters of it; and such launches give the values of a context
with records, bit for bit in FP64.  Memory is made short by a tensor that
leaves 12 GB."""
import ctypes as C
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def short_memory():
    """Fills device memory up to 12 GB; freed again whatever the test does."""
    import torch
    held = []

    def fill():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held.append(torch.empty(max(1, torch.cuda.mem_get_info()[0] - (12 << 30)), dtype=torch.uint8, device="cuda"))

    def free():
        held.clear()
        torch.cuda.empty_cache()

    yield fill, free
    free()


@pytest.mark.parametrize("style", ["eam/spline", "meam/spline"])
def test_candidates_per_launch_when_memory_binds(style, short_memory):
    import torch
    from meamzilla_b200 import synth
    from meamzilla_b200._lib import check, lib
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED, Database, Evaluator, PotentialFile
    meam = style == "meam/spline"
    spec = synth.in_range_variant(synth.teacher_potential(style, 1, 5.5, seed=2))
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    grid = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    frac = ((grid + np.array([[0, 0, 0], [.5, .5, .5]])) / 3).reshape(-1, 3)
    cells = [synth.Cell(lattice=np.eye(3) * 9.6, types=np.zeros(54, dtype=int), pos=frac * 9.6 + rng.normal(0, 0.08, (54, 3)),
                        force0=rng.normal(0, 0.3, (54, 3)), energy0=-1.0, stress0=np.zeros(6))
             for _ in range(400 if meam else 1600)]
    db = Database.from_cells(cells, pot, device=0)
    stats = db.stats()
    fill, unfill = short_memory
    fill()
    free = torch.cuda.mem_get_info()[0]
    ev = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=100000)
    one = torch.zeros(1, dtype=torch.float64, device="cuda")
    p = C.c_void_p(one.data_ptr())
    assert lib().mz_objective_device(ev._h, 100000, p, MZ_FP64, p, None, None) != 0
    holds = int(re.search(r"\((\d+)\)", lib().mz_last_error().decode()).group(1))
    # one candidate: V, the adjoint's five sums a slot (meam), 19 numbers an
    # atom, the residuals, 17 a cell; tables for at most 8 CTAs of 8 warps an SM
    table = sum(2 * s.nknots + 2 for g in spec.groups for s in g)
    per = 8 * ((3 + (5 if meam else 0)) * stats["npairs"] + 19 * stats["natoms"] + ev.esize + 17 * stats["ncells"]
               + table * (2048 + 9 * 148 * 8))
    fixed = 180 * stats["npairs"]  # the database's own arrays
    assert holds >= 0.97 * (0.6 * (free - fixed)) / per
    n = holds
    X = synth.perturbed(pot.coeffs(), n, 0.01, seed=5)
    x = torch.tensor(X, device="cuda")
    obj = torch.empty(n, dtype=torch.float64, device="cuda")
    E = torch.empty((n, ev.esize), dtype=torch.float64, device="cuda")
    ev.objective_device(x, obj, MZ_FP64, errvec=E)
    ev.sync()
    mixed = torch.empty(n, dtype=torch.float64, device="cuda")
    ev.objective_device(x, mixed, MZ_MIXED)
    ev.sync()
    grad = torch.empty((n, ev.ncoeff), dtype=torch.float64, device="cuda")
    ev.objective_grad_device(x, obj, grad, MZ_FP64)
    ev.sync()
    obj, E, grad, mixed = (t.cpu().numpy() for t in (obj, E, grad, mixed))
    del ev, x, one
    unfill()
    ref = Evaluator(db, pot, 1.0, 1.0, 0, max_candidates=2)
    for c in (0, n // 2, n - 1):
        r = ref.objective(X[c:c + 1], MZ_FP64, errvec=True)
        assert obj[c] == r["obj"][0] and np.array_equal(E[c], r["errvec"][0])
        g = ref.objective_grad(X[c:c + 1], MZ_FP64)[1][0]
        assert np.max(np.abs(grad[c] - g)) <= 1e-10 * np.max(np.abs(g))
        assert abs(mixed[c] - obj[c]) <= 1e-5 * abs(obj[c])
