"""Contexts of one process do not change each other's launches: a kernel's
shared-memory limit belongs to the kernel on the device, and a context of a
smaller potential must not lower it, neither by being made later nor by
launching from another thread at the same time."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _evaluator(style, ntypes, nr, ng, ncells, n=1):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import Database, Evaluator, PotentialFile
    spec = synth.in_range_variant(synth.teacher_potential(style, ntypes, 4.3, seed=2))
    for i, group in enumerate(spec.groups):
        for s in group:
            x = np.linspace(s.left, s.right, ng if i in (4, 6, 8) else nr)
            s.y = np.interp(x, np.linspace(s.left, s.right, s.nknots), s.y)
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    cells = synth.make_cells(ncells, lambda r: 40, rng, ntypes=ntypes)
    for c in cells:
        c.force0 = rng.normal(0, 0.3, c.force0.shape)
    ev = Evaluator(Database.from_cells(cells, pot), pot, 1.0, 1.0, 0, max_candidates=n)
    return ev, synth.perturbed(pot.coeffs(), n, 0.01, seed=5)


def test_a_later_smaller_context():
    """Eight species: the knot table and its gradient take 68 KB of 40 knots, 52 of 30."""
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED
    big, xb = _evaluator("eam/spline", 8, 40, 8, 3)
    first = big.objective_grad(xb, MZ_MIXED), big.objective(xb, MZ_FP64)
    small, xs = _evaluator("eam/spline", 8, 30, 8, 3)
    small.objective_grad(xs, MZ_MIXED)
    again, xb = _evaluator("eam/spline", 8, 40, 8, 3)
    small2, _ = _evaluator("eam/spline", 8, 30, 8, 3)
    for ev in (big, again):  # `again` has launched nothing yet
        assert np.array_equal(ev.objective(xb, MZ_FP64), first[1])
        obj, grad = ev.objective_grad(xb, MZ_MIXED)
        assert np.allclose(obj, first[0][0], rtol=1e-6)
        assert np.max(np.abs(grad - first[0][1])) <= 1e-5 * np.max(np.abs(grad))


def test_threads_with_contexts_of_their_own():
    import torch
    from meamzilla_b200._lib import lib
    from meamzilla_b200.potential import MZ_FP64
    work = []
    for ng in (6, 15):
        ev, X = _evaluator("meam/spline", 1, 10, ng, 3)
        x = torch.tensor(X, device="cuda")
        obj, grad = torch.zeros(1, dtype=torch.float64, device="cuda"), torch.zeros(x.shape, dtype=torch.float64, device="cuda")
        ev.objective_grad_device(x, obj, grad, MZ_FP64)
        ev.sync()
        work.append((ev, x, obj, grad, obj.clone(), grad.clone()))
    errors = []
    start = threading.Barrier(len(work))

    def loop(ev, x, obj, grad, *_):
        start.wait()
        for k in range(3000):
            st = lib().mz_objective_grad_device(ev._h, 1, C.c_void_p(x.data_ptr()), MZ_FP64, C.c_void_p(obj.data_ptr()),
                                                C.c_void_p(grad.data_ptr()))
            if st != 0:
                errors.append((k, lib().mz_last_error().decode()))
                return
            if k % 100 == 0:
                ev.sync()
        ev.sync()

    threads = [threading.Thread(target=loop, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for ev, x, obj, grad, o, g in work:
        assert torch.equal(obj, o) and torch.equal(grad, g)


def test_an_error_left_by_another_call():
    """The CUDA runtime keeps a failed call's code until somebody asks for it:
    an entry point does not take one that was there before it as its own."""
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    ev, X = _evaluator("eam/spline", 1, 10, 8, 2)
    value = ev.objective(X, MZ_FP64)
    cudart = C.CDLL("libcudart.so.12")
    assert cudart.cudaSetDevice(99) != 0
    other = Evaluator(ev.db, ev.pot, 1.0, 1.0, 0, max_candidates=1)
    assert np.array_equal(other.objective(X, MZ_FP64), value)
    assert cudart.cudaSetDevice(99) != 0
    assert np.array_equal(ev.objective(X, MZ_FP64), value)


def test_first_call_right_after_creation():
    """What a context is made of is there when its first kernels run: sixty
    contexts of small arrays, each evaluated at once, give one value."""
    from meamzilla_b200.potential import MZ_FP64, Evaluator
    ev, X = _evaluator("meam/spline", 2, 10, 8, 2)
    obj, grad = ev.objective_grad(X, MZ_FP64)
    for _ in range(60):
        other = Evaluator(ev.db, ev.pot, 1.0, 1.0, 0, max_candidates=1)
        o, g = other.objective_grad(X, MZ_FP64)
        assert np.array_equal(o, obj) and np.array_equal(g, grad)
