"""Device calls inside a caller's capture of the context's stream, as the very
first call of their kind: nothing is timed, allocated or waited for there, the
replays give the values of an uncaptured call (to rounding; the capture runs
the variants that need no preparation), and a later uncaptured call makes its
own choice."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _evaluator(style, ntypes, n):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import Database, Evaluator, PotentialFile
    spec = synth.in_range_variant(synth.teacher_potential(style, ntypes, 4.3, seed=2))
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    cells = synth.make_cells(7, lambda r: 30 + int(r.integers(5)), rng, ntypes=ntypes)
    for c in cells:
        c.force0 = rng.normal(0, 0.3, c.force0.shape)
    # a database of its own size: no other test's tuning choice serves it
    ev = Evaluator(Database.from_cells(cells, pot), pot, 1.0, 1.0, 0, max_candidates=n)
    return ev, synth.perturbed(pot.coeffs(), n, 0.01, seed=5)


def _capture(ev, x, obj, grad, precision):
    import torch
    from meamzilla_b200._lib import check, lib
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(ev.stream())):
        p = C.c_void_p(x.data_ptr()), int(precision), C.c_void_p(obj.data_ptr())
        if grad is None:
            check(lib().mz_objective_device(ev._h, len(x), *p, None, None))
        else:
            check(lib().mz_objective_grad_device(ev._h, len(x), *p, C.c_void_p(grad.data_ptr())))
    return graph


# tolerances: FP64 sums of some 1e4 terms in another order (the parity tests'
# 1e-12 and 1e-10); mixed: two paths of FP32 slot terms, 1e-5 of the gradient
@pytest.mark.parametrize("style,ntypes,mixed", [("eam/spline", 1, False), ("meam/spline", 1, False),
                                                ("gmeam/spline", 2, False), ("jmeam/spline", 1, False),
                                                ("meam/spline", 2, True), ("eam/spline", 2, True)])
@pytest.mark.parametrize("gradient", [False, True])
def test_first_call_captured(style, ntypes, mixed, gradient):
    import torch
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED
    precision = MZ_MIXED if mixed else MZ_FP64
    n = 3
    ev, X = _evaluator(style, ntypes, n)
    x = torch.tensor(X, device="cuda")
    obj = torch.zeros(n, dtype=torch.float64, device="cuda")
    grad = torch.zeros((n, ev.ncoeff), dtype=torch.float64, device="cuda") if gradient else None
    graph = _capture(ev, x, obj, grad, precision)
    got = []
    for replay in range(2):
        obj.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        ev.sync()
        got.append([obj.clone()] + ([grad.clone()] if gradient else []))
    for k in range(2):  # uncaptured: tunes, prepares
        if gradient:
            ev.objective_grad_device(x, obj, grad, precision)
        else:
            ev.objective_device(x, obj, precision)
        ev.sync()
    rtol, gtol = (1e-6, 1e-5) if mixed else (1e-12, 1e-10)
    for g in got:
        assert torch.all((g[0] - obj).abs() <= rtol * obj.abs())
        if gradient:
            assert torch.all((g[1] - grad).abs() <= gtol * grad.abs().amax(dim=1, keepdim=True))
    assert ev.tuning(precision, gradient)["forward_block_slots"] > 0
    # and a capture after it gives exactly the uncaptured call's values (mixed sums' order is not fixed)
    ref = [obj.clone()] + ([grad.clone()] if gradient else [])
    graph = _capture(ev, x, obj, grad, precision)
    obj.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    ev.sync()
    if not mixed:
        assert torch.equal(obj, ref[0]) and (not gradient or torch.equal(grad, ref[1]))
    graph.reset()
