"""The flag that a kernel sets when it gives up a bounded wait reaches the
caller: after every replay of a captured mixed call, not the first alone, and
at an FP64 call that follows a mixed one.  The flag is set from the host
(mz_raise_device_flag); no wait runs out."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def context(monkeypatch):
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import Database, Evaluator, PotentialFile
    monkeypatch.setenv("MZ_FM", "2")  # the moment path, whose contractions wait
    spec = synth.in_range_variant(synth.teacher_potential("meam/spline", 1, 4.5, seed=2))
    pot = PotentialFile.from_spec(spec)
    rng = np.random.default_rng(6)
    cells = synth.make_cells(6, lambda r: 32, rng)
    ev = Evaluator(Database.from_cells(cells, pot), pot, 1.0, 1.0, 0, max_candidates=8)
    return ev, synth.perturbed(pot.coeffs(), 8, 0.01, seed=5)


def _raise(ev):
    from meamzilla_b200._lib import check, lib
    check(lib().mz_raise_device_flag(ev._h))


def test_flag_after_replays(context):
    import torch
    from meamzilla_b200._lib import MzError, check, lib
    from meamzilla_b200.potential import MZ_MIXED
    ev, X = context
    x = torch.tensor(X, device="cuda")
    obj = torch.empty(8, dtype=torch.float64, device="cuda")
    ev.objective_device(x, obj, MZ_MIXED)  # picks the variant
    ev.sync()
    assert ev.moment_path(MZ_MIXED, grad=False) >= 2
    first = obj.clone()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(ev.stream())):
        check(lib().mz_objective_device(ev._h, 8, C.c_void_p(x.data_ptr()), MZ_MIXED, C.c_void_p(obj.data_ptr()),
                                        None, None))
    for replay in range(3):
        obj.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        ev.sync()
        assert torch.equal(obj, first)
    for replay in range(2):
        graph.replay()
        torch.cuda.synchronize()
        _raise(ev)
        with pytest.raises(MzError, match="timed out"):
            ev.sync()
        ev.sync()  # cleared


def test_flag_at_a_following_fp64_call(context):
    import torch
    from meamzilla_b200._lib import MzError
    from meamzilla_b200.potential import MZ_FP64, MZ_MIXED
    ev, X = context
    value = ev.objective(X, MZ_FP64)
    for k in range(2):
        x = torch.tensor(X, device="cuda")
        obj = torch.empty(8, dtype=torch.float64, device="cuda")
        ev.objective_device(x, obj, MZ_MIXED)
        _raise(ev)
        with pytest.raises(MzError, match="timed out"):
            ev.objective(X, MZ_FP64)
        assert np.array_equal(ev.objective(X, MZ_FP64), value)
        _raise(ev)
        with pytest.raises(MzError, match="timed out"):
            ev.objective(X, MZ_MIXED)
        ev.objective(X, MZ_MIXED)
