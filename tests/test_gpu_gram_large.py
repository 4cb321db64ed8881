"""mz_gram_device at the row counts where the number of k ranges changes: tiles
about as many as multiprocessors, half as many, more, and few (one thread or
one warp per output adds the ranges).  Against FP64 products, 1e-13 of
sum_k |a_k b_k| as for the smaller shapes; and no shape leaves half of the
multiprocessors idle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ev():
    from meamzilla_b200 import synth
    from meamzilla_b200.potential import Database, Evaluator, PotentialFile
    spec, cells = synth.make_workload("eam54", seed=3, ncells=2)
    pot = PotentialFile.from_spec(spec)
    return Evaluator(Database.from_cells(cells, pot), pot, 1.0, 1.0, 0)


@pytest.mark.parametrize("na,nb,n", [(65, 65, 5000), (136, 136, 1000), (321, 321, 2111), (640, 640, 1500), (760, 760, 1501),
                                     (1057, 1057, 700), (1200, 1200, 333), (700, 300, 1000), (1100, 65, 640), (64, 64, 31)])
def test_products(ev, na, nb, n):
    import torch
    g = torch.Generator(device="cuda").manual_seed(na + n)
    A = torch.randn((na, n), generator=g, dtype=torch.float64, device="cuda")
    B = A if na == nb else torch.randn((nb, n), generator=g, dtype=torch.float64, device="cuda")
    out = torch.empty((na, nb), dtype=torch.float64, device="cuda")
    ev.gram_device(A, B, out)
    ev.sync()
    first = out.clone()
    assert torch.all((out - A @ B.T).abs() <= 1e-13 * (A.abs() @ B.abs().T))
    if A is B:
        assert torch.equal(out, out.T)
    ev.gram_device(A, B, out)
    ev.sync()
    assert torch.equal(out, first)


def test_time_follows_the_work(ev):
    """760 rows are 1.17 times the products of 704 (12 and 11 tiles a side).  With
    one range a tile they took 1.95 times as long, on half of the
    multiprocessors; 1.5 lies well between."""
    import torch
    st = torch.cuda.ExternalStream(ev.stream())

    def time(n):
        A = torch.randn((n, 65000), dtype=torch.float64, device="cuda")
        out = torch.empty((n, n), dtype=torch.float64, device="cuda")
        ev.gram_device(A, A, out)
        ev.sync()
        ms = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(st)
            ev.gram_device(A, A, out)
            b.record(st)
            b.synchronize()
            ms.append(a.elapsed_time(b))
        return float(np.median(ms))

    assert time(760) < 1.5 * time(704)
