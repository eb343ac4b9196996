"""The server's admission unit covers the device memory that a solve takes,
tables of the order and workspaces included."""
import pytest

from aran_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("maxbox", [20, 64])
@pytest.mark.parametrize("precision,order", [("mixed", 4), ("mixed", 10), ("mixed", 12), ("mixed", 16),
                                             ("fp64", 8), ("fp64", 18), ("fp64", 26), ("fp64", 30)])
def test_covers_a_solve(aran, precision, order, maxbox):
    import torch
    torch.zeros(1, device="cuda")
    for n in (1000, 20_000, 100_000):
        for gen, lb in ((W.uniform, 0.0), (W.plummer, -1.0)):
            x, q = gen(n, 1)
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            with aran.Solver3d([lb] * 3, [1.0] * 3, maxbox=maxbox, order=order,
                               precision=precision) as s:
                s.solve(x, q)
                taken = free - torch.cuda.mem_get_info()[0]
            need = aran.footprint_bytes(n, maxbox=maxbox, order=order, precision=precision)
            assert taken <= need, (n, gen.__name__, taken, need)
