"""Products whose launch overlaps the end of the one before it in the stream: a chain of A x and
A'y through two buffers, each product reading what the one before wrote and overwriting what it
read, equals the chain with a synchronisation after every product, bit for bit. The sizes are
grids of a few blocks, of either side of 2 x 148 and of all resident blocks, with long rows too."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,m,n,per_col", [("uniform", 40, 70, 3), ("uniform", 2000, 5000, 5), ("uniform", 14000, 60000, 9),
                                              ("uniform", 60000, 14000, 40), ("uniform", 50021, 100003, 10),
                                              ("powerlaw", 30000, 60000, 10)])
def test_chain_without_waits_equals_chain_with(engine, instances, kind, m, n, per_col):
    inst = (instances.lp_uniform(5, m, n, per_col) if kind == "uniform" else instances.lp_powerlaw(5, m, n, per_col * n))
    A = engine.Matrix.from_instance(inst)
    L = engine.lib()
    start = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    ends = []
    for wait in (True, False):
        x, y = start.clone(), torch.zeros(m, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(30):
            assert L.sankhya_cuda_spmv_device_f64(A.handle, x.data_ptr(), y.data_ptr()) == 0
            if wait:
                torch.cuda.synchronize()
            assert L.sankhya_cuda_spmv_transpose_device_f64(A.handle, y.data_ptr(), x.data_ptr()) == 0
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        ends.append((x.cpu(), y.cpu()))
    assert torch.isfinite(ends[0][0]).all()
    assert torch.equal(ends[0][0], ends[1][0]) and torch.equal(ends[0][1], ends[1][1])
