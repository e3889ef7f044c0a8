"""After a mesh, the last-update queries describe the mesh's last update, in whatever order its
groups ran."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import engine, interferometer  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


def _last(n, d, chi, precision, layers, workers):
    _, bs, _ = interferometer.circuit(n, 31)
    ops = [b for b in bs if b[0] < layers]
    with engine.MPOSimulator(n, d, chi) as sim:
        sim.set_precision(precision)
        sim.set_workers(workers)
        sim.init_single_photons(range(0, n, 2), 0.37)
        sim.run_mesh([b[1] for b in ops], [b[2] for b in ops], [b[3] for b in ops])
        return sim.last_update_info(), sim.last_update_work()


# the ends of the chain hold few candidates and the centre more than chi, so a layer's updates
# take two SVD routes; a mesh that ends with a layer of either parity
@pytest.mark.parametrize("precision", ["fp64", "fp64-gram"])
@pytest.mark.parametrize("n,d,chi", [(14, 4, 40), (20, 3, 24)])
@pytest.mark.parametrize("layers", [7, 8])
@pytest.mark.parametrize("workers", [2, 8, 32])
def test_last_update_of_a_mesh(n, d, chi, precision, layers, workers):
    """The same answers as with the updates one by one (which compute the same bits)."""
    want, work = _last(n, d, chi, precision, layers, 1)
    got, got_work = _last(n, d, chi, precision, layers, workers)
    assert got["sectors"] == want["sectors"] and got["shape"] == want["shape"] and got["kept"] == want["kept"]
    assert got["trunc_weight"] == want["trunc_weight"]
    for a, b in zip(got["sigma"], want["sigma"]):
        assert np.array_equal(a, b)
    assert got_work["gemm_flops"] == work["gemm_flops"] and got_work["min_bytes"] == work["min_bytes"]
