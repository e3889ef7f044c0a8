"""Workspaces of an update."""
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


def test_only_preconditioned_sectors_take_eigenvector_space():
    """Two sectors of 1,080 x 1,000 (preconditioned) and two of 1,080 x 1,160, beyond the eigenvector
    kernels' largest.  Bytes held: what the sectors need, each buffer rounded up to a power of two."""
    d, L, K = 2, 1080, 30
    R = 1160
    chi = R
    rng = np.random.default_rng(0)
    gamma = np.zeros((3, chi, chi), dtype=np.complex128)
    gamma[0, :L, :K] = rng.standard_normal((L, K))
    gamma[1, :K, :R] = rng.standard_normal((K, R))
    gamma[2, :R, 0] = 1.0
    lam = np.zeros((2, chi))
    lam[0, :K] = 1.0
    lam[1, :R] = 1.0
    charge = np.full((4, chi, 2), d, dtype=np.int32)
    charge[0, :L] = 1
    charge[1, :K] = 0
    charge[2, :1000] = 0
    charge[2, 1000:R] = (0, 1)
    charge[3, 0] = 0
    with engine.MPOSimulator(3, d, chi) as sim:
        sim.load_host(gamma, lam, charge)
        sim.bs_update(0, interferometer.t_block(0.7, 0.4))
        info, held = sim.last_update_info(), sim.workspace_stats()
    shapes = [(1080, 1000), (1080, 1160)]
    assert sorted(info["shape"]) == sorted(shapes * 2)

    def room(n):
        return 1 << int(np.ceil(np.log2(n + 256)))

    m, n, w = 1080, 1000, 1160
    need = [16 * m * R,                                        # Theta
            16 * 2 * (m * n + m * w),                          # C
            16 * 2 * (2 * m * n + (m + w) * m),                # Jacobi matrices
            16 * 2 * (n * n + m * w), 16 * 2 * (m * n + m * m),  # W, V
            16 * 2 * n * n, 16 * 2 * n * n, 8 * 2 * n * n, 32 * 2 * n * n, 2 * n * n]   # of the 1,000 alone
    rounds = 80 << 20     # the blocked rounds' Grams, tables and vectors
    assert held[2] <= sum(room(x) for x in need) + rounds
