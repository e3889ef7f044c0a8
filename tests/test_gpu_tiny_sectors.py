"""Rounding of the smallest sectors' singular values."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import interferometer  # noqa: E402
from oracle import fock  # noqa: E402
from test_gpu_sector_sizes import PHI, THETA, _two_sites, _update  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


def _values(T):
    """Singular values of one or two columns in extended precision."""
    if T.shape[0] < T.shape[1]:
        T = T.conj().T
    G = T.conj().T @ T
    if T.shape[1] == 1:
        return np.sqrt(G[0].real)
    mean, half = (G[0, 0] + G[1, 1]).real / 2, (G[0, 0] - G[1, 1]).real / 2
    big = mean + np.sqrt(half ** 2 + np.abs(G[0, 1]) ** 2)
    det = (G[0, 0] * G[1, 1] - G[0, 1] * G[1, 0]).real
    return np.sqrt(np.array([big, det / big]))


@pytest.mark.parametrize("shape", [(1, 1), (8, 1), (1, 8), (2, 2), (10, 2)], ids=lambda s: "%dx%d" % s)
def test_one_and_two_columns(shape):
    """Mean error over 96 sectors, relative to the sector's norm.  Three complex products to an
    entry and its scaling (u = eps / 2 each, uniformly distributed: about 1.1 u rms), the sum of
    squares and the root (0.6 u): 1.25 u rms, and the mean magnitude is below that.  Reflectors
    applied on the way would add about 1 u each."""
    L, R = shape
    d, K, u = 2, max(shape), np.finfo(float).eps / 2
    U = fock.update_tensor(interferometer.t_block(THETA, PHI), d).astype(np.clongdouble)
    errors = []
    for seed in range(24):
        top, q, gl, gr, lam = _two_sites(np.random.default_rng(7000 + seed), L, K, R, d, spread=1.0)
        info, _, _, _ = _update("fp64", d, top, q, gl, gr, lam, 4 * K)
        a = np.array(q)
        for (c0, c1), s in zip(info["sectors"], info["sigma"]):
            w = U[top - c0, c0, top - a[:, 0]] * np.conj(U[top - c1, c1, top - a[:, 1]])
            want = _values((gl.astype(np.clongdouble) * w) @ gr.astype(np.clongdouble) * lam.astype(np.longdouble))
            errors.append(float(np.sqrt(np.sum((s - want) ** 2) / np.sum(want ** 2))))
    assert len(errors) == 96 and np.mean(errors) <= 1.25 * u
