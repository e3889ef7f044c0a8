"""The left vectors and the new sites of single updates on the plain and the preconditioned path."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import interferometer  # noqa: E402
from oracle import fock  # noqa: E402
from test_gpu_sector_sizes import ONE_CTA, PHI, THETA, _two_sites, _update  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


def _check(shape, chi, spread, all_kept):
    """Per sector, with T = C diag(lam) and its values s: V^H V = 1 whatever s is (pair tests
    relative to the columns' norms): 4 eps sqrt(rows) k; W = V^H C, so the rows of W diag(lam) have
    norm s and, where every vector is kept, V W diag(lam) = T: products of length rows and K on
    matrices of norm s[0], 16 eps (sqrt(rows) + sqrt(K)) k of s[0]."""
    L, R = shape
    d, k, eps = 2, min(shape), np.finfo(float).eps
    K = max(40, k)
    top, q, gl, gr, lam = _two_sites(np.random.default_rng(L * 3000 + R), L, K, R, d, spread=spread)
    info, g, _, _ = _update("fp64", d, top, q, gl, gr, lam, max(chi, L, R, K))
    U = fock.update_tensor(interferometer.t_block(THETA, PHI), d)
    a, at, kept = np.array(q), 0, sum(info["kept"])
    assert kept == 4 * k if all_kept else 0 < kept <= chi
    for (c0, c1), s, n in zip(info["sectors"], info["sigma"], info["kept"]):
        w = U[top - c0, c0, top - a[:, 0]] * np.conj(U[top - c1, c1, top - a[:, 1]])
        T = (gl * w) @ gr * lam
        v, x = g[0][:L, at:at + n], g[1][at:at + n, :R] * lam
        tol = 16 * eps * (np.sqrt(max(shape)) + np.sqrt(K)) * k * s[0]
        assert np.abs(v.conj().T @ v - np.eye(n)).max(initial=0.0) <= 4 * eps * np.sqrt(max(shape)) * k + 4 * eps
        assert np.abs(np.linalg.norm(x, axis=1) - s[:n]).max(initial=0.0) <= tol
        left = T - v @ x
        assert np.linalg.norm(left, 2) <= tol + (0.0 if n == k else s[n])
        at += n


@pytest.mark.parametrize("shape", ONE_CTA, ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("spread", [1.0, 8.0])
def test_one_cta(shape, spread):
    _check(shape, 4 * min(shape), spread, all_kept=True)


@pytest.mark.parametrize("shape", [(66, 66), (70, 100), (100, 70), (150, 160), (180, 150)], ids=lambda s: "%dx%d" % s)
def test_blocked(shape):
    _check(shape, 4 * min(shape), 6.0, all_kept=True)


@pytest.mark.parametrize("shape", [(66, 66), (70, 100), (100, 70), (150, 160), (180, 150), (440, 450), (470, 435)],
                         ids=lambda s: "%dx%d" % s)
def test_preconditioned(shape):
    _check(shape, 2 * min(shape), 2.0, all_kept=False)
