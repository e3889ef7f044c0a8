"""Relative accuracy of small singular values that an update keeps (default precision)."""
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


def _values(A):
    """Singular values by one-sided Jacobi (circle order) in extended precision."""
    A = A if A.shape[0] >= A.shape[1] else A.conj().T
    A = A[:, np.argsort(-(np.abs(A) ** 2).sum(0).astype(float))]
    A = np.concatenate([A, np.zeros((A.shape[0], A.shape[1] & 1), A.dtype)], 1)
    n = A.shape[1]
    at = list(range(n))
    for _ in range(40):
        worst = 0.0
        for _ in range(n - 1):
            p, q = np.array(at[:n // 2]), np.array(at[:n // 2 - 1:-1])
            X, Y = A[:, p], A[:, q]
            a, b = (np.abs(X) ** 2).sum(0), (np.abs(Y) ** 2).sum(0)
            g = (X.conj() * Y).sum(0)
            size, limit = np.abs(g), np.sqrt(a * b)
            worst = max(worst, float((size / np.where(limit > 0, limit, 1)).max()))
            turn = size > 1e-18 * limit
            zeta = (b - a) / np.where(turn, 2 * size, 1)
            t = np.where(turn, np.where(zeta >= 0, 1, -1) / (np.abs(zeta) + np.sqrt(1 + zeta ** 2)), 0)
            c = 1 / np.sqrt(1 + t * t)
            w = c * t * np.where(turn, g / np.where(turn, size, 1), 1)
            A[:, p], A[:, q] = X * c - Y * w.conj(), X * w + Y * c
            at = [at[0], at[-1]] + at[1:-1]
        if worst < 1e-17:
            break
    return np.sort(np.sqrt((np.abs(A) ** 2).sum(0)))[::-1]


# rows, columns, rank, decades over which the right Lambda spreads, chi: candidates 4 min(rows,
# columns) above chi; kept fewer than chi (the rank's 4 times), or cut by chi far down, or near
# the top (where the blocked form starts from a preconditioned matrix)
@pytest.mark.parametrize("L,R,K,decades,chi", [(120, 100, 90, 8, 380), (100, 120, 90, 8, 380),
                                               (120, 100, 90, 7, 340), (100, 120, 90, 7, 340), (100, 90, 120, 3, 200),
                                               (90, 100, 120, 3, 200), (110, 66, 120, 9, 260)])
def test_kept_values(L, R, K, decades, chi):
    """T = C diag(lam): columns of C rounded relative to themselves, and Jacobi rotations that
    keep that, move a singular value by eps kappa(C) at most, relatively (kappa over the rank);
    64 of them for the products of length K and the rotations."""
    d, eps = 2, np.finfo(float).eps
    top, q, gl, gr, lam = _two_sites(np.random.default_rng(L * 10 + R), L, K, R, d, spread=float(decades))
    info, _, _, _ = _update("fp64", d, top, q, gl, gr, lam, max(chi, L, R, K))
    U = fock.update_tensor(interferometer.t_block(THETA, PHI), d).astype(np.clongdouble)
    a = np.array(q)
    i = info["sectors"].index((1, 0))
    w = U[top - 1, 1, top - a[:, 0]] * np.conj(U[top, 0, top - a[:, 1]])
    C = (gl.astype(np.clongdouble) * w) @ gr.astype(np.clongdouble)
    n = info["kept"][i]
    want = _values(C * lam.astype(np.longdouble))[:n]
    s = np.linalg.svd(C.astype(complex), compute_uv=False)
    kappa = float(s[0] / s[min(K, L, R) - 1])
    assert 0 < n <= min(K, L, R)
    assert np.max(np.abs(info["sigma"][i][:n] - want) / want) <= 64 * eps * kappa


@pytest.mark.parametrize("k,size", [(66, 90), (100, 100), (150, 70), (200, 240)])
@pytest.mark.parametrize("near", [0.0, 1e-9, 0.3])
def test_nearly_equal_values(k, size, near):
    """Sectors whose columns are orthogonal or nearly so: all values the same, or within `near`.
    Singular values within 64 eps sqrt(size) of the largest, kept vectors orthonormal."""
    d, L, R, eps = 2, k, size, np.finfo(float).eps
    n = min(L, R)
    rng = np.random.default_rng(k + size)
    gl = np.linalg.qr(rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L)))[0][:, :n]
    gr = (np.linalg.qr(rng.standard_normal((R, R)) + 1j * rng.standard_normal((R, R)))[0][:n] *
          (1 + near * rng.random(n))[:, None])
    q = [(0, 0)] * n
    chi = 2 * n
    info, g, _, _ = _update("fp64", d, d - 1, q, gl, gr, np.ones(R), max(chi, L, R))
    U = fock.update_tensor(interferometer.t_block(THETA, PHI), d)
    at = 0
    for (c0, c1), s, m in zip(info["sectors"], info["sigma"], info["kept"]):
        T = gl @ gr * (U[1 - c0, c0, 1] * np.conj(U[1 - c1, c1, 1]))
        want = np.linalg.svd(T, compute_uv=False)
        assert np.abs(s - want).max() <= 64 * eps * np.sqrt(max(L, R)) * want[0]
        v = g[0][:L, at:at + m]
        assert np.abs(v.conj().T @ v - np.eye(m)).max(initial=0.0) <= 4 * eps * np.sqrt(max(L, R)) * n
        at += m
