"""The single-sector contraction with centre entries in any order."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import _capi  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


def _contract(d, cc, u, glc, gcr, cl, q, cr):
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (u, glc, gcr, cl, q, cr)]
    out = torch.full((glc.shape[0], gcr.shape[1]), complex("nan"), dtype=torch.complex128, device="cuda")
    p = [ctypes.c_void_p(x.data_ptr()) for x in dev]
    _capi.check(_capi.lib().bsmpo_contract_sector(d, cc[0], cc[1], p[0], p[1], p[2], p[3], p[4], p[5], glc.shape[0],
                                                  glc.shape[1], gcr.shape[1], ctypes.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


# below and above d^2 + 1 runs, windows of 1,024 entries and a last one of a few; every d; charges
# past the cutoff, which no term uses
@pytest.mark.parametrize("d", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("size", [(1, 3, 1), (33, 20, 17), (40, 70, 40), (31, 1023, 15), (64, 1100, 33), (5, 2100, 50)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("order", ["sorted", "random", "alternating"])
def test_any_order(d, size, order):
    """Against the element-wise sum; len_c products of magnitude at most max|Glc| max|Gcr| max|u|^2,
    8 eps each."""
    L, K, R = size
    rng = np.random.default_rng(d * 100 + L + K)
    glc = rng.standard_normal((L, K)) + 1j * rng.standard_normal((L, K))
    gcr = rng.standard_normal((K, R)) + 1j * rng.standard_normal((K, R))
    u = rng.standard_normal((d, d, d)) + 1j * rng.standard_normal((d, d, d))
    cl, cr = (rng.integers(0, d + 1, size=(n, 2)).astype(np.int32) for n in (L, R))
    q = rng.integers(0, d + 1, size=(K, 2)).astype(np.int32)
    if order == "sorted":
        q = np.array(sorted(map(tuple, q.tolist())), dtype=np.int32)
    elif order == "alternating":
        q = q[np.arange(K) % 2]
    cc = (d // 2, (d - 1) // 2)
    got = _contract(d, cc, u, glc, gcr, cl, q, cr)
    want = np.zeros((L, R), dtype=complex)
    rows = (cl < d).all(1) & (cl >= cc).all(1)
    cols = (cr < d).all(1) & (cr <= cc).all(1)
    for r in np.flatnonzero(cols):
        b = cr[r]
        for l in np.flatnonzero(rows):
            a = cl[l]
            ok = (q < d).all(1) & (q <= a).all(1) & (q >= b).all(1)
            w = u[a[0] - cc[0], cc[0] - b[0], a[0] - q[ok, 0]] * u[a[1] - cc[1], cc[1] - b[1], a[1] - q[ok, 1]].conj()
            want[l, r] = (w * glc[l, ok] * gcr[ok, r]).sum()
    tol = 8 * np.finfo(float).eps * K * np.abs(glc).max() * np.abs(gcr).max() * max(np.abs(u).max(), 1.0) ** 2
    assert np.abs(got - want).max() <= tol
