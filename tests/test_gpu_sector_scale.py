"""The one-CTA sector SVD of matrices of any magnitude."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_sector_sizes import _two_sites, _update  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


@pytest.mark.parametrize("shape", [(1, 1), (3, 3), (16, 16), (17, 9), (40, 40), (30, 64), (64, 60), (12, 300)],
                         ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("power", [-520, -470, -300, -99, 99, 300, 450])
def test_power_of_two_scales_out(shape, power):
    """Sites times 2^power give singular values times 2^power, the same kept counts and
    orthonormal left vectors.  Tolerances: 64 eps sqrt(size) of the largest value, and for the
    vectors (computed from columns of relative accuracy) 64 eps size."""
    L, R = shape
    K, eps = max(40, min(L, R)), np.finfo(float).eps
    chi = max(4 * min(L, R), L, R, K)
    top, q, gl, gr, lam = _two_sites(np.random.default_rng(L * 77 + R), L, K, R, 2, spread=2.0)
    a, _, _, _ = _update("fp64", 2, top, q, gl, gr, lam, chi)
    b, g, l, _ = _update("fp64", 2, top, q, np.ldexp(1.0, power) * gl, gr, lam, chi)
    assert a["kept"] == b["kept"] and sum(a["kept"]) == 4 * min(L, R)
    at = 0
    for x, y, n in zip(a["sigma"], b["sigma"], a["kept"]):
        assert np.all(np.abs(np.ldexp(y, -power) - x) <= 64 * eps * np.sqrt(max(K, L, R)) * x[0])
        v = g[0][:L, at:at + n]
        assert np.abs(v.conj().T @ v - np.eye(n)).max() <= 64 * eps * max(K, L, R)
        at += n
