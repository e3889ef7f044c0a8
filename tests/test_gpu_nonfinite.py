"""Updates of states and gates with a NaN or an infinity: the singular values they get, and that
the handle computes the next, finite state as a new one does."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import engine, interferometer  # noqa: E402
from oracle import fock  # noqa: E402

THETA, PHI, D = 0.7, 0.4, 2


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


def _state(L, K, R, chi):
    """Every centre charge is a sector of L x R (left charges (1, 1), right ones (0, 0))."""
    rng = np.random.default_rng(L * 100 + R)
    q = np.array(sorted((int(a), int(b)) for a, b in rng.integers(0, D, size=(K, 2))))
    gamma = np.zeros((3, chi, chi), dtype=np.complex128)
    gamma[0, :L, :K] = rng.standard_normal((L, K)) + 1j * rng.standard_normal((L, K))
    gamma[1, :K, :R] = rng.standard_normal((K, R)) + 1j * rng.standard_normal((K, R))
    gamma[2, :R, 0] = 1.0
    lam = np.zeros((2, chi))
    lam[0, :K] = 1.0
    lam[1, :R] = np.sort(10.0 ** -rng.random(R))[::-1]
    charge = np.full((4, chi, 2), D, dtype=np.int32)
    charge[0, :L] = 1
    charge[1, :K] = q
    charge[2, :R] = 0
    charge[3, 0] = 0
    return gamma, lam, charge


def _update(sim, state):
    sim.load_host(*state)
    sim.bs_update(0, interferometer.t_block(THETA, PHI))
    return sim.last_update_info(), [x.cpu().numpy() for x in sim.store()]


# one CTA (up to 64 columns), tall, square and wide; the blocked form
SHAPES = [(1, 1), (4, 3), (3, 4), (16, 16), (40, 20), (20, 40), (64, 64), (60, 300), (90, 80), (80, 90)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("site", [0, 1])
def test_nan_in_a_site(shape, site):
    """No column of a matrix with a NaN is rotated: the finite columns' norms are its singular
    values, in descending order, a column with a NaN counts as -1 (and is not kept).
    Tolerance: sums of K products and of L or R squares, 8 eps each."""
    L, R = shape
    K = max(L, R)
    chi = 4 * K
    good = _state(L, K, R, chi)
    bad = [x.copy() for x in good]
    bad[0][site][(L // 2, 0) if site == 0 else (0, R // 2)] = np.nan
    with engine.MPOSimulator(3, D, chi) as sim, engine.MPOSimulator(3, D, chi) as other:
        info, _ = _update(sim, bad)
        U = fock.update_tensor(interferometer.t_block(THETA, PHI), D)
        q = bad[2][1, :K]
        assert info["shape"] == [shape] * 4
        for (c0, c1), s, n in zip(info["sectors"], info["sigma"], info["kept"]):
            w = U[1 - c0, c0, 1 - q[:, 0]] * np.conj(U[1 - c1, c1, 1 - q[:, 1]])
            T = (bad[0][0, :L, :K] * w) @ bad[0][1, :K, :R] * bad[1][1, :R]
            X = T if L >= R else T.conj().T
            norms = np.sqrt((np.abs(X) ** 2).sum(0))
            want = np.concatenate([np.sort(norms[np.isfinite(norms)])[::-1], -np.ones(np.count_nonzero(np.isnan(norms)))])
            assert np.count_nonzero(want < 0) in ((1,) if (site == 0) == (L < R) else (len(norms),))
            np.testing.assert_allclose(s, want, rtol=16 * np.finfo(float).eps * K, atol=0)
            assert n == np.count_nonzero(want > 0)
        # the same handle afterwards
        a, b = _update(sim, good), _update(other, good)
        assert a[0]["kept"] == b[0]["kept"] and sum(a[0]["kept"]) == 4 * min(L, R)
        for x, y in zip(a[1], b[1]):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("value", [np.inf, 1e200])
def test_infinities_and_overflow(shape, value):
    """An infinity, and entries whose squares overflow: nothing is asked of the values but that
    kept vectors are counted within the bond, and that the next update is right."""
    L, R = shape
    K = max(L, R)
    chi = 4 * K
    good = _state(L, K, R, chi)
    bad = [x.copy() for x in good]
    bad[0][0][L // 2, :K] = value
    with engine.MPOSimulator(3, D, chi) as sim, engine.MPOSimulator(3, D, chi) as other:
        info, _ = _update(sim, bad)
        assert all(0 <= n <= min(L, R) for n in info["kept"])
        for x, y in zip(_update(sim, good)[1], _update(other, good)[1]):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp64", "fp64-gram", "tf32x3"])
def test_nan_angle(precision):
    """A mesh with a NaN angle, then the same mesh without it on the same handle."""
    n, d, chi = 10, 4, 90
    _, bs, _ = interferometer.circuit(n, 5)
    ops = [b for b in bs if b[0] < 7]
    modes, theta, phi = [b[1] for b in ops], [b[2] for b in ops], [b[3] for b in ops]
    bad = list(theta)
    bad[len(bad) // 2] = float("nan")
    out = []
    for angles in ([bad, theta], [theta]):
        with engine.MPOSimulator(n, d, chi) as sim:
            sim.set_precision(precision)
            for th in angles:
                sim.init_single_photons(range(0, n, 2), 0.37)
                try:
                    sim.run_mesh(modes, th, phi)
                except RuntimeError:
                    assert th is bad     # an update that cannot be formed may be refused
            out.append([x.cpu().numpy() for x in sim.store()] + [sim.mesh_truncation()])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
