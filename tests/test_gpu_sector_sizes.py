"""The sector SVD at the sizes where its paths change: single updates whose four sectors all
have a chosen shape, against numpy's SVD of the same matrices, and the invariances of groups."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import cuda_kernels, engine, interferometer  # noqa: E402
from oracle import fock, mpo as om  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


THETA, PHI = 0.7, 0.4


def _two_sites(rng, L, K, R, d, rank=None, spread=3.0):
    """Two sites whose left bond carries L entries of charge (d-1, d-1), the right one R of
    (0, 0) and the centre K of random charges: every centre charge is a sector of L x R."""
    top = d - 1
    q = sorted((int(a), int(b)) for a, b in rng.integers(0, d, size=(K, 2)))
    gl = (rng.standard_normal((L, K)) + 1j * rng.standard_normal((L, K))) / np.sqrt(K)
    gr = (rng.standard_normal((K, R)) + 1j * rng.standard_normal((K, R))) / np.sqrt(K)
    if rank is not None:
        gl[:, rank:] = 0.0
    lam = np.sort(10.0 ** (-spread * rng.random(R)))[::-1]
    return top, q, gl, gr, lam


def _expected(d, top, q, gl, gr, lam):
    U = fock.update_tensor(interferometer.t_block(THETA, PHI), d)
    out = {}
    qa = np.array(q)
    for c0 in range(d):
        for c1 in range(d):
            w = U[top - c0, c0, top - qa[:, 0]] * np.conj(U[top - c1, c1, top - qa[:, 1]])
            out[(c0, c1)] = np.linalg.svd((gl * w[None, :]) @ gr * lam[None, :], compute_uv=False)
    return out


def _update(precision, d, top, q, gl, gr, lam, chi):
    """Sector singular values, kept counts and the new Lambda of the update."""
    L, K = gl.shape
    R = gr.shape[1]
    gamma = np.zeros((3, chi, chi), dtype=np.complex128)
    gamma[0, :L, :K] = gl
    gamma[1, :K, :R] = gr
    gamma[2, :R, 0] = 1.0
    lamb = np.zeros((2, chi))
    lamb[0, :K] = 1.0
    lamb[1, :R] = lam
    charge = np.full((4, chi, 2), d, dtype=np.int32)
    charge[0, :L] = top
    charge[1, :K] = q
    charge[2, :R] = 0
    charge[3, 0] = 0
    with engine.MPOSimulator(3, d, chi) as sim:
        sim.set_precision(precision)
        sim.load_host(gamma, lamb, charge)
        sim.bs_update(0, interferometer.t_block(THETA, PHI))
        info = sim.last_update_info()
        g, l, c = (x.cpu().numpy() for x in sim.store())
    return info, g, l, c


# resident classes' edges, the hand-over from the streamed rows, and the limits of the
# one-CTA SVD; tall and wide (X = T and X = T^H)
SHAPES = [(28, 28), (29, 31), (56, 60), (57, 57), (113, 120), (114, 114), (158, 150), (159, 161), (224, 224), (225, 230),
          (310, 310), (311, 311), (430, 430), (431, 440), (452, 452), (17, 257), (256, 17), (33, 193), (192, 48), (49, 64),
          (9, 400), (1, 50), (50, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("precision", ["fp64", "fp64-gram"])
def test_singular_values_by_shape(shape, precision):
    """Largest chi of 4 k candidates (d = 2).  Plain path: absolute error within 64 eps sqrt(k)
    of a sector's largest (the rounding of products of length k and of the rotations); Gram
    route: eigenvalue errors of 64 eps k, so sigma^2 within 64 eps k of the largest's square."""
    L, R = shape
    d, K = 2, 40
    chi = max(L, R, K)
    rng = np.random.default_rng(L * 1000 + R)
    args = _two_sites(rng, L, K, R, d)
    want = _expected(d, *args)
    info, g, lam, _ = _update(precision, d, *args, chi)
    k, eps = min(L, R), np.finfo(np.float64).eps
    assert info["shape"] == [(L, R)] * 4
    gram = precision == "fp64-gram" and 4 * k > chi
    for cc, s in zip(info["sectors"], info["sigma"]):
        w = want[cc]
        if gram:
            tol = 64 * eps * max(k, K) * w[0] ** 2
            assert np.all(np.abs(s ** 2 - w ** 2) <= tol + np.where(s == 0, 32 * eps * k * w[0] ** 2 * 4, 0.0))
        else:
            assert np.all(np.abs(s - w) <= 64 * eps * np.sqrt(max(k, K, L, R)) * w[0])
    kept = sum(info["kept"])
    assert 0 < kept <= chi
    # the kept vectors are orthonormal, and V W restores the kept part: the squared norm of
    # W diag(lam_r) per row is sigma^2
    V = g[0][:L, :kept]
    at = 0
    for cc, n in zip(info["sectors"], info["kept"]):
        v = V[:, at:at + n]
        # a kept singular value sigma is known to eps (sigma_1 / sigma)^2 / 2 on the Gram route
        smin = min([x for x in info["sigma"][info["sectors"].index(cc)][:n]], default=1.0)
        loss = (want[cc][0] / smin) ** 2 if gram else want[cc][0] / smin
        assert np.abs(v.conj().T @ v - np.eye(n)).max(initial=0.0) <= 64 * eps * max(k, K) * max(loss, 1.0)
        at += n


# the one-CTA SVD's own limits: columns 1, 2, 16, 17, 64, 65; rows where its registers and its
# shared memory end, tall and wide
ONE_CTA = [(1, 1), (2, 2), (3, 17), (16, 16), (17, 16), (32, 33), (48, 33), (64, 64), (63, 128), (128, 64), (64, 65), (65, 64),
           (65, 65), (130, 56), (56, 130), (17, 512), (512, 17), (513, 17), (16, 800), (800, 16), (13, 1024), (1024, 13), (2, 1025)]


@pytest.mark.parametrize("shape", ONE_CTA, ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("rank", [None, 5])
def test_one_cta_svd(shape, rank):
    """Graded sectors (right weights over eight decades) that keep every vector: singular values
    within 64 eps sqrt(size) of the largest, zeros below the numerical rank, and orthonormal
    kept vectors.  A vector of sigma carries the rounding of its matrix, eps sigma_1 / sigma."""
    L, R = shape
    d, k, eps = 2, min(L, R), np.finfo(np.float64).eps
    K = max(40, k)
    rng = np.random.default_rng(L * 2000 + R)
    args = _two_sites(rng, L, K, R, d, rank=rank, spread=8.0)
    want = _expected(d, *args)
    info, g, lam, _ = _update("fp64", d, *args, max(4 * k, L, R, K))
    V, at = g[0][:L], 0
    for i, cc in enumerate(info["sectors"]):
        s, w, n = info["sigma"][i], want[cc], info["kept"][i]
        assert np.all(np.abs(s - w) <= 64 * eps * np.sqrt(max(K, L, R)) * w[0])
        v = V[:, at:at + n]
        loss = w[0] / min(s[:n], default=1.0)
        assert np.abs(v.conj().T @ v - np.eye(n)).max(initial=0.0) <= 64 * eps * max(k, K) * max(loss, 1.0)
        at += n


@pytest.mark.parametrize("precision", ["fp64", "fp64-gram"])
@pytest.mark.parametrize("rank", [0, 3, 17])
def test_rank_deficient_sectors(precision, rank):
    """Sectors of 120 x 130 and rank at most `rank`: the rest of the spectrum is zero, and a
    zero matrix keeps nothing."""
    L, R, K, d = 120, 130, 40, 2
    rng = np.random.default_rng(rank)
    args = _two_sites(rng, L, K, R, d, rank=rank)
    want = _expected(d, *args)
    if rank == 0:
        info, _, lam, _ = _update(precision, d, *args, 130)
        assert sum(info["kept"]) == 0 and not lam[0].any()
        return
    info, _, lam, _ = _update(precision, d, *args, 130)
    eps = np.finfo(np.float64).eps
    for cc, s, n in zip(info["sectors"], info["sigma"], info["kept"]):
        tol = np.sqrt(64 * eps * L) if precision == "fp64-gram" else 64 * eps * np.sqrt(L)
        assert np.all(np.abs(s - want[cc]) <= tol * want[cc][0])
        if precision == "fp64":
            assert np.count_nonzero(s) <= rank


def test_selection_beyond_its_shared_memory():
    """9 sectors of 590 candidates each (5,310 keys): the oracle's selection of the same
    singular values."""
    L = R = 590
    d, K = 3, 60
    rng = np.random.default_rng(5)
    args = _two_sites(rng, L, K, R, d)
    info, _, lam, _ = _update("fp64-gram", d, *args, L)
    keys = om.selection_keys(info["sectors"], info["sigma"])
    assert info["kept"] == om.select_top(info["sectors"], keys, L, 0.0, info["sigma"])
    assert np.count_nonzero(lam[0]) == sum(info["kept"])
    cut = sum(float(np.sum(s[n:] ** 2)) for s, n in zip(info["sigma"], info["kept"]))
    assert abs(info["trunc_weight"] - cut) <= 1e-13 * sum(float(np.sum(s ** 2)) for s in info["sigma"])


@pytest.mark.parametrize("precision,chi", [("fp64", 48), ("fp64", 130), ("fp64-gram", 130), ("tf32x3", 64)])
def test_groups_of_any_size_agree_bitwise(precision, chi):
    """A layer's updates in groups of 1, 2 and many: the same bits, on every route."""
    n, d = 14, 4
    _, bs, _ = interferometer.circuit(n, 21)
    ops = [b for b in bs if b[0] < 9]
    out = []
    for workers in (1, 4, 32):
        with engine.MPOSimulator(n, d, chi) as sim:
            sim.set_precision(precision)
            sim.set_workers(workers)
            sim.init_single_photons(range(0, n, 2), 0.37)
            sim.run_mesh([b[1] for b in ops], [b[2] for b in ops], [b[3] for b in ops])
            out.append([x.cpu().numpy() for x in sim.store()] + [sim.mesh_truncation()])
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("shape", [(1, 1, 1), (33, 1500, 31), (64, 7, 65), (100, 40, 3)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("order", ["sorted", "random"])
def test_sector_contraction_any_centre_order(shape, order):
    """Runs of equal centre charge in any order (every entry its own run at worst), beyond the
    1,024 entries whose runs are listed at once, against the element-wise sum.  Tolerance:
    len_c products of magnitude at most max|Glc| max|Gcr|, 8 eps each."""
    L, K, R = shape
    d, cc = 4, (2, 1)
    rng = np.random.default_rng(L + K + R)
    glc = rng.standard_normal((L, K)) + 1j * rng.standard_normal((L, K))
    gcr = rng.standard_normal((K, R)) + 1j * rng.standard_normal((K, R))
    cl, cr, q = (rng.integers(0, d + 1, size=(s, 2)) for s in (L, R, K))
    if order == "sorted":
        q = np.array(sorted(map(tuple, q.tolist())))
    U = fock.reference_random_tensor(3, d, 0.6)
    first = [i for i in range(K) if i == 0 or tuple(q[i]) != tuple(q[i - 1])]
    C = cuda_kernels.update_MPO(d, *cc, *(torch.from_numpy(x).cuda() for x in (U.real.copy(), U.imag.copy(), glc, gcr, cl, cr)),
                                q[first].T, np.array(first)).cpu().numpy()
    want = np.zeros((L, R), dtype=np.complex128)
    for l in range(L):
        for r in range(R):
            a, b = cl[l], cr[r]
            if a.max() >= d or b.max() >= d or (a < cc).any() or (b > cc).any():
                continue
            ok = (q <= a).all(1) & (q >= b).all(1) & (q < d).all(1)
            w = np.array([U[a[0] - cc[0], cc[0] - b[0], a[0] - x[0]] * np.conj(U[a[1] - cc[1], cc[1] - b[1], a[1] - x[1]])
                          for x in q[ok]])
            want[l, r] = (w * glc[l, ok] * gcr[ok, r]).sum() if ok.any() else 0.0
    tol = 8 * np.finfo(np.float64).eps * K * np.abs(glc).max() * np.abs(gcr).max()
    assert np.abs(C - want).max() <= tol
