"""An update that returns an error leaves the state as it was, and the handle usable."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from bosonsampling_b200 import engine, interferometer  # noqa: E402

N, D, CHI = 12, 4, 60


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    torch.cuda.set_device(0)


def _mesh(layers, first=0):
    _, bs, _ = interferometer.circuit(N, 9)
    ops = [b for b in bs if first <= b[0] < layers]
    return [b[1] for b in ops], [b[2] for b in ops], [b[3] for b in ops]


@pytest.fixture(scope="module")
def state():
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.init_single_photons(range(0, N, 2), 0.37)
        sim.run_mesh(*_mesh(6))
        return [x.cpu().numpy() for x in sim.store()]


def _host(sim):
    return [x.cpu().numpy() for x in sim.store()]


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# an expired wait of the asynchronous pipelines, a small sector that does not converge (the
# words are set from the host behind the SVD)
@pytest.mark.parametrize("word,message", [("1", "wait expired"), ("2", "did not converge")])
@pytest.mark.parametrize("precision", ["fp64", "fp64-gram"])
def test_update_that_fails(word, message, precision, state, monkeypatch):
    monkeypatch.setenv("BSMPO_TEST_ERROR", word)
    S = interferometer.t_block(0.7, 0.4)
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.set_precision(precision)
        sim.load_host(*state)
        dims = sim.bond_dims()
        with pytest.raises(RuntimeError, match=message):
            sim.bs_update(5, S)
        assert _equal(_host(sim), state) and sim.bond_dims() == dims
        sim.bs_update(5, S)
        got = _host(sim)
    monkeypatch.delenv("BSMPO_TEST_ERROR")
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.set_precision(precision)
        sim.load_host(*state)
        sim.bs_update(5, S)
        assert _equal(_host(sim), got) and not _equal(got, state)


@pytest.mark.parametrize("word", ["1", "2"])
@pytest.mark.parametrize("workers", [2, 16])
def test_mesh_that_fails(word, workers, state, monkeypatch):
    """A group that fails changes none of its bonds: the block sizes the host plans with stay those
    of the charges, and the next mesh computes from the state what a new handle does."""
    monkeypatch.setenv("BSMPO_TEST_ERROR", word)
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.set_workers(workers)
        sim.load_host(*state)
        with pytest.raises(RuntimeError):
            sim.run_mesh(*_mesh(8, 6))
        after = _host(sim)
        occupied = [int(np.count_nonzero(after[2][b, :, 0] < D)) for b in range(N + 1)]
        assert sim.bond_dims() == occupied
        sim.run_mesh(*_mesh(8, 6))
        got = _host(sim)
    monkeypatch.delenv("BSMPO_TEST_ERROR")
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.load_host(*after)
        sim.run_mesh(*_mesh(8, 6))
        assert _equal(_host(sim), got)


def test_expired_wait_of_the_last_gemm(state, monkeypatch):
    """W = V^H C on the tensor cores: a wait of its own that expires is this update's error."""
    monkeypatch.setenv("BSMPO_TC_MASK", "3")
    monkeypatch.setenv("BSMPO_TEST_ERROR", "3")
    S = interferometer.t_block(0.7, 0.4)
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.set_precision("tf32x3")
        sim.load_host(*state)
        with pytest.raises(RuntimeError, match="wait expired"):
            sim.bs_update(5, S)
        assert _equal(_host(sim), state)
        sim.bs_update(5, S)
        got = _host(sim)
    monkeypatch.delenv("BSMPO_TEST_ERROR")
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.set_precision("tf32x3")
        sim.load_host(*state)
        sim.bs_update(5, S)
        assert _equal(_host(sim), got)


@pytest.mark.parametrize("precision", ["fp64", "fp64-gram"])
def test_every_allocation_that_fails(precision, state, monkeypatch):
    """Whichever workspace cannot be had, small sectors' kernels beside the others included: an
    error, the state as it was, and the next update as in a new handle."""
    S = interferometer.t_block(0.7, 0.4)
    with engine.MPOSimulator(N, D, CHI) as sim:
        sim.set_precision(precision)
        sim.load_host(*state)
        sim.bs_update(5, S)
        want = _host(sim)
    failed = 0
    for m in range(60):
        monkeypatch.setenv("BSMPO_TEST_ERROR", str(10 + m))
        with engine.MPOSimulator(N, D, CHI) as sim:
            sim.set_precision(precision)
            sim.load_host(*state)
            try:
                sim.bs_update(5, S)
            except RuntimeError as e:
                assert "allocation" in str(e)
                failed += 1
                assert _equal(_host(sim), state)
                sim.bs_update(5, S)
            assert _equal(_host(sim), want)
    assert 10 <= failed < 60


@pytest.mark.parametrize("precision", ["fp64", "fp64-gram"])
def test_next_update_follows_a_failed_one_at_once(precision, state, monkeypatch):
    """The tables of an update that fails behind another's kernels are not overwritten by the
    next update's while their copy is queued."""
    S = interferometer.t_block(0.7, 0.4)
    results = []
    for m in (None, *range(60)):
        if m is not None:
            monkeypatch.setenv("BSMPO_TEST_ERROR", str(10 + m))
        with engine.MPOSimulator(N, D, CHI) as sim:
            sim.set_precision(precision)
            sim.load_host(*state)
            for mode in (4, 5, 6, 2, 3):
                try:
                    sim.bs_update(mode, S)
                except RuntimeError as e:
                    assert "allocation" in str(e)
                    sim.bs_update(mode, S)
            results.append(_host(sim))
    assert all(_equal(results[0], r) for r in results[1:])


@pytest.mark.parametrize("workers", [1, 4])
def test_preconditioned_form_that_does_not_converge(workers, monkeypatch):
    """Its updates are done again from the matrices themselves: no error, and the result without the
    failure to rounding (Lambda within 1e-12 of the largest).  Where those do not converge either
    the preconditioned result stands."""
    n, d, chi = 16, 4, 300
    _, bs, _ = interferometer.circuit(n, 4)
    ops = [b for b in bs if b[0] < 9]
    out = []
    for word in (None, "4", "5"):
        if word:
            monkeypatch.setenv("BSMPO_TEST_ERROR", word)
        with engine.MPOSimulator(n, d, chi) as sim:
            sim.set_workers(workers)
            sim.init_single_photons(range(0, n, 2), 0.37)
            sim.run_mesh([b[1] for b in ops], [b[2] for b in ops], [b[3] for b in ops])
            out.append((_host(sim), sim.observables()))
    (a, oa), (b, ob), (c, oc) = out
    assert not np.array_equal(a[0], b[0]) and _equal(a, c)
    assert np.abs(np.sort(a[1], axis=1) - np.sort(b[1], axis=1)).max() <= 1e-12 * a[1].max()
    assert np.abs(oa[1] - ob[1]).max() <= 1e-12 * abs(oa[0])
