"""Performance cases: what a user of the simulator has it do, from one beam splitter on a
short chain to whole layers of the 64-mode chi = 1024 circuit.

A case is a dict of plain values; ``kind`` says which public entry points it goes through:

  update       one beam splitter, gate by gate, as a rank of a partitioned chain steps it:
               the two sites and the bond are put into the handle, updated and taken out
  circuit      a whole circuit from its product state: initial state, mesh, output phases,
               trace and marginals
  layers       consecutive layers of a circuit already under way, on a device-resident
               state, then the observables
  host         one layer over a host-resident (page-locked) state, copies included
  batch        several small circuits of uneven size side by side (``engine.run_batch``)
  gradient     loss and gradient of a circuit's marginals in every angle and in eta
  sector       the reference's kernel call: one centre-charge sector of the contraction
  observables  trace and marginals of a large state

The updated site tensors are defined up to a unitary within each (near-)degenerate group of
singular vectors, so what is returned is what does not depend on that choice: Lambda and
charges of the new bond, trace, marginals, gradients.
"""
from math import comb, factorial, sqrt

import numpy as np
import torch

from bosonsampling_b200 import adjoint, cuda_kernels, engine, interferometer


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: one gate of a short chain, where launches and host work count
        dict(name="update_chi32_fp64", kind="update", n=12, d=3, chi=32, start=6, precision="fp64"),
        # one gate at the chain's centre at the benchmark's size, nothing beside it
        dict(name="update_chi1024_gram", kind="update", n=64, d=5, chi=1024, start=8, precision="fp64-gram"),
        # a small whole circuit on the default path (the size of a check against theory)
        dict(name="circuit_n9_chi50_fp64", kind="circuit", n=9, d=4, chi=50, precision="fp64"),
        # the default path on a middle-sized circuit (24 modes, 12 photons, cutoff 4)
        dict(name="circuit_n24_chi256_fp64", kind="circuit", n=24, d=4, chi=256, precision="fp64"),
        # the mixed form on a middle-sized circuit (32 modes, 496 beam splitters)
        dict(name="circuit_n32_chi256_gram", kind="circuit", n=32, d=4, chi=256, precision="fp64-gram"),
        # the benchmark: layers of the 64-mode chi = 1024 circuit once its bonds are full
        dict(name="layers_n64_chi1024_gram", kind="layers", n=64, d=5, chi=1024, start=8, count=2, precision="fp64-gram"),
        # the same circuit on the default path
        dict(name="layer_n64_chi1024_fp64", kind="layers", n=64, d=5, chi=1024, start=8, count=1, precision="fp64"),
        # a state kept in host memory between layers
        dict(name="host_n40_chi500_gram", kind="host", n=40, d=4, chi=500, start=8, count=1, precision="fp64-gram"),
        # many small independent circuits (a scan over inputs)
        dict(name="batch_8_chi64_gram", kind="batch", circuits=8, n=16, d=4, chi=64, precision="fp64-gram"),
        # fitting a circuit: forward and backward
        dict(name="gradient_n6_chi27", kind="gradient", n=6, d=3, chi=27),
        # one sector of a chi = 1024 bond through the reference's own call
        dict(name="sector_443x1024x389", kind="sector", d=5, l=443, c=1024, r=389),
        # the output of a large run
        dict(name="observables_n64_chi1024", kind="observables", n=64, d=5, chi=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["update", "update", "circuit", "circuit", "layers", "layers", "host", "batch", "gradient",
                       "sector", "observables"])
    precision = rng.choice(["fp64", "fp64-gram"])
    if kind == "update":
        chi = _log_int(rng, 32, 1024)
        return dict(kind=kind, n=rng.randint(12, 20 if chi < 200 else 48), d=rng.randint(3, 4) if chi < 300 else rng.randint(4, 5),
                    chi=chi, start=rng.randint(6, 9), precision=precision)
    if kind == "circuit":
        chi = _log_int(rng, 40, 256)
        return dict(kind=kind, n=rng.randint(8, 24), d=rng.randint(3, 4), chi=chi, precision=precision)
    if kind == "layers":
        chi = _log_int(rng, 128, 1024)
        return dict(kind=kind, n=rng.randint(20, 64), d=rng.randint(4, 5) if chi < 600 else 5, chi=chi, start=rng.randint(7, 9),
                    count=1, precision=precision)
    if kind == "host":
        return dict(kind=kind, n=rng.randint(16, 48), d=rng.randint(4, 5), chi=_log_int(rng, 100, 600), start=rng.randint(7, 9),
                    count=1, precision="fp64-gram")
    if kind == "batch":
        return dict(kind=kind, circuits=rng.randint(3, 8), n=rng.randint(10, 16), d=rng.randint(3, 4), chi=_log_int(rng, 32, 72),
                    precision=precision)
    if kind == "gradient":
        return dict(kind=kind, n=rng.randint(4, 6), d=3, chi=rng.randint(16, 32))
    if kind == "sector":
        return dict(kind=kind, d=rng.randint(3, 6), l=_log_int(rng, 20, 700), c=_log_int(rng, 40, 1024), r=_log_int(rng, 20, 700))
    return dict(kind=kind, n=rng.randint(8, 64), d=rng.randint(3, 6), chi=_log_int(rng, 64, 1024))


# ------------------------------------------------------------------------------- inputs
def _eta(seed):
    """A transmissivity of its own for every seed, clear of 0.5 (where lossy single photons
    have exactly degenerate multiplets, any basis of which is right)."""
    return float(np.random.default_rng(seed).uniform(0.25, 0.42))


def _photons(n):
    return list(range(0, n, 2))


def _target(case, seed):
    return np.random.default_rng(seed).dirichlet(np.ones(case["d"]), size=case["n"])


def _mesh(ops):
    return [b[1] for b in ops], [b[2] for b in ops], [b[3] for b in ops]


def _under_way(case, seed):
    """A handle whose circuit has run its first ``start`` layers, and the layers after them."""
    n, start = case["n"], case["start"]
    _, bs, _ = interferometer.circuit(n, seed)
    sim = engine.MPOSimulator(n, case["d"], case["chi"])
    sim.set_workers(16)
    sim.set_precision("fp64-gram" if case["chi"] >= 128 else "fp64")
    sim.init_single_photons(_photons(n), _eta(seed))
    sim.run_mesh(*_mesh([b for b in bs if b[0] < start]))
    sim.set_precision(case["precision"])
    return sim, [b for b in bs if b[0] >= start]


def _centre(bs, n):
    """The beam splitter of the first layer of ``bs`` nearest the chain's centre."""
    layer = min(b[0] for b in bs)
    return min((b for b in bs if b[0] == layer), key=lambda b: (abs(b[1] - (n // 2 - 1)), b[1]))


def _charges(g, size, d):
    """Sorted (ket, bra) charges of a bond: small ones are commoner, and the two agree mostly."""
    ket = torch.randint(0, d, (size,), generator=g) + torch.randint(0, d, (size,), generator=g)
    ket = torch.minimum(ket // 2, torch.tensor(d - 1))
    bra = (ket + torch.randint(-1, 2, (size,), generator=g)).clamp(0, d - 1)
    return torch.tensor(sorted(zip(ket.tolist(), bra.tolist())), dtype=torch.int32)


def _sector_inputs(case, seed, dev):
    d, L, K, R = case["d"], case["l"], case["c"], case["r"]
    g = torch.Generator().manual_seed(seed)
    cc = (d // 2, d // 2)

    def matrix(m, n):
        return torch.complex(torch.randn(m, n, generator=g, dtype=torch.float64),
                             torch.randn(m, n, generator=g, dtype=torch.float64)) / sqrt(K)

    glc, gcr = matrix(L, K), matrix(K, R)
    cl = torch.maximum(_charges(g, L, d), torch.tensor(cc, dtype=torch.int32))     # rows a >= cc
    cr = torch.minimum(_charges(g, R, d), torch.tensor(cc, dtype=torch.int32))     # columns b <= cc
    cl, cr = (torch.tensor(sorted(map(tuple, x.tolist())), dtype=torch.int32) for x in (cl, cr))
    q = _charges(g, K, d)
    first = [i for i in range(K) if i == 0 or q[i].tolist() != q[i - 1].tolist()]
    theta, phi = torch.rand(2, generator=g, dtype=torch.float64).tolist()
    u = torch.from_numpy(_bs_tensor(_block(0.3 + theta, 6.0 * phi).T, d))
    parts = [x.to(dev) for x in (u.real.contiguous(), u.imag.contiguous(), glc, gcr, cl, cr)]
    return dict(cc=cc, parts=parts, q=q, changes=np.array([q[i].tolist() for i in first]).T, idx=np.array(first), u=u)


def _random_state(case, seed, dev):
    """A full chain for the observables: charges of every bond, Lambda, and site tensors of
    one sign's weight, so that the trace is no sum of cancelling terms."""
    n, d, chi = case["n"], case["d"], case["chi"]
    g = torch.Generator().manual_seed(seed)
    charge = torch.stack([_charges(g, chi, d) for _ in range(n + 1)])
    lam = torch.rand(n - 1, chi, generator=g, dtype=torch.float64) + 0.1
    gd = torch.Generator(device=dev).manual_seed(seed)
    gamma = torch.complex(torch.rand(n, chi, chi, generator=gd, device=dev, dtype=torch.float64),
                          0.3 * torch.randn(n, chi, chi, generator=gd, device=dev, dtype=torch.float64))
    gamma *= 6.0 / chi
    return gamma, lam.to(dev), charge.to(dev)


def _batch_specs(case, seed):
    rng = np.random.default_rng(seed)
    specs = []
    for i in range(case["circuits"]):
        n = case["n"] - (i * 5) % 6                                  # uneven sizes, the same for every seed
        chi = case["chi"] - (i * 7) % 13 * case["chi"] // 25
        _, bs, ph = interferometer.circuit(n, seed * 100 + i)
        specs.append(dict(n=n, d=case["d"], chi=chi, eta=float(rng.uniform(0.25, 0.42)), photon_modes=_photons(n), mesh=bs,
                          phases=ph))
    return specs


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    if kind == "update":
        sim, bs = _under_way(case, seed)
        _, m, th, ph = _centre(bs, case["n"])
        S = interferometer.t_block(th, ph)
        return dict(kind=kind, sim=sim, m=m, S=S, sites=[sim.get_site(m), sim.get_site(m + 1)], bond=sim.get_bond(m + 1))
    if kind == "circuit":
        n = case["n"]
        _, bs, ph = interferometer.circuit(n, seed)
        sim = engine.MPOSimulator(n, case["d"], case["chi"])
        sim.set_precision(case["precision"])
        return dict(kind=kind, sim=sim, photons=_photons(n), eta=_eta(seed), mesh=_mesh(bs), phases=ph)
    if kind == "layers":
        sim, bs = _under_way(case, seed)
        return dict(kind=kind, sim=sim, state=sim.store(), mesh=_mesh([b for b in bs if b[0] < case["start"] + case["count"]]))
    if kind == "host":
        sim, bs = _under_way(case, seed)
        state = tuple(x.cpu().pin_memory() for x in sim.store())
        out = tuple(torch.empty_like(x).pin_memory() for x in state)
        return dict(kind=kind, sim=sim, state=state, out=out, mesh=_mesh([b for b in bs if b[0] < case["start"] + case["count"]]))
    if kind == "batch":
        return dict(kind=kind, specs=_batch_specs(case, seed), precision=case["precision"])
    if kind == "gradient":
        n = case["n"]
        _, bs, ph = interferometer.circuit(n, seed)
        circuit = adjoint.DiffCircuit(n, case["d"], case["chi"], _photons(n), bs, ph)
        return dict(kind=kind, circuit=circuit, theta=[b[2] for b in bs], phi=[b[3] for b in bs], eta=_eta(seed),
                    target=_target(case, seed))
    if kind == "sector":
        return dict(kind=kind, d=case["d"], **_sector_inputs(case, seed, dev))
    sim = engine.MPOSimulator(case["n"], case["d"], case["chi"])
    sim.load(*_random_state(case, seed, dev))
    return dict(kind=kind, sim=sim)


# ------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "update":
        sim, m = s["sim"], s["m"]
        sim.put_site(m, s["sites"][0])
        sim.put_site(m + 1, s["sites"][1])
        sim.put_bond(m + 1, *s["bond"])
        sim.bs_update(m, s["S"])
        sim.get_site(m)
        sim.get_site(m + 1)
        return dict(zip(("lambda", "charge"), sim.get_bond(m + 1)))
    if kind == "circuit":
        sim = s["sim"]
        sim.init_single_photons(s["photons"], s["eta"])
        sim.run_mesh(*s["mesh"])
        sim.apply_phases(s["phases"])
        return _observables(sim)
    if kind == "layers":
        sim = s["sim"]
        sim.load(*s["state"])
        sim.run_mesh(*s["mesh"])
        return _observables(sim)
    if kind == "host":
        s["sim"].run_mesh_host(*s["mesh"], s["state"], s["out"])
        return _observables(s["sim"])
    if kind == "batch":
        return [dict(trace=np.array([t]), marginals=p) for t, p in engine.run_batch(s["specs"], concurrency=4,
                                                                                    precision=s["precision"], workers=4)]
    if kind == "gradient":
        loss, th, ph, eta = s["circuit"].loss_and_grad(s["theta"], s["phi"], s["eta"], s["target"])
        return dict(loss=loss, theta=th, phi=ph, eta=eta)
    if kind == "sector":
        u_r, u_i, glc, gcr, cl, cr = s["parts"]
        return cuda_kernels.update_MPO(s["d"], s["cc"][0], s["cc"][1], u_r, u_i, glc, gcr, cl, cr, s["changes"], s["idx"])
    return _observables(s["sim"])


def _observables(sim):
    trace, marginals = sim.observables()
    return dict(trace=np.array([trace]), marginals=marginals)


# ------------------------------------------------------------------------------- minimum work
def _bond(b, n, layer, chi):
    """Bond dimension, roughly: it grows by a factor of about four per layer and per mode from
    the chain's end, up to chi."""
    return min(float(chi), 4.0 ** min(b, n - b, layer + 1))


def _update_work(l, c, r, kept, d):
    """One update: the two sites in and out; the block products of the contraction (about an
    eighth of the charge triples are allowed) and W; the reduction of the sectors' matrices
    (about 2.7 chi candidates over d^2 sectors of uneven size)."""
    m = 2.7 * kept
    return (16.0 * (l * c + c * r + (l + r) * kept), 8.0 * l * c * r / 8.0 + 8.0 * l * kept * r / 6.0 + 16.0 / 3.0 * m ** 3 * 2.0 / d ** 4)


def _mesh_work(n, d, chi, layers):
    by = fl = 0.0
    for layer in layers:
        for m in range(layer % 2, n - 1, 2):
            l, c, r = (_bond(b, n, layer, chi) for b in (m, m + 1, m + 2))
            b, f = _update_work(l, c, r, _bond(m + 1, n, layer + 1, chi), d)
            by, fl = by + b, fl + f
    return by, fl


def work(case):
    kind = case["kind"]
    if kind == "update":
        c = float(case["chi"])
        by, fl = _update_work(c, c, c, c, case["d"])
        return dict(bytes=by, flops=fl)
    if kind in ("layers", "host"):
        by, fl = _mesh_work(case["n"], case["d"], case["chi"], range(case["start"], case["start"] + case["count"]))
        state = 16.0 * case["n"] * case["chi"] ** 2
        return dict(bytes=max(by, 2 * state), flops=fl)
    if kind in ("circuit", "gradient"):
        by, fl = _mesh_work(case["n"], case["d"], case["chi"], range(case["n"]))
        f = 3.0 if kind == "gradient" else 1.0
        return dict(bytes=f * by, flops=f * fl)
    if kind == "batch":
        by, fl = _mesh_work(case["n"] - 2, case["d"], 0.75 * case["chi"], range(case["n"] - 2))
        return dict(bytes=case["circuits"] * by, flops=case["circuits"] * fl)
    if kind == "sector":
        l, c, r = case["l"], case["c"], case["r"]
        return dict(bytes=16.0 * (l * c + c * r + l * r), flops=8.0 * l * c * r / 4.0)
    n, chi = case["n"], case["chi"]
    return dict(bytes=16.0 * n * chi ** 2, flops=16.0 * n * chi ** 2)


# ------------------------------------------------------------------------------- in 64 bits
def _block(theta, phi):
    """T(theta, phi) = [[e^{i phi} cos, -sin], [e^{i phi} sin, cos]]."""
    c, s, e = np.cos(theta), np.sin(theta), np.exp(1j * phi)
    return np.array([[e * c, -s], [e * s, c]])


def _bs_tensor(M, d):
    """U[n, m, l] = <l, n+m-l| Gamma(M) |n, m> of a single-particle matrix M."""
    U = np.zeros((d, d, d), dtype=np.complex128)
    for n in range(d):
        for m in range(d):
            for l in range(max(0, n + m + 1 - d), min(d, n + m + 1)):
                norm = sqrt(factorial(l) * factorial(n + m - l) / (factorial(n) * factorial(m)))
                U[n, m, l] = norm * sum(comb(n, k) * comb(m, l - k) * M[0, 0] ** k * M[1, 0] ** (n - k) * M[0, 1] ** (l - k)
                                        * M[1, 1] ** (m - l + k) for k in range(max(0, l - m), min(l, n) + 1))
    return U


class _Chain:
    """The chain in plain numpy: per bond the occupied charges and Lambda, per site a dense
    matrix over the occupied entries."""

    def __init__(self, n, d, chi, photons, eta):
        self.n, self.d, self.chi = n, d, chi
        rho = [{(0, 0): 1.0 - eta, (1, 1): eta} if i in photons else {(0, 0): 1.0} for i in range(n)]
        bonds = [None] * n + [[(0, 0)]]
        for b in range(n - 1, -1, -1):
            bonds[b] = sorted({(q0 + o0, q1 + o1) for (q0, q1) in bonds[b + 1] for (o0, o1) in rho[b]
                               if q0 + o0 < d and q1 + o1 < d})
        bonds[0] = [(c, c) for c in range(d)]
        self.q = [np.array(x).reshape(-1, 2) for x in bonds]
        self.lam = [np.ones(len(x)) for x in bonds]
        self.g = [np.array([[rho[i].get((a0 - b0, a1 - b1), 0.0) for (b0, b1) in bonds[i + 1]] for (a0, a1) in bonds[i]],
                           dtype=np.complex128) for i in range(n)]
        for m in range(n - 2, -1, -1):
            self.update(m, np.eye(2))

    def update(self, m, S):
        d, U = self.d, _bs_tensor(np.asarray(S, dtype=np.complex128).T, self.d)
        ql, qc, qr, lr = self.q[m], self.q[m + 1], self.q[m + 2], self.lam[m + 2]
        gl, gr = self.g[m], self.g[m + 1]
        found = []
        for c0 in range(qr[:, 0].min(), ql[:, 0].max() + 1):
            for c1 in range(qr[:, 1].min(), ql[:, 1].max() + 1):
                rows = np.nonzero((ql[:, 0] >= c0) & (ql[:, 1] >= c1))[0]
                cols = np.nonzero((qr[:, 0] <= c0) & (qr[:, 1] <= c1))[0]
                if not len(rows) or not len(cols):
                    continue
                C = np.zeros((len(rows), len(cols)), dtype=np.complex128)
                for x in sorted(set(map(tuple, qc))):
                    k = np.nonzero((qc == x).all(1))[0]
                    i0 = ql[rows, 0] - x[0]
                    i1 = ql[rows, 1] - x[1]
                    ok = ((i0 >= 0) & (i1 >= 0))[:, None] & ((qr[cols, 0] <= x[0]) & (qr[cols, 1] <= x[1]))[None, :]
                    w0 = U[(ql[rows, 0] - c0)[:, None], (c0 - qr[cols, 0])[None, :], np.maximum(i0, 0)[:, None]]
                    w1 = U[(ql[rows, 1] - c1)[:, None], (c1 - qr[cols, 1])[None, :], np.maximum(i1, 0)[:, None]]
                    C += np.where(ok, w0 * w1.conj(), 0.0) * (gl[np.ix_(rows, k)] @ gr[np.ix_(k, cols)])
                T = C * lr[cols][None, :]
                V, s, _ = np.linalg.svd(T, full_matrices=False)
                s[s <= 16 * np.finfo(float).eps * sqrt(max(T.shape)) * np.linalg.norm(T)] = 0.0
                found.append([(c0, c1), s, V, C, rows, cols])
        # the largest chi; a ket / bra swapped pair of sectors is cut at the same place
        at = {f[0]: i for i, f in enumerate(found)}
        cand = []
        for i, f in enumerate(found):
            o = found[at[f[0][::-1]]][1] if f[0][::-1] in at else f[1]
            key = f[1].copy()
            p = min(len(key), len(o))
            key[:p] = np.maximum(key[:p], o[:p])
            cand += [(-v, i, j) for j, v in enumerate(key) if v > 0]
        kept = [0] * len(found)
        for _, i, j in sorted(cand)[: self.chi]:
            kept[i] = max(kept[i], j + 1)
        kept = [min(k, int((f[1] > 0).sum())) for k, f in zip(kept, found)]
        kept = [min(k, kept[at[f[0][::-1]]]) if f[0][::-1] in at else k for k, f in zip(kept, found)]
        total = sum(kept)
        GL, GR = np.zeros((len(ql), total), dtype=np.complex128), np.zeros((total, len(qr)), dtype=np.complex128)
        q, lam, at = [], [], 0
        for k, (cc, s, V, C, rows, cols) in zip(kept, found):
            sl = np.arange(at, at + k)
            GL[np.ix_(rows, sl)] = V[:, :k]
            GR[np.ix_(sl, cols)] = V[:, :k].conj().T @ C
            q += [cc] * k
            lam += list(s[:k])
            at += k
        self.g[m], self.g[m + 1] = GL, GR
        self.q[m + 1], self.lam[m + 1] = np.array(q).reshape(-1, 2), np.array(lam)

    def observables(self):
        return _chain_observables(self.g, self.q, self.d)


def _chain_observables(g, q, d):
    n = len(g)
    diag = [(x[:, 0] == x[:, 1]).astype(np.float64) for x in q]
    R, L = [None] * n + [diag[n]], [diag[0]]
    for i in range(n - 1, -1, -1):
        R[i] = diag[i] * (g[i] @ R[i + 1])
    for i in range(n):
        L.append(diag[i + 1] * (L[i] @ g[i]))
    P = np.zeros((n, d), dtype=np.complex128)
    for i in range(n):
        occ = q[i][:, 0][:, None] - q[i + 1][:, 0][None, :]
        M = L[i][:, None] * g[i] * R[i + 1][None, :]
        for k in range(d):
            P[i, k] = M[occ == k].sum()
    return dict(trace=np.array([R[0].sum()]), marginals=P)


def _exact_circuit(n, d, chi, eta, bs):
    chain = _Chain(n, d, chi, _photons(n), eta)
    for _, m, th, ph in bs:
        chain.update(m, _block(th, ph))
    return chain


def _exact_sector(case, seed):
    x = _sector_inputs(case, seed, torch.device("cpu"))
    _, _, glc, gcr, cl, cr = (t.numpy() for t in x["parts"])
    q, U, (c0, c1) = x["q"].numpy(), x["u"].numpy(), x["cc"]
    C = np.zeros((case["l"], case["r"]), dtype=np.complex128)
    for p in sorted(set(map(tuple, q.tolist()))):
        k = np.nonzero((q == p).all(1))[0]
        i0, i1 = cl[:, 0] - p[0], cl[:, 1] - p[1]
        ok = ((i0 >= 0) & (i1 >= 0))[:, None] & ((cr[:, 0] <= p[0]) & (cr[:, 1] <= p[1]))[None, :]
        w0 = U[(cl[:, 0] - c0)[:, None], (c0 - cr[:, 0])[None, :], np.maximum(i0, 0)[:, None]]
        w1 = U[(cl[:, 1] - c1)[:, None], (c1 - cr[:, 1])[None, :], np.maximum(i1, 0)[:, None]]
        C += np.where(ok, w0 * w1.conj(), 0.0) * (glc[:, k] @ gcr[k])
    return torch.from_numpy(C)


def exact(case, seed):
    """The same in plain numpy; None where that takes more than about 20 seconds (the larger
    circuits), and for the gradients, which no 64-bit value is at hand for."""
    kind = case["kind"]
    if kind == "sector":
        return _exact_sector(case, seed)
    if kind == "observables":
        gamma, _, charge = _random_state(case, seed, torch.device("cuda", torch.cuda.current_device()))
        return _chain_observables([x.cpu().numpy() for x in gamma], [x.cpu().numpy() for x in charge], case["d"])
    n, d, chi = case["n"], case["d"], case["chi"]
    if kind == "batch" or chi > 64 or n > 16:
        return None
    # the mesh is an input: its angles are data that the program has before the call
    _, bs, _ = interferometer.circuit(n, seed)
    if kind == "update":
        chain = _exact_circuit(n, d, chi, _eta(seed), [b for b in bs if b[0] < case["start"]])
        _, m, th, ph = _centre([b for b in bs if b[0] >= case["start"]], n)
        chain.update(m, _block(th, ph))
        lam = np.zeros(chi)
        lam[: len(chain.lam[m + 1])] = chain.lam[m + 1]
        return {"lambda": torch.from_numpy(lam), "charge": None}
    chain = _exact_circuit(n, d, chi, _eta(seed), bs)
    out = chain.observables()
    if kind == "circuit":
        return out
    P = out["marginals"].real / out["trace"][0].real
    return dict(loss=float(((P - _target(case, seed)) ** 2).sum()), theta=None, phi=None, eta=None)
