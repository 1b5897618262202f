"""Performance cases of the impurity solver: the calls a program makes through
the package's public entry points, over the sizes the configurations, tests and
benchmark of this repository use (6 to 16 orbitals per spin, half filling and
the sectors next to it, one and two impurity orbitals, both vector types).

kind "hv":       one H*v of an (N_up, N_dn) sector
kind "ground":   both Lanczos passes, E0 and the eigenvector
kind "green":    one continued-fraction chain on a given start vector, G(i w_n)
kind "solve":    a whole impurity solve over a window of sectors
kind "nambu_hv", "nambu_green": the same on a Nambu (superconducting) sector
kind "vertex":   the local vertex for a batch of frequency triples
kind "grad":     the gradient of E0 + G with respect to the bath parameters
"""
import math

import numpy as np
import torch

from ed_solver_b200 import edk, vertex
from ed_solver_b200.model import matsubara, nambu_star_model, star_model

BETA = 50.0


def listed():
    return [
        # the smallest calls: a sector of a few thousand states, as a fit over baths of 7 levels makes them
        dict(name="hv_ns8_f64", kind="hv", ns=8, nup=4, ndn=4, nc=1, dtype="f64"),
        # two orbitals with spin-flip and pair-hopping terms, the largest sector of a 12-orbital multiplet scan
        dict(name="hv_kanamori_ns12_f64", kind="hv", ns=12, nup=6, ndn=6, nc=2, dtype="f64"),
        # rows of odd length (6,435 states per spin): no two rows share an alignment
        dict(name="hv_odd_ns15_f64", kind="hv", ns=15, nup=7, ndn=8, nc=1, dtype="f64"),
        # the largest sector in single precision
        dict(name="hv_ns16_f32", kind="hv", ns=16, nup=8, ndn=8, nc=1, dtype="f32"),
        # ground state of a mid-sized sector to a small residual
        dict(name="ground_ns12_f64", kind="ground", ns=12, nup=6, ndn=6, nc=1),
        # a Green chain in double precision, 10.3 million states
        dict(name="green_ns14_f64", kind="green", ns=14, nup=8, ndn=7, nc=1, dtype="f64", steps=200, nw=512),
        # a Green chain of the largest solve, in single precision: where that solve spends its time
        dict(name="green_ns16_f32", kind="green", ns=16, nup=9, ndn=8, nc=1, dtype="f32", steps=200, nw=512),
        # a whole solve: sectors around half filling, Boltzmann window, Green functions, double occupancy
        dict(name="solve_kanamori_ns8", kind="solve", ns=8, nc=2, width=2, steps=200, nw=512),
        # superconducting bath, the largest sector that the tests and the benchmark time in double precision
        dict(name="nambu_hv_ns14_f64", kind="nambu_hv", ns=14, npart=14, dtype="f64"),
        dict(name="nambu_green_ns10_f64", kind="nambu_green", ns=10, npart=11, dtype="f64", steps=200, nw=512),
        # the local vertex for a slice of a frequency grid
        dict(name="vertex_ns4_512", kind="vertex", ns=4, nf=512),
        # backward: the gradient a bath fit asks for
        dict(name="grad_ns10_f64", kind="grad", ns=10, nup=5, ndn=5, steps=100, nw=256),
    ]


def draw(rng):
    kind = rng.choice(["hv", "hv", "hv", "ground", "green", "green", "solve", "nambu_hv", "nambu_green", "vertex",
                       "grad"])
    if kind in ("hv", "green", "ground"):
        ns = rng.randint(6, {"hv": 16, "green": 15, "ground": 13}[kind])
        nc = 2 if ns <= 12 and rng.random() < 0.3 else 1
        nup = max(1, min(ns - 1, ns // 2 + rng.randint(-1, 2)))
        ndn = max(1, min(ns - 1, ns // 2 + rng.randint(-1, 1)))
        c = dict(kind=kind, ns=ns, nup=nup, ndn=ndn, nc=nc)
        if kind == "ground":
            return c
        c["dtype"] = rng.choice(["f64", "f32"]) if ns >= 12 else "f64"
        if kind == "green":
            c["steps"] = rng.randint(50, 300 if ns < 15 else 100)
            c["nw"] = rng.choice([200, 512, 1001])
        return c
    if kind == "solve":
        return dict(kind=kind, ns=rng.randint(5, 9), nc=rng.choice([1, 2]), width=rng.randint(1, 2),
                    steps=rng.randint(100, 200), nw=rng.choice([128, 333, 512]))
    if kind in ("nambu_hv", "nambu_green"):
        ns = rng.randint(5, 13 if kind == "nambu_hv" else 10)
        c = dict(kind=kind, ns=ns, npart=ns + rng.randint(-1, 2), dtype=rng.choice(["f64", "f64", "f32"]))
        if kind == "nambu_green":
            c.update(dtype="f64", steps=rng.randint(50, 250), nw=rng.choice([200, 512]))
        return c
    if kind == "vertex":
        return dict(kind=kind, ns=rng.choice([3, 4]), nf=int(math.exp(rng.uniform(math.log(8), math.log(512)))))
    ns = rng.randint(6, 11)
    return dict(kind="grad", ns=ns, nup=ns // 2, ndn=ns - ns // 2, steps=rng.randint(40, 120), nw=rng.choice([64, 256]))


# ---------------------------------------------------------------------------
# models and inputs
# ---------------------------------------------------------------------------

def _model(case, seed):
    """A seeded star model: bath levels and hybridisations as the synthetic
    configurations draw them; two orbitals: Kanamori U, J at half filling."""
    rng = np.random.default_rng(seed)
    ns, nc = case["ns"], case.get("nc", 1)
    nb = ns - nc
    eb = np.sort(rng.uniform(-2.0, 2.0, nb))
    v = rng.uniform(0.15, 0.45, nb)
    if nc == 1:
        return star_model(-1.25, 2.5, eb, v)
    U, J = 3.5, 0.6
    return star_model(-(3 * U - 5 * J) / 2, U, eb, v, orbital_of_bath=[k % nc for k in range(nb)], nc=nc, J=J)


def _nambu(case, seed):
    rng = np.random.default_rng(seed)
    nb = case["ns"] - 1
    return nambu_star_model(-1.0, 2.0, rng.uniform(-2.0, 2.0, nb), rng.uniform(0.2, 0.5, nb),
                            rng.uniform(0.1, 0.4, nb))


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tdtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.float64


def _noise(n, seed, dtype):
    g = torch.Generator(device=_dev())
    g.manual_seed(seed)
    return torch.randn(n, generator=g, device=_dev(), dtype=dtype)


def _occupations(ns, n):
    """(states, ns) occupation numbers of one spin species' basis, increasing order."""
    s = np.arange(1 << ns, dtype=np.int64)
    bits = (s[:, None] >> np.arange(ns)) & 1
    return bits[bits.sum(1) == n]


def _start(case, seed, dtype):
    """A vector with the weight distribution of c+|ground state>: random signs
    and amplitudes that fall off with the one-body energy of the configuration."""
    m = _model(case, seed)
    w = []
    for s, n in ((0, case["nup"]), (1, case["ndn"])):
        e = _occupations(m.ns, n) @ np.concatenate([np.diag(m.eb[s]), np.diag(m.ec[s]) + 0.5 * m.u[0, 0]])
        w.append(torch.tensor(np.exp(-0.7 * (e - e.min())), device=_dev()).to(dtype))
    x = _noise(len(w[0]) * len(w[1]), seed, dtype)
    x.view(len(w[1]), len(w[0])).mul_(w[1][:, None]).mul_(w[0][None, :])
    return x


def _e0(m, nup, ndn):
    """The chains' energy origin: 0.5 below the Hartree estimate of the sector's lowest energy."""
    t = np.zeros((m.ns, m.ns))
    t[:m.nb, :m.nb], t[m.nb:, m.nb:] = m.eb[0], m.ec[0] + 0.5 * np.diag(np.diag(m.u))
    t[:m.nb, m.nb:], t[m.nb:, :m.nb] = m.vbc[0], m.vbc[0].T
    e = np.linalg.eigvalsh(t)
    return float(e[:nup].sum() + e[:ndn].sum() - 0.25 * np.trace(m.u) - 0.5)


def _nambu_matrix(nm):
    """One-body matrix over the up orbitals and the down holes (baths first in each half)."""
    m = nm.base
    nb, ns = m.nb, m.ns
    t = np.zeros((2 * ns, 2 * ns))
    for blk, s, sg in ((slice(0, ns), 0, 1.0), (slice(ns, 2 * ns), 1, -1.0)):
        h = np.zeros((ns, ns))
        h[:nb, :nb], h[nb:, nb:], h[:nb, nb:], h[nb:, :nb] = m.eb[s], m.ec[s], m.vbc[s], m.vbc[s].T
        t[blk, blk] = sg * h
    t[:nb, ns:ns + nb], t[ns:ns + nb, :nb] = nm.pb, nm.pb.T
    return t


def _nambu_start(case, seed):
    """As _start and _e0, for a Nambu sector."""
    nm = _nambu(case, seed)
    t, u, ns, nb = _nambu_matrix(nm), float(nm.base.u[0, 0]), nm.ns, nm.nb
    t[nb, nb] += 0.5 * u
    t[ns + nb, ns + nb] -= 0.5 * u
    st = _popcount_states(2 * ns, case["npart"], _dev())
    e = torch.zeros(len(st), dtype=torch.float64, device=_dev())
    for o in range(2 * ns):
        e += float(t[o, o]) * ((st >> o) & 1).double()
    x = _noise(len(st), seed, torch.float64) * torch.exp(-0.7 * (e - e.min()))
    return x.to(_tdtype(case)), float(np.linalg.eigvalsh(t)[:case["npart"]].sum() + 0.25 * u - 0.5)


def _triples(nf, beta, seed):
    rng = np.random.default_rng(seed)
    nu = 1j * (2 * rng.integers(-8, 8, (nf, 3)) + 1) * np.pi / beta
    nu[::3, 2] = -nu[::3, 1]                       # the diagonal of the grid: w2 + w3 = 0
    return nu


def _sectors(case):
    """The sectors around half filling, as a program that tracks its sectors scans them."""
    ns, d = case["ns"], case["width"]
    h = ns // 2
    return [(a, b) for a in range(h - d, h + d + 1) for b in range(h - d, h + d + 1) if 0 <= a <= ns and 0 <= b <= ns]


def _grad_chains():
    return [(0, 0, True), (0, 0, False)]


_CTX = []


def _ctx():
    """The one context a program keeps; single-precision sectors sum their hops in single precision, as the
    mixed-precision benchmark does."""
    if not _CTX:
        c = edk.Context(0)
        c.set_fp32_sums(True)
        _CTX.append(c)
    return _CTX[0]


# ---------------------------------------------------------------------------
# the timed calls
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind, ctx = case["kind"], _ctx()
    s = dict(kind=kind, case=case, ctx=ctx)
    if kind in ("hv", "green", "ground"):
        s["model"] = _model(case, seed)
        s["h"] = edk.Hamiltonian(ctx, s["model"], case["nup"], case["ndn"])
    elif kind in ("nambu_hv", "nambu_green"):
        s["h"] = edk.HamiltonianSz(ctx, _nambu(case, seed), case["npart"])
    if kind in ("hv", "nambu_hv"):
        s["x"] = _noise(s["h"].dim, seed, _tdtype(case)) / math.sqrt(s["h"].dim)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "green":
        s["x"] = _start(case, seed, _tdtype(case))
        s["e0"], s["wn"] = _e0(s["model"], case["nup"], case["ndn"]), matsubara(BETA, case["nw"])
    elif kind == "nambu_green":
        s["x"], s["e0"] = _nambu_start(case, seed)
        s["wn"] = matsubara(BETA, case["nw"])
    elif kind == "solve":
        s["model"], s["sectors"] = _model(case, seed), _sectors(case)
    elif kind == "vertex":
        n = case["ns"] // 2
        m = _model(case, seed)
        s["E"], s["M"] = vertex.vertex_inputs(ctx, m, n, n)
        s["beta"], s["n"], s["w"] = 10.0, n, _triples(case["nf"], 10.0, seed)
        s["Z"], s["gs"] = vertex.partition(s["E"], s["beta"])
    elif kind == "grad":
        m = _model(case, seed)
        s["h"] = edk.Hamiltonian(ctx, m, case["nup"], case["ndn"])
        r = s["h"].lanczos_e0("f64", tolerance=1e-14, residual_tol=1e-12)
        s["psi"], s["e0"] = s["h"].lanczos_gs(r["vecp"][0]), float(r["E"][0])
        s["params"], s["wn"] = edk.star_params(m), matsubara(BETA, case["nw"])
        s["gbar"] = _gbar(case, seed)
    return s


def _gbar(case, seed):
    rng = np.random.default_rng(seed + 1)
    return (rng.normal(size=(2, case["nw"])) + 1j * rng.normal(size=(2, case["nw"]))) / case["nw"]


def run(s):
    kind, case = s["kind"], s["case"]
    if kind in ("hv", "nambu_hv"):
        return s["h"].hmult(s["x"], out=s["y"])
    if kind in ("green", "nambu_green"):
        # the coefficients past the first converged Ritz value follow the rounding of every step before them, so a
        # program uses G alone; a chain in single precision gives G to that precision, and is kept in it
        G = s["h"].green_chain(s["x"], case["steps"], s["e0"], 1, s["wn"], cutoff_dynamic=0.0)[0]
        return G.astype(np.complex64) if case["dtype"] == "f32" else G
    if kind == "ground":
        r = s["h"].lanczos_e0("f64", tolerance=1e-14, residual_tol=1e-11)
        return dict(e0=float(r["E"][0]), psi=s["h"].lanczos_gs(r["vecp"][0]))
    if kind == "solve":
        r = edk.solve(s["ctx"], s["model"], s["sectors"], BETA, case["nw"], nitergreen=case["steps"],
                      tolerance=1e-14, residual_tol=1e-11)
        return dict(e0=r["e0"], z=r["z"], G=r["G"], docc=r["docc"])
    if kind == "vertex":
        pd, pu = edk.chiloc(s["ctx"], s["E"], s["M"], s["w"], s["beta"], s["Z"], s["gs"], case["ns"], s["n"], s["n"])
        return dict(dndn=pd, updn=pu)
    grad, G, _ = s["h"].grad_green(s["psi"], s["e0"], _grad_chains(), case["steps"], s["wn"], s["gbar"], s["params"],
                                   e0bar=1.0, cg_tol=1e-12)
    return dict(grad=grad, G=G)


def _dim(case):
    if "npart" in case:
        return math.comb(2 * case["ns"], case["npart"])
    return math.comb(case["ns"], case["nup"]) * math.comb(case["ns"], case["ndn"])


def work(case):
    """Bytes: vectors in and out (H*v), or three vector streams a Lanczos step;
    operations: one multiply-add per non-zero element of H."""
    kind, ns = case["kind"], case["ns"]
    if kind == "vertex":
        d = math.comb(ns, ns // 2) ** 2
        return dict(bytes=14 * 8 * d * d + case["nf"] * 80, flops=case["nf"] * 35 * 8 * d ** 3)
    if kind == "solve":
        dim = sum(math.comb(ns, a) * math.comb(ns, b) for a, b in _sectors(case))
        steps, size = 2 * 60, 8
        return dict(bytes=3 * dim * size * steps, flops=dim * 2 * (ns + 3) * steps)
    dim, size = _dim(case), 4 if case.get("dtype") == "f32" else 8
    terms = (2 * ns if "npart" in case else ns) + 1
    if kind in ("hv", "nambu_hv"):
        return dict(bytes=2 * dim * size, flops=2 * dim * terms)
    steps = {"ground": 2 * 60, "grad": 2 * 2 * case.get("steps", 0)}.get(kind, case.get("steps", 0))
    return dict(bytes=3 * dim * size * steps, flops=2 * dim * terms * steps)


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------

def _parity(s, lo, hi):
    """Sign of the occupied bits strictly between lo and hi."""
    v = s & (((1 << hi) - 1) & ~((2 << lo) - 1))
    for k in (16, 8, 4, 2, 1):
        v = v ^ (v >> k)
    return (1 - 2 * (v & 1)).double()


def _popcount_states(bits, n, dev):
    s = torch.arange(1 << bits, device=dev, dtype=torch.int32)
    c = torch.zeros_like(s, dtype=torch.int8)
    for k in range(bits):
        c += ((s >> k) & 1).to(torch.int8)
    return s[c == n].contiguous()


def _hop(states, a, b):
    """(rows, columns, signs) of c+_a c_b over a sorted list of states, a != b."""
    ok = (((states >> b) & 1) == 1) & (((states >> a) & 1) == 0)
    src = torch.nonzero(ok).flatten()
    s = states[src]
    t = (s ^ ((1 << a) | (1 << b))).contiguous()
    return torch.searchsorted(states, t), src, _parity(s, min(a, b), max(a, b))


def _sparse(n, parts, dev):
    if not parts:
        parts = [(torch.zeros(0, dtype=torch.int64, device=dev),) * 2 + (torch.zeros(0, dtype=torch.float64, device=dev),)]
    i = torch.stack([torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])])
    return torch.sparse_coo_tensor(i, torch.cat([p[2] for p in parts]), (n, n)).coalesce().to_sparse_csr()


class _Exact:
    """H of an (N_up, N_dn) sector as sums of Kronecker products of one-spin operators."""

    def __init__(self, m, nup, ndn):
        dev = _dev()
        nb, nc, ns = m.nb, m.nc, m.ns
        self.T, diag, occ, moves = [], [], [], []
        for s, n in ((0, nup), (1, ndn)):
            t = np.zeros((ns, ns))
            t[:nb, :nb], t[nb:, nb:], t[:nb, nb:], t[nb:, :nb] = m.eb[s], m.ec[s], m.vbc[s], m.vbc[s].T
            st = _popcount_states(ns, n, dev)
            parts = []
            for a in range(ns):
                for b in range(ns):
                    if a != b and abs(t[a, b]) > m.cutoff:
                        r, c, g = _hop(st, a, b)
                        parts.append((r, c, g * t[a, b]))
            self.T.append(_sparse(len(st), parts, dev))
            o = torch.stack([((st >> k) & 1).double() for k in range(ns)])
            diag.append((torch.tensor(np.diag(t).copy(), device=dev)[:, None] * o).sum(0))
            occ.append(o[nb:])
            moves.append({(a, b): _sparse(len(st), [_hop(st, nb + a, nb + b)], dev)
                          for a in range(nc) for b in range(nc) if a != b})
        self.D = diag[1][:, None] + diag[0][None, :]
        pairs = [(a, b) for a in range(nc) for b in range(a + 1, nc) if m.u[a, b] != 0]
        for c in range(nc):
            self.D += m.u[c, c] * occ[1][c][:, None] * occ[0][c][None, :]
        for a, b in pairs:
            na = occ[1][a][:, None] + occ[0][a][None, :]
            nb_ = occ[1][b][:, None] + occ[0][b][None, :]
            self.D += m.u[a, b] * na * nb_ - m.jj[a, b] * ((occ[1][a] * occ[1][b])[:, None] +
                                                         (occ[0][a] * occ[0][b])[None, :])
        self.hund = []
        if abs(m.jhund) > 1e-5:
            for a, b in pairs:
                for p, q in ((a, b), (b, a)):
                    self.hund.append((float(m.jj[p, q]), moves[0][p, q], moves[1][q, p]))   # spin flip
                    self.hund.append((float(m.jj[p, q]), moves[0][p, q], moves[1][p, q]))   # pair hopping
        self.shape = tuple(self.D.shape)

    def up(self, A, x):
        return (A @ x.t().contiguous()).t()

    def __call__(self, v):
        x = v.view(self.shape)
        y = self.D * x
        y += self.T[1] @ x
        y += self.up(self.T[0], x)
        for j, u, d in self.hund:
            y += j * (d @ self.up(u, x).contiguous())
        return y.reshape(-1)


class _ExactSz:
    """H of a Nambu sector: one species of 2*ns orbitals, particle-hole transformed down spins."""

    def __init__(self, nm, npart, keep):
        m, dev = nm.base, _dev()
        nb, ns = m.nb, m.ns
        t = _nambu_matrix(nm)
        self.st = _popcount_states(2 * ns, npart, dev)
        self.terms = [(a, b, t[a, b]) for a in range(2 * ns) for b in range(2 * ns) if a != b and abs(t[a, b]) > m.cutoff]
        self.D = torch.zeros(len(self.st), dtype=torch.float64, device=dev)
        for o in range(2 * ns):
            self.D += float(t[o, o]) * ((self.st >> o) & 1).double()
        self.D += float(m.u[0, 0]) * (((self.st >> nb) & 1) * (1 - ((self.st >> (ns + nb)) & 1))).double()
        self.A = None
        if keep:
            self.A = _sparse(len(self.st), [(r, c, g * h) for r, c, g, h in
                                            ((*_hop(self.st, a, b), h) for a, b, h in self.terms)], dev)

    def __call__(self, v):
        y = self.D * v
        if self.A is not None:
            return y + self.A @ v
        for a, b, h in self.terms:
            r, c, g = _hop(self.st, a, b)
            y[r] += h * g * v[c]
        return y


def _lanczos(op, v, steps, keep=False):
    """Plain Lanczos: |v|, alpha, beta (and the vectors, orthogonalised against each other when kept)."""
    nrm = float(v.norm())
    v = v / nrm
    al, be, V, prev = [], [], [v], torch.zeros_like(v)
    for k in range(steps):
        w = op(v)
        if be:
            w -= be[-1] * prev
        a = float(w @ v)
        w -= a * v
        if keep:
            Q = torch.stack(V)
            for _ in range(2):
                w -= Q.t() @ (Q @ w)
        al.append(a)
        b = float(w.norm())
        if k == steps - 1 or b < 1e-12 * abs(a) + 1e-14:
            break
        be.append(b)
        prev, v = v, w / b
        if keep:
            V.append(v)
    return nrm, np.array(al), np.array(be), V


def _cf(nrm, al, be, z):
    g = np.zeros_like(z)
    for k in range(len(al) - 1, -1, -1):
        g = 1.0 / (z - al[k] - (be[k] ** 2 * g if k < len(be) else 0.0))
    return nrm ** 2 * g


def _ground(op, dim, seed=3):
    """Lowest eigenpair by restarted Lanczos with full orthogonalisation."""
    if dim == 1:
        v = torch.ones(1, dtype=torch.float64, device=_dev())
        return float(op(v)[0]), v
    v = _noise(dim, seed, torch.float64)
    for _ in range(40):
        _, al, be, V = _lanczos(op, v, min(dim, 80), keep=True)
        e, c = np.linalg.eigh(np.diag(al) + np.diag(be[:len(al) - 1], 1) + np.diag(be[:len(al) - 1], -1))
        v = torch.tensor(c[:, 0], device=_dev()) @ torch.stack(V[:len(al)])
        v /= v.norm()
        r = op(v)
        e0 = float(r @ v)
        if float((r - e0 * v).norm()) < 3e-13 * max(1.0, abs(e0)) * 4:
            break
    return e0, v


def _apply(m, nup, ndn, spin, create, site, x):
    """c+ or c of one impurity orbital (per-spin Jordan-Wigner order)."""
    n = (nup, ndn)[spin]
    dev, bit = _dev(), m.nb + site
    src = _popcount_states(m.ns, n, dev)
    tgt = _popcount_states(m.ns, n + (1 if create else -1), dev)
    ok = ((src >> bit) & 1) == (0 if create else 1)
    i = torch.nonzero(ok).flatten()
    s = src[i]
    j = torch.searchsorted(tgt, (s ^ (1 << bit)).contiguous())
    sg = _parity(s, bit, m.ns)
    x = x.view(-1, math.comb(m.ns, nup))
    if spin == 0:
        y = torch.zeros((x.shape[0], len(tgt)), dtype=x.dtype, device=dev)
        y[:, j] = x[:, i] * sg
    else:
        y = torch.zeros((len(tgt), x.shape[1]), dtype=x.dtype, device=dev)
        y[j] = x[i] * sg[:, None]
    return y.reshape(-1)


def _exact_solve(case, seed):
    m = _model(case, seed)
    z = 1j * matsubara(BETA, case["nw"])
    found = []
    for nu, nd in _sectors(case):
        op = _Exact(m, nu, nd)
        e, v = _ground(op, math.comb(m.ns, nu) * math.comb(m.ns, nd))
        found.append((e, nu, nd, v))
    e0 = min(f[0] for f in found)
    kept = [f for f in found if f[0] <= e0 + 5.0 / BETA]
    Z = sum(math.exp(-BETA * (f[0] - e0)) for f in kept)
    G = np.zeros((2, m.nc, case["nw"]), complex)
    for e, nu, nd, v in kept:
        w = math.exp(-BETA * (e - e0)) / Z
        for spin in (0, 1):
            for create in (True, False):
                d = 1 if create else -1
                tu, td = (nu + d, nd) if spin == 0 else (nu, nd + d)
                if not (0 <= tu <= m.ns and 0 <= td <= m.ns):
                    continue
                op = _Exact(m, tu, td)
                for c in range(m.nc):
                    r = _lanczos(op, _apply(m, nu, nd, spin, create, c, v), min(case["steps"], op.D.numel()))
                    g = _cf(r[0], r[1], r[2], (z if create else -z) + e)
                    G[spin, c] += w * (g if create else -g)
    return dict(e0=e0, z=Z, G=G, docc=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("vertex", "grad"):
        # 35 four-state sums, and a derivative through a ground state: no short 64-bit form
        return None
    if kind == "solve":
        return _exact_solve(case, seed)
    if kind in ("hv", "green", "ground"):
        m = _model(case, seed)
        op = _Exact(m, case["nup"], case["ndn"])
        if kind == "ground":
            return dict(e0=_ground(op, _dim(case))[0], psi=None)      # the eigenvector's sign is free
        if kind == "hv":
            return op((_noise(_dim(case), seed, _tdtype(case)) / math.sqrt(_dim(case))).double())
        x, e0 = _start(case, seed, _tdtype(case)).double(), _e0(m, case["nup"], case["ndn"])
    else:
        op = _ExactSz(_nambu(case, seed), case["npart"], kind == "nambu_green")
        if kind == "nambu_hv":
            return op((_noise(_dim(case), seed, _tdtype(case)) / math.sqrt(_dim(case))).double())
        x, e0 = _nambu_start(case, seed)
        x = x.double()
    r = _lanczos(op, x, min(case["steps"], _dim(case)))
    return _cf(r[0], r[1], r[2], 1j * matsubara(BETA, case["nw"]) + e0)
