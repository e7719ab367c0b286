"""The work that is timed: what a program that uses this library has it do, at the sizes it does it.

Strings come in three families, the ones this repository is tested and benchmarked on:

* ``fci``   every string of the orbital space (all C(norb, n): the 8- and 12-orbital full CI sets);
* ``sci``   synthetic selected sets (``synth.py``'s law: weight 0.3^k for excitation rank k from the
            Hartree-Fock string), about one single and tens of doubles per string;
* ``mol``   sets selected the way a molecule's are: the strings of lowest orbital-energy sum with
            some spread.  Their singles and doubles per string (39 / 403 at 18 orbitals, 7 electrons,
            4,041 strings; 48 / 574 at 24 orbitals, 5 electrons, 5,514) are those of the published
            N2 (40.9 / 410) and H2O (51.1 / 622) sets of the same sizes.

Integrals are ``synth.py``'s, from the seed.  Vectors are random numbers damped by the excitation
rank of both strings, normalised, as CI vectors are: the large entries sit on few determinants.
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sbd-pub_b200", "python")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import sbd_tpb  # noqa: E402
import synth  # noqa: E402
ORBITAL_GAP = 5.0
REPULSION = 0.4


def _case(name, kind, family, norb, na_el, nb_el, na, nb, dtype, form="", **more):
    c = dict(kind=kind, family=family, norb=norb, na_el=na_el, nb_el=nb_el, na=na, nb=nb, dtype=dtype, form=form)
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a 4,900-determinant full CI, as in unit tests and embedding loops: one sigma is a few short
        # launches, so the call itself is what costs
        _case("sigma_fci8_f64", "sigma", "fci", 8, 4, 4, 70, 70, "f64", "general"),
        # the 12-orbital full CI (853,776 determinants), FP64: dense singles and doubles in a small vector
        _case("sigma_fci12_f64", "sigma", "fci", 12, 6, 6, 924, 924, "f64", "general"),
        # the same space in the step of a mixed-precision solve: FP32, exchange-symmetric vector
        _case("sigma_fci12_sym_f32", "sigma", "fci", 12, 6, 6, 924, 924, "f32", "symmetric"),
        # a host program that calls sigma on its own (pinned) memory in the reference's convention, with
        # unequal electron and string counts and odd rows
        _case("sigma_sci24_host_f64", "sigma", "sci", 24, 8, 7, 4001, 2999, "f64", "host"),
        # one step of a mixed solve at 1e8 determinants
        _case("sigma_sci28_sym_f32", "sigma", "sci", 28, 9, 9, 10000, 10000, "f32", "symmetric"),
        # the benchmark's headline sigma: 4e8 determinants, FP64
        _case("sigma_sci32_f64", "sigma", "sci", 32, 10, 10, 20000, 20000, "f64", "general"),
        # sigma on a molecular set of the size of the published N2 1e-5 one (1.6e7 determinants, odd rows)
        _case("sigma_mol18_f64", "sigma", "mol", 18, 7, 7, 4041, 4041, "f64", "general"),
        # one step of a mixed solve on a set of the size of the published H2O 1e-5 one (3.0e7 determinants)
        _case("sigma_mol24_sym_f32", "sigma", "mol", 24, 5, 5, 5514, 5514, "f32", "symmetric"),
        # a Davidson cycle of ten steps from the Hartree-Fock determinant on a set of the size of the
        # published N2 1e-4 one (1.9e6 determinants), with the CI vector read back
        _case("davidson_mol18_f64", "davidson", "mol", 18, 7, 7, 1387, 1387, "f64", steps=10, vector=True),
        # ten mixed-precision steps at 1.6e7 determinants, energy and occupations only
        _case("davidson_sci24_mixed", "davidson", "sci", 24, 8, 8, 4000, 4000, "mixed", steps=10, vector=False),
        # the whole application on a small molecule: tables, solve, CI vector and RDMs in one call
        _case("diag_mol18_rdm_f64", "diag", "mol", 18, 7, 7, 642, 642, "f64", steps=10),
        # 1- and 2-RDMs of a vector held by the host
        _case("rdm_mol18", "rdm", "mol", 18, 7, 7, 1387, 1387, "f64"),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sigma", "sigma", "sigma", "sigma", "davidson", "davidson", "diag", "rdm"])
    family = rng.choice(["fci", "sci", "sci", "mol", "mol", "mol"]) if kind == "sigma" else rng.choice(["sci", "mol"])
    if family == "fci":
        norb, n = rng.choice([(8, 4), (9, 4), (10, 5), (11, 5), (12, 6), (12, 5)])
        na = nb = math.comb(norb, n)
        ea = eb = n
    elif family == "sci":
        norb = rng.randint(20, 34)
        ea = rng.randint(6, norb // 3)
        na = logint(300, {"sigma": 16000, "davidson": 6000}.get(kind, 2000))
        eb, nb = ea, na
    else:
        norb = rng.randint(16, 26)
        ea = {16: 6, 17: 6, 18: 7, 19: 6, 20: 6}.get(norb, 5)
        na = logint(150, {"sigma": 3900, "davidson": 1300}.get(kind, 600))
        eb, nb = ea, na
    form = ""
    if kind == "sigma":
        form = rng.choice(["general", "general", "symmetric", "symmetric", "host"])
        if form == "host":
            na = nb = min(na, 3000) if family != "fci" else na
        if family != "fci" and form != "symmetric" and rng.random() < 0.5:
            eb = max(3, ea - rng.randint(0, 2))
            nb = max(100, int(na * rng.uniform(0.4, 1.0)))
    dtype = rng.choice(["f64", "f32"]) if kind == "sigma" else rng.choice(["f64", "mixed"]) if kind == "davidson" else "f64"
    more = {}
    if kind in ("davidson", "diag"):
        more["steps"] = rng.randint(5, 10)
    if kind == "davidson":
        more["vector"] = rng.random() < 0.5
    return _case("", kind, family, norb, ea, eb, na, nb, dtype, form, **more)


# ---- inputs -------------------------------------------------------------------------------------


def _sci_strings(norb, n, count, rng):
    """The Hartree-Fock string and distinct strings of excitation rank k with weight 0.3^k."""
    kmax = min(n, norb - n)
    ks = np.arange(1, kmax + 1)
    w = np.array([math.comb(n, int(k)) * math.comb(norb - n, int(k)) * 0.3 ** int(k) for k in ks])
    got = np.array([(1 << n) - 1], np.uint64)
    while len(got) < count:
        m = 2 * (count - len(got)) + 64
        k = rng.choice(ks, size=m, p=w / w.sum())
        holes = np.argsort(rng.random((m, n)), axis=1)[:, :kmax].astype(np.uint64)
        parts = (np.argsort(rng.random((m, norb - n)), axis=1)[:, :kmax] + n).astype(np.uint64)
        use = (np.arange(kmax)[None, :] < k[:, None]).astype(np.uint64)
        flip = np.bitwise_or.reduce((use << holes) | (use << parts), axis=1)
        new = np.setdiff1d(got[0] ^ flip, got)
        got = np.concatenate([got, rng.permutation(new)[: count - len(got)]])
    return np.sort(got)


def _mol_strings(norb, n, count, rng):
    """The Hartree-Fock string and the strings of lowest sum of equally spaced orbital energies, with noise."""
    idx = np.fromiter(itertools.chain.from_iterable(itertools.combinations(range(norb), n)), np.int64).reshape(-1, n)
    s = (np.int64(1) << idx).sum(axis=1).astype(np.uint64)
    score = idx.sum(axis=1) + 2.0 * rng.gumbel(size=len(s))
    score[0] = -np.inf
    return np.sort(s[np.argsort(score, kind="stable")[: min(count, len(s))]])


def _strings(case, spin, seed):
    norb, n, count = case["norb"], case["nb_el" if spin else "na_el"], case["nb" if spin else "na"]
    same = (case["na_el"], case["na"]) == (case["nb_el"], case["nb"])
    rng = np.random.default_rng([seed, 11, 0 if same else spin])
    if case["family"] == "sci" and count < math.comb(norb, n):
        return _sci_strings(norb, n, count, rng)
    if case["family"] == "mol":
        return _mol_strings(norb, n, count, rng)
    return synth.sample_strings(norb, n, count)


def _problem(case, seed):
    h1, eri, core = synth.synthetic_hamiltonian(case["norb"], seed=1729 + seed)
    if "steps" in case:
        # a solve: orbital energies that outweigh the random repulsion, as a molecule's do, so that the
        # Hartree-Fock determinant is the lowest one and no E - H_ii comes near zero
        h1 = h1 + np.diag(ORBITAL_GAP * np.arange(case["norb"]))
        eri *= REPULSION
    return sbd_tpb.Problem(norb=case["norb"], nelec=case["na_el"] + case["nb_el"], core=core, h1=h1,
                           eri_packed=eri, astr=_strings(case, 0, seed), bstr=_strings(case, 1, seed))


def _vector(case, prob, seed):
    """[na, nb] float64 on the GPU: N(0, 1) times 0.5^(rank of both strings), norm 1."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(len(prob.astr), len(prob.bstr), dtype=torch.float64, device="cuda", generator=g)
    for s, shape in ((prob.astr, (-1, 1)), (prob.bstr, (1, -1))):
        rank = np.bitwise_count(s & ~np.uint64(s[0])).astype(np.float64)
        x *= torch.from_numpy(0.5 ** rank).cuda().reshape(shape)
    if case["form"] == "symmetric":
        x = x + x.T
    return x.div_(x.norm())


def _params(case):
    """A solve from the Hartree-Fock determinant of a fixed number of steps."""
    return sbd_tpb.default_params(max_it=1, max_nb=case["steps"], eps=1e-14,
                                  precision=sbd_tpb.MIXED if case["dtype"] == "mixed" else sbd_tpb.FP64)


def prepare(case, seed):
    prob = _problem(case, seed)
    st = dict(case=case, prob=prob)
    if case["kind"] == "diag":  # one call does everything
        st["params"] = _params(case)
        return st
    h = sbd_tpb.Handle(torch.cuda.current_device())
    h.set_problem(prob)
    st["handle"] = h
    if case["kind"] == "davidson":
        st["params"] = _params(case)
        return st
    x = _vector(case, prob, seed)
    if case["dtype"] == "f32":
        x = x.float()
    x = x.contiguous().reshape(-1)
    if case["kind"] == "rdm":
        st["W"] = x.cpu().numpy()
    elif case["form"] == "host":
        st["C"] = x.cpu().pin_memory().numpy()
        st["out"] = torch.zeros(x.numel(), dtype=x.dtype, pin_memory=True).numpy()
    else:
        st["C"], st["out"] = x, torch.zeros_like(x)
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "sigma":
        if case["form"] == "host":
            return state["handle"].sigma(state["C"], state["out"])
        return state["handle"].sigma_device(state["C"], state["out"], symmetric=case["form"] == "symmetric")
    if case["kind"] == "davidson":
        r = state["handle"].davidson(state["params"], want_vector=case["vector"])
        out = dict(energy=r["energy"], density=r["density"])
        if case["vector"]:
            out["W"] = r["W"]
        return out
    if case["kind"] == "diag":
        r = sbd_tpb.diag(state["prob"], state["params"], want_rdm=True)
        return dict(energy=r["energy"], density=r["density"], W=r["W"], one=r["one"], two=r["two"])
    one, two = state["handle"].rdm(state["W"])
    return dict(one=one, two=two)


# ---- what a pass cannot do without -----------------------------------------------------------------


def _connections(s):
    """Mean singles and doubles of a string, from up to 256 rows."""
    rows = s if len(s) <= 256 else s[np.linspace(0, len(s) - 1, 256).astype(int)]
    d = np.bitwise_count(rows[:, None] ^ s[None, :])
    return float((d == 2).sum()) / len(rows), float((d == 4).sum()) / len(rows)


def work(case):
    """One sigma reads C and writes sigma; it multiplies and adds once per connected pair (same-spin
    singles and doubles of each spin, and alpha-single x beta-single pairs) and once for the diagonal.
    A solve is its sigmas; the RDMs multiply and add once per connected pair of determinants."""
    a, b = _strings(case, 0, 0), _strings(case, 1, 0)
    n = float(len(a)) * len(b)
    (sa, da), (sb, db) = _connections(a), _connections(b)
    flops = 2.0 * n * (1.0 + sa + da + sb + db + sa * sb)
    size = 8 if case["dtype"] == "f64" else 4
    if case["kind"] == "sigma":
        return {"bytes": 2 * n * size, "flops": flops}
    rdm = 4 * 8.0 * case["norb"] ** 4
    if case["kind"] == "rdm":
        return {"bytes": n * 8 + rdm, "flops": flops}
    k = case["steps"]
    solve = {"bytes": 2 * n * size * k + 2 * n * 8, "flops": flops * (k + 1)}
    if case["kind"] == "diag":
        return {"bytes": solve["bytes"] + rdm + n * 8, "flops": solve["flops"] + flops}
    return solve


def tolerance(case):
    # about four times the largest difference from exact() that the cases show: rounding of sums taken
    # in another order (FP64 sigma 2.4e-16, RDMs 1.2e-15, FP32 sigma 8.5e-8), carried through the
    # steps of a solve
    if case["kind"] == "sigma":
        return {"rel": 1e-15} if case["dtype"] == "f64" else {"rel": 4e-7}
    if case["kind"] == "rdm":
        return {"rel": 5e-15}
    return {"rel": 1e-12} if case["dtype"] == "f64" else {"rel": 1e-5}


# ---- the same in plain torch, 64 bits ----------------------------------------------------------------


def _popc(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    return ((x * 0x0101010101010101) >> 56) & 0xFF


def _low(x):  # index of the lowest set bit
    return _popc((x & -x) - 1)


def _moved(I, p, q):
    """Sign of moving an electron of string I from orbital p to orbital q."""
    lo, hi = torch.minimum(p, q), torch.maximum(p, q)
    one = torch.ones_like(I)
    between = ((one << hi) - 1) & ~((one << (lo + 1)) - 1)
    return (1 - 2 * (_popc(I & between) & 1)).double()


class _Spin:
    """Connected pairs of one spin's strings: singles (bra, ket, cr, an, sign) and the matrix of
    everything that does not depend on the other spin."""

    def __init__(self, strings, h1, g):
        s = torch.from_numpy(strings.astype(np.int64)).cuda()
        self.s, self.n, L = s, len(s), h1.shape[0]
        self.occ = ((s[:, None] >> torch.arange(L, device="cuda")[None, :]) & 1).double()
        jd = torch.einsum("ppqq->pq", g) - torch.einsum("pqqp->pq", g)
        self.e = self.occ @ torch.diagonal(h1) + 0.5 * torch.einsum("ip,pq,iq->i", self.occ, jd, self.occ)
        bra, ket, bra2, ket2 = [], [], [], []
        step = max(1, 20_000_000 // self.n)
        for r in range(0, self.n, step):
            d = _popc(s[r:r + step, None] ^ s[None, :])
            for which, bb, kk in ((2, bra, ket), (4, bra2, ket2)):
                i, j = torch.nonzero(d == which, as_tuple=True)
                bb.append(i + r)
                kk.append(j)
            del d
        self.bra, self.ket = torch.cat(bra), torch.cat(ket)
        I, J = s[self.bra], s[self.ket]
        self.cr, self.an = _low(I & ~J), _low(J & ~I)
        self.sign = _moved(I, self.cr, self.an)
        pair = torch.einsum("pqkk->pqk", g) - torch.einsum("pkkq->pqk", g)  # (pq|kk) - (pk|kq)
        v1 = self.sign * (h1[self.an, self.cr] + (pair[self.an, self.cr] * self.occ[self.bra]).sum(1))
        self.bra2, self.ket2 = torch.cat(bra2), torch.cat(ket2)
        I, J = s[self.bra2], s[self.ket2]
        c, a = I & ~J, J & ~I
        c0, a0 = _low(c), _low(a)
        c1, a1 = _low(c & (c - 1)), _low(a & (a - 1))
        one = torch.ones_like(I)
        self.sign2 = _moved(I, c0, a0) * _moved(I ^ (one << c0) ^ (one << a0), c1, a1)
        self.lab2 = (c0, c1, a0, a1)
        v2 = self.sign2 * (g[a0, c0, a1, c1] - g[a0, c1, a1, c0])
        self.H = _csr(torch.cat([self.bra, self.bra2]), torch.cat([self.ket, self.ket2]), torch.cat([v1, v2]), self.n)


def _csr(i, j, v, n):
    return torch.sparse_coo_tensor(torch.stack([i, j]), v, (n, n)).coalesce().to_sparse_csr()


class _Exact:
    def __init__(self, prob):
        L = prob.norb
        self.L, self.core = L, prob.core
        self.h1 = torch.from_numpy(np.asarray(prob.h1)).cuda()
        self.g = torch.from_numpy(synth.unpack_eri(prob.eri_packed, L)).cuda()
        self.a = _Spin(prob.astr, self.h1, self.g)
        same = len(prob.astr) == len(prob.bstr) and bool((prob.astr == prob.bstr).all())
        self.b = self.a if same else _Spin(prob.bstr, self.h1, self.g)
        self.J = torch.einsum("ppqq->pq", self.g)
        # sign of the reference's interleaved determinant against alpha-then-beta: a beta electron
        # passes every alpha electron of a higher orbital
        above = self.a.occ.flip(1).cumsum(1).flip(1) - self.a.occ
        self.D = 1 - 2 * torch.remainder(above @ self.b.occ.T, 2) if len(prob.astr) * len(prob.bstr) < 5e7 else None
        self.hii = self.a.occ @ self.J @ self.b.occ.T + self.core
        self.hii += self.a.e[:, None] + self.b.e[None, :]
        self.pairs = [(x, y) for x in range(L) for y in range(L) if x != y]

    def sigma(self, C):
        out = self.hii * C
        out += torch.sparse.mm(self.a.H, C)
        for spin, other, X, flip in ((self.b, self.a, C.T.contiguous(), True), (self.a, self.b, C, False)):
            acc = torch.sparse.mm(spin.H, X) if flip else torch.zeros_like(X)
            key = spin.an * self.L + spin.cr
            order = torch.argsort(key, stable=True)
            cut = torch.searchsorted(key[order], torch.arange(self.L ** 2 + 1, device="cuda")).tolist()
            jk = torch.einsum("pqkk->pqk", self.g)
            for pq in range(self.L ** 2):
                if cut[pq + 1] == cut[pq]:
                    continue
                e = order[cut[pq]:cut[pq + 1]]
                an, cr = divmod(pq, self.L)
                Y = X[spin.ket[e]]
                # the other spin's number operators ...
                z = Y * (other.occ @ jk[an, cr])[None, :]
                if not flip and len(other.bra):  # ... and, once, its singles
                    M = _csr(other.bra, other.ket, other.sign * self.g[an, cr][other.an, other.cr], other.n)
                    z += torch.sparse.mm(M, Y.T.contiguous()).T
                acc.index_add_(0, spin.bra[e], z * spin.sign[e][:, None])
            out += acc.T if flip else acc
        return out

    def davidson(self, steps):
        C = torch.zeros_like(self.hii)
        C[0, 0] = 1.0
        S, H = [C], []
        for k in range(steps):
            H.append(self.sigma(S[k]))
            T = torch.tensor([[float((x * y).sum()) for y in H] for x in S], dtype=torch.float64)
            w, u = torch.linalg.eigh(0.5 * (T + T.T))
            u0 = u[:, 0].tolist()
            W = sum(c * x for c, x in zip(u0, S))
            if k + 1 < steps:
                r = sum(c * x for c, x in zip(u0, H)) - float(w[0]) * W
                d = float(w[0]) - self.hii
                t = torch.where(d.abs() > 1e-12, r / d, r / (d - 1e-12))
                for _ in range(2):
                    for x in S:
                        t -= float((x * t).sum()) * x
                S.append(t / t.norm())
        W = W / W.norm()
        return W if W[0, 0] > 0 else -W

    def energy(self, W):
        return float((W * self.sigma(W)).sum())

    def density(self, W):
        w2 = W * W
        return torch.stack([self.a.occ.T @ w2.sum(1), self.b.occ.T @ w2.sum(0)], 1).reshape(-1)

    def rdm(self, W):
        """(one, two) laid out as sbd_tpb_rdm does: one[s][p + L q], two[s + 2 t][p + L q + L^2 r + L^3 u]."""
        L = self.L
        one = torch.zeros(2, L, L, dtype=torch.float64, device="cuda")        # [s, q, p]
        two = torch.zeros(2, 2, L, L, L, L, dtype=torch.float64, device="cuda")  # [t, s, u, r, q, p]

        def put(s, t, p, q, r, u, x):
            flat = ((((t * 2 + s) * L + u) * L + r) * L + q) * L + p
            two.view(-1).index_add_(0, flat.reshape(-1), x.reshape(-1))

        ar = torch.arange(L, device="cuda")
        for s, spin, other, X in ((0, self.a, self.b, W), (1, self.b, self.a, W.T.contiguous())):
            rho = (X * X).sum(1)
            n2 = torch.einsum("i,ip,iq->pq", rho, spin.occ, spin.occ)
            one[s, ar, ar] += rho @ spin.occ
            n2.fill_diagonal_(0.0)
            p, q = torch.meshgrid(ar, ar, indexing="ij")
            put(s, s, p, q, p, q, n2)
            put(s, s, p, q, q, p, -n2)
            if s == 0:
                m = spin.occ.T @ (X * X) @ other.occ
                put(0, 1, p, q, p, q, m)
                put(1, 0, q, p, q, p, m)
            gram = X @ X.T
            x = spin.sign * gram[spin.bra, spin.ket]
            one[s].view(-1).index_add_(0, spin.an * L + spin.cr, x)
            # a single with a number operator of its own spin, then of the other
            nj = spin.occ[spin.bra].clone()
            nj[torch.arange(len(spin.bra), device="cuda"), spin.cr] = 0.0
            key = spin.an * L + spin.cr
            acc = torch.zeros(L * L, L, dtype=torch.float64, device="cuda").index_add_(0, key, nj * x[:, None])
            oth = torch.zeros_like(acc)
            for e in torch.split(torch.arange(len(spin.bra), device="cuda"), max(1, 50_000_000 // X.shape[1])):
                oth.index_add_(0, key[e], spin.sign[e][:, None] * ((X[spin.bra[e]] * X[spin.ket[e]]) @ other.occ))
            an, cr, j = torch.meshgrid(ar, ar, ar, indexing="ij")
            for t, z in ((s, acc), (1 - s, oth)):
                z = z.reshape(L, L, L)
                put(s, t, cr, j, an, j, z)
                put(t, s, j, cr, j, an, z)
            z = acc.reshape(L, L, L)
            put(s, s, cr, j, j, an, -z)
            put(s, s, j, cr, an, j, -z)
            c0, c1, a0, a1 = spin.lab2
            x = spin.sign2 * gram[spin.bra2, spin.ket2]
            put(s, s, c0, c1, a0, a1, x)
            put(s, s, c1, c0, a1, a0, x)
            put(s, s, c0, c1, a1, a0, -x)
            put(s, s, c1, c0, a0, a1, -x)
        # alpha single x beta single, placed by the spin-orbital order of the four indices
        a, b = self.a, self.b
        if len(a.bra) and len(b.bra):
            bkey = b.an * L + b.cr
            X2 = torch.zeros(L * L, L * L, dtype=torch.float64, device="cuda")
            akey = a.an * L + a.cr
            for pq in torch.unique(akey).tolist():
                e = torch.nonzero(akey == pq)[:, 0]
                # P[Ib, Jb] = sum_e sign W[Ia, Ib] W[Ja, Jb], then summed by the label of (Ib, Jb)
                P = (W[a.bra[e]] * a.sign[e][:, None]).T @ W[a.ket[e]]
                X2[pq].index_add_(0, bkey, b.sign * P[b.bra, b.ket])
            ana, cra, anb, crb = torch.meshgrid(ar, ar, ar, ar, indexing="ij")
            x = X2.reshape(L, L, L, L)
            i, jj, aa, bb = 2 * cra, 2 * crb + 1, 2 * ana, 2 * anb + 1
            I, J = torch.minimum(i, jj), torch.maximum(i, jj)
            A, B = torch.minimum(aa, bb), torch.maximum(aa, bb)
            si, sj, sa = I % 2, J % 2, A % 2
            oi, oj, oa, ob = I // 2, J // 2, A // 2, B // 2
            r1, u1 = torch.where(si == sa, oi, oj), torch.where(si == sa, oj, oi)
            put(si, sj, oa, ob, r1, u1, x)
            put(sj, si, ob, oa, u1, r1, x)
        return one.reshape(-1).cpu().numpy(), two.reshape(-1).cpu().numpy()


def exact(case, seed):
    prob = _problem(case, seed)
    X = _Exact(prob)
    if case["kind"] in ("sigma", "rdm"):
        C = _vector(case, prob, seed)
        if case["dtype"] == "f32":
            C = C.float().double()
        if case["form"] == "host" or case["kind"] == "rdm":
            C = C * X.D  # vectors that cross the host boundary are in the reference's convention
        if case["kind"] == "rdm":
            one, two = X.rdm(C)
            return dict(one=one, two=two)
        y = X.sigma(C)
        return (y * X.D if case["form"] == "host" else y).reshape(-1).cpu().numpy()
    W = X.davidson(case["steps"])
    out = dict(energy=X.energy(W), density=X.density(W).cpu().numpy())
    if case["kind"] == "diag" or case["vector"]:
        out["W"] = (W * X.D).reshape(-1).cpu().numpy()
    if case["kind"] == "diag":
        out["one"], out["two"] = X.rdm(W)
    return out
