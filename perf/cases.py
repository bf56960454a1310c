"""The engine's work as its users have it do it, one case per kind of call and size.

Systems are the ones of the tests and the benchmark: periodic XXZ chains, J1-J2
chains and square-lattice tori at fixed Sz, reduced by translations and, where
the sector is half filled, spin inversion.  Every case goes through the
package's public classes (Sector, Hamiltonian, Batch) or the C ABI entry point
that a driver of the reference calls.  Random inputs (vectors, anisotropies,
coupling sets) come from the seed.  exact() restates the physics in FP64 torch
on bit strings, without the package.
"""
import ctypes
import math

import numpy as np
import torch

import qmbcuda_b200 as q

A = q._capi
_DEV = "cuda"


# ------------------------------------------------------------------ systems
def _sys(case):
    """(L, n_up, N1, N2) of a case; a chain is N1 = L, N2 = 1."""
    N1, N2 = case["N1"], case["N2"]
    return N1 * N2, (N1 * N2) // 2, N1, N2


def _bonds(case):
    """[(site, site)] and the coupling of each."""
    L, _, N1, N2 = _sys(case)
    if N2 > 1:
        b = []
        for i in range(N1):
            for j in range(N2):
                b += [(i * N2 + j, ((i + 1) % N1) * N2 + j), (i * N2 + j, i * N2 + (j + 1) % N2)]
        return b, [1.0] * len(b)
    b = [(i, (i + 1) % L) for i in range(L)]
    J = [1.0] * L
    if case["model"] == "j1j2":
        b += [(i, (i + 2) % L) for i in range(L)]
        J += [0.5] * L
    return b, J


def _delta(case, seed):
    """The Sz Sz anisotropy: near the case's value, from the seed."""
    return case["delta"] * (1.0 + 0.02 * float(np.random.default_rng(seed).uniform(-1, 1)))


def _chars(case):
    """Characters over e = z * G + g of the case's momentum (and, with flip, even inversion parity)."""
    _, _, N1, N2 = _sys(case)
    kx, ky = divmod(case["k"], N2)
    c = np.array([np.exp(2j * np.pi * (kx * a / N1 + ky * b / N2)) for a in range(N1) for b in range(N2)])
    return np.concatenate([c, c]) if case["flip"] else c


def _real(case):
    return bool(np.abs(_chars(case).imag).max() < 1e-12)


def _group(case):
    """(permutations, case's character row) as a user takes them from the package."""
    _, _, N1, N2 = _sys(case)
    perm, ch = q.translation_group(N1, N2)
    row = ch[case["k"]]
    return perm, (q.with_spin_flip(row, 1) if case["flip"] else row)


def _sector(case):
    L, n_up, _, _ = _sys(case)
    perm, row = _group(case)
    return q.Sector(L, n_up, perm, spin_flip=case["flip"]).set_irrep(row)


def _terms(case, seed):
    b, J = _bonds(case)
    d = _delta(case, seed)
    return q.xxz_terms(b, J, [j * d for j in J])


def _dtype(case):
    if _real(case):
        return torch.float64 if case["prec"] == 64 else torch.float32
    return torch.complex128 if case["prec"] == 64 else torch.complex64


def _prec(case):
    return A.PREC_FP64 if case["prec"] == 64 else A.PREC_FP32


def _vector(n, dtype, seed):
    g = torch.Generator(device=_DEV).manual_seed(1000 + seed)
    return torch.randn(n, dtype=dtype, device=_DEV, generator=g)


# -------------------------------------------------------------------- cases
def _case(kind, N1, N2=1, model="xxz", k=0, flip=False, prec=64, delta=1.0, **more):
    return dict(kind=kind, N1=N1, N2=N2, model=model, k=k, flip=flip, prec=prec, delta=delta, **more)


def listed():
    return [
        # One product of a small momentum sector inside somebody's own solver or
        # time evolution: launch latency is all there is.
        dict(_case("hv", 20, k=3), name="hv_chain20_k3_c64"),
        # The stored product of a mid-sized complex sector (vectors in L2).
        dict(_case("hv", 4, 6, k=8, prec=32), name="hv_torus4x6_c32"),
        # The stored product where the entries stream from HBM, in both precisions.
        dict(_case("hv", 32, model="j1j2", flip=True, prec=32), name="hv_j1j2_32_f32"),
        dict(_case("hv", 30, model="j1j2", k=0, prec=64), name="hv_j1j2_30_f64"),
        # The matrix-free product, for sectors whose matrix is not kept: the
        # benchmark's 32-site J1-J2 chain, and a complex torus sector in FP64.
        dict(_case("mf", 32, model="j1j2", flip=True, prec=32), name="mf_j1j2_32_f32"),
        dict(_case("mf", 4, 6, k=8, prec=64), name="mf_torus4x6_c64"),
        # A new sector and its matrix, as a driver builds them for every lattice,
        # momentum and filling before the first product.
        dict(_case("build", 28, model="j1j2", flip=True, prec=32), name="build_j1j2_28"),
        # A whole ground-state solve of one sector whose vectors fit L2.
        dict(_case("solve", 24, flip=True, delta=0.5, mode=A.MODE_FP64), name="solve_chain24_f64"),
        # Full reorthogonalisation for a fixed number of steps on a sector without
        # symmetry; returns the state too.
        dict(_case("reorth", 16, sym=False, steps=150), name="reorth_chain16"),
        # Many coupling sets over all momenta: the batched mixed-precision solve.
        dict(_case("batch", 20, sets=128, mode=A.MODE_MIXED), name="batch_chain20_128_mixed"),
        # Structure factor at every momentum and the correlators from site 0.
        dict(_case("expval", 24, hops=0), name="expval_chain24"),
        # The reference driver's own call: fixed FP32 Lanczos steps on a caller's
        # row-major ELL.
        dict(_case("ref_ell", 20, k=7, steps=50), name="ref_ell_chain20_k7"),
    ]


def draw(rng):
    kind = rng.choice(["hv", "hv", "mf", "build", "solve", "reorth", "batch", "expval", "ref_ell"])
    prec = rng.choice([32, 64])
    delta = round(rng.uniform(0.3, 1.7), 2)
    if rng.random() < 0.3 and kind in ("hv", "mf", "build", "solve", "expval"):
        N1, N2 = rng.choice([(3, 4), (4, 4), (3, 5), (4, 5), (3, 7), (2, 9), (4, 6), (5, 5)])
        model = "xxz"
    else:
        top = {"hv": 30, "mf": 28, "build": 28, "solve": 26, "reorth": 18, "batch": 17, "expval": 24, "ref_ell": 22}[kind]
        N1, N2, model = rng.randint({"reorth": 12, "batch": 9}.get(kind, 10), top), 1, rng.choice(["xxz", "j1j2"])
    L = N1 * N2
    flip = L % 2 == 0 and rng.random() < 0.5
    k = 0 if rng.random() < 0.4 else rng.randrange(L)
    c = _case(kind, N1, N2, model, k, flip, prec, delta)
    if kind == "batch":
        c.update(k=0, flip=False, prec=64, sets=int(round(2 ** rng.uniform(0, 7.5))), mode=rng.choice([A.MODE_FP64, A.MODE_MIXED]))
    elif kind == "solve":
        c.update(k=0, prec=64, mode=rng.choice([A.MODE_FP64, A.MODE_MIXED]))
    elif kind == "reorth":
        sym = rng.random() < 0.5
        c.update(prec=64, sym=sym, steps=rng.randint(60, 150) if not sym and L <= 16 else rng.randint(40, 90))
        c.update(k=0, flip=c["flip"] and sym, N1=L if sym or L <= 16 else 16)
        c["flip"] = c["flip"] and c["N1"] % 2 == 0
    elif kind == "ref_ell":
        c.update(prec=32, flip=False, steps=rng.randint(30, 80))
    elif kind == "expval":
        c.update(k=0, prec=64, hops=rng.choice([0, 1]))
    return c


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind in ("hv", "mf"):
        # the handle, the input vector and a buffer for the product
        st["sec"] = _sector(case)
        st["h"] = q.Hamiltonian(st["sec"], _terms(case, seed), prec=_prec(case))
        n = st["h"].info.n_rows
        st["x"] = _vector(n, _dtype(case), seed)
        st["y"] = torch.empty_like(st["x"])
        st["stream"] = torch.cuda.current_stream().cuda_stream
    elif kind == "build":
        st["group"] = _group(case)
        st["terms"] = _terms(case, seed)
        st["x"] = _vector(_n_rows(case), _dtype(case), seed)
        st["stream"] = torch.cuda.current_stream().cuda_stream
    elif kind == "solve":
        st["sec"] = _sector(case)
        st["h"] = q.Hamiltonian(st["sec"], _terms(case, seed))
        st["seed"] = 20261203 + seed
    elif kind == "reorth":
        L, n_up, _, _ = _sys(case)
        if case["sym"]:
            st["sec"] = _sector(case)
        else:
            st["sec"] = q.Sector(L, n_up, np.arange(L, dtype=np.uint32)[None, :]).set_irrep([1.0])
        st["h"] = q.Hamiltonian(st["sec"], _terms(case, seed), prec=A.PREC_FP64)
        st["seed"] = 20261203 + seed
    elif kind == "batch":
        L, n_up, _, _ = _sys(case)
        perm, ch = q.translation_group(L)
        st["secs"] = [q.Sector(L, n_up, perm).set_irrep(ch[a]) for a in range(L)]
        b, J = _bonds(case)
        st["b"] = q.Batch(st["secs"], q.xxz_terms(b, J, 0.0, part="xy"), q.xxz_terms(b, 0.0, J, part="z"), case["sets"])
        st["cxy"], st["cz"] = _couplings(case, seed)
    elif kind == "expval":
        st["sec"] = _sector(case)
        st["h"] = q.Hamiltonian(st["sec"], _terms(case, seed), prec=A.PREC_FP64)
        psi = _vector(st["h"].info.n_rows, torch.float64, seed)
        st["psi"] = psi / psi.norm()
        st["ops"] = [q.operator_terms(o) for o in _operators(case)]
    elif kind == "ref_ell":
        L, n_up, _, _ = _sys(case)
        sec = _sector(case)
        terms = _terms(case, seed)
        W = 2 * len(_bonds(case)[0]) + 1
        ind, val, tr = q.export_ref(sec, terms, W)
        st["R"], st["W"] = ind.shape
        st["cplx"] = 0 if _real(case) else 1
        v = val.real.astype(np.float32) if not st["cplx"] else val.astype(np.complex64)
        st["ind"] = torch.from_numpy(ind.view(np.int32)).to(_DEV)
        st["val"] = torch.from_numpy(v).to(_DEV)
        st["tr"] = torch.from_numpy(tr).to(_DEV)
        st["seed"] = 2212456 + seed
    else:
        raise ValueError(kind)
    return st


def _couplings(case, seed):
    r = np.random.default_rng(seed)
    D = r.uniform(0.1, 2.0, case["sets"])
    J = r.uniform(0.5, 1.5, case["sets"])
    return J, J * D


def _operators(case):
    """S(q) at the chain's momenta (all of a torus's sites as one chain of phases) and <Sz_0 Sz_j>; with hops, <S+_0 S-_j>."""
    L = case["N1"] * case["N2"]
    ops = []
    for m in range(L):
        ops.append([(np.exp(2j * np.pi * m * (i - j) / L) / L, [("Sz", i), ("Sz", j)]) for i in range(L) for j in range(L)])
    ops += [[(1.0, [("Sz", 0), ("Sz", j)])] for j in range(L)]
    if case["hops"]:
        ops += [[(1.0, [("Sp", 0), ("Sm", j)])] for j in range(L)]
    return ops


# ---------------------------------------------------------------------- run
def run(st):
    kind, case = st["kind"], st["case"]
    if kind in ("hv", "mf"):
        st["h"].hv_dev(st["x"].data_ptr(), st["y"].data_ptr(), _prec(case), st["stream"], matrix_free=kind == "mf")
        return st["y"]
    if kind == "build":
        L, n_up, _, _ = _sys(case)
        perm, row = st["group"]
        s = q.Sector(L, n_up, perm, spin_flip=case["flip"]).set_irrep(row)
        h = q.Hamiltonian(s, st["terms"], prec=_prec(case))
        i = h.info
        y = torch.empty_like(st["x"])
        h.hv_dev(st["x"].data_ptr(), y.data_ptr(), _prec(case), st["stream"])
        h.close()
        s.close()
        return {"y": y, "rows": int(i.n_rows), "entries": int(i.nnz_offdiag), "widest": int(i.max_row)}
    if kind == "solve":
        return st["h"].lanczos(mode=case["mode"], tol=1e-12, seed=st["seed"]).E0
    if kind == "reorth":
        r = st["h"].lanczos(mode=A.MODE_FP64, tol=0.0, max_iter=case["steps"], reorth=2, want_vector=1,
                            check_every=case["steps"], seed=st["seed"], allow_unconverged=True)
        return {"E0": r.E0, "psi": st["h"].ground_state()}
    if kind == "batch":
        E, _ = st["b"].solve(st["cxy"], st["cz"], mode=case["mode"], tol=1e-12)
        return E
    if kind == "expval":
        return st["h"].expval(st["ops"], psi_dev=st["psi"].data_ptr())
    E = ctypes.c_float()
    vp = ctypes.c_void_p
    q.check(q.lib().qmb_lanczos_ref_ell(ctypes.byref(E), case["steps"], st["R"], st["W"], st["seed"], vp(st["ind"].data_ptr()),
                                        vp(st["val"].data_ptr()), vp(st["tr"].data_ptr()), st["cplx"], None, 0, None))
    return np.float32(E.value)


# --------------------------------------------------------------------- work
def _sizes(case, sym=True):
    """(rows, off-diagonal entries) of the case's sector, from counting all its strings."""
    L, k, N1, N2 = _sys(case)
    n = math.comb(L, k) / ((N1 * N2 * (2 if case["flip"] else 1)) if sym else 1)
    n = max(1.0, n)
    return n, n * len(_bonds(case)[0]) * 2.0 * k * (L - k) / (L * (L - 1))


def work(case):
    kind = case["kind"]
    n, nnz = _sizes(case, case.get("sym", True))
    cx = 1 if _real(case) else 2
    sv = case["prec"] // 8 * cx
    mul = 2 if cx == 1 else 8
    hv = nnz * 4 + n * 3 * sv  # an entry's column and value code, the diagonal, x and y
    if kind == "hv":
        return {"bytes": hv, "flops": nnz * mul}
    if kind == "mf":
        return {"bytes": n * (4 + 2 * sv), "flops": nnz * mul}
    if kind == "build":
        L, k, _, _ = _sys(case)
        return {"bytes": math.comb(L, k) / 8 + n * 8 + nnz * (4 + sv) + hv, "flops": nnz * mul}
    if kind == "solve":
        return {"bytes": 50 * (hv + 3 * n * sv), "flops": 50 * (nnz * mul + 8 * n)}
    if kind == "reorth":
        m = case["steps"]
        return {"bytes": m * (hv + 3 * n * sv) + m * m * n * sv, "flops": m * nnz * mul + 2.0 * m * m * n * cx * cx}
    if kind == "batch":
        # all momenta: as many rows as the unreduced sector; steps of the FP64
        # solve, five passes over a complex vector each
        L, k, _, _ = _sys(case)
        rows = math.comb(L, k) * case["sets"]
        return {"bytes": 60.0 * rows * 5 * (8 if case["mode"] == A.MODE_MIXED else 16), "flops": 60.0 * rows * 8 * 0.53 * L}
    if kind == "expval":
        L = case["N1"] * case["N2"]
        return {"bytes": n * 16 + 16.0 * L * L, "flops": n * 2.0 * L * (L - 1) / 2 + case["hops"] * n * 4.0 * L * L}
    return {"bytes": case["steps"] * (hv + 3 * n * sv), "flops": case["steps"] * nnz * mul}


# -------------------------------------------------------------------- exact
def _states(L, k):
    """All L-bit strings with k ones, ascending, from their two halves."""
    h = L // 2
    lo = torch.arange(1 << h, device=_DEV)
    hi = torch.arange(1 << (L - h), device=_DEV)

    def pop(v, bits):
        c = torch.zeros_like(v)
        for b in range(bits):
            c += (v >> b) & 1
        return c
    pl, ph = pop(lo, h), pop(hi, L - h)
    order = torch.argsort(pl, stable=True)
    cnt = torch.bincount(pl, minlength=h + 1)
    start = torch.cumsum(cnt, 0) - cnt
    keep = (ph <= k) & (k - ph <= h)
    hi, need = hi[keep], (k - ph)[keep]
    c, s = cnt[need], start[need]
    first = torch.cumsum(c, 0) - c
    rep = torch.repeat_interleave(torch.arange(len(hi), device=_DEV), c)
    at = torch.arange(len(rep), device=_DEV) - first[rep] + s[rep]
    return (hi[rep] << h) | lo[order][at]


def _image(case, t, e):
    """Element e's image of the strings t."""
    for f, y in _images(case, t, e):
        return y


def _images(case, t, only=None):
    """Every element's image of the strings t: (e, image), e = z * G + g; element (nx, ny) moves site (i, j) to (i - nx, j - ny)."""
    L, _, N1, N2 = _sys(case)
    full = (1 << L) - 1
    for nx in range(N1):
        if only is not None and only % (N1 * N2) // N2 != nx:
            continue
        r = (N1 - nx) % N1 * N2
        y = ((t << r) | (t >> (L - r))) & full if r else t
        for ny in range(N2):
            if only is not None and only % N2 != ny:
                continue
            c = (N2 - ny) % N2
            low = sum(1 << s for s in range(L) if s % N2 < N2 - c)
            z = ((y & low) << c) | ((y & (full ^ low)) >> (N2 - c)) if c else y
            if only is None or only < N1 * N2:
                yield nx * N2 + ny, z
            if case["flip"] and (only is None or only >= N1 * N2):
                yield N1 * N2 + nx * N2 + ny, z ^ full


class _Sector:
    """Representatives (orbit minima), norms and matrix of a case's sector."""

    def __init__(self, case, sym=True):
        self.case, self.sym = case, sym
        L, k, _, _ = _sys(case)
        self.chi = torch.tensor(_chars(case), device=_DEV)
        s = _states(L, k)
        if sym:
            ne = len(self.chi)
            for e in range(ne):  # keep what no element maps lower, one element at a time
                s = s[_image(case, s, e) >= s]
            stab = torch.zeros(len(s), dtype=torch.complex128, device=_DEV)
            for e, y in _images(case, s):
                stab += torch.where(y == s, self.chi[e], torch.zeros_like(self.chi[e]))
            norm = torch.sqrt(stab.real.abs() * ne) / ne
            live = norm >= 1e-5
            s, self.norm = s[live], norm[live]
        else:
            self.norm = torch.ones(len(s), dtype=torch.float64, device=_DEV)
        self.reps = s
        self.n = len(s)

    def rep_of(self, t):
        best, be = t.clone(), torch.zeros_like(t)
        if self.sym:
            for e, y in _images(self.case, t):
                m = y < best
                best = torch.where(m, y, best)
                be = torch.where(m, torch.full_like(be, e), be)
        return best, be

    def hops(self):
        """Per bond: (bond, rows, columns, values with unit coupling) of the spin exchange."""
        for b, (i, j) in enumerate(_bonds(self.case)[0]):
            rows = torch.nonzero(((self.reps >> i) ^ (self.reps >> j)) & 1).flatten()
            src = self.reps[rows]
            t, e = self.rep_of(src ^ ((1 << i) | (1 << j)))
            c = torch.searchsorted(self.reps, t).clamp(max=self.n - 1)
            ok = self.reps[c] == t
            rows, c, e = rows[ok], c[ok], e[ok]
            v = 0.5 * (self.norm[c] / self.norm[rows]).to(torch.complex128)
            if self.sym:
                v = v * self.chi[e].conj()
            yield b, rows, c, v

    def zz(self, i, j):
        return 0.25 - 0.5 * (((self.reps >> i) ^ (self.reps >> j)) & 1).to(torch.float64)

    def csr(self, xy, real=False):
        """The exchange part sum_b xy_b as a sparse matrix."""
        R, C, V = [], [], []
        for b, r, c, v in self.hops():
            R.append(r)
            C.append(c)
            V.append(v * xy[b])
        v = torch.cat(V)
        m = torch.sparse_coo_tensor(torch.stack([torch.cat(R), torch.cat(C)]), v.real.contiguous() if real else v, (self.n, self.n))
        return m.coalesce().to_sparse_csr()


def _n_rows(case):
    """Active orbits of the case's sector by Burnside's count weighted with the characters."""
    L, k, N1, N2 = _sys(case)
    chi = _chars(case)
    total = 0.0
    for nx in range(N1):
        for ny in range(N2):
            seen, cyc = set(), []
            for s in range(L):
                m, t = 0, s
                while t not in seen:
                    seen.add(t)
                    m += 1
                    i, j = divmod(t, N2)
                    t = ((i + nx) % N1) * N2 + (j + ny) % N2
                if m:
                    cyc.append(m)
            poly = [1] + [0] * L
            for m in cyc:
                for d in range(L, m - 1, -1):
                    poly[d] += poly[d - m]
            g = nx * N2 + ny
            total += chi[g].real * poly[k]
            if case["flip"]:
                # complement: every cycle of even length alternates in two ways
                total += chi[N1 * N2 + g].real * (2 ** len(cyc) if all(m % 2 == 0 for m in cyc) else 0)
    return int(round(total / len(chi)))


def _apply(sec, case, d, x):
    b, J = _bonds(case)
    y = torch.zeros_like(x)
    for (i, j), Jb in zip(b, J):
        y += (Jb * d) * sec.zz(i, j) * x
    for k, r, c, v in sec.hops():
        y[r] += J[k] * v * x[c]
    return y


def _lowest(sec, case, d, steps, start=None):
    """Lowest eigenvalue and its vector: FP64 Lanczos with full reorthogonalisation."""
    b, J = _bonds(case)
    real = _real(case) or not sec.sym
    M = sec.csr(J, real)
    diag = sum((Jb * d) * sec.zz(i, j) for (i, j), Jb in zip(b, J))
    dt = torch.float64 if real else torch.complex128
    if start is None:
        g = torch.Generator(device=_DEV).manual_seed(77)
        start = torch.randn(sec.n, dtype=dt, device=_DEV, generator=g)
    v = start.to(dt) / start.norm()
    first = v
    steps = min(steps, sec.n)
    Q = torch.zeros(steps, sec.n, dtype=dt, device=_DEV)
    al, be = [], []
    for j in range(steps):
        Q[j] = v
        w = M @ v + diag * v
        al.append(float(torch.vdot(v, w).real))
        for _ in range(2):
            w = w - Q[: j + 1].T @ (Q[: j + 1].conj() @ w)
        nb = float(w.norm())
        if nb < 1e-12:
            break
        be.append(nb)
        v = w / nb
    T = torch.diag(torch.tensor(al, dtype=torch.float64))
    m = len(al)
    for i in range(m - 1):
        T[i, i + 1] = T[i + 1, i] = be[i]
    w, U = torch.linalg.eigh(T)
    psi = Q[:m].T @ U[:, 0].to(dt).to(_DEV)
    psi = psi / psi.norm()
    s = torch.vdot(first, psi)
    return float(w[0]), (psi if float(s.real) >= 0 else -psi)


def _splitmix_start(n, seed, cplx):
    """The documented start vector: uniform(-1, 1) from splitmix64(seed + i)."""
    m = (2 if cplx else 1) * n
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.arange(m, dtype=np.uint64) + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    u = (z >> np.uint64(11)).astype(np.float64) * (2.0 / 9007199254740992.0) - 1.0
    return torch.from_numpy(u.view(np.complex128) if cplx else u).to(_DEV)


def _batch_energies(case, seed):
    """Lowest level of every (set, momentum): plain FP64 Lanczos of all sets of a sector at once."""
    J, cz = (torch.tensor(v, device=_DEV) for v in _couplings(case, seed))
    L = case["N1"]
    E = np.zeros((case["sets"], L))
    b, Jb = _bonds(case)
    for k in range(L):
        c = dict(case, k=k)
        sec = _Sector(c)
        if sec.n <= 320:
            M = sec.csr(Jb).to_dense()
            D = sum(Jk * sec.zz(i, j) for (i, j), Jk in zip(b, Jb))
            H = J[:, None, None] * M[None] + torch.diag_embed(cz[:, None] * D[None]).to(torch.complex128)
            E[:, k] = torch.linalg.eigvalsh(H)[:, 0].cpu().numpy()
            continue
        M = sec.csr(Jb)
        D = sum(Jk * sec.zz(i, j) for (i, j), Jk in zip(b, Jb))[:, None]
        g = torch.Generator(device=_DEV).manual_seed(5)
        w = torch.randn(sec.n, case["sets"], dtype=torch.complex128, device=_DEV, generator=g)
        v0, beta = torch.zeros_like(w), w.norm(dim=0)
        al, be = [], []
        for _ in range(min(220, sec.n)):
            v = w / beta
            w = J * (M @ v) + cz * (D * v) - beta * v0 * (1.0 if al else 0.0)
            a = (v.conj() * w).sum(0).real
            w = w - a * v
            v0, beta = v, w.norm(dim=0)
            al.append(a)
            be.append(beta)
        T = torch.diag_embed(torch.stack(al, 1))
        o = torch.stack(be[:-1], 1)
        T = T + torch.diag_embed(o, offset=1) + torch.diag_embed(o, offset=-1)
        E[:, k] = torch.linalg.eigvalsh(T.cpu())[:, 0].numpy()
    return E


def _expvals(case, seed):
    """<psi|A|psi> over the unreduced strings: a k = 0 state has its orbit's amplitude over the square root of the orbit's size."""
    sec = _Sector(case)
    L, k, _, _ = _sys(case)
    psi = _vector(sec.n, torch.float64, seed)
    psi = psi / psi.norm()
    s = _states(L, k)
    t, _ = sec.rep_of(s)
    o = torch.searchsorted(sec.reps, t)
    size = torch.bincount(o, minlength=sec.n).to(torch.float64)
    c = (psi / size.sqrt())[o]
    p = c * c
    bits = [((s >> i) & 1).to(torch.float64) - 0.5 for i in range(L)]
    G = torch.zeros(L, L, dtype=torch.float64, device=_DEV)
    for i in range(L):
        for j in range(i, L):
            G[i, j] = G[j, i] = (p * bits[i] * bits[j]).sum()
    ph = torch.arange(L, device=_DEV, dtype=torch.float64)
    out = [((torch.exp(2j * math.pi * m * (ph[:, None] - ph[None, :]) / L) / L) * G).sum() for m in range(L)]
    out += [G[0, j].to(torch.complex128) for j in range(L)]
    if case["hops"]:
        for j in range(L):
            # <S+_0 S-_j>: strings with site j up and site 0 down (j = 0: site 0 up)
            if j == 0:
                out.append((p * (bits[0] + 0.5)).sum().to(torch.complex128))
                continue
            r = torch.nonzero((bits[j] > 0) & (bits[0] < 0)).flatten()
            z = torch.searchsorted(s, s[r] ^ (1 | (1 << j)))
            out.append((c[z] * c[r]).sum().to(torch.complex128))
    return torch.stack(out).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("hv", "mf", "build"):
            sec = _Sector(case)
            x = _vector(sec.n, _dtype(case), seed)
            y = _apply(sec, case, _delta(case, seed), x.to(torch.complex128))
            y = y.real.contiguous() if _real(case) else y
            return {"y": y, "rows": None, "entries": None, "widest": None} if kind == "build" else y
        if kind == "solve":
            return _lowest(_Sector(case), case, _delta(case, seed), 130)[0]
        if kind == "reorth":
            sec = _Sector(case, case["sym"])
            cplx = case["sym"] and not _real(case)
            start = _splitmix_start(sec.n, 20261203 + seed, cplx)
            E, psi = _lowest(sec, case, _delta(case, seed), case["steps"], start)
            return {"E0": E, "psi": psi.cpu().numpy()}
        if kind == "batch":
            return _batch_energies(case, seed)
        if kind == "expval":
            return _expvals(case, seed)
        if kind == "ref_ell":
            return np.float64(_lowest(_Sector(case), case, _delta(case, seed), 130)[0])
    return None
