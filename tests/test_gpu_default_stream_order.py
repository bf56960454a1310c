"""Calls on caller-owned device arrays that take no stream run after what the caller
queued on the default stream, on first and on repeated calls.  (Both contents of
every array are valid tables, so a call that did not wait would only give the
other energy.)"""
import ctypes as C

import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi
L, SEED, STEPS = 14, 2212456, 50
DELAY = 20_000_000  # clock cycles, about 10 ms: longer than the calls


def _ell(Jz):
    import torch
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[0])
    ind, val, tr = q.export_ref(s, q.xxz_terms(q.chain_bonds(L), 1.0, Jz), 2 * L + 1)
    return [torch.tensor(ind.astype(np.int64)).to(torch.int32).cuda(), torch.tensor(val.real.astype(np.float32)).cuda(),
            torch.tensor(tr.astype(np.int16)).cuda()]


def _solve(t, check):
    E, r, kry = C.c_float(), C.c_float(), np.zeros(STEPS, np.float32)
    q.check(q.lib().qmb_lanczos_ref_ell(C.byref(E), STEPS, *t[0].shape, SEED, *(C.c_void_p(x.data_ptr()) for x in t), 0,
                                        A.ptr(kry), check, C.byref(r)))
    return E.value, kry, r.value


def _eigvec(t, kry, psi):
    q.check(q.lib().qmb_eigvec_from_seed_ref(SEED, C.c_void_p(psi.data_ptr()), A.ptr(kry), STEPS, *t[0].shape,
                                             *(C.c_void_p(x.data_ptr()) for x in t), 0))


@pytest.mark.parametrize("check", [0, 1])
def test_reference_solve(check):
    import torch
    a, b = _ell(1.0), _ell(0.3)
    torch.cuda.synchronize()
    want = _solve(b, check)
    live = [x.clone() for x in a]
    for _ in range(3):
        for x, y in zip(live, a):
            x.copy_(y)
        torch.cuda.synchronize()
        torch.cuda._sleep(DELAY)
        for x, y in zip(live, b):
            x.copy_(y)
        got = _solve(live, check)
        assert got[0] == want[0] and got[2] == want[2] and np.array_equal(got[1], want[1])


def test_reference_eigenvector():
    import torch
    a = _ell(1.0)
    torch.cuda.synchronize()
    kry = _solve(a, 0)[1]
    psi = torch.zeros(a[0].shape[0], device="cuda")
    _eigvec(a, kry, psi)
    want = psi.clone()
    for _ in range(3):
        torch.cuda._sleep(DELAY)
        psi.fill_(7.0)  # work on the array queued before the call
        _eigvec(a, kry, psi)
        torch.cuda.synchronize()
        assert torch.equal(psi, want)


def test_observables():
    import torch
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[0])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    g = torch.Generator(device="cuda").manual_seed(5)
    p1, p2 = (torch.randn(h.info.n_rows, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    op = q.operator_terms([(1.0, [("Sz", 0), ("Sz", 1)]), (0.5, [("Sp", 0), ("Sm", 3)])])
    want = h.expval(op, p2.data_ptr())
    live = p1.clone()
    for _ in range(3):
        live.copy_(p1)
        torch.cuda._sleep(DELAY)
        live.copy_(p2)
        assert h.expval(op, live.data_ptr()) == want
