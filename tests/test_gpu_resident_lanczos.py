"""Lanczos steps of sectors of few rows in one resident kernel: row counts at the
edges of warps, row blocks and splits, real and complex, every mode, with and
without reorthogonalisation, against dense diagonalisation; and the states they
return against their own product."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi

# (L, n_up, lattice or None, k): 1, 5, 32, 33, 253, 276 and 495 rows without a
# group, complex sectors of 25 and 810 rows
SIZES = [(6, 6, None, 0), (5, 1, None, 0), (32, 1, None, 0), (33, 1, None, 0), (23, 2, None, 0), (24, 2, None, 0),
         (12, 4, None, 0), (10, 5, (10, 1), 3), (16, 8, (16, 1), 5)]


@pytest.mark.parametrize("L,n_up,lattice,k", SIZES)
@pytest.mark.parametrize("mode,reorth", [(A.MODE_FP64, 0), (A.MODE_FP64, 1), (A.MODE_FP64, 2), (A.MODE_MIXED, 0),
                                         (A.MODE_MIXED, 2), (A.MODE_FP32, 0), (A.MODE_FP32, 2)])
def test_energies_and_states(L, n_up, lattice, k, mode, reorth):
    if lattice is None:
        perm, ch = np.arange(L, dtype=np.uint32)[None, :], np.ones((1, 1), complex)
        bonds = [(i, i + 1) for i in range(L - 1)]  # open, with a gradient: no degenerate levels
        t = q.xxz_terms(bonds, np.linspace(0.7, 1.3, len(bonds)), 0.8)
    else:
        perm, ch = q.translation_group(*lattice)
        t = q.xxz_terms(q.chain_bonds(L), 1.0, 0.8)
    s = q.Sector(L, n_up, perm).set_irrep(ch[k])
    h = q.Hamiltonian(s, t)
    sec = O.build_sector(oracle_group(perm, ch), n_up)
    rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), k, 2 * t.n_terms + 1)
    M = O.ell_to_csr(ind, val, tr, O.active_rows(sec, k))
    e = O.ground_energy_dense(M)
    r = h.lanczos(mode=mode, tol=1e-12, reorth=reorth, max_iter=200, want_vector=1, allow_unconverged=True)
    assert abs(r.E0 - e) <= (2e-5 if mode == A.MODE_FP32 else 1e-10) * max(1.0, abs(e))
    psi = h.ground_state()
    res = np.linalg.norm(h.hv_host(psi) - r.E0 * psi) / np.linalg.norm(psi)
    assert res <= (2e-3 if mode == A.MODE_FP32 else 1e-5) * max(1.0, abs(e))
    assert abs(res - r.residual) <= 1e-6 * max(1.0, abs(e))


@pytest.mark.parametrize("check_every", [1, 7, 60])
def test_steps_do_not_depend_on_the_launches(check_every):
    """60 steps in launches of 1, 7 or 60: the same coefficients."""
    L = 14
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[3])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    for reorth in (0, 2):
        o = dict(mode=A.MODE_FP64, tol=0.0, max_iter=60, reorth=reorth, allow_unconverged=True)
        r0, c0 = h.lanczos(n_coeffs=60, check_every=10, **o)
        r1, c1 = h.lanczos(n_coeffs=60, check_every=check_every, **o)
        assert r0.E0 == r1.E0 and np.array_equal(c0, c1)


def test_regenerated_state_is_the_stored_one(monkeypatch):
    """A ring that wraps regenerates the basis with the same kernel: the same bits."""
    L = 12
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[0])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    r = h.lanczos(tol=1e-12, want_vector=1)
    a = h.ground_state()
    monkeypatch.setenv("QMB_LZ_RING_MAX", "3")
    h2 = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    r2 = h2.lanczos(tol=1e-12, want_vector=1)
    assert r2.E0 == r.E0 and r2.n_hv > r.n_hv
    assert np.abs(h2.ground_state() - a).max() <= 4e-15
