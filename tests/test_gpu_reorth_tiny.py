"""Reorthogonalised solves of sectors with fewer rows than steps, where the Krylov
space ends early: energies against dense diagonalisation."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


# 1 to 38 rows, with degenerate levels (no group) and without
@pytest.mark.parametrize("L,n_up,k", [(4, 2, 0), (5, 4, None), (6, 3, 1), (6, 2, None), (9, 5, 2), (8, 4, None), (10, 5, 3), (12, 6, 5)])
@pytest.mark.parametrize("mode", [A.MODE_FP64, A.MODE_MIXED, A.MODE_FP32])
@pytest.mark.parametrize("reorth", [1, 2])
@pytest.mark.parametrize("check_every", [1, 10])
def test_energies(L, n_up, k, mode, reorth, check_every):
    if k is None:
        perm, ch = np.arange(L, dtype=np.uint32)[None, :], np.ones((1, 1), complex)
    else:
        perm, ch = q.translation_group(L)
    s = q.Sector(L, n_up, perm).set_irrep(ch[k or 0])
    t = q.xxz_terms(q.chain_bonds(L), 1.0, 0.8)
    h = q.Hamiltonian(s, t)
    sec = O.build_sector(oracle_group(perm, ch), n_up)
    rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), k or 0, 2 * t.n_terms + 1)
    e = O.ground_energy_dense(O.ell_to_csr(ind, val, tr, O.active_rows(sec, k or 0)))
    for tol in (1e-10, 0.0):
        r = h.lanczos(mode=mode, tol=tol, reorth=reorth, max_iter=300, refine_max_iter=300, check_every=check_every,
                      want_vector=1, allow_unconverged=True)
        assert abs(r.E0 - e) <= (2e-5 if mode == A.MODE_FP32 else 1e-9) * max(1.0, abs(e)), (tol, r.E0, e)
        psi = h.ground_state()
        res = np.linalg.norm(h.hv_host(psi) - r.E0 * psi) / np.linalg.norm(psi)
        assert res <= (2e-3 if mode == A.MODE_FP32 else 1e-5) * max(1.0, abs(e))
