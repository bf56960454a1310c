"""Batches over sectors of one to a few rows, whose Krylov spaces end within the first
steps: every energy against dense diagonalisation."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("L,n_up", [(2, 1), (3, 2), (5, 1), (8, 0), (9, 1), (10, 9), (4, 2), (6, 2), (6, 3)])
@pytest.mark.parametrize("n_sets", [3, 40])
@pytest.mark.parametrize("mode", [A.MODE_FP64, A.MODE_MIXED, A.MODE_FP32])
def test_energies(L, n_up, n_sets, mode):
    perm, ch = q.translation_group(L)
    sec = O.build_sector(oracle_group(perm, ch), n_up)
    ks = [k for k in range(L) if len(O.active_rows(sec, k))]
    secs = [q.Sector(L, n_up, perm).set_irrep(ch[k]) for k in ks]
    bonds = q.chain_bonds(L)
    b = q.Batch(secs, q.xxz_terms(bonds, 1.0, 0.0, part="xy"), q.xxz_terms(bonds, 0.0, 1.0, part="z"), n_sets)
    J, D = np.linspace(0.6, 1.4, n_sets), np.linspace(-1.3, 1.7, n_sets)
    E, r = b.solve(J, J * D, mode=mode, tol=1e-10, allow_unconverged=True)
    b.close()
    for i in range(0, n_sets, 1 if n_sets < 5 else 13):
        t = q.xxz_terms(bonds, J[i], J[i] * D[i])
        for c, k in enumerate(ks):
            rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), k, 2 * t.n_terms + 1)
            e = O.ground_energy_dense(O.ell_to_csr(ind, val, tr, O.active_rows(sec, k)))
            assert abs(E[i, c] - e) <= (1e-5 if mode == A.MODE_FP32 else 1e-8) * max(1.0, abs(e)), (i, k, E[i, c], e)
