"""Sectors with conjugate matrices (momenta k and -k of a real Hamiltonian)
are solved once in a batch.  Every energy is still its own sector's."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


def _dense(perm, ch, n_up, a, t):
    g = oracle_group(perm, ch)
    sec = O.build_sector(g, n_up)
    rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), a, 2 * t.n_terms + 1)
    return O.ground_energy_dense(O.ell_to_csr(ind, val, tr, O.active_rows(sec, a)))


@pytest.mark.parametrize("L,order,phase,shared", [
    (9, list(range(9)), 0.0, True),            # odd length: one real momentum, four pairs
    (10, [7, 3, 0, 3, 9, 5, 1], 0.0, True),    # pairs out of order, a momentum twice, one without its partner
    (9, list(range(9)), 0.3, False),           # complex hopping: k and -k have different spectra
])
@pytest.mark.parametrize("mode", [A.MODE_FP64, A.MODE_MIXED])
def test_conjugate_sectors_have_their_own_energies(L, order, phase, shared, mode):
    perm, ch = q.translation_group(L)
    n_up, bonds, n_sets = L // 2, q.chain_bonds(L), 5
    hop = np.exp(1j * phase) if phase else 1.0
    secs = [q.Sector(L, n_up, perm).set_irrep(ch[a]) for a in order]
    b = q.Batch(secs, q.xxz_terms(bonds, hop, 0.0, part="xy"), q.xxz_terms(bonds, 0.0, 1.0, part="z"), n_sets)
    J, D = np.linspace(0.6, 1.4, n_sets), np.linspace(0.3, 1.7, n_sets)
    E, r = b.solve(J, J * D, mode=mode, tol=1e-12)
    for i in (0, n_sets - 1):
        for c, a in enumerate(order):
            e = _dense(perm, ch, n_up, a, q.xxz_terms(bonds, J[i] * hop, J[i] * D[i]))
            assert abs(E[i, c] - e) <= 1e-10 * abs(e), (i, a, E[i, c], e)
    pairs = [(c, d) for c, a in enumerate(order) for d, e in enumerate(order) if c < d and (a + e) % L == 0 and a != e]
    assert pairs
    same = [np.array_equal(E[:, c], E[:, d]) for c, d in pairs]
    assert all(same) if shared else not any(same)
    b.close()
