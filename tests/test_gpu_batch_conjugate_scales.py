"""Which sectors count as conjugates is judged for the hopping and the diagonal part
apart: a diagonal part of far larger entries does not hide that the hopping parts
of momenta k and -k differ."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


def _dense(perm, ch, n_up, a, t):
    sec = O.build_sector(oracle_group(perm, ch), n_up)
    rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), a, 2 * t.n_terms + 1)
    return O.ground_energy_dense(O.ell_to_csr(ind, val, tr, O.active_rows(sec, a)))


@pytest.mark.parametrize("scale", [1e14, 1.0, 1e-14])
@pytest.mark.parametrize("mode", [A.MODE_FP64, A.MODE_MIXED])
def test_complex_hopping_beside_a_scaled_diagonal(scale, mode):
    L, n_up, order = 9, 4, [3, 6, 1, 8]  # (at half filling inversion gives k and -k the same levels)
    perm, ch = q.translation_group(L)
    bonds, hop = q.chain_bonds(L), np.exp(0.3j)
    secs = [q.Sector(L, n_up, perm).set_irrep(ch[a]) for a in order]
    b = q.Batch(secs, q.xxz_terms(bonds, hop, 0.0, part="xy"), q.xxz_terms(bonds, 0.0, scale, part="z"), 2)
    J = np.array([1.0, 0.8])
    E, r = b.solve(J, np.zeros(2), mode=mode, tol=1e-12)  # the diagonal part is switched off
    for c, a in enumerate(order):
        e = _dense(perm, ch, n_up, a, q.xxz_terms(bonds, J[1] * hop, 0.0))
        assert abs(E[1, c] - e) <= 1e-10 * abs(e), (a, E[1, c], e)
    assert abs(E[0, 0] - E[0, 1]) > 1e-6  # k and -k differ
    b.close()
