"""Solves whose coefficients come over in one copy and, from larger step limits on, in
separate ones: the same energies and states, with a test after every step too."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("L,k", [(12, 0), (14, 3)])
@pytest.mark.parametrize("mode,reorth", [(A.MODE_FP64, 0), (A.MODE_FP64, 2), (A.MODE_MIXED, 0), (A.MODE_FP32, 0)])
def test_step_limits(L, k, mode, reorth):
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[k])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    got = []
    # (two limits around 16 KB of coefficients, and the largest)
    for limit, every in ((200, 10), (1021, 10), (1022, 10), (1023, 10), (4096, 10), (1022, 1), (4096, 1)):
        r = h.lanczos(mode=mode, reorth=reorth, tol=1e-10, max_iter=limit, refine_max_iter=limit, check_every=every,
                      want_vector=1, allow_unconverged=True)
        got.append((every, r.E0, h.ground_state()))
    for every, e, psi in got:
        if every == 10:
            assert e == got[0][1] and np.array_equal(psi, got[0][2])
        else:
            assert abs(e - got[0][1]) <= (1e-5 if mode == A.MODE_FP32 else 1e-9) * abs(e)
