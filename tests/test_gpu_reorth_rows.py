"""Reorthogonalised solves on both sides of the row counts up to which the resident
kernel runs them: energies against a plain solve, and the same coefficients from
launches of 3 and of 10 steps."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


# real 54,264 and 65,780 rows, complex 43,263 and 112,632 (lines at 57,344 and 81,920)
@pytest.mark.parametrize("L,n_up,k", [(21, 6, None), (26, 5, None), (25, 8, 3), (24, 12, 5)])
@pytest.mark.parametrize("mode", [A.MODE_FP64, A.MODE_FP32])
def test_solves_around_the_line(L, n_up, k, mode):
    if k is None:  # open, with a gradient: no degenerate levels
        perm, chars = np.arange(L, dtype=np.uint32)[None, :], np.ones(1)
        bonds = [(i, i + 1) for i in range(L - 1)]
        t = q.xxz_terms(bonds, np.linspace(0.7, 1.3, len(bonds)), 0.8)
    else:
        perm, ch = q.translation_group(L)
        chars, t = ch[k], q.xxz_terms(q.chain_bonds(L), 1.0, 0.8)
    s = q.Sector(L, n_up, perm).set_irrep(chars)
    h = q.Hamiltonian(s, t)
    e = h.lanczos(tol=1e-12, max_iter=600).E0
    o = dict(mode=mode, reorth=2, tol=0.0, max_iter=60, want_vector=1, allow_unconverged=True)
    r, c = h.lanczos(n_coeffs=60, **o)
    psi = h.ground_state()
    r3, c3 = h.lanczos(n_coeffs=60, check_every=3, **o)
    assert r3.E0 == r.E0 and np.array_equal(c3, c) and np.array_equal(h.ground_state(), psi)
    res = np.linalg.norm(h.hv_host(psi) - r.E0 * psi) / np.linalg.norm(psi)
    assert abs(res - r.residual) <= 1e-6 * max(1.0, abs(e))
    # an eigenvalue lies within the residual of E0, and E0 above the lowest one
    assert e - (2e-5 if mode == A.MODE_FP32 else 1e-10) * abs(e) <= r.E0 <= e + res + 1e-3 * abs(e)
