"""Products whose rows are dealt to several threads, at the row counts where the
split changes and at ragged ends, against the oracle's matrix."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


def _case(L, n_up, lattice, k):
    if lattice is None:
        return np.arange(L, dtype=np.uint32)[None, :], np.ones((1, 1), complex), 0
    perm, ch = q.translation_group(*lattice)
    return perm, ch, k


# rows: 1, 7 (one slice), 33..., just below and above 16,384 and 131,072
SIZES = [(6, 6, None, 0), (7, 1, None, 0), (11, 4, None, 0), (10, 5, (10, 1), 3), (12, 6, (4, 3), 7),
         (16, 7, None, 0), (17, 7, None, 0), (18, 7, None, 0), (19, 9, None, 0), (20, 9, None, 0)]


@pytest.mark.parametrize("L,n_up,lattice,k", SIZES)
@pytest.mark.parametrize("prec", [A.PREC_FP32, A.PREC_FP64])
def test_split_products_equal_the_oracle(L, n_up, lattice, k, prec):
    import torch
    perm, ch, k = _case(L, n_up, lattice, k)
    bonds = q.chain_bonds(L) if lattice is None or lattice[1] == 1 else q.square_bonds(*lattice)
    # exchange terms, and a three-site term, which the matrix-free product takes through its general loop
    xxz = q.xxz_terms(bonds, 1.0, 0.7)
    three = q.operator_terms([(0.3, [("Sz", i), ("Sp", (i + 1) % L), ("Sm", (i + 2) % L)]) for i in range(L)] +
                             [(0.3, [("Sz", i), ("Sm", (i + 1) % L), ("Sp", (i + 2) % L)]) for i in range(L)])
    for t in (xxz, xxz + three) if L <= 12 and lattice is None else (xxz,):
        s = q.Sector(L, n_up, perm).set_irrep(ch[k])
        h = q.Hamiltonian(s, t, prec=prec)
        sec = O.build_sector(oracle_group(perm, ch), n_up)
        rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), k, 2 * t.n_terms + 1)
        M = O.ell_to_csr(ind, val, tr, O.active_rows(sec, k))
        n = M.shape[0]
        rng = np.random.default_rng(n)
        cplx = h.info.is_complex
        x = (rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)).astype(h.dtype(prec))
        eps = 2.3e-16 if prec == A.PREC_FP64 else 1.2e-7
        bound = 2 * (h.info.max_row + 4) * eps * (np.abs(M) @ np.abs(x)).max()
        want = M @ x if cplx else (M @ x).real
        xd = torch.from_numpy(x).cuda()
        for mf in (False, True):
            y = torch.full_like(xd, float("nan"))
            h.hv_dev(xd.data_ptr(), y.data_ptr(), prec, matrix_free=mf)
            torch.cuda.synchronize()
            assert np.abs(y.cpu().numpy() - want).max() <= bound, (mf, n)
