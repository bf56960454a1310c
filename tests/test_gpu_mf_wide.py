"""Matrix-free products on strings beyond 32 sites, hop form and general terms, at the
row counts of every split, against the stored product."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


# (lattice, n_up, k or None without a group): 1, 16, 3,930, 15,180, 91,390, 278,256 and 658,008 rows
@pytest.mark.parametrize("lattice,n_up,k", [((33, 1), 1, 5), ((33, 1), 2, 0), ((6, 6), 4, 7), ((36, 1), 5, 0), ((40, 1), 4, None),
                                            ((34, 1), 5, None), ((40, 1), 5, None)])
@pytest.mark.parametrize("general", [False, True])
def test_wide_strings(lattice, n_up, k, general):
    import torch
    L = lattice[0] * lattice[1]
    if k is None:
        perm, chars = np.arange(L, dtype=np.uint32)[None, :], np.ones(1)
    else:
        perm, ch = q.translation_group(*lattice)
        chars = ch[k]
    s = q.Sector(L, n_up, perm).set_irrep(chars)
    bonds = q.square_bonds(*lattice) if lattice[1] > 1 else q.chain_bonds(L)
    t = q.xxz_terms(bonds, 1.0, 0.7)
    if general:  # S+ S- Sz: not a two-site exchange
        terms = [(0.3, [("Sp", i), ("Sm", j), ("Sz", (i + 5) % L)]) for i, j in bonds]
        t = t + q.operator_terms(terms + [(0.3, [("Sp", j), ("Sm", i), ("Sz", (i + 5) % L)]) for i, j in bonds])
    h = q.Hamiltonian(s, t)
    n = h.info.n_rows
    for prec, eps in ((A.PREC_FP64, 2.3e-16), (A.PREC_FP32, 1.2e-7)):
        dt = {np.dtype("f4"): torch.float32, np.dtype("f8"): torch.float64, np.dtype("c8"): torch.complex64,
              np.dtype("c16"): torch.complex128}[np.dtype(h.dtype(prec))]
        x = torch.randn(n, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
        y, z = torch.empty_like(x), torch.empty_like(x)
        h.hv_dev(x.data_ptr(), y.data_ptr(), prec)
        h.hv_dev(x.data_ptr(), z.data_ptr(), prec, matrix_free=True)
        torch.cuda.synchronize()
        # rows of up to some tens of entries, each with a value of rounded factors
        assert float((y - z).abs().max()) <= 8 * (h.info.max_row + 4) * eps * float(x.abs().max())
    if n > 1:
        o = dict(tol=1e-11, max_iter=400, allow_unconverged=True)
        assert abs(h.lanczos(**o).E0 - h.lanczos(hv=A.HV_MATRIX_FREE, **o).E0) <= 1e-8 * L
