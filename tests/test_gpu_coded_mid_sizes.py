"""Coded entries of matrices whose plain entries take some tens of MB (all of it
in L2), against the matrix-free product."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("lattice,k,prec,coded", [((24, 1), 0, A.PREC_FP64, True), ((4, 6), 8, A.PREC_FP32, True),
                                                  ((24, 1), 5, A.PREC_FP32, True), ((23, 1), 0, A.PREC_FP32, False),
                                                  ((26, 1), 0, A.PREC_FP32 | A.PREC_FP64, True)])
def test_coded_product(lattice, k, prec, coded):
    import torch
    L = lattice[0] * lattice[1]
    perm, ch = q.translation_group(*lattice)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[k])
    if lattice[1] == 1:
        t = q.xxz_terms(q.chain_bonds(L) + q.chain_bonds(L, 2), [1.0] * L + [0.5] * L, 0.7)
    else:
        t = q.xxz_terms(q.square_bonds(*lattice), 1.0, 0.7)
    h = q.Hamiltonian(s, t, prec=prec)
    i = h.info
    for p in (A.PREC_FP32, A.PREC_FP64):
        if not prec & p:
            continue
        assert bool(i.coded if p == A.PREC_FP32 else i.coded_fp64) == coded
        dt = {np.dtype("f4"): torch.float32, np.dtype("f8"): torch.float64, np.dtype("c8"): torch.complex64,
              np.dtype("c16"): torch.complex128}[np.dtype(h.dtype(p))]
        x = torch.randn(i.n_rows, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
        y, z = torch.empty_like(x), torch.empty_like(x)
        h.hv_dev(x.data_ptr(), y.data_ptr(), p)
        h.hv_dev(x.data_ptr(), z.data_ptr(), p, matrix_free=True)
        torch.cuda.synchronize()
        eps = 1.2e-7 if p == A.PREC_FP32 else 2.3e-16
        assert float((y - z).abs().max()) <= 4 * (i.max_row + 4) * eps * float(x.abs().max())
