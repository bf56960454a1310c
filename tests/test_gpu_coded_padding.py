"""Padding of coded entries gathers the row's own x, as that of the plain entries:
an infinity in one element reaches the rows that hold its column and no others."""
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("L,k,prec", [(24, 0, A.PREC_FP64), (24, 5, A.PREC_FP32), (26, 0, A.PREC_FP32)])
def test_infinity_in_the_first_element(L, k, prec, monkeypatch):
    import torch
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[k])
    t = q.xxz_terms(q.chain_bonds(L) + q.chain_bonds(L, 2), [1.0] * L + [0.5] * L, 0.7)
    out = []
    for coded in (True, False):
        if not coded:
            monkeypatch.setenv("QMB_COLUMN_BLOCKS", "0")
        h = q.Hamiltonian(s, t, prec=prec)
        i = h.info
        assert bool(i.coded if prec == A.PREC_FP32 else i.coded_fp64) == coded
        assert i.padded > i.nnz_offdiag  # there is padding
        dt = {(A.PREC_FP64, 0): torch.float64, (A.PREC_FP32, 0): torch.float32,
              (A.PREC_FP32, 1): torch.complex64}[(prec, i.is_complex)]
        x = torch.ones(i.n_rows, dtype=dt, device="cuda")
        x[0] = float("inf")
        y = torch.empty_like(x)
        h.hv_dev(x.data_ptr(), y.data_ptr(), prec)
        torch.cuda.synchronize()
        out.append(torch.isfinite(torch.view_as_real(y)).all(1) if i.is_complex else torch.isfinite(y))
        h.close()
    assert torch.equal(out[0], out[1])
    n_bad = int((~out[0]).sum())
    assert 1 <= n_bad <= 4 * L + 1  # the rows connected to row 0
