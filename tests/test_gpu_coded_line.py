"""Where real FP32 entries become coded (70 MB of plain entries): products on both
sides of the line against the matrix-free ones."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


# 54.5, 65.3 and 74.3 MB of plain entries
@pytest.mark.parametrize("L,n_up,k,j2,coded", [(21, 9, None, 0.5, 0), (26, 11, 0, 0.5, 0), (22, 11, None, 0.0, 1)])
def test_real_fp32(L, n_up, k, j2, coded):
    import torch
    perm, ch = (np.arange(L, dtype=np.uint32)[None, :], np.ones((1, 1))) if k is None else q.translation_group(L)
    s = q.Sector(L, n_up, perm).set_irrep(ch[k or 0])
    bonds = q.chain_bonds(L) + (q.chain_bonds(L, 2) if j2 else [])
    h = q.Hamiltonian(s, q.xxz_terms(bonds, [1.0] * L + [j2] * (len(bonds) - L), 0.5), prec=A.PREC_FP32)
    i = h.info
    assert not i.is_complex and i.coded == coded
    x = torch.randn(i.n_rows, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    y, z = torch.empty_like(x), torch.empty_like(x)
    h.hv_dev(x.data_ptr(), y.data_ptr(), A.PREC_FP32)
    h.hv_dev(x.data_ptr(), z.data_ptr(), A.PREC_FP32, matrix_free=True)
    torch.cuda.synchronize()
    assert float((y - z).abs().max()) <= 4 * (i.max_row + 4) * 1.2e-7 * float(x.abs().max())
