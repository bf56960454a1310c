"""Matrix build: the dictionary collected on the device (samples, values that
the samples miss, more values than it holds) and values filled in one pass in
every precision."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("L,n_up,n_couplings,coded", [
    (13, 6, 1, True),    # 1,716 rows: two column blocks of 1,024, the last ragged
    (14, 7, 14, True),   # one value per bond
    (15, 7, 105, True),  # all pairs, one value each: some are rare in the sample
    (24, 3, 276, False), # more than 255 values: no coded layout
])
@pytest.mark.parametrize("prec", [A.PREC_FP32, A.PREC_FP64, A.PREC_FP32 | A.PREC_FP64])
def test_coded_build_equals_the_oracle(L, n_up, n_couplings, coded, prec, monkeypatch):
    monkeypatch.setenv("QMB_CB_SHIFT", "10")
    pairs = [(i, j) for i in range(L) for j in range(i + 1, L)]
    bonds = pairs if n_couplings > L else q.chain_bonds(L)
    J = np.linspace(0.5, 1.5, len(bonds)) if n_couplings > 1 else np.ones(len(bonds))
    perm = np.arange(L, dtype=np.uint32)[None, :]
    t = q.xxz_terms(bonds, J, 0.7)
    s = q.Sector(L, n_up, perm).set_irrep([1.0])
    h = q.Hamiltonian(s, t, prec=prec)
    g = oracle_group(perm, np.ones((1, 1)))
    sec = O.build_sector(g, n_up)
    rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), 0, 2 * t.n_terms + 1)
    M = O.ell_to_csr(ind, val, tr, O.active_rows(sec, 0)).real
    i = h.info
    off = M.copy()
    off.setdiag(0)
    off.eliminate_zeros()
    assert (i.n_rows, i.nnz_offdiag, i.max_row) == (M.shape[0], off.nnz, int(np.diff(off.indptr).max()))
    assert i.coded == int(coded and bool(prec & A.PREC_FP32) and i.n_rows > 1024)
    x = np.random.default_rng(L).standard_normal(M.shape[0])
    scale = np.abs(M).dot(np.abs(x)).max()
    if prec & A.PREC_FP64:
        # a row sums at most max_row + 1 products in FP64
        assert np.abs(h.hv_host(x) - M @ x).max() <= (i.max_row + 2) * 2.3e-16 * scale
    if prec & A.PREC_FP32:
        x32 = x.astype(np.float32)
        assert np.abs(h.hv_host(x32, A.PREC_FP32) - M @ x32.astype(np.float64)).max() <= (i.max_row + 2) * 1.2e-7 * scale
