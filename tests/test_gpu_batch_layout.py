"""Vectors of a batch: the sectors of a kind lie in the caller's order, whichever of
them a solve runs, and the product acts on each sector in its place."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("L,order,n_sets", [(10, [7, 3, 0, 9, 5, 1], 3), (9, [5, 4, 8, 1, 2, 7, 0], 33), (8, [3, 5], 40),
                                            (8, [0, 4], 2)])
@pytest.mark.parametrize("prec", [A.PREC_FP64, A.PREC_FP32])
def test_offsets_and_product(L, order, n_sets, prec, monkeypatch):
    import torch
    monkeypatch.setenv("QMB_MERGE_REAL", "0")
    perm, ch = q.translation_group(L)
    bonds = q.chain_bonds(L)
    secs = [q.Sector(L, L // 2, perm).set_irrep(ch[a]) for a in order]
    b = q.Batch(secs, q.xxz_terms(bonds, 1.0, 0.0, part="xy"), q.xxz_terms(bonds, 0.0, 1.0, part="z"), n_sets)
    J, D = np.linspace(0.7, 1.3, n_sets), np.linspace(0.2, 1.1, n_sets)
    b.solve(J, J * D, tol=1e-8)  # sets the couplings of the product
    off, cplx = b.layout()
    stride = b.info.set_stride
    at = [0, sum(stride * s.info.n_active for s, c in zip(secs, cplx) if not c)]  # real kind, then complex
    for i, s in enumerate(secs):
        assert off[i] == at[cplx[i]], (i, off, cplx)
        at[cplx[i]] += stride * s.info.n_active * (2 if cplx[i] else 1)
    assert off[-1] == at[1]
    real = torch.float64 if prec == A.PREC_FP64 else torch.float32
    x = torch.randn(int(off[-1]), dtype=real, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    y = torch.zeros_like(x)
    b.hv_dev(x.data_ptr(), y.data_ptr(), prec)
    torch.cuda.synchronize()
    xh, yh = x.cpu().double().numpy(), y.cpu().double().numpy()
    for i, s in enumerate(secs):
        n, m = s.info.n_active, 2 if cplx[i] else 1
        cut = lambda v: v[off[i]:off[i] + n * stride * m]
        xs, ys = ((cut(v).view(np.complex128) if m == 2 else cut(v)).reshape(n, stride) for v in (xh, yh))
        for j in (0, n_sets - 1):
            h = q.Hamiltonian(s, q.xxz_terms(bonds, J[j], J[j] * D[j]), prec=A.PREC_FP64)
            want = h.hv_host(xs[:, j].copy() if m == 1 or h.info.is_complex else xs[:, j].real.copy())
            eps = 2.3e-16 if prec == A.PREC_FP64 else 1.2e-7
            assert np.abs(ys[:, j] - want).max() <= 8 * (2 * L + 4) * eps * np.abs(xs[:, j]).max()
    b.close()
