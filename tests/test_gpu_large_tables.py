"""Matrix-free products and solves whose term and group tables fill a block's shared
memory almost to its limit, against the stored product."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("n_terms", [1500, 3400, 3700])
def test_general_terms(n_terms):
    L, n_up = 13, 6
    mirror = np.arange(L, dtype=np.uint32)[::-1]
    # 96 times the group of a mirror: 96 KB of tables, 36 bytes a term
    perm = np.concatenate([np.stack([np.arange(L, dtype=np.uint32), mirror])] * 96)
    s = q.Sector(L, n_up, perm).set_irrep(np.ones(192))
    rng = np.random.default_rng(n_terms)
    terms = []
    while len(terms) < n_terms:  # a term, its adjoint and both mirror images
        a = [int(v) for v in rng.permutation(L)[:3]]
        c = rng.standard_normal() / n_terms
        for x in (a, [L - 1 - v for v in a]):
            for i, j in ((x[0], x[1]), (x[1], x[0])):
                terms.append((c, [("Sp", i), ("Sm", j), ("Sz", x[2])]))
    terms[0] = (terms[0][0], terms[0][1] + [("I", 0)] * 5)  # eight columns
    h = q.Hamiltonian(s, q.operator_terms(terms), prec=A.PREC_FP64)
    import torch
    n = h.info.n_rows
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    y, z = torch.empty_like(x), torch.empty_like(x)
    h.hv_dev(x.data_ptr(), y.data_ptr(), A.PREC_FP64)
    h.hv_dev(x.data_ptr(), z.data_ptr(), A.PREC_FP64, matrix_free=True)
    torch.cuda.synchronize()
    assert float((y - z).abs().max()) <= 1e-14 * float(y.abs().max()) * 100
    e = h.lanczos(tol=1e-11, max_iter=600).E0
    m = h.lanczos(tol=1e-11, max_iter=600, hv=A.HV_MATRIX_FREE).E0
    assert abs(e - m) <= 1e-9 * abs(e)
