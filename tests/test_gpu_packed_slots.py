"""The packed slot order of built matrices (a term's entries share a slot where
they fit) against the oracle's matrix, at the widths and row counts where it
changes course."""
import numpy as np
import pytest

import oracle as O
import qmbcuda_b200 as q
from helpers import oracle_group, oracle_terms

pytestmark = pytest.mark.gpu
A = q._capi


def _pairs(L, n):
    return [(i, j) for d in range(1, L) for i in range(L - d) for j in [i + d]][:n]


# (group sizes, L, n_up, bonds, momentum): rows 1, 31..33 (slice edges), slices up
# to 32, 33, 64 and 65 wide, null orbits, more than 1,024 mobile terms
CASES = [
    ("one_row", (1, 1), 6, 6, q.chain_bonds(6), 0),
    ("rows_3", (3, 1), 3, 1, q.chain_bonds(3), 1),
    ("rows_35", (1, 1), 7, 3, q.chain_bonds(7), 0),
    ("null_orbits", (12, 1), 12, 6, q.chain_bonds(12) + q.chain_bonds(12, 2), 3),
    ("torus", (4, 4), 16, 8, q.square_bonds(4, 4), 5),
    ("width_32", (1, 1), 12, 4, _pairs(12, 66), 0),
    ("width_36", (1, 1), 12, 6, _pairs(12, 66), 0),
    ("width_64", (1, 1), 16, 8, _pairs(16, 120), 0),
    ("width_72", (1, 1), 17, 8, _pairs(17, 136), 0),
    ("terms_1104", (1, 1), 24, 2, _pairs(24, 276) * 2, 0),
]


@pytest.mark.parametrize("name,lattice,L,n_up,bonds,k", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("prec", [A.PREC_FP32, A.PREC_FP64])
def test_packed_matrix_equals_the_oracle(name, lattice, L, n_up, bonds, k, prec):
    if lattice == (1, 1):
        perm, ch = np.arange(L, dtype=np.uint32)[None, :], np.ones((1, 1), complex)
    else:
        perm, ch = q.translation_group(*lattice)
    t = q.xxz_terms(bonds, np.linspace(0.8, 1.2, len(bonds)) if lattice == (1, 1) else 1.0, 0.6)
    s = q.Sector(L, n_up, perm).set_irrep(ch[k])
    h = q.Hamiltonian(s, t, prec=prec)
    sec = O.build_sector(oracle_group(perm, ch), n_up)
    rc, ind, val, tr = O.ell_terms(sec, oracle_terms(t), k, 2 * t.n_terms + 1)
    rows = O.active_rows(sec, k)
    M = O.ell_to_csr(ind, val, tr, rows)
    i = h.info
    assert (i.n_rows, i.nnz_offdiag, i.max_row) == (len(rows), int(np.sum(tr[rows] - 1)), int(np.max(tr[rows] - 1)))
    rng = np.random.default_rng(3)
    x = rng.standard_normal(len(rows)) + (1j * rng.standard_normal(len(rows)) if i.is_complex else 0)
    eps = 2.3e-16 if prec == A.PREC_FP64 else 1.2e-7
    x = x.astype(h.dtype(prec))
    # a row sums max_row + 1 products, each component of a complex one two more
    bound = 2 * (i.max_row + 3) * eps * (np.abs(M) @ np.abs(x)).max()
    assert np.abs(h.hv_host(x, prec) - (M @ x if i.is_complex else (M @ x).real)).max() <= bound
