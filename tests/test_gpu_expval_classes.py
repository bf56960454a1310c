"""Observables by classes of terms: products of Sz over up to eight sites at the
numbers of masks and rows where the sign sums change shape, on strings of up to
and beyond 32 sites, against direct sums over the strings."""
import itertools

import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu


def _strings(L, n_up):
    return np.array([sum(1 << b for b in c) for c in itertools.combinations(range(L), n_up)], dtype=np.uint64)


def _sz(states, i):
    return ((states >> np.uint64(i)) & np.uint64(1)).astype(float) - 0.5


@pytest.mark.parametrize("L,n_up", [(5, 5), (8, 1), (9, 4), (13, 6), (32, 2), (33, 2), (40, 3), (64, 1)])
@pytest.mark.parametrize("n_ops", [1, 7, 8, 9, 40])
def test_products_of_sz_without_a_group(L, n_up, n_ops):
    perm = np.arange(L, dtype=np.uint32)[None, :]
    s = q.Sector(L, n_up, perm).set_irrep([1.0])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.5))
    states = np.sort(_strings(L, n_up))
    rng = np.random.default_rng(L + n_ops)
    psi = rng.standard_normal(len(states))
    h.set_ground_state(psi)
    ops, want = [], []
    p = psi * psi / (psi @ psi)
    for k in range(n_ops):
        terms, w = [], 0.0
        for _ in range(3):
            sites = rng.integers(0, L, size=rng.integers(0, 9))  # repeated sites among them
            c = complex(rng.standard_normal(), rng.standard_normal())
            terms.append((c, [("Sz", int(i)) for i in sites]))
            w += c * np.sum(p * np.prod([_sz(states, int(i)) for i in sites], axis=0) if len(sites) else p)
        ops.append(q.operator_terms(terms))
        want.append(w)
    # sums of len(states) terms of at most 3 in FP64
    assert np.abs(h.expval(ops) - np.array(want)).max() <= 1e-14 * (10 + np.sqrt(len(states)))


def test_inversion_makes_odd_products_vanish():
    L = 8
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm, spin_flip=True).set_irrep(q.with_spin_flip(ch[0], 1))
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.7))
    n = h.info.n_rows
    psi = np.random.default_rng(2).standard_normal(n)
    h.set_ground_state(psi)
    odd = [q.operator_terms([(1.0, [("Sz", i)]), (0.5, [("Sz", i), ("Sz", 1), ("Sz", 2)])]) for i in range(3, L)]
    assert np.abs(h.expval(odd)).max() == 0.0
    # S+_0 Sz_2 S-_4 and its image under inversion have opposite values
    a = h.expval([q.operator_terms([(1.0, [("Sp", 0), ("Sz", 2), ("Sm", 4)])]),
                  q.operator_terms([(1.0, [("Sm", 0), ("Sz", 2), ("Sp", 4)])])])
    assert abs(a[0] + a[1]) <= 1e-15


def test_slabs_of_rows():
    """More rows than one pass of the sign sums takes (2^23): <Sz Sz> of a uniform state."""
    L, n_up = 26, 12  # 9,657,700 strings
    perm = np.arange(L, dtype=np.uint32)[None, :]
    s = q.Sector(L, n_up, perm).set_irrep([1.0])
    h = q.Hamiltonian(s, q.xxz_terms([(0, 1)], 1.0, 0.5), prec=q._capi.PREC_FP32)
    n = h.info.n_rows
    h.set_ground_state(np.ones(n))
    m = 2 * n_up - L
    corr = (m * m - L) / (4.0 * L * (L - 1))  # two distinct sites of a uniform superposition
    v = h.expval([q.operator_terms([(1.0, [("Sz", 0), ("Sz", j)])]) for j in (1, 13, 25)])
    assert np.abs(v - corr).max() <= 1e-14
