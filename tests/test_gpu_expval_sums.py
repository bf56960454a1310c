"""Operators that share some of their hopping terms: values of one call against
those of calls with one operator each, where every term belongs to that
operator's sum; and an operator of more terms than one launch takes."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu


def _handle(L, k, grouped):
    perm, ch = q.translation_group(L) if grouped else (np.arange(L, dtype=np.uint32)[None, :], np.ones((1, 1), complex))
    s = q.Sector(L, L // 2, perm).set_irrep(ch[k])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.7))
    n = h.info.n_rows
    rng = np.random.default_rng(L + k)
    h.set_ground_state(rng.standard_normal(n) + (1j * rng.standard_normal(n) if h.info.is_complex else 0))
    return h, rng


def _term(L, rng):
    a = [int(v) for v in rng.permutation(L)[:rng.integers(2, 5)]]
    return complex(*rng.standard_normal(2)), [("Sp", a[0]), ("Sm", a[1])] + [("Sz", v) for v in a[2:]]


@pytest.mark.parametrize("L,k,grouped", [(8, 0, False), (10, 0, True), (10, 3, True)])
@pytest.mark.parametrize("n_ops", [2, 3, 9])
def test_shared_terms(L, k, grouped, n_ops):
    h, rng = _handle(L, k, grouped)
    pool = [_term(L, rng) for _ in range(6)]
    ops, size = [], 0.0
    for i in range(n_ops):
        own = [_term(L, rng) for _ in range(i % 3)]
        shared = [(c * (i + 1), f) for c, f in pool[i % 4:i % 4 + 3]]
        diag = [(0.5, [("Sz", 0), ("Sz", i % L)])]
        ops.append(q.operator_terms(own + shared + diag))
        size = max(size, sum(abs(c) for c, _ in own + shared + diag))
    got = h.expval(ops)
    want = np.array([h.expval(o) for o in ops])
    # a term's value is at most 1, its sum over the rows one of some hundred FP64 products
    assert np.abs(got - want).max() <= 1e-14 * size


def test_more_terms_than_one_launch_takes():
    L = 16
    h, rng = _handle(L, 0, True)
    terms = [_term(L, rng) for _ in range(700)]  # up to 11,200 images, some 7,000 a launch
    whole = h.expval(q.operator_terms(terms))
    parts = sum(h.expval(q.operator_terms(terms[i:i + 50])) for i in range(0, 700, 50))
    assert abs(whole - parts) <= 1e-14 * sum(abs(c) for c, _ in terms)
