"""Freed device buffers are kept and handed out again: results with reuse
across handles, streams and threads, and the bound on what is kept."""
import threading

import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


def _sector(L, k=0):
    perm, ch = q.translation_group(L)
    return q.Sector(L, L // 2, perm).set_irrep(ch[k])


def _product(L, k=0, seed=0):
    s = _sector(L, k)
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    n = h.info.n_rows
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(n) + (1j * rng.standard_normal(n) if h.info.is_complex else 0)
    y = h.hv_host(x)
    e = h.lanczos(tol=1e-12).E0
    h.close()
    s.close()
    return y, e


def test_reuse_in_threads_gives_the_same_results():
    sizes = [(10, 0), (13, 2), (16, 5), (12, 6)]
    want = {c: _product(*c) for c in sizes}
    bad = []

    def work(t):
        for r in range(6):
            c = sizes[(t + r) % len(sizes)]
            y, e = _product(*c)
            if not (np.array_equal(y, want[c][0]) and e == want[c][1]):
                bad.append((t, r, c))

    th = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not bad


def test_handle_closed_while_its_products_run():
    """Closing a handle waits for products on the caller's stream: its buffers
    go to the next handle only when they are idle."""
    import torch
    L = 22
    s = _sector(L)
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8), prec=A.PREC_FP64)
    n = h.info.n_rows
    x = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    want = torch.empty_like(x)
    h.hv_dev(x.data_ptr(), want.data_ptr(), A.PREC_FP64)
    torch.cuda.synchronize()
    ys = [torch.empty_like(x) for _ in range(64)]
    st = torch.cuda.Stream()
    for y in ys:
        h.hv_dev(x.data_ptr(), y.data_ptr(), A.PREC_FP64, st.cuda_stream)
    h.close()
    s.close()
    s2 = _sector(L, 3)  # takes the freed buffers
    h2 = q.Hamiltonian(s2, q.xxz_terms(q.chain_bonds(L), 1.0, 0.3))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want) for y in ys)
    h2.close()
    s2.close()


def test_kept_memory_is_bounded():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    _product(10)
    free0 = torch.cuda.mem_get_info()[0]
    for L in (20, 22, 24, 26, 23, 25):
        _product(L)
    # 512 MB are kept at most; two allocation granules of slack for each buffer size
    assert free0 - torch.cuda.mem_get_info()[0] <= (512 + 64) << 20


def test_trim_gives_kept_memory_back():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    s = _sector(24)
    q.trim()
    free0 = torch.cuda.mem_get_info()[0]
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(24), 1.0, 0.8))
    h.lanczos(tol=1e-10)
    h.close()
    assert torch.cuda.mem_get_info()[0] < free0  # kept for reuse
    q.trim()
    # (kernels loaded meanwhile may hold a few allocation granules)
    assert free0 - torch.cuda.mem_get_info()[0] <= 8 << 20
    with pytest.raises(q.QMBError):
        q.trim(99)


def test_observables_where_memory_is_short():
    """9,657,700 rows with 48 MB of device memory left: the sign sums' scratch
    (100 MB with memory to spare) shrinks, and the values stay."""
    import torch
    L, n_up = 26, 12
    s = q.Sector(L, n_up, np.arange(L, dtype=np.uint32)[None, :]).set_irrep([1.0])
    h = q.Hamiltonian(s, q.xxz_terms([(0, 1)], 1.0, 0.5), prec=A.PREC_FP32)
    h.set_ground_state(np.ones(h.info.n_rows))
    ops = [q.operator_terms([(1.0, [("Sz", 0), ("Sz", j)])]) for j in (1, 13, 25)]
    want = h.expval(ops)
    q.trim()
    torch.cuda.empty_cache()
    rest = torch.cuda.mem_get_info()[0] - (48 << 20)
    hog = torch.empty(rest, dtype=torch.uint8, device="cuda")
    try:
        got = h.expval(ops)
    finally:
        del hog
        torch.cuda.empty_cache()
    m = 2 * n_up - L
    assert np.abs(got - want).max() <= 1e-14
    assert np.abs(got - (m * m - L) / (4.0 * L * (L - 1))).max() <= 1e-14
