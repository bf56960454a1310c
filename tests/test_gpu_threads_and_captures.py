"""Calls of the library while another thread captures a graph in thread-local mode:
the capture is left alone, a batched solve's own loop among them."""
import threading

import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


def _under_capture(call):
    """Runs call() while another thread captures two additions, which then replay."""
    import torch
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    started, done, broke = threading.Event(), threading.Event(), []

    def capture():
        try:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.stream(torch.cuda.Stream()):
                g.capture_begin(capture_error_mode="thread_local")
                x.add_(1.0)
                started.set()
                done.wait(60)
                x.add_(1.0)
                g.capture_end()
            g.replay()
            torch.cuda.synchronize()
        except Exception as e:  # a capture that was invalidated
            broke.append(str(e))

    t = threading.Thread(target=capture)
    t.start()
    assert started.wait(20)
    try:
        r = call()
    finally:
        done.set()
        t.join()
    assert not broke, broke
    assert x.tolist() == [2.0] * 8
    return r


def _handles(L=12, k=0):
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[k])
    return s, q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))


def _batch(L=10, n_sets=5):
    perm, ch = q.translation_group(L)
    ss = [q.Sector(L, L // 2, perm).set_irrep(ch[k]) for k in (0, 2, 3)]
    return q.Batch(ss, q.xxz_terms(q.chain_bonds(L), 1.0, 0.0, "xy"), q.xxz_terms(q.chain_bonds(L), 0.0, 1.0, "z"), n_sets)


J, D = np.linspace(0.8, 1.2, 5), np.linspace(0.3, 1.1, 5)


def _build_and_solve():
    s, h = _handles(14, 3)
    op = q.operator_terms([(1.0, [("Sz", 0), ("Sz", 1)]), (0.5, [("Sp", 0), ("Sm", 3)])])
    out = [h.lanczos(tol=1e-11, want_vector=1).E0, h.lanczos(tol=1e-11, reorth=2, mode=A.MODE_MIXED).E0,
           h.lanczos(tol=1e-11, hv=A.HV_MATRIX_FREE).E0, h.expval(op), float(s.orbit_map().sum()), s.active()[-1]]
    h.close()
    s.close()
    b = _batch()
    for mode in (A.MODE_FP64, A.MODE_MIXED):
        out.extend(b.solve(J, J * D, mode=mode, tol=1e-10)[0].ravel())
    b.close()
    q.trim()
    return out


def test_builds_and_solves_leave_a_thread_local_capture_alone():
    want = _build_and_solve()
    assert _under_capture(_build_and_solve) == want


def test_batched_solves_while_another_thread_builds():
    b = _batch()
    want = b.solve(J, J * D, tol=1e-10)[0]
    stop, errors = threading.Event(), []

    def build():
        try:
            while not stop.is_set():
                s, h = _handles(13, 2)
                h.lanczos(tol=1e-10)
                h.close()
                s.close()
        except q.QMBError as e:
            errors.append(str(e))

    t = threading.Thread(target=build)
    t.start()
    try:
        for _ in range(20):
            assert np.array_equal(b.solve(J, J * D, tol=1e-10)[0], want)
    finally:
        stop.set()
        t.join()
    b.close()
    assert not errors, errors
