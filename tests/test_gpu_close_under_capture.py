"""Closing a handle while another thread captures a graph: a capture of its own
thread's mode is left alone, and the handle's memory is not handed out."""
import threading

import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


def test_close_leaves_a_thread_local_capture_alone():
    import torch
    perm, ch = q.translation_group(12)
    s = q.Sector(12, 6, perm).set_irrep(ch[0])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(12), 1.0, 0.8))
    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    started, closed, broke = threading.Event(), threading.Event(), []

    def capture():
        try:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.stream(torch.cuda.Stream()):
                g.capture_begin(capture_error_mode="thread_local")
                x.add_(1.0)
                started.set()
                closed.wait(20)
                x.add_(1.0)
                g.capture_end()
            g.replay()
            torch.cuda.synchronize()
        except Exception as e:  # a capture that was invalidated
            broke.append(str(e))

    t = threading.Thread(target=capture)
    t.start()
    assert started.wait(20)
    h.close()
    s.close()
    closed.set()
    t.join()
    assert not broke, broke
    assert x.tolist() == [2.0] * 8
