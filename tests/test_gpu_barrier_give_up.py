"""A grid barrier of the resident Lanczos kernel that gives up: the call reports a
timeout, and the handle solves as before afterwards."""
import ctypes as C

import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi
L = 18  # 2,704 rows in 43 row blocks


@pytest.mark.parametrize("mode,reorth", [(A.MODE_FP64, 0), (A.MODE_FP64, 2), (A.MODE_MIXED, 0)])
def test_handle_after_a_timeout(mode, reorth, monkeypatch):
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[0])
    h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
    o = dict(mode=mode, reorth=reorth, tol=1e-11, max_iter=200, want_vector=1)
    want = h.lanczos(**o).E0
    psi = h.ground_state()
    monkeypatch.setenv("QMB_LZ_BAR_SPINS", "0")  # one poll
    with pytest.raises(q.QMBError) as e:
        h.lanczos(**o)
    assert e.value.status == A.QMB_ERR_TIMEOUT
    assert np.array_equal(h.ground_state(), psi)  # the state of the last solve that ended
    monkeypatch.delenv("QMB_LZ_BAR_SPINS")
    assert h.lanczos(**o).E0 == want
    assert np.array_equal(h.ground_state(), psi)


def test_static_scratch_after_a_timeout(monkeypatch):
    import torch
    perm, ch = q.translation_group(L)
    s = q.Sector(L, L // 2, perm).set_irrep(ch[0])
    ind, val, tr = q.export_ref(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8), 2 * L + 1)
    t = [torch.tensor(ind.astype(np.int64)).to(torch.int32).cuda(), torch.tensor(val.real.astype(np.float32)).cuda(),
         torch.tensor(tr.astype(np.int16)).cuda()]
    torch.cuda.synchronize()

    def call(f, *extra):
        E, r, kry = C.c_float(), C.c_float(), np.zeros(60, np.float32)
        st = f(C.byref(E), 60, *ind.shape, 7, *(C.c_void_p(x.data_ptr()) for x in t), 0, A.ptr(kry), 1, C.byref(r), *extra)
        return st, E.value, r.value, kry.tobytes()

    for f, extra in ((q.lib().qmb_lanczos_ref_ell, ()), (q.lib().qmb_lanczos_ref_ell_noalloc, (None,))):
        want = call(f, *extra)
        assert want[0] == A.QMB_OK
        monkeypatch.setenv("QMB_LZ_BAR_SPINS", "0")
        assert call(f, *extra)[0] == A.QMB_ERR_TIMEOUT
        monkeypatch.delenv("QMB_LZ_BAR_SPINS")
        assert call(f, *extra) == want
