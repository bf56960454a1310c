"""Solves of different step limits in several threads at once: the reorthogonalised
kernel's shared memory grows with the limit, and each launch gets its own."""
import threading

import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi


@pytest.mark.parametrize("L,mode", [(10, A.MODE_FP64), (12, A.MODE_MIXED)])
def test_step_limits_in_threads(L, mode):
    perm, ch = q.translation_group(L)
    errors, energies = [], []

    def work(limits):
        s = q.Sector(L, L // 2, perm).set_irrep(ch[0])
        h = q.Hamiltonian(s, q.xxz_terms(q.chain_bonds(L), 1.0, 0.8))
        try:
            for i in range(60):
                energies.append(h.lanczos(mode=mode, tol=1e-11, reorth=2, max_iter=limits[i % len(limits)]).E0)
        except q.QMBError as e:
            errors.append(str(e))
        h.close()
        s.close()

    th = [threading.Thread(target=work, args=(m,)) for m in ([4000], [70], [3300], [80, 2000])]
    [t.start() for t in th]
    [t.join() for t in th]
    assert not errors, errors
    assert len(energies) == 240 and max(energies) - min(energies) <= 1e-10 * abs(energies[0])
