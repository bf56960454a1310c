"""Matrix-free products through the window lookup (QMB_MF_WINDOW=0: the bucket
search) against the stored product: chains with all rotations (odd keys), the
same with inversion, tori and no group (all keys), null orbits, general terms."""
import numpy as np
import pytest

import qmbcuda_b200 as q

pytestmark = pytest.mark.gpu
A = q._capi

# (lattice or L, n_up, flip, momentum)
CASES = [((12, 1), 6, True, 0), ((12, 1), 6, True, 6), ((13, 1), 5, False, 0), ((12, 1), 6, False, 4), ((9, 1), 1, False, 2),
         ((9, 1), 9, False, 0), ((10, 1), 0, False, 0), ((4, 4), 8, False, 5), ((3, 5), 7, False, 0), ((2, 9), 9, True, 3),
         ((32, 1), 2, False, 0), ((31, 1), 3, False, 7), (14, 7, False, 0), (32, 2, False, 0), ((20, 1), 10, True, 0)]


@pytest.mark.parametrize("lattice,n_up,flip,k", CASES)
@pytest.mark.parametrize("general", [False, True])
def test_window_lookup(lattice, n_up, flip, k, general, monkeypatch):
    import torch
    if isinstance(lattice, int):
        L = lattice
        perm, ch, row = np.arange(L, dtype=np.uint32)[None, :], None, np.ones(1, complex)
        bonds = q.chain_bonds(L)
    else:
        L = lattice[0] * lattice[1]
        perm, ch = q.translation_group(*lattice)
        row = ch[k]
        bonds = q.chain_bonds(L) if lattice[1] == 1 else q.square_bonds(*lattice)
    t = q.xxz_terms(bonds, 1.0, 0.7)
    if general:  # a term that is no plain exchange: the general loop
        t = t + q.operator_terms([(0.2, [("Sz", i), ("Sz", (i + 1) % L), ("Sp", i), ("Sm", (i + 1) % L)]) for i in range(L)])
    s = q.Sector(L, n_up, perm, spin_flip=flip).set_irrep(q.with_spin_flip(row, 1) if flip else row)
    if s.info.n_active == 0:
        return
    ys = []
    for win in ("1", "0"):
        monkeypatch.setenv("QMB_MF_WINDOW", win)
        h = q.Hamiltonian(s, t)
        n = h.info.n_rows
        dt = h.dtype(A.PREC_FP64)
        rng = np.random.default_rng(5)
        x = (rng.standard_normal(n) + (1j * rng.standard_normal(n) if h.info.is_complex else 0)).astype(dt)
        xd = torch.from_numpy(x).cuda()
        y = torch.full_like(xd, float("nan"))
        h.hv_dev(xd.data_ptr(), y.data_ptr(), A.PREC_FP64, matrix_free=True)
        torch.cuda.synchronize()
        ys.append(y.cpu().numpy())
        want = h.hv_host(x)
        # sums of at most 3 L products of values below 3
        assert np.abs(ys[-1] - want).max() <= 3 * L * 2.3e-16 * 9 * np.abs(x).max()
    assert np.array_equal(ys[0], ys[1])


@pytest.mark.parametrize("L,n_up,flip", [(1, 1, False), (2, 1, True), (7, 3, False), (8, 4, True), (8, 8, False), (8, 0, False),
                                         (17, 8, False), (22, 11, True), (32, 3, False)])
def test_chain_representatives(L, n_up, flip):
    """Representatives of all rotations: the minima of every orbit, by counting and checking each."""
    perm, _ = q.translation_group(L)
    s = q.Sector(L, n_up, perm, spin_flip=flip)
    reps = s.reps()
    full = (1 << L) - 1
    seen = 0
    for r in (int(v) for v in reps[:: max(1, len(reps) // 2000)]):
        im = {((r << k) | (r >> (L - k))) & full for k in range(L)}
        if flip:
            im |= {v ^ full for v in im}
        assert min(im) == r
    for r in (int(v) for v in reps) if len(reps) <= 5000 else ():
        im = {((r << k) | (r >> (L - k))) & full for k in range(L)}
        seen += len(im | ({v ^ full for v in im} if flip else set()))
    if seen:
        assert seen == s.info.n_states
