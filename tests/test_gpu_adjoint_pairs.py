"""
The differentiable run's pair list by cells against the all-pairs build: the
same pairs in the same order (dense and sparse boxes, three cells per axis and
many, uneven boxes, positions outside the box by whole periods).
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,box,g", [(1, (4.0, 4.0, 4.0), (3, 3, 3)), (63, (4.0, 4.2, 5.4), (3, 3, 4)),
                                     (65, (9.2, 4.0, 4.0), (7, 3, 3)), (700, (9.7, 9.2, 10.5), (7, 7, 8)),
                                     (700, (40.0, 41.0, 42.0), (10, 10, 10)), (5000, (18.3, 17.0, 19.6), (14, 13, 15))])
def test_cells_equal_all_pairs(gpu, n, box, g):
    import torch
    from taichimps_gb300 import _device, _lib
    L, st = _device.lib(), _device.stream()
    rng = np.random.default_rng(n)
    prd, lo = np.array(box), np.array([1.5, -3.0, 0.0])
    r = rng.uniform(0.4, 0.6, size=n)
    skin = 0.1
    assert (prd / np.array(g) > 2 * 0.6 + skin).all()
    x = lo + rng.random((n, 3)) * prd
    x[::3] += prd * rng.integers(-2, 3, size=x[::3].shape)
    x[: n // 8, 0] = lo[0]  # on the seam
    rec = _lib.AdjRec()
    rec.lo[:], rec.prd[:] = lo.tolist(), prd.tolist()
    d_rec = torch.from_numpy(np.frombuffer(bytes(rec), dtype=np.uint8).copy()).cuda()
    d_x, d_r = torch.from_numpy(np.ascontiguousarray(x.T)).cuda(), torch.from_numpy(r).cuda()
    work = torch.empty(int(L.tmps_adj_cells_bytes(n, int(np.prod(g)))), dtype=torch.uint8, device="cuda")
    got = []
    for cells in (False, True):
        def call(*out):
            args = (n, d_x.data_ptr(), d_r.data_ptr(), d_rec.data_ptr(), skin)
            rc = (L.tmps_adj_pairs_cells(*args, *g, work.data_ptr(), *out, st) if cells
                  else L.tmps_adj_pairs(*args, *out, st))
            assert rc == _lib.TMPS_OK
        count = torch.zeros(n, dtype=torch.int32, device="cuda")
        call(count.data_ptr(), None, None, None)
        ibeg = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        ibeg[1:] = torch.cumsum(count, 0).to(torch.int32)
        m = int(ibeg[-1])
        pi, pj = (torch.full((max(m, 1),), -1, dtype=torch.int32, device="cuda") for _ in range(2))
        call(None, ibeg.data_ptr(), pi.data_ptr(), pj.data_ptr())
        got.append([a.cpu().numpy() for a in (count, ibeg, pi, pj)])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    if n > 1 and max(box) < 20.0:
        assert got[0][1][-1] > 0
    assert ctypes.sizeof(_lib.AdjRec) == len(bytes(rec))


def test_reverse_across_lists_of_unequal_length(gpu):
    """A run whose pair lists differ in length by more than a page of the workspace, against the same
    run on one wide list: the reverse's running values do not depend on a list's number of pairs."""
    import torch
    from taichimps_gb300.adjoint import stress_curve
    from taichimps_gb300.packing import compress_packing
    from test_gpu_adjoint import BASE, _run
    pk = compress_packing(343, seed=11)
    v = np.random.default_rng(4).normal(0.0, 3.0, size=pk["x"].shape)
    got = []
    for skin in (0.01, 0.3):
        run = _run(pk, 80, 20, 30, skin=skin, v=v)
        ps = {k: torch.tensor(a, dtype=torch.float64, requires_grad=True) for k, a in BASE.items()}
        r = torch.tensor(pk["radius"], dtype=torch.float64, device="cuda", requires_grad=True)
        q = stress_curve(run, ps["kn"], ps["kt"], ps["gamman"], ps["gammat"], ps["xmu"], r)
        (q ** 2).sum().backward()
        got.append((run, {k: float(a.grad) for k, a in ps.items()}, r.grad))
    (few, g, gr), (one, h, hr) = got
    counts = [p.npairs for p in few.lists]
    assert one.rebuilds == 0 and max(abs(a - b) for a, b in zip(counts, counts[1:])) >= 32, counts
    for k in BASE:  # the tolerance of the comparison with autograd
        assert abs(g[k] - h[k]) <= 1e-8 * abs(h[k]) + 1e-12, (k, g[k], h[k])
    assert (gr - hr).abs().max() <= 1e-8 * hr.abs().max()
