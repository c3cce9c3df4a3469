"""
The calls of the differentiable run's C interface: each is ordered after whatever was queued before it (its
kernels read ahead of their dependency wait only what their own call's earlier launches settled), the queue's
last finished step, and the reverse one step a call (tmps_adj_step_back) against the queued reverse.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _job(steps=12, every=4, ckpt=5, skin=0.1, v=0.5):
    from taichimps_gb300.adjoint import AdjointRun
    from taichimps_gb300.packing import compress_packing
    pk = compress_packing(512, seed=5)
    axes = {"x": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
            "y": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1}, "z": {"style": "erate", "rate": -1e-3}}
    return AdjointRun(pk["x"], pk["radius"], pk["density"], pk["lo"], pk["lo"] + pk["L"], dt=5e-5, steps=steps, axes=axes,
                      max_rate=1e-2, sample_every=every, checkpoint_every=ckpt, skin=skin,
                      v=np.random.default_rng(8).normal(0.0, v, size=pk["x"].shape))


PRM = dict(kn=1.0e5, kt=1.0e5 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5)


def test_first_half_after_a_queued_run(gpu):
    """tmps_adj_initial right behind tmps_adj_forward, whose last kernel writes the positions that are both its
    state and its reference: the largest displacement is |dt v|, never one to other positions."""
    import torch
    from taichimps_gb300 import _device
    from taichimps_gb300.adjoint import _p, _Tapes
    job = _job(steps=8, ckpt=8)
    job.forward(**PRM)
    L, st = _device.lib(), _device.stream()
    state, li = job.ckpt[0][0], job.ckpt[0][2]
    pairs = job.lists[li]
    queue, disp = torch.zeros(2, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    work = job._work(pairs.npairs)
    a, b = _Tapes(1, job.n, pairs.npairs, job.dev), _Tapes(1, job.n, pairs.npairs, job.dev)
    for rep in range(20):
        s = {k: t.clone() for k, t in state.items()}
        shear = job.ckpt[0][1].clone()
        sys = job._sys(s, pairs, shear)
        assert L.tmps_adj_forward(sys, job.prm, job.servo, a.cstruct(), 0, 0, job.rec.data_ptr(), 1, 6, _p(s["x"]),
                                  float("inf"), _p(queue), _p(work), st) == 0
        disp.zero_()
        assert L.tmps_adj_initial(sys, job.prm, b.cstruct(), _p(s["x"]), _p(disp), st) == 0
        want = ((b.field(0, "xh") - s["x"]) ** 2).sum(0).max()
        got = disp.view(torch.float64)[0]
        # (x + dt v) - x, squared and summed, in another order
        assert float((got - want).abs()) <= 1e-14 * float(want), (rep, float(got), float(want))
        assert queue.tolist() == [0, 6]


def test_reverse_one_step_a_call(gpu, monkeypatch):
    import torch
    from taichimps_gb300 import _device, _lib, adjoint
    job = _job(skin=0.002, v=3.0)  # a rebuild on the way
    q = job.forward(**PRM)
    assert job.rebuilds > 0
    qbar = torch.linspace(1.0, 2.0, len(q), dtype=torch.float64)
    want = {k: v.clone() if torch.is_tensor(v) else v for k, v in job.backward(qbar).items()}
    lib = _device.lib()

    def reverse(sys, prm, servo, tape, astride, pstride, rec, first, last, fprev, tprev, xprev, linked, qb, bar, work, st):
        n = last - first + 2
        q = np.ctypeslib.as_array(ctypes.cast(qb, ctypes.POINTER(ctypes.c_double)), (n,))

        def at(k):
            t = _lib.AdjTape()
            for name, _ in _lib.AdjTape._fields_:
                step = {"shear": 24 * pstride, "mask": pstride}.get(name, 8 * astride)
                setattr(t, name, getattr(tape, name) + step * k)
            return t

        for s in range(last, first - 1, -1):
            t = at(s - first)
            f, tq = (fprev, tprev) if s == first else (at(s - first - 1).f, at(s - first - 1).t)
            own = _lib.AdjSys.from_buffer_copy(sys)
            rc = lib.tmps_adj_step_back(own, prm, servo, t, rec, s, f, tq, float(q[s - first + 1]), bar, work, st)
            if rc:
                return rc
        return 0

    class Calls:
        tmps_adj_reverse = staticmethod(reverse)

        def __getattr__(self, name):
            return getattr(lib, name)

    monkeypatch.setattr(adjoint._device, "lib", lambda: Calls())
    got = job.backward(qbar)
    for k, w in want.items():
        w, g = torch.as_tensor(w).cpu(), torch.as_tensor(got[k]).cpu()
        assert float((w - g).abs().max()) <= 1e-12 * float(w.abs().max()), k


def test_queue_follows_the_rebuilds(gpu):
    """Frequent rebuilds under one long checkpoint: the launches stay near five a step, and the run is that of
    short checkpoints bit for bit."""
    from taichimps_gb300 import _device
    got = []
    for ckpt in (300, 7):
        job = _job(steps=300, every=50, ckpt=ckpt, skin=0.005, v=3.0)
        n0 = _device.lib().tmps_launch_count()
        q = job.forward(**PRM)
        got.append((q.cpu().numpy(), job.q_all(), job.rebuilds, _device.lib().tmps_launch_count() - n0))
    (qa, ra, na, la), (qb, rb, nb, _) = got
    assert na == nb >= 10
    np.testing.assert_array_equal(qa, qb)
    np.testing.assert_array_equal(ra, rb)
    # five launches a step, a remap per queue, a pair list (some 20 launches) per rebuild, and as much again
    # for what is queued past a rebuild
    assert la < 2 * (6 * 300 + 20 * na), la
