"""
Runs of a few steps on a list that stands: what the host waits for, and that the contact path follows the list.
"""

import numpy as np
import pytest

from _twin import dense_packing, gpu_state, make_twin

pytestmark = pytest.mark.gpu


def _sim(oracle, lo=0.50, hi=0.56):
    rng = np.random.default_rng(6)
    x, r = dense_packing(rng, 343, 7.0, lo, hi)
    sim, _ = make_twin(oracle, x, r, 2.5, [0.0] * 3, [7.0] * 3, v=rng.normal(scale=0.1, size=x.shape),
                       pair="hertz/history", dt=5e-5, skin=0.1, cundall=(0.7, 0.7))
    return sim


def test_one_wait_a_run(gpu, oracle, monkeypatch):
    """FP64 runs on the list of the run before: one read-back each, at the end (the counts were read with the
    list).  A build drops them."""
    from taichimps_gb300 import _device
    sim = _sim(oracle)
    sim.run(2)
    kept = sim.neighbor.counts
    assert kept is not None and sim.last_engine.rows
    sim.run_pre = False
    calls = []
    pull = _device.pull_many
    monkeypatch.setattr(_device, "pull_many", lambda items: (calls.append(len(items)), pull(items))[1])
    for k in range(1, 4):
        sim.run(1)
        assert len(calls) == k and sim.last_engine.rows and sim.neighbor.counts == kept
    sim.reneighbor_if_needed(force=True)
    assert sim.neighbor.counts is None
    sim.run(1)
    nnb = sim.neighbor.nnb.cpu().numpy()
    assert sim.neighbor.counts[1] * 2 == int(nnb.sum())


@pytest.mark.parametrize("loose_first", [True, False])
def test_path_follows_the_list(gpu, oracle, loose_first):
    """Radii changed between runs with a build: the next list is counted anew."""
    sim = _sim(oracle)
    r = sim.atom.radius.to_numpy()[:343].copy()
    for loose in (loose_first, not loose_first):
        sim.atom.radius.from_numpy(r * (0.8 if loose else 1.0))
        sim.run(3)
        assert sim.last_engine.rows == (not loose)
    assert np.isfinite(gpu_state(sim)["f"]).all()


def test_few_mixed_steps_stay_screened(gpu, oracle):
    """The shortest runs do not number the pairs; the two paths agree within the mixed form's rounding."""
    runs = []
    for steps in (4, 5):
        sim = _sim(oracle)
        sim.precision = "mixed"
        sim.run(steps)
        assert sim.last_engine.rows == (steps == 5)
        assert (sim.neighbor.counts is not None) == (steps == 5)
        runs.append(sim)
    whole, parts = _sim(oracle), runs[0]
    whole.precision = "mixed"
    whole.run(5)
    parts.run_pre = False
    parts.run(1)
    a, b = gpu_state(whole), gpu_state(parts)
    for k in ("x", "v", "f"):
        assert np.abs(a[k] - b[k]).max() <= 1e-4 * np.abs(a[k]).max(), k


@pytest.mark.parametrize("steps,fused", [(2, False), (11, False), (12, True)])
def test_few_steps_with_walls_go_hook_by_hook(gpu, steps, fused):
    """Setting the fused step up costs what a dozen steps with walls save; the results are the hooks' either way."""
    import taichimps_gb300 as G

    def run(on):
        rng = np.random.default_rng(2)
        g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5
        dom = G.Domain(boxlo=[0.0] * 3, boxhi=[4.0] * 3, boundary=("f", "f", "f"))
        atom = G.AtomSystem(max_atoms=64)
        atom.add_particles(x=g + rng.uniform(-0.04, 0.04, size=g.shape), radius=rng.uniform(0.48, 0.52, size=64),
                           density=np.full(64, 2.5), v=rng.normal(0.0, 1.0, size=g.shape))
        law = dict(kn=2e5, kt=2e5 * 2 / 7, gamman=50.0, gammat=25.0, xmu=0.5)
        sim = G.Simulation(domain=dom, atom=atom, neighbor=G.NeighborList(domain=dom, skin=0.02, max_atoms=64),
                           history=G.ContactHistory(max_atoms=64), pair=G.GranHookeHistory(domain=dom, dampflag=1, **law),
                           dt=1e-4)
        sim.add_fix(G.FixNVESphere(domain=dom))
        sim.add_fix(G.FixWallGran(domain=dom, wall_axis=2, wall_side=-1, wall_coord=0.0, max_atoms=64, **law))
        sim.fused = on
        for _ in range(3):
            sim.run(steps)
            sim.run_pre = False
        assert (getattr(sim, "last_engine", None) is not None) == (on and fused)
        return gpu_state(sim)

    a, b = run(True), run(False)
    for k in ("x", "v", "omega", "f", "torque", "virial"):
        # two orders of FP64 sums over at most 36 steps
        assert np.abs(a[k] - b[k]).max() <= 1e-11 * max(np.abs(b[k]).max(), 1e-300), k
