"""
Granular walls in the fused step (tmps_fused_walls) against the hook-by-hook path: planes and cylinders,
one and several walls, with and without history and damping, atom counts around the warp and block edges,
through neighbor rebuilds; and the configurations that must stay hook by hook.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

K = dict(kn=2e5, gamman=50.0, xmu=0.5)
T = dict(kt=2e5 * 2 / 7, gammat=25.0)


def _walls(G, dom, kind, n):
    plane = lambda axis, side, at, **kw: G.FixWallGran(domain=dom, wall_axis=axis, wall_side=side, wall_coord=at,
                                                       max_atoms=n, **dict(K, **T, **kw))
    tube = lambda **kw: G.FixWallGranRegion(domain=dom, max_atoms=n, **dict(dict(axis="z", c1=4.0, c2=4.0, radius=3.9, side="in",
                                                                       fstyle="hooke/history", **K), **kw))
    return {"planes": [plane(2, -1, 0.0), plane(2, 1, 8.0, history=False), plane(0, -1, 0.0, shear_axis=1, shear_vel=0.5)],
            "tube": [tube()], "hertz": [tube(fstyle="hertz/history", axis_lo=1.0, axis_hi=7.0)],
            "post": [tube(side="out", radius=1.2), plane(2, -1, 0.0)]}[kind]


def _sim(n, kind, fused, cundall=False, first=True, precision="fp64", extra=()):
    import taichimps_gb300 as G
    rng = np.random.default_rng(n)
    g = np.stack(np.meshgrid(*[np.arange(8)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5
    x = rng.permutation(g)[:n] + rng.uniform(-0.04, 0.04, size=(n, 3))
    r = rng.uniform(0.48, 0.52, size=n)
    dom = G.Domain(boxlo=[0.0] * 3, boxhi=[8.0] * 3, boundary=("f", "f", "f"))
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=x, radius=r, density=np.full(n, 2.5), v=rng.normal(0.0, 1.5, size=(n, 3)))
    sim = G.Simulation(domain=dom, atom=atom, neighbor=G.NeighborList(domain=dom, skin=0.02, max_atoms=n),
                       history=G.ContactHistory(max_atoms=n), pair=G.GranHookeHistory(domain=dom, dampflag=1, **K, **T), dt=1e-4,
                       precision=precision)
    sim.add_fix(G.FixNVESphere(domain=dom))
    damp = [G.FixDampingCundall(domain=dom, gamma_lin=0.3, gamma_ang=0.2)] if cundall else []
    walls = _walls(G, dom, kind, n)
    for f in (damp + walls if first else walls + damp) + [e(G, dom) for e in extra]:
        sim.add_fix(f)
    sim.fused = fused
    return sim, walls


@pytest.mark.parametrize("n,kind,cundall,path", [
    (1, "planes", False, "auto"), (31, "tube", False, "auto"), (32, "planes", True, "auto"), (33, "post", False, "auto"),
    (129, "hertz", True, "auto"), (512, "planes", True, "auto"), (511, "tube", False, "auto"), (511, "planes", True, "rows"),
    (257, "tube", False, "screened")])
def test_fused_walls_match_hooks(gpu, n, kind, cundall, path):
    out = []
    for fused in (True, False):
        sim, walls = _sim(n, kind, fused, cundall)
        sim.contact_path = path
        sim.run(90)
        sim.run_pre = False
        sim.run(70)
        assert (getattr(sim, "last_engine", None) is not None) == fused
        st = {k: getattr(sim.atom, k).to_numpy()[:n] for k in ("x", "v", "omega", "f", "torque")}
        out.append((st, walls, sim.neighbor.build_count))
    (a, wa, ba), (b, wb, bb) = out
    assert ba == bb and (n == 1 or ba > 2)
    for k in a:  # two orders of FP64 sums over 160 steps, as against the oracle
        scale = np.abs(b[k]).max()
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * scale + 1e-300, (k, np.abs(a[k] - b[k]).max(), scale)
    touched = 0
    for p, q in zip(wa, wb):
        assert getattr(p, "elapsed", 0.0) == getattr(q, "elapsed", 0.0)
        s, t = p.shear.cpu().numpy(), q.shear.cpu().numpy()
        np.testing.assert_array_equal(p.touch.cpu().numpy(), q.touch.cpu().numpy())
        assert np.abs(s - t).max() <= 1e-10 * max(np.abs(t).max(), 1e-12)
        touched += int(q.touch.sum())
    assert touched > 0 or n < 33


def test_what_stays_hook_by_hook(gpu):
    from taichimps_gb300.engine import fusable
    import taichimps_gb300 as G
    ok = lambda **kw: fusable(_sim(33, kw.pop("kind", "planes"), True, **kw)[0], walls=True)
    wall = lambda **kw: (lambda G, dom: G.FixWallGran(domain=dom, wall_axis=2, wall_side=1, wall_coord=8.0, max_atoms=33,
                                                      **dict(K, **T, **kw)))
    servo = lambda G, dom: G.FixDeformPressure(domain=dom, axes={"z": {"style": "erate", "rate": -0.1}}, remap="x")
    assert ok() and ok(cundall=True) and ok(extra=[wall()] * 5)
    assert not ok(cundall=True, first=False)                                       # damping after the walls
    assert not ok(extra=[wall(wiggle_amplitude=0.01, wiggle_period=0.02)])         # a moving wall
    assert not ok(extra=[wall()] * 6)                                              # more than one kernel takes
    assert not ok(extra=[servo])                                                   # a servo reads the virial
    assert not fusable(_sim(33, "planes", True)[0])                                # batches and the mixed form
    with pytest.raises(NotImplementedError):
        _sim(33, "planes", True, precision="mixed")[0].run(1)


@pytest.mark.parametrize("steps", [1, 2, 60])
def test_pressure_after_a_run_with_walls(gpu, steps):
    """The pressure tensor after a run is the last step's, through the fused step as hook by hook."""
    import taichimps_gb300 as G
    got = []
    for fused in (True, False):
        sim, _ = _sim(512, "planes", fused)
        sim.run(40)
        early = sim.atom.virial.to_numpy().copy()
        sim.run_pre = False
        sim.run(steps)
        got.append((G.Computes().compute_pressure_tensor(sim.atom, sim.domain), sim.atom.virial.to_numpy()[:512].copy()))
        assert np.abs(sim.atom.virial.to_numpy() - early).max() > 0.0
    (p, v), (q, w) = got
    assert np.abs(w).max() > 0.0
    # two orders of FP64 sums over the run, as the states
    assert np.abs(p - q).max() <= 1e-10 * np.abs(q).max()
    assert np.abs(v - w).max() <= 1e-10 * np.abs(w).max()
