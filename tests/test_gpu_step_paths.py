"""
Paths of the fused step that a state or an option chooses: batches without a servo, kinetic sums kept and dropped
as contacts come and go under a servo, and the image velocities of remap v on both contact paths.
"""

import numpy as np
import pytest

from _twin import dense_packing, gpu_state, make_twin, oracle_state, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_without_a_servo(gpu, oracle, precision):
    """The contact kernel closes the step while the batch's servo launch still runs (for an instance that has a
    servo beside those that have none): every instance as its own single run, bit for bit, rebuilds included."""
    import taichimps_gb300 as G
    shape = (2, 2)

    def systems():
        rng = np.random.default_rng(61)
        out = []
        for k, (n, box) in enumerate([(1, 3.0), (64, 5.0), (343, 8.2), (33, 4.2), (512, 9.0)]):
            x, r = dense_packing(rng, n, box, 0.45, 0.56)
            v = rng.normal(scale=8.0 if k % 2 else 0.05, size=x.shape)
            servo = dict(axes={"x": {"style": "erate", "rate": -0.1}}, remap="x") if k == 2 else None
            sim, _ = make_twin(oracle, x, r, 2.5, [0.0] * 3, [box] * 3, v=v, pair="hertz/history", dt=5e-5, deform=servo)
            sim.precision = precision
            sim.launch_shape = shape
            out.append(sim)
        return out

    batch, single = systems(), systems()
    eng = G.BatchedEngine(batch, precision=precision, chunk=16, launch_shape=shape)
    for steps in (60, 7):
        eng.run(steps)
        for s in single:
            s.contact_path = "screened"
            s.run(steps)
        for a, b in zip(batch, single):
            assert a.timestep == b.timestep and a.neighbor.build_count == b.neighbor.build_count
            p, q = gpu_state(a), gpu_state(b)
            for k in ("x", "v", "omega", "f", "torque"):
                np.testing.assert_array_equal(p[k], q[k], err_msg=k)
    assert eng.rebuilds > 0 and max(np.abs(gpu_state(s)["f"]).max() for s in batch) > 0


@pytest.mark.parametrize("path", ["screened", "rows"])
def test_kept_kinetic_sums_as_contacts_come_and_go(gpu, oracle, path):
    """A thin gas under a servo: 32-atom groups gain their first contact, lose it and gain it again, and every
    step's pressure is the oracle's.  Tolerance: 160 steps of sums rounded in two orders, as the states
    (a few 2^-53 each, grown by the collisions)."""
    n, box, steps = 343, 10.0, 160
    rng = np.random.default_rng(5)
    x, r = dense_packing(rng, n, box, 0.40, 0.50, jitter=0.2)
    v = rng.normal(scale=8.0, size=x.shape)
    sim, osim = make_twin(oracle, x, r, 2.5, [0.0] * 3, [box] * 3, v=v, pair="hooke/history", dt=1e-4, skin=0.4,
                          deform=dict(axes={d: {"style": "pressure", "ptarget": 1.0, "pgain": 1e-3} for d in "xyz"},
                                      max_rate=1e-1, remap="x"))
    sim.contact_path = path
    fix = sim.fixes[-1]
    fix.record_pressure(steps)
    osim.setup(steps)
    want, groups = [], []
    for _ in range(steps):
        osim.step()
        want.append(np.array(osim.last_pressure, dtype=np.float64).reshape(-1)[:6])
        f = np.abs(osim.atoms.f).max(axis=1) != 0.0
        groups.append([f[g:g + 32].any() for g in range(0, n, 32)])
    groups = np.array(groups)
    # (atoms keep their order until the list is rebuilt: groups here are those of the insertion order, a witness
    # that most of a step's atoms are free and contacts come and go)
    turns = np.abs(np.diff(groups.astype(int), axis=0)).sum(axis=0)
    assert (turns >= 2).sum() >= 4 and groups.mean() < 0.7
    sim.run(steps)
    got = fix.pressure_history(range(1, steps + 1))
    for k in range(steps):
        assert rel_err(got[k], want[k]) < 1e-10, k
    g, o = gpu_state(sim), oracle_state(osim)
    for k in ("x", "v", "omega"):
        assert rel_err(g[k], o[k]) < 1e-10, k
    assert sim.neighbor.build_count == osim.neighbor.build_count


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,box", [(27, 3.0), (343, 7.0)])
def test_image_velocity_on_both_paths(gpu, oracle, precision, n, box):
    """remap v shifts a partner's velocity by the box's rate where the pair crosses a face: the pair path as the
    screened one, bit for bit, and (FP64) as the oracle."""
    states = []
    for path in ("screened", "rows"):
        rng = np.random.default_rng(9)
        x, r = dense_packing(rng, n, box, 0.50, 0.56)
        v = rng.normal(scale=0.3, size=x.shape)
        axes = {"x": {"style": "erate", "rate": -2.0}, "y": {"style": "erate", "rate": 1.0}, "z": {"style": "erate", "rate": -1.0}}
        sim, osim = make_twin(oracle, x, r, 2.5, [0.0] * 3, [box] * 3, v=v, pair="hertz/history", dt=5e-5, skin=0.05,
                              deform=dict(axes=axes, remap="v"))
        sim.precision = precision
        sim.contact_path = path
        sim.run(40)
        assert sim.last_engine.rows == (path == "rows")
        states.append((gpu_state(sim), np.array(sim.domain.prd), sim.neighbor.build_count))
    (a, pa, ba), (b, pb, bb) = states
    assert ba == bb and np.abs(a["f"]).max() > 0
    np.testing.assert_array_equal(pa, pb)
    for k in ("x", "v", "omega", "f", "torque"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    if precision == "fp64":
        osim.run(40)
        o = oracle_state(osim)
        for k in ("x", "v", "f"):
            assert rel_err(b[k], o[k]) < 1e-10, k
