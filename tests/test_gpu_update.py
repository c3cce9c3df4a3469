"""
The update kernel of the fused step where atoms carry no force: velocities left in
memory as they are, kinetic sums kept between passes (FP64 form), and the skin
check's displacement from the bits of the positions -- against the oracle.
"""

import numpy as np
import pytest

from _twin import gpu_state, make_twin, oracle_state, rel_err

pytestmark = pytest.mark.gpu

# x, v and the pressure of a force-free flight are sums of a few rounded products per step: 64 steps of
# 2^-53 relative, with room for the order of the sums
TOL = 1e-13
MIXED_X = 1e-9  # the mixed form's positions, as tests/test_gpu_fused.py states them


def _gas(rng, n, box, sigma):
    """n small spheres, no two within reach of one another for the length of a test."""
    side = int(np.ceil(n ** (1.0 / 3.0)))
    g = (np.arange(side) + 0.5) * (box / side)
    x = np.array([[a, b, c] for a in g for b in g for c in g])[:n]
    return x, rng.uniform(0.05, 0.1, size=n), rng.normal(scale=sigma, size=(n, 3)), rng.normal(scale=sigma, size=(n, 3))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 31, 33, 343])
def test_force_free_flight_pressure_every_step(gpu, oracle, precision, n):
    """No contacts: every step's pressure is kinetic alone, read back from the kept sums after the
    first two passes; across a second run the sums are formed anew from the velocities then held."""
    rng = np.random.default_rng(n)
    box = 8.0
    x, r, v, w = _gas(rng, n, box, 0.3)
    deform = dict(axes={"x": {"style": "erate", "rate": -0.1}, "y": {"style": "erate", "rate": 0.2}}, remap="x")
    sim, osim = make_twin(oracle, x, r, 2.5, [0.0] * 3, [box] * 3, v=v, w=w, dt=1e-4, deform=deform)
    sim.precision = precision
    fix = sim.fixes[-1]
    fix.record_pressure(64)
    tol = TOL if precision == "fp64" else 1e-6  # the mixed form's kinetic terms are FP32 products
    for rep in range(2):
        sim.run(32)
        rows = fix.pressure_history(range(32 * rep + 1, 32 * rep + 33))
        # one step at a time leaves the oracle's setup pass at each run's start only
        osim.setup(32)
        for k in range(32):
            vol = float(np.prod(osim.domain.prd))  # the box the step's pressure is taken in
            osim.step()
            m, ov = osim.atoms.rmass, osim.atoms.v
            kin = np.einsum("i,ia,ib->ab", m, ov, ov)
            want = np.array([kin[0, 0], kin[1, 1], kin[2, 2], kin[0, 1], kin[0, 2], kin[1, 2]]) / vol
            assert rel_err(rows[k], want) < tol, (rep, k)
        g, o = gpu_state(sim), oracle_state(osim)
        for k in ("x", "v", "omega"):
            lim = MIXED_X if precision == "mixed" and k == "x" else TOL
            assert rel_err(g[k], o[k]) < lim, (k, rel_err(g[k], o[k]))
        # other velocities before the next run, on both sides
        v = rng.normal(scale=0.2, size=v.shape)
        sim.atom.v.from_numpy(v)
        osim.atoms.v[:] = v


@pytest.mark.parametrize("offset", [0.0, 64.0, -64.0, 1.0e-3, 1000.25, -4096.0])
def test_skin_check_fires_on_the_oracles_step(gpu, oracle, offset):
    """One fast atom starting at an odd place near `offset` (signs and powers of two crossed on the way)
    trips the skin check on exactly the oracle's step, for many starts."""
    rng = np.random.default_rng(int(abs(offset)) + 3)
    for k in range(6):
        start = offset + rng.uniform(-0.03, 0.03, size=3)
        far = offset + np.array([2.0, 2.0, 2.0])
        x = np.stack([start, far])
        v = np.stack([rng.normal(scale=20.0, size=3), np.zeros(3)])
        lo = [offset - 4.0] * 3
        hi = [offset + 4.0] * 3
        sim, osim = make_twin(oracle, x, np.array([0.1, 0.1]), 2.5, lo, hi, v=v, dt=1e-5, skin=0.02)
        sim.run(200)
        osim.run(200)
        assert osim.neighbor.build_count > 1
        assert sim.neighbor.build_count == osim.neighbor.build_count
        assert sim.neighbor.last_build_step == osim.neighbor.last_build_step
        assert rel_err(gpu_state(sim)["x"], oracle_state(osim)["x"]) < TOL
