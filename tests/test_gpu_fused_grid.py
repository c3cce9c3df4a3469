"""
The grids of the FP64 step spread a small system over the SMs, one 32-atom group a block up to a wave, with a
servo as without one.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("servo", [False, True])
@pytest.mark.parametrize("n", [33, 500, 4000])
def test_one_group_a_block(gpu, n, servo):
    import taichimps_gb300 as G
    from taichimps_gb300 import _device, _lib
    from taichimps_gb300.packing import make_packing
    p = make_packing(n, 0.9, 1.1, 0.35, 3, jitter=0.02)
    dom = G.Domain(boxlo=[0.0] * 3, boxhi=[p["L"]] * 3, boundary=("p", "p", "p"))
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=p["x"], radius=p["radius"], density=2.5)
    sim = G.Simulation(domain=dom, atom=atom, neighbor=G.NeighborList(domain=dom, skin=0.1, max_atoms=n),
                       history=G.ContactHistory(max_atoms=n),
                       pair=G.GranHertzHistory(domain=dom, kn=2e5, kt=2e5 * 2 / 7, gamman=50.0, gammat=25.0, xmu=0.5,
                                               dampflag=1), dt=5e-5)
    sim.add_fix(G.FixNVESphere(domain=dom))
    if servo:
        sim.add_fix(G.FixDeformPressure(domain=dom, axes={d: {"style": "pressure", "ptarget": 1.0, "pgain": 1e-3}
                                                          for d in "xyz"}, couple="xyz", max_rate=1e-4, remap="x"))
    sim.run(2)
    e = sim.last_engine
    a_b, c_b = ctypes.c_int32(), ctypes.c_int32()
    assert _device.lib().tmps_fused_shape(n, int(sim.pair_style.params.style), 0, 0, 0, ctypes.byref(a_b),
                                          ctypes.byref(c_b)) == _lib.TMPS_OK
    assert (e.a_blocks, e.c_blocks) == (a_b.value, c_b.value)
    assert c_b.value == (n + 31) // 32  # (none of these fills a wave)
    assert np.isfinite(atom.x.to_numpy()).all()
