"""
The contact kernel right behind the bounds kernel, as a rebuild step of a C host queues them: no synchronisation
in between, every group screened (no gap order), the flag words of an earlier pass still there.  Every atom's force
is written or cleared.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cull", [0, 1])
def test_contacts_behind_the_bounds(gpu, precision, cull):
    import numpy as np
    import torch
    import taichimps_gb300 as G
    from taichimps_gb300 import _device, _lib
    from taichimps_gb300.engine import FusedEngine
    n = 3000
    rng = np.random.default_rng(2)
    g = np.stack(np.meshgrid(*[np.arange(15)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] + 0.5
    dom = G.Domain(boxlo=[0.0] * 3, boxhi=[15.0] * 3, boundary=("p", "p", "p"))
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=g + rng.uniform(-0.05, 0.05, size=g.shape), radius=rng.uniform(0.42, 0.52, size=n), density=2.5)
    sim = G.Simulation(domain=dom, atom=atom, neighbor=G.NeighborList(domain=dom, skin=0.1, max_atoms=n),
                       history=G.ContactHistory(max_atoms=n),
                       pair=G.GranHooke(domain=dom, kn=2e5, kt=0.0, gamman=50.0, gammat=25.0, xmu=0.5, dampflag=1), dt=1e-4,
                       precision=precision)
    sim.add_fix(G.FixNVESphere(domain=dom))
    sim.init_simulation()
    eng = FusedEngine(sim, precision, cull=bool(cull), contact_path="screened")
    eng.begin()
    L, st = _device.lib(), _device.stream()
    atoms, nl, par = eng.atoms(), sim.history.cstruct(sim.neighbor), sim.pair_style.params
    force = eng.f32 if eng.mixed else atom.buffers.f

    def once(sync):
        force.fill_(7.0)
        _lib.check(L.tmps_fused_bounds(atoms, nl, sim.domain.dbox, eng._eng.data_ptr(), par, cull, eng.part.data_ptr(), st),
                   "tmps_fused_bounds")
        if sync:
            torch.cuda.synchronize()
        _lib.check(L.tmps_fused_c(atoms, nl, sim.domain.dbox, eng._eng.data_ptr(), par, eng.c_blocks, eng.part.data_ptr(),
                                  st), "tmps_fused_c")
        return force.clone()

    want = once(True)
    touching = int((want.reshape(3, -1) != 0).any(0).sum())
    assert 0 < touching < n and float(want.abs().max()) != 7.0
    for _ in range(40):
        assert torch.equal(once(False), want)
