"""
The FP64 form's states bit for bit: a jammed packing with fast rolling and sliding contacts, a dozen steps of
every pair style, through the fused step (every contact path) and hook by hook, against digests stored from the
form that makes each division and square root by the compiler's own operation.  The laws' quotients and roots
(quot64, sqrt64) are rounded as those, and every atom's sums run in slot order, so nothing may differ.
"""

import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "fp64_states.json"
STYLES = ("hooke", "hooke/history", "hertz", "hertz/history", "granular", "granular/rolling")
PATHS = ("auto", "screened", "rows", "hooks")


def digests(style, path):
    import taichimps_gb300 as G
    from taichimps_gb300.packing import dense_cell
    c = dense_cell()
    # a slab of the compressed cell, periodic in x and y, open in z
    keep = c["x"][:, 2] < c["lo"][2] + 3.0
    x, r = c["x"][keep], c["radius"][keep]
    n = len(r)
    rng = np.random.default_rng(23)
    hi = [float(c["lo"][k] + c["L"][k]) for k in range(3)]
    dom = G.Domain(boxlo=[float(a) for a in c["lo"]], boxhi=hi, boundary=("p", "p", "f"))
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=x, radius=r, density=2.5, v=rng.normal(0.0, 0.5, size=(n, 3)), omega=rng.normal(0.0, 2.0, size=(n, 3)))
    nl = G.NeighborList(domain=dom, skin=0.1, max_atoms=n, max_neighbors_per_atom=32)
    hist = G.ContactHistory(max_atoms=n, max_neighbors=32)
    soft = dict(kn=2.0e3, kt=2.0e3 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.1, dampflag=1)
    stiff = dict(soft, kn=2.0e5, kt=2.0e5 * 2.0 / 7.0)
    if style.startswith("granular"):
        roll = dict(rolling="epsd", rolling_coeffs=[1.0e3, 50.0, 0.1]) if style.endswith("rolling") else {}
        pair = G.PairGranular(domain=dom, normal="hertz/material", normal_coeffs=[2.73e5, 0.5, 0.3],
                              damping="coeff_restitution", tangential="mindlin", tangential_coeffs=[None, 1.0, 0.1], **roll)
    else:
        pair = {"hooke": G.GranHooke, "hooke/history": G.GranHookeHistory, "hertz": G.GranHertz,
                "hertz/history": G.GranHertzHistory}[style](domain=dom, **(soft if style.startswith("hooke") else stiff))
    sim = G.Simulation(domain=dom, atom=atom, neighbor=nl, history=hist, pair=pair, dt=5e-5)
    sim.add_fix(G.FixNVESphere(domain=dom))
    sim.add_fix(G.FixDampingCundall(domain=dom, gamma_lin=0.2, gamma_ang=0.1))
    if path == "hooks":
        sim.fused = False
    else:
        sim.contact_path = path
    sim.run(12)
    out = {k: np.ascontiguousarray(getattr(atom, k).to_numpy()) for k in ("x", "v", "omega", "f", "torque")}
    assert np.abs(out["f"]).max() > 1.0
    return {k: hashlib.sha256((a + 0.0).tobytes()).hexdigest() for k, a in out.items()}


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("style", STYLES)
def test_states(gpu, style, path):
    want = json.loads(GOLDEN.read_text())
    assert digests(style, path) == want[f"{style} {'hooks' if path == 'hooks' else 'fused'}"]
