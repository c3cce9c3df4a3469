"""
The differentiable run at calibration size (31,250 spheres of a jammed packing) against stored values.

The overlap ra + rb - |d| of a barely touching pair cancels its leading digits, so a last bit of a position,
a distance or (through the servo) the pressure moves that sphere's dL/d(radius) by 1e-9 to 1e-7 of the
largest.  The forward therefore keeps every rounding and the order of its sums; the stored records are of the
run's plainest form (one thread per pair and per atom, the compiler's divisions and square roots, blocks of
256), and the forward has to give them bit for bit.  The reverse is linear in what the forward recorded: its
sums may be ordered anew, which moves a gradient by some 1e-15 of its scale; 1e-12 is asked for.
"""

from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "adjoint_31250.npz"
STEPS, EVERY, CHECKPOINT = 40, 10, 25


def forward_and_gradients():
    import torch
    from taichimps_gb300.adjoint import AdjointRun, stress_curve
    from taichimps_gb300.packing import dense_cell, tile_packing
    p = tile_packing(dense_cell(), (2, 1, 1))
    rng = np.random.default_rng(17)
    order = rng.permutation(len(p["radius"]))
    x, r = p["x"][order], p["radius"][order]
    axes = {"x": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
            "y": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1}, "z": {"style": "erate", "rate": -1.0e-3}}
    run = AdjointRun(x, r, p["density"], p["lo"], p["lo"] + p["L"], dt=5e-5, steps=STEPS, axes=axes, max_rate=1.0e-2,
                     sample_every=EVERY, checkpoint_every=CHECKPOINT, v=rng.normal(0.0, 0.02, size=x.shape))
    prm = dict(kn=2.0e5, kt=2.0e5 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5)
    ps = {k: torch.tensor(a, dtype=torch.float64, requires_grad=True) for k, a in prm.items()}
    rad = torch.tensor(r, dtype=torch.float64, device="cuda", requires_grad=True)
    q = stress_curve(run, ps["kn"], ps["kt"], ps["gamman"], ps["gammat"], ps["xmu"], rad)
    (q ** 2).sum().backward()
    out = {k: t.grad.cpu().numpy() for k, t in ps.items()}
    return dict(out, radius=rad.grad.cpu().numpy(), records=run.records())


def test_forward_bits_and_gradients(gpu):
    want, got = np.load(GOLDEN), forward_and_gradients()
    np.testing.assert_array_equal(got["records"], want["records"])
    for k in ("kn", "kt", "gamman", "gammat", "xmu", "radius"):
        scale = np.abs(want[k]).max()
        assert np.abs(got[k] - want[k]).max() <= 1e-12 * scale, (k, np.abs(got[k] - want[k]).max() / scale)
