"""
Compressed packings kept as data (packing.compress_packing): read for the arguments they were made with,
a packing with the radii of those arguments, at the pressure asked for; any other argument, and regenerate=True,
makes the run.
"""

import numpy as np
import pytest


def test_stored_packing_is_what_its_arguments_say():
    from taichimps_gb300 import packing
    p = packing.compress_packing(512, seed=5)
    site = packing.make_packing_box(512, 0.8, 1.2, 0.3, 5, jitter=0.3)
    np.testing.assert_array_equal(p["radius"], site["radius"])
    d = p["x"][:, None] - p["x"][None]
    d -= p["L"] * np.round(d / p["L"])
    gap = np.sqrt((d * d).sum(-1)) - (p["radius"][:, None] + p["radius"][None])
    np.fill_diagonal(gap, np.inf)
    touching = (gap < 0).sum(1)
    # rattlers aside a frictional packing holds each sphere by about four contacts, overlaps of p / kn ~ 1e-4
    assert gap.min() > -0.01 and 3.0 < touching[touching > 0].mean() < 6.0
    assert abs(np.mean(p["pressure"][:3]) - 1.0) < 0.1
    assert p["phi"] == pytest.approx(float((4 / 3 * np.pi * p["radius"] ** 3).sum() / np.prod(p["L"])))


def test_other_arguments_are_not_the_stored_ones():
    from taichimps_gb300 import packing
    same = dict(dmin=0.8, dmax=1.2, density=2.5, kn=1.0e5, xmu=0.5, ptarget=1.0, pgain=1.0, max_rate=0.005, cycles=100,
                relax_cycles=10, cycle_steps=2000, dt=5e-4, precision="fp64", phi0=0.3, jitter=0.3)
    assert packing._stored_packing(343, 11, same) is not None
    assert packing._stored_packing(343, 12, same) is None
    for k, v in dict(dmin=0.7, kn=2.0e5, cycles=99, precision="mixed", dt=2e-4).items():
        assert packing._stored_packing(343, 11, dict(same, **{k: v})) is None


@pytest.mark.gpu
def test_regenerated_packing(gpu):
    from taichimps_gb300.packing import compress_packing
    kept = compress_packing(343, seed=11)
    p = compress_packing(343, seed=11, regenerate=True)
    np.testing.assert_array_equal(p["radius"], kept["radius"])
    assert abs(np.mean(p["pressure"][:3]) - 1.0) < 0.2 and abs(p["phi"] - kept["phi"]) < 0.02
