"""
The contact-dense path of the fused step (tmps_fused_c_pairs): every pair style
at sizes around a 32-atom group and a block, forced on, against the screened
path; rebuilds every few steps (histories out of the pair buffer and back), and
boxes of one and two bins.
"""

import numpy as np
import pytest

from _twin import dense_packing, gpu_state, make_twin

pytestmark = pytest.mark.gpu

STYLES = ["hooke", "hooke/history", "hertz", "hertz/history", "granular/linear_history", "granular/nohistory",
          "granular/rolling"]


def _states(oracle, n, box, pair, precision, steps, check=True, skin=0.1, w_scale=0.5):
    out = []
    for path in ("screened", "rows"):
        rng = np.random.default_rng(n)
        x, r = dense_packing(rng, n, box, 0.48, 0.56)
        v = rng.normal(scale=0.3, size=x.shape)
        w = rng.normal(scale=w_scale, size=x.shape)
        sim, _ = make_twin(oracle, x, r, 2.5, [0.0] * 3, [box] * 3, v=v, w=w, pair=pair, dt=5e-5, skin=skin,
                           cundall=(0.7, 0.7))
        sim.precision = precision
        sim.contact_path = path
        sim.neighbor.check = check
        sim.neighbor.every = 1 if check else 7
        sim.run(steps)
        assert sim.last_engine.rows == (path == "rows")
        h = sim.history
        st = dict(gpu_state(sim), builds=sim.neighbor.build_count, touch=h.touch.cpu().numpy(),
                  shear=h.shear.cpu().numpy())
        if h.rolling is not None:
            st["rolling"] = h.rolling.cpu().numpy()
        out.append(st)
    return out


def _same(a, b, exact, tol):
    assert a["builds"] == b["builds"]
    np.testing.assert_array_equal(a["touch"], b["touch"])
    live = ((a["touch"][None, :] >> np.arange(a["shear"].shape[1], dtype=np.int64)[:, None]) & 1) == 1
    for k in ("x", "v", "omega", "f", "torque", "shear", "rolling"):
        if k not in a:
            continue
        p, q = (a[k][:, live], b[k][:, live]) if k in ("shear", "rolling") else (a[k], b[k])
        if exact:
            np.testing.assert_array_equal(p, q, err_msg=k)
        elif p.size:
            assert np.abs(p - q).max() <= tol * max(np.abs(p).max(), 1e-300), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("pair", STYLES)
def test_pairs_equal_screened(gpu, oracle, precision, pair):
    """The legacy styles run the same instructions per contact in both paths: bit for bit.  pair granular
    may contract sums of products differently (FP64 a few 2^-53 per step over 21 steps; mixed 2^-24)."""
    a, b = _states(oracle, 343, 7.0, pair, precision, 21, check=False)
    assert a["builds"] == 4  # one at the setup, then every seven steps
    assert np.abs(a["f"]).max() > 0
    _same(a, b, not pair.startswith("granular"), 1e-12 if precision == "fp64" else 1e-4)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,box", [(1, 2.0), (2, 2.2), (8, 2.0), (31, 4.0), (33, 4.0), (127, 5.1), (257, 6.4), (1025, 10.2)])
def test_pairs_sizes(gpu, oracle, precision, n, box):
    """Around a group and a block of atoms; the smallest boxes have one bin (FP32 image) per axis."""
    a, b = _states(oracle, n, box, "hertz/history", precision, 15, skin=0.05)
    _same(a, b, True, 0.0)
