"""
The pair path of the fused step where the device has no room for its buffer.
"""

import numpy as np
import pytest

from _twin import dense_packing, gpu_state, make_twin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_no_room_for_the_pairs(gpu, oracle, precision, monkeypatch):
    """Where the pair path's buffer does not fit the device, the run takes the screened path: it ran before there
    was a pair path, and its results are the same."""
    import torch
    from taichimps_gb300 import engine

    def run(full):
        rng = np.random.default_rng(4)
        x, r = dense_packing(rng, 343, 7.0, 0.50, 0.56)
        sim, _ = make_twin(oracle, x, r, 2.5, [0.0] * 3, [7.0] * 3, v=rng.normal(scale=0.3, size=x.shape),
                           pair="hertz/history", dt=5e-5, skin=0.05, cundall=(0.7, 0.7))
        sim.precision = precision
        with monkeypatch.context() as m:
            if full:
                class Full:
                    def __getattr__(self, name):
                        return getattr(torch, name)

                    @staticmethod
                    def empty(*a, **kw):
                        if kw.get("dtype") is torch.uint8 and "pin_memory" not in kw:
                            raise torch.OutOfMemoryError("no room")
                        return torch.empty(*a, **kw)

                m.setattr(engine, "torch", Full())
            sim.run(30)
        assert sim.last_engine.rows == (not full)
        h = sim.history
        return gpu_state(sim), h.touch.cpu().numpy(), sim.neighbor.build_count

    (a, ta, ba), (b, tb, bb) = run(False), run(True)
    assert ba == bb and np.abs(a["f"]).max() > 0
    np.testing.assert_array_equal(ta, tb)
    for k in ("x", "v", "omega", "f", "torque"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
