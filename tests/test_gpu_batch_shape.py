"""
A batch asked for the default grids (launch shape 0, 0) takes one 32-atom group per warp, in both forms: every
instance as its own single run of that shape.
"""

import numpy as np
import pytest

from _twin import dense_packing, gpu_state, make_twin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_default_grids_of_a_batch(gpu, oracle, precision):
    import taichimps_gb300 as G

    def systems(shape):
        rng = np.random.default_rng(71)
        out = []
        for n, box in ((33, 4.2), (343, 8.2), (512, 9.0)):
            x, r = dense_packing(rng, n, box, 0.45, 0.56)
            deform = dict(axes={d: {"style": "pressure", "ptarget": 1.0, "pgain": 1e-3} for d in "xyz"}, couple="xyz",
                          max_rate=1e-1, remap="x")
            sim, _ = make_twin(oracle, x, r, 2.5, [0.0] * 3, [box] * 3, pair="hertz/history", dt=5e-5, deform=deform)
            sim.precision, sim.launch_shape, sim.contact_path = precision, shape, "screened"
            out.append(sim)
        return out

    batch, single = systems((0, 0)), systems((1, 1))
    eng = G.BatchedEngine(batch, precision=precision, chunk=8, launch_shape=(0, 0))
    assert eng.launch_shape == (1, 1)
    eng.run(20)
    for e, b, s in zip(eng.engines, batch, single):
        s.run(20)
        n = b.atom.nlocal
        assert (e.a_blocks, e.c_blocks) == ((n + 255) // 256, (n + 127) // 128)
        p, q = gpu_state(b), gpu_state(s)
        for k in ("x", "v", "f"):
            np.testing.assert_array_equal(p[k], q[k], err_msg=k)
        np.testing.assert_array_equal(b.domain.prd, s.domain.prd)


@pytest.mark.parametrize("mixed", [0, 1])
def test_default_blocks_of_the_c_interface(gpu, mixed):
    """tmps_batch_blocks: the grids of one group per warp, up to the wave."""
    import ctypes
    from taichimps_gb300 import _device, _lib
    L = _device.lib()
    for n in (1, 33, 500, 16000, 1_000_000):
        got, want = [(ctypes.c_int32(), ctypes.c_int32()) for _ in range(2)]
        assert L.tmps_batch_blocks(n, 3, mixed, *map(ctypes.byref, got)) == _lib.TMPS_OK
        assert L.tmps_fused_shape(n, 3, mixed, 1, 1, *map(ctypes.byref, want)) == _lib.TMPS_OK
        assert [v.value for v in got] == [v.value for v in want]
        if n <= 16000:
            assert [v.value for v in got] == [(n + 255) // 256, (n + 127) // 128]
