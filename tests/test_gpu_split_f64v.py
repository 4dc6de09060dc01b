"""The FP64 velocity form from 60,000 nodes on, whose products with constants
run in integer arithmetic, against the oracle: operands whose products leave
the integer path's exponent range at either end (subnormal results among
them), zero and negative factors, both z = 0 rows, all walls and sources.
Tolerance 0: the result is defined to the bit.
"""
import numpy as np
import pytest

from test_gpu_split import TABLE, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-100, 1e-305, 1e220])
@pytest.mark.parametrize("shape,modes,sign", [((41, 37, 41), ("corrected", "absorbing", "line"), 1),
                                              ((33, 65, 33), ("reference", "absorbing", "wall"), 1),
                                              ((44, 36, 39), ("corrected", "rigid", "wall"), -1)])
def test_integer_products_equal_oracle(gpu_lib, oracle, scale, shape, modes, sign):
    from phonomena_gb300.device import DeviceSimulation

    assert np.prod(shape) >= 60000
    surface, bc, source = modes
    steps = 14  # a graph chunk and a remainder
    sp, ids, dt, src = _problem(shape, sum(shape), steps)
    table = TABLE.copy()
    table[2, [2, 5, 10]] *= sign
    src = src * scale
    prob = oracle.OracleProblem(sp, ids, table, dt, src, surface_mode=int(surface == "corrected"), bc=int(bc == "rigid"),
                                source_mode=int(source == "wall"))
    want, want_surf = oracle.run_f64v(prob, record_every=2)
    with DeviceSimulation(sp, ids, table, dt, precision="f64v", surface_mode=surface, bc=bc, source_mode=source,
                          max_steps=steps, record_every=2) as sim:
        sim.set_source(src)
        sim.step(steps)
        sim.sync()
        for key, w in zip(("ux", "uy", "uz"), want.u):
            assert np.array_equal(sim.download(key), w), key
        assert np.array_equal(sim.read_surface(), want_surf)
