"""The FP64 two-launch step outside the exponent range of its integer path:
against the tile pass, whose products and quotients are FP64 instructions, to
the bit (the sign of a zero included), and against the oracle.

Sources whose fields, stresses or results are huge, subnormal or underflow to
zero, and states of zeros of either sign with a few values among them; stress
passes of one, two and six threads a point, materials whose normal stresses
share terms and others, negative and zero stiffnesses, spacings below and
above 1/2 and 2 (factors whose records borrow from the sign bit and do not).
"""
import numpy as np
import pytest

from test_gpu_split import TABLE, _problem

pytestmark = pytest.mark.gpu

# six, two and one thread a stress point
CASES = [((9, 17, 33), ("corrected", "absorbing", "line")), ((28, 29, 31), ("reference", "rigid", "wall")),
         ((44, 36, 39), ("corrected", "absorbing", "line"))]


def _table(shared):
    table = TABLE.copy()
    if shared:
        table[0, [1, 2, 3, 5, 6, 7]] = 64e9
    table[2, [4, 9, 11]] *= -1
    return table


def _runs(precision, sp, ids, table, dt, src, modes, state=None):
    """Bits of the final state and of the surface: default handle, tile pass."""
    from phonomena_gb300.device import DeviceSimulation

    surface, bc, source = modes
    for kw in ({}, {"tile_j": 8, "x_segment": 8}):
        with DeviceSimulation(sp, ids, table, dt, precision=precision, surface_mode=surface, bc=bc, source_mode=source,
                              max_steps=src.size, record_every=2, **kw) as sim:
            sim.set_source(src)
            for k in sim.state_fields if state else ():
                sim.upload(k, state[k])
            sim.step(src.size)
            sim.sync()
            yield {**{k: sim.download(k) for k in sim.state_fields}, "surface": sim.read_surface()}


def _same_bits(a, b):
    for k in a:
        assert np.array_equal(a[k].view(np.uint64), b[k].view(np.uint64)), k


@pytest.mark.parametrize("scale", [1e-100, 1e-235, 1e-305, 1e220])
@pytest.mark.parametrize("shape,modes", CASES)
@pytest.mark.parametrize("shared", [True, False])
def test_extreme_sources(gpu_lib, oracle, scale, shape, shared, modes):
    sp, ids, dt, src = _problem(shape, sum(shape), 14)
    table, src = _table(shared), src * scale
    prob = oracle.OracleProblem(sp, ids, table, dt, src, surface_mode=int(modes[0] == "corrected"),
                                bc=int(modes[1] == "rigid"), source_mode=int(modes[2] == "wall"))
    want, want_surf = oracle.run_f64(prob, record_every=2)
    got, tiles = _runs("f64", sp, ids, table, dt, src, modes)
    for key, w in zip(("ux", "uy", "uz"), want.u):
        assert np.array_equal(got[key], w), key
    assert np.array_equal(got["surface"], want_surf)
    _same_bits(got, tiles)


@pytest.mark.parametrize("precision", ["f64", "f64v"])
@pytest.mark.parametrize("shape,modes", CASES)
@pytest.mark.parametrize("spacing", [1.0, 3e5])
def test_zeros_of_either_sign(gpu_lib, precision, shape, spacing, modes):
    from phonomena_gb300.device import field_shape

    sp, ids, dt, _ = _problem(shape, sum(shape), 1)
    sp = {k: v * spacing for k, v in sp.items()}
    rng = np.random.default_rng(sum(shape))
    names = ("ux", "uy", "uz", "ux_old", "uy_old", "uz_old") if precision == "f64" else \
        ("ux", "uy", "uz", "vx", "vy", "vz", "cx", "cy", "cz")
    state = {}
    for q, k in enumerate(names):
        f = rng.choice([0.0, -0.0], field_shape(*shape, q % 3))
        some = rng.random(f.shape) < 0.01
        state[k] = np.where(some, rng.standard_normal(f.shape) * 1e-9, f)
    got, tiles = _runs(precision, sp, ids, _table(True), dt, np.array([-0.0, 0.0, -0.0]), modes, state)
    _same_bits(got, tiles)
