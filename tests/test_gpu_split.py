"""The two-launch step (default tile shape) against the oracle and the tile pass.

Sizes where its flattened boxes, face lists and stress window can go wrong:
the smallest meshes (three nodes per axis, where faces meet), extents around
the block size, and a mesh whose window holds only part of the planes.
Tolerance 0: every scheme's result is defined to the bit.
"""
import numpy as np
import pytest

from phonomena_gb300 import crystal

pytestmark = pytest.mark.gpu

TABLE = np.array([[224e9, 64e9, 60e9, 66e9, 220e9, 64e9, 62e9, 64e9, 226e9, 80e9, 78e9, 82e9, 2330.0],
                  [0.0] * 12 + [2330.0],
                  [520e9, 200e9, 200e9, 200e9, 520e9, 200e9, 200e9, 200e9, 520e9, 160e9, 160e9, 160e9, 19300.0]])


def _problem(shape, seed, steps):
    rng = np.random.default_rng(seed)
    sp = {}
    for a, n in zip("xyz", shape):
        fd = 1e-5 * rng.choice([0.5, 0.75, 1.0, 1.0 + 2.0 ** -52], n - 1)
        sp["fd" + a], sp["sd" + a] = fd, (fd[1:] + fd[:-1]) / 2
    ids = rng.choice(3, shape, p=[0.7, 0.2, 0.1]).astype(np.uint8)
    ids[0, 0, 0] = 0
    return sp, ids, 2e-10, rng.standard_normal(steps)


@pytest.mark.parametrize("precision", ["f64", "f32k", "f64v"])
@pytest.mark.parametrize("shape,modes", [
    ((3, 3, 3), ("corrected", "absorbing", "line")), ((4, 3, 6), ("reference", "absorbing", "wall")),
    ((3, 4, 3), ("corrected", "rigid", "line")), ((5, 4, 4), ("reference", "absorbing", "line")),
    ((3, 33, 9), ("corrected", "absorbing", "line")), ((40, 5, 33), ("corrected", "rigid", "wall")),
    ((9, 17, 65), ("reference", "absorbing", "line"))])
def test_two_launch_step_equals_oracle(gpu_lib, oracle, precision, shape, modes):
    from phonomena_gb300.device import DeviceSimulation

    surface, bc, source = modes
    steps = 26  # two graph chunks and a remainder
    sp, ids, dt, src = _problem(shape, sum(shape), steps)
    prob = oracle.OracleProblem(sp, ids, TABLE, dt, src, surface_mode=int(surface == "corrected"),
                                bc=int(bc == "rigid"), source_mode=int(source == "wall"))
    run = {"f64": oracle.run_f64, "f32k": oracle.run_f32k, "f64v": oracle.run_f64v}[precision]
    want, want_surf = run(prob, record_every=4)
    with DeviceSimulation(sp, ids, TABLE, dt, precision=precision, surface_mode=surface, bc=bc, source_mode=source,
                          max_steps=steps, record_every=4) as sim:
        sim.set_source(src)
        sim.step(steps)
        sim.sync()
        for key, w in zip(("ux", "uy", "uz"), want.u):
            assert np.array_equal(sim.download(key), w), key
        assert np.array_equal(sim.read_surface(), want_surf)


@pytest.mark.parametrize("flip", [None, 3, 6, 1, 7, 2, 5])
def test_shared_stress_terms(gpu_lib, oracle, flip):
    """Materials whose normal stresses share terms, and the same with one of
    the stiffnesses a little different or a zero of the other sign."""
    from phonomena_gb300.device import DeviceSimulation

    sp, ids, dt, src = _problem((13, 12, 37), 3, 20)
    tab = TABLE.copy()
    tab[0, [3, 6]], tab[0, [1, 7]], tab[0, [2, 5]] = 61e9, 63e9, 65e9
    if flip is not None:
        tab[0, flip] *= 1 + 2.0 ** -40
        tab[1, flip] = -0.0
    prob = oracle.OracleProblem(sp, ids, tab, dt, src, surface_mode=1)
    want, _ = oracle.run_f64(prob)
    with DeviceSimulation(sp, ids, tab, dt, precision="f64", surface_mode="corrected", max_steps=20) as sim:
        sim.set_source(src)
        sim.step(20)
        sim.sync()
        for key, w in zip(("ux", "uy", "uz"), want.u):
            assert np.array_equal(sim.download(key), w), key


@pytest.mark.parametrize("precision", ["f64", "f64v"])
def test_chunked_window_equals_tile_pass(gpu_lib, precision):
    """A mesh of several chunks (77 planes of 270 x 180 nodes: 128 MB hold 57)."""
    from phonomena_gb300.device import DeviceSimulation

    spec = crystal.CrystalSpec(cells=(76, 269, 179), lattice=12, radius=(0.2, 0.4), tungsten_frac=0.25, seed=4, steps=26,
                               record_every=5)
    g, m = crystal.build(spec)
    src = crystal.sin_source(40e6, m.dt, spec.steps)
    out = []
    for kw in ({}, {"tile_j": 8, "x_segment": 19}):
        with DeviceSimulation(g.spacing(), m.ids, m.table, m.dt, precision=precision, surface_mode="corrected",
                              max_steps=spec.steps, record_every=5, **kw) as sim:
            sim.set_source(src)
            sim.step(spec.steps)
            sim.sync()
            out.append([sim.download(k) for k in ("ux", "uy", "uz")] + [sim.read_surface()])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["f64", "f32k"])
def test_switching_forms_mid_run(gpu_lib, precision, tmp_path):
    """From the two-launch form to tiles and, through a checkpoint, back."""
    from phonomena_gb300.device import DeviceSimulation

    sp, ids, dt, src = _problem((21, 19, 37), 5, 40)

    def make():
        sim = DeviceSimulation(sp, ids, TABLE, dt, precision=precision, surface_mode="corrected", max_steps=40)
        sim.set_source(src)
        return sim

    with make() as sim:
        sim.step(40)
        sim.sync()
        want = [sim.download(k) for k in sim.state_fields]
    with make() as sim:
        sim.step(13)
        ck = sim.checkpoint()
        sim.set_tiling(8, 4)
        sim.step(27)
        sim.sync()
        for k, w in zip(sim.state_fields, want):
            assert np.array_equal(sim.download(k), w), k
    with DeviceSimulation.from_checkpoint(ck) as sim:
        sim.step(27)
        sim.sync()
        for k, w in zip(sim.state_fields, want):
            assert np.array_equal(sim.download(k), w), k


@pytest.mark.parametrize("precision,shape", [("f64", {}), ("f32k", {}), ("f64v", {}), ("f32k", {"tile_j": 4, "x_segment": 8}),
                                             ("f64", {"tile_j": 8, "x_segment": 8})])
def test_handles_through_a_batch(gpu_lib, precision, shape):
    """Odd step counts in, through and out of a batch, where FP32 handles take
    other tiles, and the tile pass, which keeps v and the Kahan term in other
    buffers than the two-launch form."""
    from phonomena_gb300.batch import Batch
    from phonomena_gb300.device import DeviceSimulation

    tj = 4 if precision == "f32k" else 8
    probs = [_problem(s, 7, 40) for s in ((21, 19, 37), (30, 12, 9))]

    def make(p):
        sim = DeviceSimulation(p[0], p[1], TABLE, p[2], precision=precision, surface_mode="corrected", max_steps=40, **shape)
        sim.set_source(p[3])
        return sim

    for leave in ("remove", "close"):
        sims = [make(p) for p in probs]
        b = Batch(2, precision=precision, tile_j=tj)
        for s in sims:
            s.step(5)
        slots = [b.add(s, 13) for s in sims]
        b.step(13)
        b.sync()
        for slot in slots if leave == "remove" else ():
            b.remove(slot)
        b.close()
        for s, p in zip(sims, probs):
            s.step(22)
            s.sync()
            with make(p) as ref:
                ref.step(40)
                ref.sync()
                for k in s.state_fields:
                    assert np.array_equal(s.download(k), ref.download(k)), (leave, k)
            s.close()


def test_batch_that_grows(gpu_lib):
    """A small instance whose segments are cut anew, in mid-run, when a large
    one joins, and again when it has left."""
    from phonomena_gb300.batch import Batch
    from phonomena_gb300.device import DeviceSimulation

    small, large = _problem((30, 21, 13), 2, 90), _problem((260, 250, 40), 3, 90)

    def make(p):
        sim = DeviceSimulation(p[0], p[1], TABLE, p[2], precision="f32k", surface_mode="corrected", max_steps=90)
        sim.set_source(p[3])
        return sim

    with make(small) as a, make(large) as b, Batch(3, precision="f32k", tile_j=4) as batch:
        batch.add(a, 77)
        batch.step(25)
        batch.add(b, 26)
        batch.step(26)
        batch.step(26)
        batch.sync()
        for sim, p, n in ((a, small, 77), (b, large, 26)):
            with make(p) as ref:
                ref.step(n)
                ref.sync()
                for k in sim.state_fields:
                    assert np.array_equal(sim.download(k), ref.download(k)), (n, k)
