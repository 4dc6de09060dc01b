"""Face points written by the FP32 tile pass (heights 8 and 16) against the
oracle: rows and planes next to a face at the edges of tiles and segments, a
last segment of one plane (its ux row is finished by the segment before), the
row counts around the smallest that takes this path, z = N at every place of a
thread's four points.  Alone, in the persistent batch and on streams.
Tolerance 0: the result is defined to the bit.
"""
import numpy as np
import pytest

from test_gpu_split import TABLE, _problem

pytestmark = pytest.mark.gpu

SHAPES = [(6, 3, 5), (6, 4, 5), (5, 5, 4), (4, 6, 6), (3, 7, 7), (7, 9, 33), (6, 10, 34), (9, 17, 35), (5, 18, 36),
          (12, 19, 65), (26, 34, 9)]


@pytest.mark.parametrize("tile_j,segments", [(4, 24), (8, 1), (8, "short"), (16, 24), (16, 2)])
@pytest.mark.parametrize("modes", [("corrected", "absorbing", "line"), ("reference", "absorbing", "wall"),
                                   ("corrected", "rigid", "wall")])
def test_tile_faces_equal_oracle(gpu_lib, oracle, tile_j, segments, modes):
    from phonomena_gb300.batch import Batch
    from phonomena_gb300.device import DeviceSimulation

    surface, bc, source = modes
    steps = 14  # a graph chunk and a remainder
    for shape in SHAPES:
        sp, ids, dt, src = _problem(shape, sum(shape), steps)
        prob = oracle.OracleProblem(sp, ids, TABLE, dt, src, surface_mode=int(surface == "corrected"),
                                    bc=int(bc == "rigid"), source_mode=int(source == "wall"))
        want, want_surf = oracle.run_f32k(prob, record_every=2)
        seg = segments if segments != "short" else ([shape[0] - 2, 1] if shape[0] > 2 else 24)

        def sim(x_segment):
            s = DeviceSimulation(sp, ids, TABLE, dt, precision="f32k", surface_mode=surface, bc=bc, source_mode=source,
                                 max_steps=steps, record_every=2, tile_j=tile_j,
                                 x_segment=x_segment if isinstance(x_segment, int) else 24)
            if not isinstance(x_segment, int):
                s.set_tiling(tile_j, x_segment)
            s.set_source(src)
            return s

        def check(s, how):
            for key, w in zip(("ux", "uy", "uz"), want.u):
                assert np.array_equal(s.download(key), w), (shape, key, how)
            assert np.array_equal(s.read_surface(), want_surf), (shape, how)

        with sim(seg) as s:
            s.step(steps)
            s.sync()
            check(s, "alone")
        if shape[1] < 4:
            continue
        for streams in (0, 2):
            with sim(seg) as s, sim(24) as t, Batch(2, precision="f32k", tile_j=tile_j, streams=streams) as batch:
                batch.add(s, steps)
                batch.add(t, steps)
                batch.step(steps)
                batch.sync()
                check(s, streams)
                check(t, streams)
