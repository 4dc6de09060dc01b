"""Material ids through the stage of their upload (256 KB and more) and below
it: rows around multiples of the 8 bytes a thread writes, an upload of several stages (a last one of few
rows) and rows longer than half a stage.  The ids read back are those uploaded,
and a refused upload leaves them.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 5, 7), (9, 6, 33), (120, 781, 7), (300, 310, 3), (99, 83, 32), (91, 90, 33), (161, 160, 164), (3, 3, 3000001),
                                   (3, 3, 4200001)])
def test_ids_round_trip(gpu_lib, shape):
    from phonomena_gb300.device import DeviceSimulation

    rng = np.random.default_rng(sum(shape))
    table = np.ones((256, 13))
    sp = {k + a: np.full(n - 1 - (k == "sd"), 1e-5) for a, n in zip("xyz", shape) for k in ("fd", "sd")}
    ids = rng.integers(0, 256, shape, dtype=np.uint8)
    with DeviceSimulation(sp, ids, table, 1e-10, precision="f32k", max_steps=1) as s:
        assert np.array_equal(s.download_materials(), ids)
        ids = rng.integers(0, 256, shape, dtype=np.uint8)
        s.set_materials(ids, table)
        assert np.array_equal(s.download_materials(), ids)
        bad = ids.copy()
        bad[-1, -1, -1] = 255
        with pytest.raises(Exception, match="out of range"):
            s.set_materials(bad, table[:255])
        assert np.array_equal(s.download_materials(), ids)


def test_uploads_of_several_threads(gpu_lib):
    """Handles of several threads share the stage; the last one gives it back."""
    import threading

    from phonomena_gb300.device import DeviceSimulation

    shape, failed = (70, 90, 61), []
    table = np.ones((256, 13))
    sp = {k + a: np.full(n - 1 - (k == "sd"), 1e-5) for a, n in zip("xyz", shape) for k in ("fd", "sd")}

    def work(seed):
        rng = np.random.default_rng(seed)
        for _ in range(4):
            ids = rng.integers(0, 256, shape, dtype=np.uint8)
            with DeviceSimulation(sp, ids, table, 1e-10, precision="f32k", max_steps=1) as s:
                for _ in range(4):
                    if not np.array_equal(s.download_materials(), ids):
                        failed.append(seed)
                    ids = rng.integers(0, 256, shape, dtype=np.uint8)
                    s.set_materials(ids, table)

    threads = [threading.Thread(target=work, args=(q,)) for q in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
