"""Host code of the C ABI on a stand-in CUDA runtime."""
import ctypes
import threading

import numpy as np
import pytest

from host_abi import Handle, compile_host_abi


@pytest.fixture(scope="module")
def lib():
    return compile_host_abi()


@pytest.fixture
def L(lib):
    lib.fake_reset()
    return lib


def test_handles_do_not_wait_for_another_ones_steps(L):
    """While an upload waits for the steps its own handle has queued, handles
    of another thread are made, given ids of any size and destroyed."""
    busy = Handle(L, (80, 70, 60), max_steps=1)  # ids above 256 KB: staged
    L.fake_hold(busy.stream(), 1)
    done = threading.Event()

    def others():
        for shape in ((9, 8, 7), (81, 70, 60)):
            h = Handle(L, shape, max_steps=1)
            assert h.rc == 0 and h.set_ids(5) == 0 and h.ids_arrived()
            h.close()
        done.set()

    upload = threading.Thread(target=busy.set_ids, args=(3,))
    upload.start()
    upload.join(0.2)
    assert upload.is_alive()
    worker = threading.Thread(target=others)
    worker.start()
    free = done.wait(5.0)
    L.fake_hold(busy.stream(), 0)
    upload.join()
    worker.join()
    assert free and busy.ids_arrived()
    busy.close()
    assert L.fake_bytes(0) == 0 and L.fake_broken() == 0


def test_calls_with_another_device_current(L):
    """Uploads of ids and reads into pinned memory use the handle's device and
    leave the caller's current."""
    shape = (80, 70, 60)
    h = Handle(L, shape, max_steps=1)
    field = np.random.default_rng(1).standard_normal((79, 70, 60)).astype(np.float32)
    assert L.phono_upload(h.h, 0, field.ctypes.data, field.nbytes) == 0
    got = np.zeros_like(field)
    L.fake_pin(got.ctypes.data, got.nbytes)
    small = Handle(L, (9, 8, 7), max_steps=1)
    L.fake_device(1)
    try:
        assert h.set_ids(7) == 0, L.phono_last_error()
        assert h.ids_arrived()
        reads = L.fake_count(b"readback")
        assert L.phono_download(h.h, 0, got.ctypes.data, got.nbytes) == 0, L.phono_last_error()
        assert L.fake_count(b"readback") == reads + 1 and np.array_equal(got, field)
        assert L.fake_current() == 1 and L.fake_bytes(1) == 0
        h.close()
        small.close()
    finally:
        L.fake_device(0)
    assert L.fake_bytes(0) == 0 and L.fake_broken() == 0


def test_graphs_are_not_destroyed_while_they_run(L):
    """An instance whose segments are cut anew, between calls that do not wait,
    because a larger one has run out."""
    small, large = Handle(L, (30, 21, 13)), Handle(L, (200, 200, 40))
    b = ctypes.c_void_p()
    assert L.phono_batch_create(2, 1, 4, ctypes.byref(b)) == 0
    assert L.phono_batch_add(b, small.h, 90) >= 0 and L.phono_batch_add(b, large.h, 24) >= 0
    graphs = L.fake_count(b"graph")
    assert L.phono_batch_step(b, 24) == 0 and L.phono_batch_step(b, 24) == 0
    assert L.fake_count(b"graph") > graphs and L.fake_broken() == 0
    assert L.phono_batch_sync(b) == 0
    L.phono_batch_destroy(b)
    small.close()
    large.close()


def test_a_handle_is_destroyed_with_steps_queued(L):
    h = Handle(L, (30, 21, 13))
    assert L.phono_step(h.h, 24) == 0
    h.close()
    assert L.fake_broken() == 0
