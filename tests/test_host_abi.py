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


def test_memory_of_fp64_handles_with_a_tile_shape(L):
    """The stress window of the two-launch step is held by the handles that
    step that way alone, and the footprint of a handle is what it allocates."""
    shape, out = (21, 70, 60), ctypes.c_size_t()
    held = {}
    for kw in ({}, {"tile_j": 8}, {"x_segment": 12}, {"tile_j": 16, "x_segment": -4}):
        for precision, code in (("f64", 0), ("f64v", 2), ("f32k", 1)):
            h = Handle(L, shape, precision, max_steps=30, **kw)
            held[precision, bool(kw)] = L.fake_bytes(0)
            assert L.phono_footprint_shaped(*shape, code, 30, 0, kw.get("tile_j", 0), kw.get("x_segment", 0),
                                            ctypes.byref(out)) == 0
            assert out.value == L.fake_bytes(0), (precision, kw)
            if not kw:
                assert L.phono_footprint(*shape, code, 30, 0, ctypes.byref(out)) == 0 and out.value == held[precision, False]
                if precision == "f64":
                    assert L.phono_step(h.h, 13) == 0 and L.phono_set_tiling(h.h, 8, 6) == 0 and L.phono_step(h.h, 13) == 0
                    assert L.fake_bytes(0) == held["f64", False] - window(shape)
            h.close()
            assert L.fake_bytes(0) == 0 and L.fake_broken() == 0
    assert held["f64", True] == held["f64", False] - window(shape)
    assert held["f64v", True] == held["f64v", False] and held["f32k", True] == held["f32k", False]


def test_the_window_comes_after_what_a_handle_cannot_do_without(L):
    """A handle that fits the device's memory without the stress window is made,
    and steps by tiles."""
    shape, out = (21, 70, 60), ctypes.c_size_t()
    assert L.phono_footprint_shaped(*shape, 0, 30, 1, 8, 0, ctypes.byref(out)) == 0
    for spare, form in ((0, b"tile"), (window(shape) - 512, b"tile"), (window(shape), b"split")):
        L.fake_limit(out.value + spare)
        h = Handle(L, shape, "f64", max_steps=30, record_every=1)
        assert h.rc == 0, L.phono_last_error()
        n = L.fake_count(form)
        assert L.phono_step(h.h, 5) == 0 and L.fake_count(form) > n
        h.close()
    assert L.fake_bytes(0) == 0 and L.fake_broken() == 0


def window(shape):
    """Bytes of the leapfrog's window: six stresses of rows padded to 64 bytes, the first 32 of them zeros."""
    return -(-6 * shape[0] * shape[1] * -(-(4 + shape[2]) // 8) * 64 // 512) * 512


@pytest.mark.parametrize("what", ["sync", "copy", "configure"])
@pytest.mark.parametrize("shape,tile", [((30, 21, 13), 0), ((60, 70, 60), 0), ((60, 70, 60), 4)])
def test_a_failed_join_leaves_the_handle_as_it_was(L, what, shape, tile):
    ref = Handle(L, shape, tile_j=tile)
    h = Handle(L, shape, tile_j=tile)
    form = "split" if shape == (30, 21, 13) else "tile"
    b = ctypes.c_void_p()
    assert L.phono_batch_create(2, 1, 4, ctypes.byref(b)) == 0
    assert L.phono_step(h.h, 1) == 0 and L.phono_step(ref.h, 1) == 0
    for after in (1, 2):
        L.fake_fail(what.encode(), after)
        rc = L.phono_batch_add(b, h.h, 20)
        L.fake_fail(what.encode(), 0)
        if rc < 0:  # alone: the kernels it had
            n = L.fake_count(form.encode())
            assert L.phono_step(h.h, 3) == 0
            steps = L.fake_count(form.encode()) - n
            n = L.fake_count(form.encode())
            assert L.phono_step(ref.h, 3) == 0
            assert steps == L.fake_count(form.encode()) - n > 0
        else:
            assert L.phono_batch_step(b, 5) == 0 and L.phono_batch_remove(b, rc) == 0
    slot = L.phono_batch_add(b, h.h, 20)
    assert slot >= 0 and L.phono_batch_step(b, 20) == 0 and L.phono_batch_remove(b, slot) == 0
    L.phono_batch_destroy(b)
    for x in (h, ref):
        x.close()
    assert L.fake_broken() == 0


def test_segments_that_cannot_be_cut_anew(L):
    """Tensor maps that cannot be made while a batch is stepped or left: the
    call reports it, nothing is launched without maps, and a later call works."""
    small, large = Handle(L, (30, 21, 13)), Handle(L, (130, 150, 40))
    b = ctypes.c_void_p()
    assert L.phono_batch_create(2, 1, 4, ctypes.byref(b)) == 0
    slots = [L.phono_batch_add(b, h.h, 40) for h in (small, large)]
    for after in (1, 2, 5):
        L.fake_fail(b"encode", after)
        assert L.phono_batch_step(b, 5) < 0
        L.fake_fail(b"encode", 0)
    assert L.phono_batch_step(b, 5) == 0
    L.fake_fail(b"encode", 1)
    assert L.phono_batch_remove(b, slots[1]) < 0
    L.fake_fail(b"encode", 0)
    assert L.phono_step(large.h, 5) == 0  # out of the batch, in tiles that work
    assert L.phono_batch_step(b, 5) == 0 and L.phono_batch_remove(b, slots[0]) == 0
    assert L.phono_step(small.h, 20) == 0
    L.phono_batch_destroy(b)
    for h in (small, large):
        h.close()
    assert L.fake_broken() == 0


@pytest.mark.parametrize("what", ["encode", "copy", "both"])
def test_a_handle_that_cannot_take_its_form_back(L, what):
    """A default FP32 handle whose own tiles or two-launch form cannot be set up
    as it leaves a batch: reported, out of the batch, and a graph captured in
    the form it had before is not replayed on the state of another."""
    h = Handle(L, (30, 21, 13))
    b = ctypes.c_void_p()
    assert L.phono_batch_create(1, 1, 4, ctypes.byref(b)) == 0
    assert L.phono_step(h.h, 13) == 0  # 12 of them by a graph of the two-launch form
    slot = L.phono_batch_add(b, h.h, 20)
    for name in ("encode", "copy") if what == "both" else (what,):
        L.fake_fail(name.encode(), 1)
    assert L.phono_batch_remove(b, slot) < 0
    tiles, splits = L.fake_count(b"tile"), L.fake_count(b"split")
    assert L.phono_step(h.h, 13) == 0
    # 13 steps launched or captured anew, in one form
    assert (L.fake_count(b"tile") - tiles, L.fake_count(b"split") - splits) == ((0, 26) if what == "encode" else (13, 0))
    slot = L.phono_batch_add(b, h.h, 20)
    assert slot >= 0 and L.phono_batch_step(b, 20) == 0 and L.phono_batch_remove(b, slot) == 0
    L.phono_batch_destroy(b)
    h.close()
    assert L.fake_broken() == 0
