"""Fields read back into pinned host memory (a kernel writes the dense array)
against the copy into pageable memory: rows shorter and longer than a 16-byte
vector, extents off every multiple, arrays that start off a 16-byte boundary,
a fraction of a pinned block, neighbours untouched, and a field below the size
that takes the kernel.  Bytes equal.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(9, 6, 4), (300, 60, 3), (41, 33, 34), (33, 35, 130), (3, 4, 6001)]


@pytest.mark.parametrize("precision", ["f32k", "f64", "f64v"])
@pytest.mark.parametrize("lead", [0, 1, 3])
def test_pinned_equals_pageable(gpu_lib, precision, lead):
    import torch
    from phonomena_gb300.device import DeviceSimulation
    from test_gpu_split import TABLE, _problem

    for shape in SHAPES:
        sp, ids, dt, src = _problem(shape, sum(shape), 4)
        with DeviceSimulation(sp, ids, TABLE, dt, precision=precision, max_steps=4) as s:
            rng = np.random.default_rng(sum(shape))
            for f in s.state_fields:
                want = rng.standard_normal(s.download(f).shape).astype(s.dtype)
                s.upload(f, want)
                block = torch.full((want.size + 16,), 7.0, dtype=torch.float32 if precision == "f32k" else torch.float64,
                                   pin_memory=True).numpy()
                out = block[lead:lead + want.size].reshape(want.shape)
                s.download(f, out=out)
                assert np.array_equal(out, want), (shape, f)
                assert np.all(block[:lead] == 7) and np.all(block[lead + want.size:] == 7), (shape, f)
                assert np.array_equal(s.download(f), want), (shape, f)
