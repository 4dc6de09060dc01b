"""Energy of FP32 meshes large enough for the pairs-of-floats reduction.

Against numpy sums in FP64 on odd extents (ragged tiles of 8 rows and 32
columns, item edges along x), constants and spacings with full significands:
a pair is good to 2^-47 a term at random and the FP64 sums on either side to a
few 2^-53 times the square root of the number of partial sums, so 1e-13 is far
above both.  Fields outside the range the pairs are used for (all zero, tiny,
huge, not finite) must give what FP64 arithmetic gives.
"""
import numpy as np
import pytest

from test_gpu_parity import _energy_numpy

pytestmark = pytest.mark.gpu


def _mesh(shape, seed):
    rng = np.random.default_rng(seed)
    d = {"ids": rng.choice(3, shape, p=[0.8, 0.1, 0.1]).astype(np.uint8), "dt": 2e-10}
    d["ids"][0, 0, 0] = 0
    c = rng.uniform(1e10, 3e11, (3, 13))
    c[:, 12] = rng.uniform(2e3, 2e4, 3)
    c[1, :12] = 0.0
    d["table"] = c
    for a, n in zip("xyz", shape):
        fd = 1e-5 * rng.uniform(0.5, 1.0, n - 1)
        d["fd" + a], d["sd" + a] = fd, (fd[1:] + fd[:-1]) / 2
    u = [rng.standard_normal([n - (q == c) for q, n in enumerate(shape)]).astype(np.float32) for c in range(3)]
    v = [(1e8 * rng.standard_normal(f.shape)).astype(np.float32) for f in u]
    return d, u, v


def _sim(d, u, v):
    from phonomena_gb300.device import DeviceSimulation

    sp = {k: d[k] for k in ("fdx", "fdy", "fdz", "sdx", "sdy", "sdz")}
    sim = DeviceSimulation(sp, d["ids"], d["table"], d["dt"], precision="f32k", surface_mode="corrected")
    for a, f, w in zip("xyz", u, v):
        sim.upload("u" + a, f)
        sim.upload("v" + a, w)
    return sim


@pytest.mark.parametrize("shape", [(61, 59, 57), (130, 18, 98), (201, 34, 33), (12, 130, 129)])
def test_pair_energy_matches_fp64(gpu_lib, shape):
    d, u, v = _mesh(shape, sum(shape))
    assert np.prod(shape) >= 200000
    ek_ref, es_ref = _energy_numpy(d, [f.astype(np.float64) for f in u], [f.astype(np.float64) for f in v])
    with _sim(d, u, v) as sim:
        ek, es = sim.energy()
        assert sim.energy() == (ek, es)  # a fixed order: the same bits
    assert abs(ek - ek_ref) <= 1e-13 * ek_ref and abs(es - es_ref) <= 1e-13 * es_ref, (ek / ek_ref - 1, es / es_ref - 1)


@pytest.mark.parametrize("scale", [0.0, 1e-24, 1e22])
def test_energy_outside_the_pairs_range(gpu_lib, scale):
    d, u, v = _mesh((61, 59, 57), 3)
    u, v = ([(f * np.float32(scale)).astype(np.float32) for f in fs] for fs in (u, v))
    ek_ref, es_ref = _energy_numpy(d, [f.astype(np.float64) for f in u], [f.astype(np.float64) for f in v])
    with _sim(d, u, v) as sim:
        ek, es = sim.energy()
    assert abs(ek - ek_ref) <= 1e-12 * ek_ref and abs(es - es_ref) <= 1e-12 * es_ref


def test_energy_of_a_non_finite_state(gpu_lib):
    d, u, v = _mesh((61, 59, 57), 3)
    u[2][30, 30, 30] = np.inf
    with _sim(d, u, v) as sim:
        ek, es = sim.energy()
    assert np.isfinite(ek) and not np.isfinite(es)
