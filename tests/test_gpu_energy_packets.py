"""Energy of FP32 meshes of 200,000 nodes and more whose state is a few values:
no error averages out there, and every term has to be as good as FP64 makes it.

Against the sums in the host's long double.  Roundings (u = 2^-53): a kinetic
term two, 4 u allowed; a strain term three in each strain (difference,
reciprocal spacing, product), so six in a square, one in a summed stiffness,
four in the quadratic form, and the sums of at most a dozen terms: 16 u.
"""
import numpy as np
import pytest

from test_gpu_energy import _mesh, _sim
from test_gpu_parity import _energy_numpy

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("shape", [(61, 59, 57), (130, 18, 98)])
@pytest.mark.parametrize("seed", range(6))
def test_energy_of_single_values(gpu_lib, shape, seed):
    assert np.finfo(np.longdouble).nmant >= 63
    d, u, v = _mesh(shape, seed)
    d["ids"][:] = 0
    for m in range(3):  # positive definite: no cancellation between terms
        lam, mu = d["table"][0, 1] / 10, d["table"][0, 9]
        d["table"][m, :9] = np.where(np.arange(9) % 4 == 0, lam + 2 * mu, lam)
    rng = np.random.default_rng(seed)
    c = seed % 3
    at = tuple(rng.integers(3, n - 4) for n in shape)
    for fields, scale in ((u, 1e-6), (v, 1e-3)):
        keep = fields[c][at] * np.float32(scale)
        for f in fields:
            f[:] = 0
        fields[c][at] = keep
    long = {k: w.astype(np.longdouble) if w.dtype == np.float64 else w for k, w in d.items() if isinstance(w, np.ndarray)}
    ek_ref, es_ref = _energy_numpy(long, [f.astype(np.longdouble) for f in u], [f.astype(np.longdouble) for f in v])
    with _sim(d, u, v) as sim:
        ek, es = sim.energy()
    assert abs(ek - ek_ref) <= 4 * U * ek_ref, float((ek - ek_ref) / ek_ref / U)
    assert abs(es - es_ref) <= 16 * U * es_ref, float((es - es_ref) / es_ref / U)


def test_energy_of_values_that_are_not_normal(gpu_lib):
    """Subnormal and zero values of either sign among the others."""
    d, u, v = _mesh((61, 59, 57), 3)
    rng = np.random.default_rng(5)
    for f in (*u, *v):
        f[:] = np.where(rng.random(f.shape) < 0.3, rng.choice(np.array([0.0, -0.0, 1e-40, -3e-45], np.float32), f.shape), f)
    for a in range(3):
        u[a][30:34] *= np.float32(1e-38)
        v[a][30:34] *= np.float32(1e-38)
    ek_ref, es_ref = _energy_numpy(d, [f.astype(np.float64) for f in u], [f.astype(np.float64) for f in v])
    with _sim(d, u, v) as sim:
        ek, es = sim.energy()
    assert abs(ek - ek_ref) <= 1e-13 * ek_ref and abs(es - es_ref) <= 1e-13 * es_ref
    for a in range(3):  # nothing but those
        u[a][:], v[a][:] = np.float32(1e-40), rng.choice(np.array([3e-40, -2e-44], np.float32), v[a].shape)
    with _sim(d, u, v) as sim:
        ek, es = sim.energy()
    ek_ref, es_ref = _energy_numpy(d, [f.astype(np.float64) for f in u], [f.astype(np.float64) for f in v])
    assert ek > 0 and abs(ek - ek_ref) <= 1e-13 * ek_ref and es == es_ref == 0
