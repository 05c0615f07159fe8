"""Kernel smoothing (smooth_sem.F90:63-467): the oracle's restatement of the
reference's CPU loop (every pair of points, CUSTOM_REAL) and the GPU kernel
(sf2d_smooth: cells of `cutoff` standard deviations, double sums).

No reference output pins the smoothing (the reference ships no smoothed
kernel files); the oracle follows the CPU program's arithmetic and the GPU is
held to it.  Tolerance: 1e-5 relative L2 (the GPU leaves out weights below
exp(-18) and sums in double; the oracle sums in float)."""
import numpy as np
import pytest

from fwi_case import Case
from helpers import rel_l2


@pytest.fixture(scope="module")
def fields():
    c = Case(nstep=10)
    db = c.start_db()
    rng = np.random.default_rng(0)
    f = np.stack([np.ones((db.nspec, 5, 5)), c.anomaly(), rng.standard_normal((db.nspec, 5, 5)),
                  c.anomaly(2100.0, 1100.0, 150.0) * rng.uniform(0.5, 1.5, (db.nspec, 5, 5))])
    return db, f.astype(np.float32)


def test_oracle_smoothing_keeps_constants_and_averages(fields):
    import oracle

    db, f = fields
    out = oracle.smooth(db, f, 200.0, 100.0)
    assert np.abs(out[0] - 1.0).max() < 1e-6            # a normalised average of a constant
    assert out[1].max() < f[1].max() and out[1].min() >= f[1].min()
    assert out[2].std() < 0.1 * f[2].std()              # white noise averages out
    # every copy of a global point gets the value of the point
    g = db.ibool.ravel()
    v = out[1].ravel()
    first = np.full(db.nglob, -1)
    first[g[::-1]] = np.arange(g.size - 1, -1, -1)
    assert np.array_equal(v, v[first[g]])


@pytest.mark.gpu
@pytest.mark.parametrize("sigmas", [(200.0, 100.0), (150.0, 300.0)])
def test_gpu_smoothing_matches_oracle(fields, sigmas):
    import oracle

    from specfem2d_b200.runtime import smooth

    db, f = fields
    ref = oracle.smooth(db, f, *sigmas)
    got = smooth(db, f, *sigmas)
    for k in range(f.shape[0]):
        assert rel_l2(got[k], ref[k]) < 1e-5, k


@pytest.mark.gpu
@pytest.mark.parametrize("nspec, extent, size, nfields",
                         [(1, 1.0, 4.0, 1), (11, 0.5, 0.3, 2), (21, 400.0, 8.0, 4), (300, 30.0, 0.7, 3)])
def test_gpu_smoothing_of_scattered_elements(nspec, extent, size, nfields):
    """One element, more than a block's targets in one cell, few elements in a wide extent, elements larger than
    the cutoff, against all pairs in double.  A weight exp(-r2/2) is off by at most r2 x 2 x 2^-24 + 2^-22 (the
    rounding of r2 and of expf), below 5e-6 where r2 <= 36, and what lies beyond weighs below 2e-8: 1e-5."""
    from types import SimpleNamespace

    from specfem2d_b200.runtime import smooth

    rng = np.random.default_rng(nspec)
    unit = np.array([-1.0, -0.6546537, 0.0, 0.6546537, 1.0])
    mid = rng.uniform(0.0, extent, (nspec, 2))
    half = 0.5 * size * rng.uniform(0.5, 1.0, (nspec, 2))
    x = np.broadcast_to((mid[:, 0, None] + half[:, 0, None] * unit)[:, None, :], (nspec, 5, 5))
    z = np.broadcast_to((mid[:, 1, None] + half[:, 1, None] * unit)[:, :, None], (nspec, 5, 5))
    sh, sv = 1.25, 0.75
    wg = np.array([0.1, 0.5444444, 0.7111111, 0.5444444, 0.1])
    db = SimpleNamespace(nspec=nspec, ibool=np.arange(nspec * 25).reshape(nspec, 5, 5),
                         coord=np.stack([(sh * x).ravel(), (sv * z).ravel()], 1),
                         jacobian=rng.uniform(0.5, 2.0, (nspec, 5, 5)), gll=SimpleNamespace(wgll_dble=wg))
    f = rng.uniform(1.0, 2.0, (nfields, nspec, 5, 5)).astype(np.float32)
    got = smooth(db, f, sh, sv)
    sx = (db.coord[:, 0].astype(np.float32) / np.float32(sh)).astype(np.float64)
    sz = (db.coord[:, 1].astype(np.float32) / np.float32(sv)).astype(np.float64)
    r2 = (sx[:, None] - sx) ** 2 + (sz[:, None] - sz) ** 2
    g = np.where(r2 <= 36.0, np.exp(-0.5 * r2), 0.0) * (db.jacobian * np.outer(wg, wg)).ravel()
    ref = (f.reshape(nfields, -1).astype(np.float64) @ g.T / g.sum(1)).reshape(f.shape)
    assert np.abs(got / ref - 1.0).max() < 1e-5
