"""Tiles by rows: local numbering, assembly phases and kernels on meshes whose
elements do not share one orientation, and at tile sizes around one warp's
elements.

Half of the elements are turned by 180 degrees (their GLL arrays reversed, the
mapping derivatives negated): the same mesh and medium, but neighbours hold
common points at positions of one class, so that a tile needs more than the
four assembly phases of a structured mesh.  The reference is the oracle on the
mesh as it was; tolerance 1e-5 relative L2, the repository's bound for
seismograms and displacement, and for kernels the FP32 oracle's own distance
from FP64 (at least 1e-5)."""
import copy

import numpy as np
import pytest

from fwi_case import Case
from helpers import rel_l2


def turned(db, seed=0):
    out = copy.copy(db)
    t = np.random.default_rng(seed).random(db.nspec) < 0.5

    def rev(a, sign=1.0):
        a = np.array(a)
        a[t] = sign * a[t][:, ::-1, ::-1]
        return a

    out.ibool = rev(db.ibool).astype(np.int32)
    for k in ("xix", "xiz", "gammax", "gammaz"):
        setattr(out, k, rev(getattr(db, k), -1.0))
    for k in ("jacobian", "rhostore", "kappastore", "mustore", "rho_vpstore", "rho_vsstore"):
        setattr(out, k, rev(getattr(db, k)))
    if db.atten is not None:
        out.atten = {k: rev(v) for k, v in db.atten.items()}
    if db.aniso is not None:
        out.aniso = {k: (v if k == "ispec" else rev(v)) for k, v in db.aniso.items()}
    ts, tr = t[db.source_ispec], t[db.rec_ispec]
    out.sourcearrays = np.array(db.sourcearrays)
    out.sourcearrays[ts] = db.sourcearrays[ts][:, ::-1, ::-1]
    out.hxir, out.hgammar = np.array(db.hxir), np.array(db.hgammar)
    out.hxir[tr], out.hgammar[tr] = db.hxir[tr][:, ::-1], db.hgammar[tr][:, ::-1]
    return out


def _db(physics, nstep):
    c = Case(nstep=nstep, qmu=40.0 if physics.startswith("visco") else None, time_scheme=2 if "lddrk" in physics else 1)
    db = c.start_db()
    if physics.endswith(("mixed", "point")):
        # coefficients that differ inside the elements: two sets, which points
        # name, or 24,000, which are more than are shared
        f, keys = np.arange(25).reshape(5, 5) % 2 + np.zeros(db.ibool.shape), ("a1", "b1", "a2", "b2", "phi1", "phi2")
        if physics.endswith("point"):
            f, keys = np.random.default_rng(4).uniform(0.0, 50.0, db.ibool.shape), ("b1", "b2", "phi1", "phi2")
        for k in keys:
            db.atten[k] = (db.atten[k] * (1.0 + 1e-3 * f)[..., None]).astype(np.float32)
    if physics == "aniso":
        f32 = np.float32
        k, m = db.kappastore, db.mustore
        db.aniso = {"ispec": np.arange(db.nspec) % 3 == 0, "c11": (1.1 * (k + m)).astype(f32),
                    "c13": (0.9 * (k - m)).astype(f32), "c15": (0.02 * k).astype(f32), "c33": (k + m).astype(f32),
                    "c35": (-0.01 * k).astype(f32), "c55": (1.05 * m).astype(f32)}
    return db


@pytest.mark.parametrize("tile_elems", [1, 5, 16, 33, 64, 256])
def test_row_tiles_of_a_mesh_without_orientation(tile_elems):
    from specfem2d_b200 import runtime

    db = _db("iso", 10)
    assert runtime.tiling_stats(db, tile_elems)["max_phases"] <= 4
    st = runtime.tiling_stats(turned(db), tile_elems)
    assert st["max_phases"] <= 16 and (tile_elems == 1 or st["max_phases"] >= 4)


@pytest.mark.gpu
@pytest.mark.parametrize("physics,tile_elems", [("iso", 1), ("iso", 17), ("iso", 32), ("iso", 256), ("aniso", 31),
                                                ("aniso", 128), ("visco", 16), ("visco", 48), ("visco", 128),
                                                ("visco mixed", 32), ("visco point", 32),
                                                ("visco lddrk mixed", 16), ("visco lddrk point", 17)])
def test_lane_kernels_on_a_mesh_without_orientation(physics, tile_elems):
    import oracle
    from specfem2d_b200.runtime import ElasticSolver

    n = 400
    db = _db(physics, n)
    s = ElasticSolver(turned(db), tile_elems=tile_elems)
    assert s.layout_info()["max_elems"] == min(tile_elems, 128)
    seis = s.run(n)
    o = oracle.Oracle(db, 4)
    ref = o.run(n)
    assert rel_l2(seis, ref) < 1e-5
    assert rel_l2(s.get_fields()[0], o.displ) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("physics", ["iso", "visco"])
def test_lane_gradient_on_a_mesh_without_orientation(physics):
    _lane_gradient(physics, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("physics,tile_elems", [("iso", 33), ("iso", 128), ("visco", 64), ("visco", 128),
                                                ("visco point", 32)])
def test_lane_gradient_in_larger_tiles(physics, tile_elems):
    _lane_gradient(physics, tile_elems)


def _lane_gradient(physics, tile_elems):
    import oracle
    from specfem2d_b200.fwi import FWIGradient

    n = 300
    db = _db(physics, n)
    t = np.arange(n)[None, :, None] / n
    rng = np.random.default_rng(5)
    adj = np.sin(2 * np.pi * rng.uniform(2, 6, (len(db.rec_ispec), 1, 2)) * t) * np.sin(np.pi * t) ** 2
    tdb = turned(db)
    g = FWIGradient(tdb, 70, tile_elems=tile_elems)
    g.forward()
    k = g.backward(adj)
    flip = (tdb.ibool != db.ibool).any(axis=(1, 2))
    o32, o64 = (oracle.adjoint_kernels(db, adj, checkpoint_every=70, precision=p)[2:] for p in (4, 8))
    for got, r32, r64 in zip(k, o32, o64):
        got = np.array(got)
        got[flip] = got[flip][:, ::-1, ::-1]
        assert rel_l2(got, r64) < max(1e-5, 1.5 * rel_l2(r32, r64))


@pytest.mark.gpu
def test_gradient_on_tiles_of_scattered_elements(monkeypatch):
    """Elements in random order and no element centres: a tile of 128 holds more
    than 3,064 points, more than an adjoint run has shared memory for, so both
    runs take smaller tiles.  Against the ordered mesh, whose sums are in
    another order (1e-4, four times what that changes in a kernel)."""
    from specfem2d_b200 import configs, fwi, runtime

    n = 500
    db = configs.c1_homogeneous(nstep=n)
    perm = np.random.default_rng(1).permutation(db.nspec)
    mixed = copy.copy(db)
    for k in ("ibool", "xix", "xiz", "gammax", "gammaz", "jacobian", "rhostore", "kappastore", "mustore", "rho_vpstore",
              "rho_vsstore"):
        setattr(mixed, k, np.ascontiguousarray(getattr(db, k)[perm]))
    new = np.argsort(perm).astype(np.int32)
    mixed.source_ispec, mixed.rec_ispec = new[db.source_ispec], new[db.rec_ispec]
    shared = [mixed.ibool[k:k + 128].reshape(-1) for k in range(0, db.nspec, 128)]
    assert max(len(np.unique(p)) for p in shared) > 3064
    t = np.arange(n)[None, :, None] / n
    adj = np.sin(2 * np.pi * np.random.default_rng(2).uniform(2, 6, (len(db.rec_ispec), 1, 2)) * t) * np.sin(np.pi * t) ** 2

    def kernels(d, **kw):
        g = fwi.FWIGradient(d, 125, **kw)
        seis = g.forward()
        return [seis] + list(g.backward(adj))

    ref = kernels(db)

    def without_centres(*a):
        d, keep = runtime.build_desc(*a)
        d.centroid_xz = None
        return d, keep

    monkeypatch.setattr(fwi, "build_desc", without_centres)
    got = kernels(mixed, tile_elems=128)
    assert rel_l2(got[0], ref[0]) < 1e-5
    for a, b in zip(got[1:], ref[1:]):
        assert np.linalg.norm(b) > 0 and rel_l2(a, b[perm]) < 1e-4
