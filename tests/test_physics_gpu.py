"""GPU parity of the anisotropic, viscoelastic (3 SLS) and LDDRK variants of the
tile-staged elastic kernel against the CPU oracle and the reference's golden traces.

Tolerances (relative L2): seismograms and displacement 1e-5 against the FP32
oracle; golden traces 1e-5 on the windows the oracle is pinned on.
"""
import numpy as np
import pytest

from helpers import load_golden, rel_l2
from specfem2d_b200.setup.from_par_file import database_from_config

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _compare(db, nstep, **solver_kw):
    import oracle
    from specfem2d_b200.runtime import ElasticSolver

    o = oracle.Oracle(db, 4)
    ref = o.run(nstep)
    sol = ElasticSolver(db, **solver_kw)
    if "tile_elems" in solver_kw:
        assert sol.layout_info()["max_elems"] == solver_kw["tile_elems"]
    s = sol.run(nstep)
    d, _, _ = sol.get_fields()
    return s, ref, d, o.displ


@pytest.mark.parametrize("threads", [256, 250])
def test_anisotropic_gpu_matches_oracle_and_golden(threads):
    cfg, golden = load_golden("anisotropic_isotropic_model")
    db = database_from_config(cfg)
    s, ref, d, d_or = _compare(db, db.nstep, threads_per_block=threads)
    assert rel_l2(s, ref) < TOL
    assert rel_l2(d, d_or) < TOL
    assert rel_l2(s[0, :, 0], golden["S0001_BXX"]) < TOL
    assert rel_l2(s[0, :, 1], golden["S0001_BXZ"]) < TOL


@pytest.mark.parametrize("tile_elems,threads", [(16, 256), (64, 256), (32, 250)])
def test_viscoelastic_newmark_gpu_matches_oracle_and_golden(tile_elems, threads):
    cfg, golden = load_golden("attenuation_viscoelastic")
    db = database_from_config(cfg, absorbing_as_stacey=True)
    s, ref, d, d_or = _compare(db, db.nstep, tile_elems=tile_elems, threads_per_block=threads)
    assert rel_l2(s, ref) < TOL
    assert rel_l2(d, d_or) < TOL
    t = float(golden["t_first"]) + float(golden["t_step"]) * np.arange(db.nstep)
    w = t <= 0.4
    assert rel_l2(s[0, w, 0], golden["S0001_BXX"][w]) < TOL
    assert rel_l2(s[0, w, 1], golden["S0001_BXZ"][w]) < TOL


def test_lddrk_elastic_gpu_matches_oracle():
    cfg, _ = load_golden("tromp2005_kernel")
    db = database_from_config(cfg, nstep=1500, time_scheme=2)
    s, ref, d, d_or = _compare(db, 1500)
    assert rel_l2(s, ref) < TOL
    assert rel_l2(d, d_or) < TOL


@pytest.mark.parametrize("threads", [256, 250])
def test_lddrk_viscoelastic_gpu_matches_oracle(threads):
    cfg, _ = load_golden("attenuation_viscoelastic")
    db = database_from_config(cfg, absorbing_as_stacey=True, time_scheme=2)
    s, ref, d, d_or = _compare(db, db.nstep, tile_elems=32, threads_per_block=threads)
    assert rel_l2(s, ref) < TOL
    assert rel_l2(d, d_or) < TOL


def test_lddrk_and_newmark_agree_to_time_discretisation_error():
    """Both schemes approximate the same wave equation: the traces of the
    viscoelastic example differ by the time-discretisation error only."""
    from specfem2d_b200.runtime import ElasticSolver

    cfg, _ = load_golden("attenuation_viscoelastic")
    nm = database_from_config(cfg, absorbing_as_stacey=True)
    lk = database_from_config(cfg, absorbing_as_stacey=True, time_scheme=2)
    a = ElasticSolver(nm).run(nm.nstep)
    b = ElasticSolver(lk).run(lk.nstep)
    assert rel_l2(b, a) < 2e-2


def test_lddrk_initial_mode_gpu_matches_oracle_and_ref_seis():
    """EXAMPLES/initial_mode_LDDRK on the fluid tile kernels (LDDRK variant, free
    surfaces on all four edges, no source): started from the analytical membrane
    mode, the GPU traces over 5500 steps lie within the FP32 band around the FP64
    oracle (as the reference's own FP32 traces do) and within 2.5x that band of
    the reference's traces.  See test_oracle_golden for the band."""
    from helpers import initial_mode_run, within_fp32_band
    from specfem2d_b200.coupled import CoupledSolver

    cfg, seis = load_golden("initial_mode_lddrk")
    db = database_from_config(cfg)
    ref = np.stack([seis["S0001_BXX"], seis["S0001_BXZ"]], axis=1)
    o32, o64 = initial_mode_run(db, 4), initial_mode_run(db, 8)
    s = CoupledSolver(db)
    f = db.initial_field
    s.set_fields(pot=f["pot"], pot_dot=f["pot_dot"], pot_dot_dot=f["pot_dot_dot"])
    gpu = s.run(db.nstep)[0]
    assert within_fp32_band(gpu, o64, o32, o64)
    for c in (0, 1):
        assert rel_l2(gpu[:, c], ref[:, c]) < 2.5 * rel_l2(o32[:, c], o64[:, c])
