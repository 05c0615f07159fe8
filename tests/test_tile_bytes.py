"""The byte count of a tile launch that the bench's roofline uses stays within
the arrays the solver holds."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("qmu,scheme", [(None, 1), (40.0, 1), (40.0, 2)])
def test_bytes_of_a_tile_launch_are_within_the_solvers_arrays(qmu, scheme):
    """A launch cannot move more than every array of the solver once and what it
    writes once more: the memory variables, the fields of the points and the
    partial sums."""
    from fwi_case import Case
    from specfem2d_b200.configs import tile_launch_bytes
    from specfem2d_b200.runtime import ElasticSolver

    db = Case(nstep=10, qmu=qmu, time_scheme=scheme).start_db()
    s = ElasticSolver(db, tile_elems=32)
    info = s.layout_info()
    n_int = db.nglob - info["nshared"]
    got = tile_launch_bytes(db.nspec, n_int, info["n_slots"], db.atten is not None, scheme)
    written = 24 * n_int + 8 * info["n_slots"]
    if scheme == 2:
        written += 16 * n_int
    if db.atten is not None:
        written += db.nspec * 25 * (48 if scheme == 1 else 72)
    # a point that several tiles touch is read by each of them
    again = 24 * (info["n_slots"] - info["nshared"])
    assert got <= info["device_bytes"] + written + again
    assert got > 600 * db.nspec

