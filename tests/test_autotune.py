"""The tile autotuner times every configuration that differs once."""
from types import SimpleNamespace

import numpy as np
import pytest


class FakeSolver:
    """Tiles as the library forms them on a mesh of 3000 elements: 0 means 8,
    96 and 128 do not fit; the time falls with the tile size."""
    built = []

    def __init__(self, db, tile_elems=0, threads_per_block=256):
        from specfem2d_b200.runtime import SF2DError

        if tile_elems > 64:
            raise SF2DError(-1, "tile too large for shared memory")
        self.te, self.nt = tile_elems or 8, threads_per_block
        FakeSolver.built.append((tile_elems, threads_per_block))

    def enqueue(self, n):
        pass

    def synchronize(self, t):
        pass

    def time_kernels(self, n):
        return [10.0 / self.te, 1.0, 10.0 / self.te + 1.0 + 1e-3 * self.nt]

    def layout_info(self):
        return {"ntiles": -(-3000 // self.te), "nshared": 7, "max_elems": self.te, "threads_per_block": 5 * self.te,
                "smem_bytes": 1}

    def close(self):
        pass


@pytest.mark.parametrize("region,threads", [(None, [256]), (np.zeros(3000, int), [256]),
                                            (np.arange(3000) % 2, [256, 512])])
def test_autotune_times_each_configuration_once(monkeypatch, region, threads):
    """Without CPML elements threads_per_block changes nothing, and 0 and 8 are the same tiles here."""
    from specfem2d_b200 import autotune, runtime

    monkeypatch.setattr(runtime, "ElasticSolver", FakeSolver)
    db = SimpleNamespace(pml=None if region is None else {"region": region})
    best, results = autotune.autotune_elastic(db, tiles=(0, 8, 32, 64, 128), threads=(256, 512))
    timed = [(r["tile_elems"], r["threads"], r["max_elems"]) for r in results if "step_ms" in r]
    assert timed == [(te, nt, te or 8) for te in (0, 32, 64) for nt in threads]
    assert [r["tile_elems"] for r in results if "error" in r] == [128] * len(threads)
    assert best == (64, 256)
