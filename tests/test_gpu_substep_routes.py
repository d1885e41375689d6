"""The default path's kernels by size: every route must give the bits of the
one-launch substep, which takes the same arithmetic through one route at all
sizes (two threads per cell in P2G; tile allocation and bucketing of their
own).  One scene steps with two threads per cell up to 640 particles per SM and
with one above; its tiles are bucketed by one kernel up to 4,096 of them and by
two above; and G2P takes a tile in up to four parts while there are at most 256
particles per SM."""
import numpy as np
import pytest

from mpm_b200 import create_mpm_mls_gpu_solver
from mpm_b200.layout import ParticleArrays

pytestmark = pytest.mark.gpu

WATER = {"lambda": 160_000.0, "mu": 0.0, "model": "water", "density": 0.02}
OIL = {"lambda": 120_000.0, "mu": 0.0, "model": "oil", "density": 0.016}
SMS = 148


def _scene(n, cells_x, cells_y, spacing):
    rng = np.random.default_rng(n)
    columns = max(1, min(n, int((cells_x - 4) * 10 / spacing)))
    r, c = np.divmod(np.arange(n), columns)
    p = ParticleArrays.empty(n)
    p.px[:] = 20 + (c + 0.5 + rng.uniform(-0.3, 0.3, n)) * spacing
    p.py[:] = 20 + (r + 0.5 + rng.uniform(-0.3, 0.3, n)) * spacing
    assert p.py.max() < cells_y * 10
    p.vx[:], p.vy[:] = rng.uniform(-40, 40, n), rng.uniform(-40, 40, n)
    p.volume[:] = spacing * spacing
    p.materials = [WATER, OIL]
    p.material[:] = (r % 40 >= 20).astype(np.int32)
    config = {"grid": {"cellsX": cells_x, "cellsY": cells_y, "cellSize": 10}, "particleMass": 0.5,
              "particleVolume": 25.0, "material": WATER}
    return p, config


@pytest.mark.parametrize("n, cells_x, cells_y, spacing", [
    (1, 20, 20, 5.0),
    (257, 17, 33, 5.0),
    (640 * SMS, 400, 400, 5.0),      # the last size with two threads per cell
    (640 * SMS + 1, 400, 400, 5.0),  # and the first with one
    (256 * SMS, 300, 250, 5.0),      # the last size whose tiles G2P divides
    (256 * SMS + 1, 300, 250, 5.0),
    (3_000, 17, 33, 3.0),            # more items than tiles
    (30_001, 1021, 509, 5.0),        # 4,096 tiles: bucketed by one kernel
    (30_001, 1021, 510, 5.0),        # 4,160
    (60_001, 120, 130, 2.5),         # 16 particles per cell: every tile above one stage
])
def test_every_route_gives_the_one_launch_bits(n, cells_x, cells_y, spacing):
    p, config = _scene(n, cells_x, cells_y, spacing)
    runs = []
    for fused in (False, True):
        solver = create_mpm_mls_gpu_solver(p, config)
        try:
            solver.set_substep_variant(fused=fused, p2g_records=False)
            solver.step_batch(9, 1 / 1500, {"x": 3.0, "y": 90.0})
            assert solver.read_status_words()[0] == 0
            runs.append(solver.read_particles_packed()[0])
        finally:
            solver.dispose()
    assert np.array_equal(np.ascontiguousarray(runs[0]).view(np.uint32), np.ascontiguousarray(runs[1]).view(np.uint32))


@pytest.mark.parametrize("cells_x, cells_y", [(509, 253), (510, 253), (509, 509), (509, 510)])
def test_bucketing_at_each_number_of_tiles(cells_x, cells_y):
    """1,024 tiles and 1,056, 2,048 and 2,080: the bucketing kernel's instances;
    particles in the first and last tiles, few enough for one CTA and a second."""
    for n in (1, 1_024, 1_025, 5_000):
        rng = np.random.default_rng(n)
        p = ParticleArrays.empty(n)
        p.px[:], p.py[:] = rng.uniform(20, cells_x * 10 - 20, n), rng.uniform(20, cells_y * 10 - 20, n)
        p.px[-1], p.py[-1] = cells_x * 10 - 5, cells_y * 10 - 5
        p.volume[:] = 25.0
        p.materials = [WATER]
        p.material[:] = 0
        config = {"grid": {"cellsX": cells_x, "cellsY": cells_y, "cellSize": 10}, "particleMass": 0.5,
                  "particleVolume": 25.0, "material": WATER}
        runs = []
        for fused in (False, True):
            solver = create_mpm_mls_gpu_solver(p, config)
            try:
                solver.set_substep_variant(fused=fused, p2g_records=False)
                solver.step_batch(5, 1 / 1500, {"x": 3.0, "y": 90.0})
                assert solver.read_status_words()[0] == 0
                runs.append(solver.read_particles_packed()[0])
            finally:
                solver.dispose()
        assert np.array_equal(np.ascontiguousarray(runs[0]).view(np.uint32), np.ascontiguousarray(runs[1]).view(np.uint32))
