"""The surface field's two routes: 512 consecutive particles are summed in
shared memory where their stencils' box holds at most 4,096 sums (one per node
and phase) and added one by one where it holds more.  The sums are integers:
the same particles uploaded in another order, so that they take the other route
(or meet in other boxes), must give the same bits."""
import numpy as np
import pytest

from mpm_b200 import create_mpm_mls_gpu_solver
from mpm_b200.layout import ParticleArrays

pytestmark = pytest.mark.gpu

WATER = {"lambda": 160_000.0, "mu": 0.0, "model": "water", "density": 0.02}
OIL = {"lambda": 120_000.0, "mu": 0.0, "model": "oil", "density": 0.016}
SOLID = {"lambda": 50_000.0, "mu": 30_000.0, "model": "fixed-corotated"}


def _field(p, config):
    solver = create_mpm_mls_gpu_solver(p, config)
    try:
        first, second = solver.gather_surface_occupancy(), solver.gather_surface_occupancy()
    finally:
        solver.dispose()
    assert np.array_equal(first.view(np.uint32), second.view(np.uint32))  # the sums start from zero again
    return first


@pytest.mark.parametrize("n, materials, box", [
    (1, [WATER], (3, 3)),
    (513, [OIL], (20, 9)),             # a second CTA of one particle; no water
    (3000, [WATER, OIL, SOLID], (40, 30)),
    (512, [WATER], (64, 64)),          # the largest box of one phase
    (512, [WATER], (65, 64)),
    (512, [WATER, OIL], (64, 32)),     # and of two
    (512, [WATER, OIL], (64, 33)),
])
def test_both_routes_give_the_same_bits(n, materials, box):
    rng = np.random.default_rng(n + box[0] + box[1])
    cells = 300
    p = ParticleArrays.empty(n)
    cx, cy = rng.integers(0, box[0] - 2, n), rng.integers(0, box[1] - 2, n)
    cx[0] = cy[0] = 0
    cx[-1], cy[-1] = box[0] - 3, box[1] - 3
    p.px[:], p.py[:] = 30 + cx * 10 + rng.uniform(1, 9, n), 30 + cy * 10 + rng.uniform(1, 9, n)
    p.F[:] = np.array([1, 0, 0, 1]) + rng.uniform(-0.1, 0.1, (n, 4))
    p.volume[:] = rng.uniform(1, 40, n)
    p.materials = materials
    p.material[:] = rng.integers(0, len(materials), n)
    config = {"grid": {"cellsX": cells, "cellsY": cells, "cellSize": 10}, "particleMass": 0.5,
              "particleVolume": 25.0, "material": materials[0]}
    near = _field(p, config)
    assert np.count_nonzero(near) > 0
    # the same particles with others far off between them: no box is small
    far = ParticleArrays.empty(2 * n)
    even = p.take(np.repeat(np.arange(n), 2).tolist())
    for name in ("px", "py", "F", "volume", "material"):
        getattr(far, name)[:] = getattr(even, name)
    far.materials = materials
    far.px[1::2], far.py[1::2] = np.where(np.arange(n) % 2, 35.0, 2905.0), 2905.0
    far.volume[1::2] = 1.0
    wide = _field(far, config)
    region = np.s_[:box[1] + 10, :box[0] + 10]
    assert np.array_equal(near[region].view(np.uint32), wide[region].view(np.uint32))
