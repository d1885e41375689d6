"""The fixed-point transfer's routes against the CPU emulation of the same
integers, word for word: 512 consecutive particles are summed in shared memory
where their stencils' box has at most 8,192 words (four per node and channel)
and added one by one where it has more, and the quotients by the particle mass
and volume take another route for a divisor whose significand is all ones."""
import numpy as np
import pytest

from mpm_b200 import create_experimental_mpm_mls_atomic_gpu_solver
from mpm_b200.layout import ParticleArrays
from oracle import emulate_fixed_point_scatter

pytestmark = pytest.mark.gpu

MATERIALS = [{"lambda": 160_000.0, "mu": 0.0, "model": "water", "density": 0.02},
             {"lambda": 120_000.0, "mu": 0.0, "model": "oil", "density": 0.016},
             {"lambda": 50_000.0, "mu": 30_000.0, "model": "fixed-corotated"}]
ALL_ONES = float(np.nextafter(np.float32(1), np.float32(0)))


def _positions(kind, n, cells, rng):
    if kind == "block":  # rows of particles, two per cell
        r, c = np.divmod(np.arange(n), 60)
        return 20 + (c + 0.5 + rng.uniform(-0.3, 0.3, n)) * 5, 20 + (r + 0.5 + rng.uniform(-0.3, 0.3, n)) * 5
    if kind == "scattered":
        return rng.uniform(20, cells * 10 - 20, n), rng.uniform(20, cells * 10 - 20, n)
    # one CTA's particles with stencils in a box of `kind` by 32 nodes
    cx, cy = rng.integers(0, kind - 2, n), rng.integers(0, 30, n)
    cx[:2], cy[:2] = (0, kind - 3), (0, 29)
    return 30 + cx * 10 + rng.uniform(1, 9, n), 30 + cy * 10 + rng.uniform(1, 9, n)


@pytest.mark.parametrize("n, cells, kind, materials, mass, volume, steps", [
    (1, 20, "block", 1, 0.5, 25.0, 0),
    (1500, 45, "block", 3, 0.5, 25.0, 5),       # all three channels in a CTA
    (513, 45, "block", 2, 0.7, 23.3, 5),        # a second CTA of one particle
    (1500, 45, "block", 3, ALL_ONES, 25.0, 5),
    (1500, 45, "block", 2, 0.7, 25 * ALL_ONES, 0),
    (2000, 200, "scattered", 3, 0.3, 25.0, 5),  # boxes far too large
    (512, 80, 64, 1, 0.5, 25.0, 0),             # 64 x 32 nodes: the largest box
    (512, 80, 65, 1, 0.5, 25.0, 0),
])
def test_words_match_the_cpu_emulation(n, cells, kind, materials, mass, volume, steps):
    rng = np.random.default_rng(n + cells)
    p = ParticleArrays.empty(n)
    p.px[:], p.py[:] = _positions(kind, n, cells, rng)
    p.vx[:], p.vy[:] = rng.uniform(-3, 3, n), rng.uniform(-3, 3, n)
    p.C[:] = rng.uniform(-0.05, 0.05, (n, 4))
    p.volume[:] = 25.0
    p.materials = MATERIALS[:materials]
    p.material[:] = rng.integers(0, materials, n)
    config = {"grid": {"cellsX": cells, "cellsY": cells, "cellSize": 10}, "particleMass": mass,
              "particleVolume": volume, "material": MATERIALS[0]}
    solver = create_experimental_mpm_mls_atomic_gpu_solver(p, config, fixed_point_shift=18)
    try:
        if steps:  # the words start from zero again after each substep
            solver.step_batch(steps, 1e-4, {"x": 3.0, "y": 90.0})
            assert solver.read_status_words()[0] == 0
        packed = solver.read_particles_packed()[0]
        words, affine = solver.probe_fixed_point(1e-4)
        again, _ = solver.probe_fixed_point(1e-4)
    finally:
        solver.dispose()
    expected, flags = emulate_fixed_point_scatter(packed, affine, 10.0, mass, volume, cells, cells, 18)
    assert flags == 0
    assert np.count_nonzero(words) > 0
    assert np.array_equal(words, expected)
    assert np.array_equal(again, expected)
