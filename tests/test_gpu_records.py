"""Particle records packed and unpacked on the device (mpm_read_particles,
mpm_write_particles): every word comes back as it was written, whole and by
index, at the sizes where the staging changes form -- one CTA of 128 records,
one pinned chunk of 1 MiB (12,483 records of 84 bytes: written straight to
pinned memory), several chunks, one device slab of 2^20 records and beyond."""
import numpy as np
import pytest

from mpm_b200 import create_mpm_mls_gpu_solver
from mpm_b200.errors import RangeError
from mpm_b200.layout import ParticleArrays

pytestmark = pytest.mark.gpu

MATERIALS = [{"lambda": 20.0, "mu": 10.0, "model": "neo-hookean"},
             {"lambda": 8.0, "mu": 0.0, "model": "water", "density": 1.0},
             {"lambda": 20.0, "mu": 10.0, "model": "powder", "frictionCoefficient": 0.55}]


def _solver(n):
    rng = np.random.default_rng(n)
    p = ParticleArrays.empty(n)
    p.px[:], p.py[:] = rng.uniform(4, 60, n), rng.uniform(4, 60, n)
    p.vx[:], p.vy[:] = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    p.C[:] = rng.uniform(-1, 1, (n, 4))
    p.F[:] += rng.uniform(-0.2, 0.2, (n, 4))
    p.plastic_volume[:] = rng.uniform(0.9, 1.1, n)
    p.volume[:] = rng.uniform(0.2, 0.3, n)
    p.materials, p.material[:] = MATERIALS, np.arange(n) % 3
    p.damage[p.material == 0] = 0.25
    config = {"grid": {"cellsX": 64, "cellsY": 64, "cellSize": 1.0}, "particleMass": 0.25, "particleVolume": 0.25,
              "material": MATERIALS[0]}
    return create_mpm_mls_gpu_solver(p, config)


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 12_483, 12_484, 60_001, (1 << 20) + 3])
def test_records_come_back_as_written(n):
    solver = _solver(n)
    try:
        first, ids = solver.read_particles_packed()
        assert np.array_equal(ids, np.zeros(n, np.uint32))
        rng = np.random.default_rng(1)
        records = first.copy()
        records[:, 0:13] += rng.uniform(0, 0.1, (n, 13)).astype(np.float32)
        records[0::3, 18] = 0.5  # damage
        solver.write_particles_packed(records)
        back, _ = solver.read_particles_packed()
        assert np.array_equal(_bits(back), _bits(records))
        # once the slots have been re-ordered, by index as in the whole
        solver.write_particles_packed(first)
        solver.step_batch(2, 1e-4, {"x": 0.0, "y": 0.0})
        whole, _ = solver.read_particles_packed()
        assert n < 100 or not np.array_equal(_bits(whole[:, 0:12]), _bits(first[:, 0:12]))
        some = rng.integers(0, n, min(n, 300))
        part, _ = solver.read_particles_packed(some)
        assert np.array_equal(_bits(part), _bits(whole[some]))
    finally:
        solver.dispose()


def test_refused_records_leave_the_state_and_new_materials_are_taken():
    solver = _solver(300)
    try:
        before, _ = solver.read_particles_packed()
        for word, value, message in ((13, 6, "particle 17 has an unsupported MPM material model 6"),
                                     (19, 4, "particle 17 has an invalid bonded triangle marker")):
            bad = before.copy()
            bad[:, 0] += 1.0
            bad.view(np.uint32)[17, word] = value
            with pytest.raises(RangeError, match=message):
                solver.write_particles_packed(bad)
            assert np.array_equal(_bits(solver.read_particles_packed()[0]), _bits(before))
        new = before.copy()
        new[5, 14] = 33.0  # a Neo-Hookean particle of another lambda
        new[7:40:3, 16] = 1.5  # water of another density
        solver.write_particles_packed(new)
        assert np.array_equal(_bits(solver.read_particles_packed()[0]), _bits(new))
    finally:
        solver.dispose()
