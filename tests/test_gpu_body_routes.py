"""Bonded-triangle bodies by number: a CTA of the field stages 128 at a time and
keeps those within the band of its tile, and pair contacts are cached up to
2,048 bodies and found again in each pass above.  Against the oracle: the
field as for the interactive scene's pebbles (the body exactly, ties included; the
float64 samples to 1e-6 in float32), and two substeps with the reference's
own bounds (position 0.02, velocity 0.025 + 5e-4 |v|)."""
import numpy as np
import pytest

from helpers import oracle_columns, packed_columns
from mpm_b200 import create_mpm_mls_gpu_solver
from mpm_b200.scenes import GATE4_FIXED_STEP_SECONDS, create_mpm_gate4_scene, create_mpm_gate4_step_config
from oracle import OracleState

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies", [1, 128, 129, 300, 2049])
def test_many_bodies_match_the_oracle(bodies):
    p, _, _ = create_mpm_gate4_scene()
    vertices = np.flatnonzero(p.bonded_vertex >= 0)[:3]
    assert list(p.bonded_vertex[vertices]) == [0, 1, 2]
    rng = np.random.default_rng(bodies)
    config = create_mpm_gate4_step_config()
    dx = config["grid"]["cellSize"]
    side = np.ptp(p.px[vertices])
    per_row = max(1, int(np.sqrt(bodies)))
    q = p.take(np.tile(vertices, bodies))
    row, column = np.divmod(np.arange(bodies), per_row)
    # some touch, some lie apart; the first rows straddle tiles of 16 x 8 nodes
    ox = 3 * dx + column * 1.4 * side + rng.uniform(0, 0.3 * side, bodies)
    oy = 3 * dx + row * 1.4 * side + rng.uniform(0, 0.3 * side, bodies)
    q.px[:] = (q.px - np.tile([p.px[vertices].min()] * 3, bodies) + np.repeat(ox, 3)).astype(np.float32)
    q.py[:] = (q.py - np.tile([p.py[vertices].min()] * 3, bodies) + np.repeat(oy, 3)).astype(np.float32)
    q.vx[:] = np.repeat(rng.uniform(-1, 1, bodies), 3).astype(np.float32)
    q.vy[:] = np.repeat(rng.uniform(-1, 1, bodies), 3).astype(np.float32)
    q.object_id[:] = np.repeat(np.arange(bodies) + 1, 3)
    cells = int(max(q.px.max(), q.py.max()) / dx) + 8
    config = dict(config, grid=dict(config["grid"], cellsX=cells, cellsY=cells + 5))
    dt = GATE4_FIXED_STEP_SECONDS / 16
    solver = create_mpm_mls_gpu_solver(q, config)
    try:
        field = solver.probe_triangle_field(dt)
        solver.step_batch(2, dt, config["gravity"])
        packed, _ = solver.read_particles_packed()
        assert solver.read_status_words()[0] == 0
    finally:
        solver.dispose()
    ref = OracleState(q, config).triangle_field(config)
    near = ref["body"] >= 0
    assert near.sum() > 0
    assert np.array_equal(field["body"], ref["body"])
    assert np.max(np.abs(field["sd"] - ref["sd"]) / (1 + np.abs(ref["sd"]))) <= 1e-6
    assert np.max(np.abs(field["normal"][near] - ref["normal"][near])) <= 1e-6
    assert np.max(np.abs(field["bary"][near] - ref["bary"][near])) <= 1e-6
    cfg = dict(config, dt=float(np.float32(dt)))
    state = OracleState(q, cfg)
    state.run(cfg, 2)
    gpu, want = packed_columns(packed), oracle_columns(state)
    assert np.max(np.abs(gpu["position"] - want["position"])) <= 0.02
    assert np.max(np.abs(gpu["velocity"] - want["velocity"]) - (0.025 + 5e-4 * np.abs(want["velocity"]))) <= 0.0
