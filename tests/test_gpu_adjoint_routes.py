"""The differentiable engine's routes: scenes of one material only (the grid
kernels leave the other's nodes alone), horizons that are no multiple of the
checkpoint interval, and one engine used again with other velocities and
intervals (the last segment's tape, the sums that every substep leaves at
zero).  Blocks that never meet have the gradients of engines of their own, and a
reused engine those of a fresh one, up to the rounding of the scattered sums:
1e-3 of the gradient, as for the checkpoint interval."""
import numpy as np
import pytest

from mpm_b200.adjoint import create_mpm_adjoint_engine, fixed_cfl_dt
from mpm_b200.scenes import ADJOINT_GRAVITY, create_adjoint_scenes

pytestmark = pytest.mark.gpu


def _gradients(engine, steps, every, dt, targets, velocities=None):
    if velocities is not None:
        engine.set_velocities(velocities)
    loss = engine.forward(steps, [dt], targets, checkpoint_every=every)
    gv, gp = engine.backward()
    return loss, gv, gp


def _near(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b)


@pytest.mark.parametrize("steps, every", [(1, 4), (7, 3), (8, 4), (9, 9)])
def test_one_material_and_a_reused_engine(steps, every):
    (p, c, t), = create_adjoint_scenes(1, seed=5, water_columns=24, water_rows=33, solid_side=17, cells=64)
    dt = float(np.float32(fixed_cfl_dt(p, c, 90.0, 0.05)))
    water = np.flatnonzero(p.material == 0)
    solid = np.flatnonzero(p.material == 1)
    both = create_mpm_adjoint_engine([(p, c)], ADJOINT_GRAVITY)
    try:
        loss, gv, gp = _gradients(both, steps, every, dt, t)
        total = 0.0
        for rows, parameters in ((water, slice(0, 1)), (solid, slice(1, 3))):
            alone = create_mpm_adjoint_engine([(p.take(rows), c)], ADJOINT_GRAVITY)
            try:
                part, part_gv, part_gp = _gradients(alone, steps, every, dt, t[rows])
            finally:
                alone.dispose()
            total += part[0]
            assert _near(gv[rows], part_gv)
            assert _near(gp[0, parameters], part_gp[0, parameters])
        assert abs(loss[0] - total) <= 1e-4 * total
        # the engine again: other velocities and interval, then the first ones
        v = np.stack([p.vx, p.vy], axis=1).astype(np.float32)
        _gradients(both, steps + 2, 2, dt, t, 0.5 * v)
        again = _gradients(both, steps, every, dt, t, v)
        assert abs(again[0][0] - loss[0]) <= 1e-4 * loss[0]
        assert _near(again[1], gv) and _near(again[2], gp)
    finally:
        both.dispose()


@pytest.mark.parametrize("every", [1, 3, 8])
def test_a_batch_above_two_ctas_per_sm_has_the_gradients_of_its_scenes(every):
    """Turning from a substep to the one before takes another instance of the
    kernel where 148 SMs hold more than two CTAs of 256 particles each; every 1
    turns nowhere."""
    scenes = create_adjoint_scenes(8, seed=5, water_columns=96, water_rows=98, solid_side=20, cells=128)
    assert sum(len(p) for p, _, _ in scenes) > 2 * 148 * 256
    dts = [float(np.float32(fixed_cfl_dt(p, c, 90.0, 0.05))) for p, c, _ in scenes]
    batch = create_mpm_adjoint_engine([(p, c) for p, c, _ in scenes], ADJOINT_GRAVITY)
    try:
        losses = batch.forward(8, dts, np.concatenate([t for _, _, t in scenes]), checkpoint_every=every)
        gv, gp = batch.backward()
    finally:
        batch.dispose()
    first = 0
    for k, (p, c, t) in enumerate(scenes):
        if k in (0, 7):
            alone = create_mpm_adjoint_engine([(p, c)], ADJOINT_GRAVITY)
            try:
                loss, own_gv, own_gp = _gradients(alone, 8, every, dts[k], t)
            finally:
                alone.dispose()
            assert abs(losses[k] - loss[0]) <= 1e-4 * loss[0]
            assert _near(gv[first:first + len(p)], own_gv) and _near(gp[k], own_gp[0])
        first += len(p)
