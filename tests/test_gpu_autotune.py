"""What the autotuner times: every distinct form of a step once, and nothing
that it may not choose unless its time is asked for."""
import ctypes

import numpy as np
import pytest

import oracle as O
from seis_b200 import Shot
from seis_b200._lib import (IN_VEL, IN_WAVELET, OP_BORN_ADJOINT, OP_MODELING, SNAP_F16, TILE_16x128, TILE_64x32,
                            TILE_SHAPES, Plan)

pytestmark = pytest.mark.gpu
STEPS = 7
# of one form without interior tiles: per timing the tables' launches, every
# step's pad launch alone and its one launch as run; a warm-up of 3 steps
ONE = {OP_MODELING: 2 + 2 * (3 + STEPS), OP_BORN_ADJOINT: 4 + 2 * (3 + STEPS)}


def plan(ctx, op, n=21):
    s = Shot(nx=n, nz=n, pml=6, nt=40, ndel=5, sx=n // 2, sz=2, dt=1e-3, dx=10.0, dz=10.0,
             gz=np.ones(n))
    p = Plan(ctx, op, [s])
    p.set(0, IN_VEL, np.full((n, n), 2000.0, np.float32))
    p.set(0, IN_WAVELET, O.ricker(s.dt, 30.0, s.ndel, s.NT))
    return p


def launches(ctx, p, ms):
    best, before = ctypes.c_int(), ctx.launches
    ctx.check(ctx.L.seis_fd_plan_autotune(p.h, STEPS, 1, ms, ctypes.byref(best)))
    return ctx.launches - before, best.value


@pytest.mark.parametrize("op", [OP_MODELING, OP_BORN_ADJOINT], ids=["modeling", "adjoint"])
def test_equal_forms_are_timed_once(ctx, op):
    with plan(ctx, op) as p:  # no interior tiles: one form per shape
        n, best = launches(ctx, p, (ctypes.c_double * len(TILE_SHAPES))())
        assert n == len(TILE_SHAPES) * ONE[op] and p.tile_shape == best


def test_fp16_adjoint_times_its_own_shape(ctx):
    with plan(ctx, OP_BORN_ADJOINT) as p:
        p.set_snapshots(2, SNAP_F16)
        n, best = launches(ctx, p, None)
        assert n == ONE[OP_BORN_ADJOINT] and best == p.tile_shape == TILE_64x32
        ms = (ctypes.c_double * len(TILE_SHAPES))()
        n, best = launches(ctx, p, ms)  # times asked for
        assert n == len(TILE_SHAPES) * ONE[OP_BORN_ADJOINT] and all(t > 0 for t in ms)
        assert best == p.tile_shape == TILE_64x32


def test_fp16_after_tuning_takes_its_shape(ctx):
    """FP16 set after a tuning by time: the plan's shape is FP16's all the same
    (sizes of which not every one is fastest in 64x32); a shape set by hand stays."""
    for n in (21, 60, 130, 300):
        with plan(ctx, OP_BORN_ADJOINT, n) as p:
            p.autotune(steps=STEPS, force=True)
            p.set_snapshots(2, SNAP_F16)
            assert p.tile_shape == TILE_64x32
    with plan(ctx, OP_BORN_ADJOINT) as p:
        p.autotune(steps=STEPS, force=True)
        p.set_tile_shape(TILE_16x128)
        p.set_snapshots(2, SNAP_F16)
        assert p.tile_shape == TILE_16x128
