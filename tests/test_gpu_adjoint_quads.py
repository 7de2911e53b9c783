"""Pad tiles of the exact adjoint: the quad-wise gathers of the ring terms
against the FP64 transpose where they can go wrong -- both pads around one row
quad, a model one column wide, pads that end inside a quad, single tile columns
and rows, strips longer than a tile -- in every tile shape.  The tolerance is
the one of the operator's own test against the same transpose (2e-5: FP32
rounding over a few hundred steps, measured 4e-6 to 5e-6 on its grids)."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_l2
from seis_b200 import Shot
from seis_b200._lib import (IN_GATHER, IN_VEL, IN_WAVELET, LAUNCH_PER_TILE, LAUNCH_PERSISTENT,
                            OP_BORN_ADJOINT, OUT_IMAGE, TILE_SHAPES, Plan)

pytestmark = pytest.mark.gpu

CASES = [(30, 1, 6), (34, 2, 7), (1, 30, 5), (3, 40, 9), (45, 31, 13), (95, 63, 1), (70, 150, 30)]


@pytest.mark.parametrize("shape", sorted(TILE_SHAPES))
@pytest.mark.parametrize("nx,nz,pml", CASES)
def test_adjoint_quads_match_fp64(ctx, nx, nz, pml, shape):
    rng = np.random.default_rng(nx + 7 * nz)
    s = Shot(nx=nx, nz=nz, pml=pml, nt=80, ndel=6, sx=nx // 2, sz=nz // 3, dt=1e-3, dx=11.0,
             dz=9.0, gz=rng.integers(0, nz, nx))
    vel = (1800 + 1500 * rng.random((nx, nz))).astype(np.float32)
    wav = O.ricker(s.dt, 40.0, s.ndel, s.NT)
    rec = rng.standard_normal((nx, s.nt)).astype(np.float32)
    want = O.born_adjoint(s, wav.astype(np.float64), vel, rec, prec="f64")
    for form in (LAUNCH_PER_TILE, LAUNCH_PERSISTENT):
        with Plan(ctx, OP_BORN_ADJOINT, [s]) as p:
            p.set_tile_shape(shape)
            p.set_launch(form)
            p.set(0, IN_VEL, vel)
            p.set(0, IN_WAVELET, wav)
            p.set(0, IN_GATHER, rec)
            p.run()
            assert rel_l2(p.get(0, OUT_IMAGE), want) < 2e-5
