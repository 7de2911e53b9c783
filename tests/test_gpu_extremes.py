"""Values at the ends of the range: the restatement's bits where a field
overflows, and the adjoint beside cells of zero velocity."""
import numpy as np
import pytest

import oracle as O
from helpers import fd_args, rel_l2
from seis_b200 import Shot, fd
from seis_b200._lib import (IN_DV, IN_VEL, IN_WAVELET, OP_BORN, OP_MODELING, OUT_GATHER,
                            TILE_SHAPES, Plan)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", sorted(TILE_SHAPES))
@pytest.mark.parametrize("sx,sz", [(40, 40), (63, 31), (9, 70)])
def test_doubling_overflows_as_by_itself(ctx, sx, sz, shape):
    """A cell above half the largest number: 2 x overflows before the sum that
    it enters."""
    s = Shot(nx=80, nz=80, pml=8, nt=8, ndel=0, sx=sx, sz=sz, dt=1e-3, dx=11.0, dz=9.0,
             gz=np.full(80, sz))
    vel = np.full((80, 80), 2000.0, np.float32)  # (v dt)^2 = 4
    dv = np.full((80, 80), 40.0, np.float32)
    wav = np.zeros(s.NT, np.float32)
    wav[0] = 6.25e37
    for op in (OP_MODELING, OP_BORN):
        with Plan(ctx, op, [s]) as p:
            p.set_tile_shape(shape)
            p.set(0, IN_VEL, vel)
            p.set(0, IN_WAVELET, wav)
            if op == OP_BORN:
                p.set(0, IN_DV, dv)
            p.run()
            got = p.get(0, OUT_GATHER)
        want = O.modeling(s, wav, vel) if op == OP_MODELING else O.born(s, wav, vel, dv)
        assert not np.isfinite(want).all()
        assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("nx,nz", [(40, 33), (70, 66)])
def test_adjoint_without_pad_beside_zero_velocity(ctx, nx, nz):
    """No pad and cells of zero velocity, on the model's edge too: the image is
    undefined (0 / 0) at those cells alone.  Tolerance as in the operator's own
    test against the same transpose."""
    rng = np.random.default_rng(nx)
    s = Shot(nx=nx, nz=nz, pml=0, nt=40, ndel=4, sx=nx // 2, sz=nz // 3, dt=1e-3, dx=11.0, dz=9.0,
             gz=rng.integers(1, nz - 1, nx))
    vel = (1800 + 1500 * rng.random((nx, nz))).astype(np.float32)
    vel[0, 5] = vel[nx - 1, 9] = vel[7, 0] = vel[11, nz - 1] = vel[nx // 2, nz // 2] = 0.0
    wav = O.ricker(s.dt, 40.0, s.ndel, s.NT)
    rec = rng.standard_normal((nx, s.nt)).astype(np.float32)
    want = O.born_adjoint(s, wav.astype(np.float64), vel, rec, prec="f64")
    got = fd.born_adjoint(*fd_args(s), wav, vel, rec, ctx=ctx)
    zero = vel == 0
    assert np.array_equal(np.isnan(want), zero) and np.array_equal(np.isnan(got), zero)
    assert rel_l2(got[~zero], want[~zero]) < 2e-5
