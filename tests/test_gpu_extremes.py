"""Values at the ends of the range: the restatement's bits where a field
overflows."""
import numpy as np
import pytest

import oracle as O
from seis_b200 import Shot
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
