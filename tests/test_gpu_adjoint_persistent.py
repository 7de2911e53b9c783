"""The adjoint's persistent interior kernel with two and more tiles per CTA: a
CTA weighs its tile's velocity in place, so the stage that the next tensor copy
refills has been written by its threads, and every tile uses the same second
weighted field.  The per-tile form's bits, and the FP64 transpose within the
operator's own tolerance against it (2e-5)."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_l2
from seis_b200 import Shot
from seis_b200._lib import (IN_GATHER, IN_VEL, IN_WAVELET, LAUNCH_OVERLAP, LAUNCH_PER_TILE,
                            LAUNCH_PERSISTENT, OP_BORN_ADJOINT, OUT_IMAGE, SNAP_BF16, SNAP_F32,
                            TILE_32x64, TILE_64x32, Plan)

pytestmark = pytest.mark.gpu
N = 1200  # some 620 interior tiles of 2048 cells; 296 CTAs (2 per SM) are resident


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(11)
    s = Shot(nx=N, nz=N, pml=9, nt=10, ndel=2, sx=N // 2, sz=N // 2, dt=1e-3, dx=11.0, dz=9.0,
             gz=N // 2 + rng.integers(-3, 4, N))
    vel = (1800 + 1500 * rng.random((N, N))).astype(np.float32)
    wav = rng.standard_normal(s.NT).astype(np.float32)
    rec = rng.standard_normal((N, s.nt)).astype(np.float32)
    return s, vel, wav, rec, O.born_adjoint(s, wav.astype(np.float64), vel, rec, prec="f64")


def image(ctx, case, shape, form, dtype):
    s, vel, wav, rec, _ = case
    with Plan(ctx, OP_BORN_ADJOINT, [s]) as p:
        p.set_snapshots(1, dtype)
        p.set_tile_shape(shape)
        p.set_launch(form)
        p.set(0, IN_VEL, vel)
        p.set(0, IN_WAVELET, wav)
        p.set(0, IN_GATHER, rec)
        p.run()
        return p.get(0, OUT_IMAGE)


@pytest.mark.parametrize("dtype", [SNAP_F32, SNAP_BF16], ids=["f32", "bf16"])
@pytest.mark.parametrize("shape", [TILE_32x64, TILE_64x32], ids=["32x64", "64x32"])
def test_persistent_adjoint_matches_per_tile(ctx, case, shape, dtype):
    one = image(ctx, case, shape, LAUNCH_PER_TILE, dtype)
    if dtype == SNAP_F32:
        assert rel_l2(one, case[4]) < 2e-5
    for form in (LAUNCH_PERSISTENT, LAUNCH_PERSISTENT | LAUNCH_OVERLAP):
        assert np.array_equal(image(ctx, case, shape, form, dtype), one)
