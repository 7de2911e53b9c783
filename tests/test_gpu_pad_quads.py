"""Pad tiles: the quad-wise absorbing update, its coefficient tables and its
branch-free quotients against the restatement, bit for bit, where they can go
wrong -- both pads in one row quad, pads that end inside a quad, no pad at all,
single tile columns, amplitudes down to denormals, coefficients outside the
quotient's range -- in every tile shape."""
import numpy as np
import pytest

import oracle as O
from seis_b200 import Shot
from seis_b200._lib import (IN_DV, IN_VEL, IN_WAVELET, LAUNCH_OVERLAP, LAUNCH_PER_TILE,
                            LAUNCH_PERSISTENT, OP_BORN, OP_MODELING,
                            OUT_GATHER, TILE_SHAPES, Plan)

pytestmark = pytest.mark.gpu

# nx, nz, pml, dt, amplitude of the wavelet
CASES = [
    (30, 1, 6, 1e-3, 1.0),     # top and bottom pad meet in one quad
    (34, 2, 7, 1e-3, 1.0),
    (1, 1, 5, 1e-3, 1.0),
    (3, 40, 9, 1e-3, 1.0),
    (40, 33, 0, 1e-3, 1.0),    # no pad
    (45, 31, 13, 1e-3, 1.0),   # the pad ends inside a quad
    (95, 63, 1, 1e-3, 1.0),    # one column and one row in the last tiles
    (70, 70, 30, 1e-3, 1.0),
    (48, 40, 12, 1e-3, 1e-30), # quotients below the fused correction's range
    (48, 40, 12, 1e-3, 1e-38), # denormals
    (48, 40, 12, 1e-9, 1e25), # 1 / (a1 + a2) out of the table's range
    (48, 40, 12, 1e-3, 1e30),
]


@pytest.mark.parametrize("shape", sorted(TILE_SHAPES))
@pytest.mark.parametrize("nx,nz,pml,dt,amp", CASES)
def test_pad_quads_match_restatement(ctx, nx, nz, pml, dt, amp, shape):
    rng = np.random.default_rng(nx + 7 * nz)
    nt, ndel = 60, 4
    lo = 1 if pml == 0 else 0
    s = Shot(nx=nx, nz=nz, pml=pml, nt=nt, ndel=ndel, sx=max(lo, nx // 2), sz=max(lo, nz // 3),
             dt=dt, dx=11.0, dz=9.0, gz=rng.integers(lo, max(nz - lo, lo + 1), nx))
    vel = (1500 + 2500 * rng.random((nx, nz))).astype(np.float32)
    dv = (40 * rng.standard_normal((nx, nz))).astype(np.float32)
    wav = (amp * rng.standard_normal(s.NT)).astype(np.float32)
    # without a pad the reference overwrites a scattering source on the frame
    # and the library adds it: Born is compared with a pad only
    for op in (OP_MODELING, OP_BORN) if pml > 0 else (OP_MODELING,):
        with Plan(ctx, op, [s]) as p:
            p.set_tile_shape(shape)
            p.set_launch(LAUNCH_PER_TILE)
            p.set(0, IN_VEL, vel)
            p.set(0, IN_WAVELET, wav)
            if op == OP_BORN:
                p.set(0, IN_DV, dv)
            p.run()
            got = p.get(0, OUT_GATHER)
        want = O.modeling(s, wav, vel) if op == OP_MODELING else O.born(s, wav, vel, dv)
        assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("amp", [1e-33, 1e-36, 1e-39, 1e-42])
def test_quotients_around_the_smallest_normal(ctx, amp):
    """Pad cells whose one-way quotients cross the smallest normal number: the
    scaled division and its second rounding, in the same bits."""
    rng = np.random.default_rng(5)
    s = Shot(nx=41, nz=37, pml=17, nt=90, ndel=4, sx=20, sz=3, dt=1e-3, dx=11.0, dz=9.0,
             gz=rng.integers(0, 37, 41))
    vel = (1500 + 2500 * rng.random((41, 37))).astype(np.float32)
    dv = (40 * rng.standard_normal((41, 37))).astype(np.float32)
    wav = (amp * rng.standard_normal(s.NT)).astype(np.float32)
    for op in (OP_MODELING, OP_BORN):
        with Plan(ctx, op, [s]) as p:
            p.set(0, IN_VEL, vel)
            p.set(0, IN_WAVELET, wav)
            if op == OP_BORN:
                p.set(0, IN_DV, dv)
            p.run()
            got = p.get(0, OUT_GATHER)
        want = O.modeling(s, wav, vel) if op == OP_MODELING else O.born(s, wav, vel, dv)
        assert np.array_equal(got, want)


@pytest.mark.parametrize("shape", [k for k, v in sorted(TILE_SHAPES.items()) if v[0] * v[1] == 2048])
def test_born_persistent_beside_pad_tiles(ctx, shape):
    """Born's persistent interior kernel at one CTA per SM, with more interior
    tiles than CTAs, beside the pad tiles: the restatement's bits."""
    rng = np.random.default_rng(shape)
    n = 800
    s = Shot(nx=n, nz=n, pml=9, nt=10, ndel=2, sx=n // 2, sz=n // 2, dt=1e-3, dx=11.0, dz=9.0,
             gz=n // 2 + rng.integers(-3, 4, n))
    vel = (1500 + 2500 * rng.random((n, n))).astype(np.float32)
    dv = (40 * rng.standard_normal((n, n))).astype(np.float32)
    wav = rng.standard_normal(s.NT).astype(np.float32)
    with Plan(ctx, OP_BORN, [s]) as p:
        p.set_tile_shape(shape)
        p.set_launch(LAUNCH_OVERLAP | LAUNCH_PERSISTENT)
        p.set(0, IN_VEL, vel)
        p.set(0, IN_WAVELET, wav)
        p.set(0, IN_DV, dv)
        p.run()
        got = p.get(0, OUT_GATHER)
    assert np.array_equal(got, O.born(s, wav, vel, dv))
