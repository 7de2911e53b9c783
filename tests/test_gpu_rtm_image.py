"""Imaging kernel of the reference RTM and the restoration of the boundary layers
fused into it, against the restatement, bit for bit, at the sizes where they
can go wrong: columns shorter than the filter, remainders of its groups of
outputs, models whose layers meet (restored by their own kernel) and the
smallest that do not, a source outside the model's columns or on its edge."""
import numpy as np
import pytest

import oracle as O
from helpers import fd_args
from seis_b200 import Shot, fd

pytestmark = pytest.mark.gpu

# nx, nz, pml, sx
CASES = [(8, 8, 3, 4), (9, 10, 5, 0), (12, 13, 9, 11), (20, 7, 6, 10), (7, 20, 6, 3), (33, 62, 1, 5),
         (16, 30, 8, -3), (24, 11, 12, 26), (40, 129, 4, 39)]


@pytest.mark.parametrize("true", [False, True], ids=["adjoint", "rtm_true"])
@pytest.mark.parametrize("nx,nz,pml,sx", CASES)
def test_image_sizes_match_restatement(ctx, nx, nz, pml, sx, true):
    rng = np.random.default_rng(nx + 13 * nz)
    s = Shot(nx=nx, nz=nz, pml=pml, nt=50, ndel=7, sx=sx, sz=min(2, nz - 1), dt=1e-3, dx=11.0,
             dz=9.0, gz=rng.integers(0, nz - 1, nx))
    vel = (1500 + 1500 * rng.random((nx, nz))).astype(np.float32)
    wav = O.ricker(s.dt, 30.0, s.ndel, s.NT)
    rec = rng.standard_normal((nx, s.nt)).astype(np.float32)
    run, ref = (fd.rtm_true, O.rtm_true) if true else (fd.adjoint, O.rtm)
    assert np.array_equal(run(*fd_args(s), wav, vel, rec, ctx=ctx), ref(s, wav, vel, rec))
