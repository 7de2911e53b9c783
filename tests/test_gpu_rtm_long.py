"""Reference RTM of columns as long as a CTA's shared memory holds: with the
filter's zeros around them (28,990 rows), without (up to 29,056), against the
restatement, bit for bit; one row more is refused."""
import numpy as np
import pytest

import oracle as O
from helpers import fd_args
from seis_b200 import SeisError, Shot, fd

pytestmark = pytest.mark.gpu


def case(NZ):
    rng = np.random.default_rng(NZ)
    nx, pml = 9, 4
    nz = NZ - 2 * pml
    s = Shot(nx=nx, nz=nz, pml=pml, nt=6, ndel=2, sx=4, sz=nz - 3, dt=1e-3, dx=11.0, dz=9.0,
             gz=rng.integers(nz - 20, nz - 1, nx))
    vel = (1500 + 1500 * rng.random((nx, nz))).astype(np.float32)
    wav = rng.standard_normal(s.NT).astype(np.float32)
    rec = rng.standard_normal((nx, s.nt)).astype(np.float32)
    return s, wav, vel, rec


@pytest.mark.parametrize("true", [False, True], ids=["adjoint", "rtm_true"])
@pytest.mark.parametrize("NZ", [28990, 28991, 29024, 29056])
def test_long_columns_match_restatement(ctx, NZ, true):
    s, wav, vel, rec = case(NZ)
    run, ref = (fd.rtm_true, O.rtm_true) if true else (fd.adjoint, O.rtm)
    want = ref(s, wav, vel, rec)
    assert np.abs(want).max() > 0
    assert np.array_equal(run(*fd_args(s), wav, vel, rec, ctx=ctx), want)


def test_longer_columns_are_refused(ctx):
    s, wav, vel, rec = case(29057)
    with pytest.raises(SeisError):
        fd.adjoint(*fd_args(s), wav, vel, rec, ctx=ctx)
    s, wav, vel, rec = case(40)  # the next call is served
    assert np.array_equal(fd.adjoint(*fd_args(s), wav, vel, rec, ctx=ctx), O.rtm(s, wav, vel, rec))
