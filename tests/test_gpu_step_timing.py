"""The step time of Plan.time_kernels is that of the steps of a run, in every
launch form."""
import time

import numpy as np
import pytest

import oracle as O
from seis_b200 import Shot
from seis_b200._lib import (IN_DV, IN_VEL, IN_WAVELET, LAUNCH_OVERLAP, LAUNCH_PERSISTENT, OP_BORN,
                            OP_MODELING, Plan)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [LAUNCH_OVERLAP, LAUNCH_OVERLAP | LAUNCH_PERSISTENT],
                         ids=["one_launch", "persistent"])
@pytest.mark.parametrize("op", [OP_MODELING, OP_BORN], ids=["modeling", "born"])
def test_step_time_is_that_of_a_run(ctx, op, flags):
    """Small shots, whose steps take microseconds: a wait between two timed steps
    would show.  A run of 4,000 steps (clearing and tables beside them: a
    hundredth) against 1,000 timed ones, the best of several each; 10% between
    them."""
    s = Shot(nx=201, nz=201, pml=40, nt=3900, ndel=100, sx=100, sz=2, dt=5e-4, dx=10.0, dz=10.0,
             gz=np.ones(201))
    with Plan(ctx, op, [s]) as p:
        p.set_launch(flags)
        p.set(0, IN_VEL, np.full((201, 201), 2000.0, np.float32))
        p.set(0, IN_WAVELET, O.ricker(s.dt, 20.0, s.ndel, s.NT))
        if op == OP_BORN:
            p.set(0, IN_DV, np.full((201, 201), 20.0, np.float32))
        p.run()
        p.sync()
        run = []
        for _ in range(3):
            t = time.perf_counter()
            p.run()
            p.sync()
            run.append((time.perf_counter() - t) / s.NT * 1e3)
        step = [p.time_kernels(1000)[0][2] for _ in range(3)]
        assert abs(min(step) / min(run) - 1.0) < 0.1
