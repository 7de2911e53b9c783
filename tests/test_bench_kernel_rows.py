"""The benchmark's kernel rows describe the launches of the timed iteration:
the adjoint's plan is tuned with the solver's snapshots, rows are timed in the
solver's shapes and forms, and DRAM figures stay with the shape they were
captured at.  Host only: plans that record their calls."""
import importlib.util
import os

import numpy as np
import pytest

from seis_b200 import _lib as S

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class FakePlan:
    """Tuned once per operator, snapshot type and build; a forced tuning finds
    another choice."""
    cache, made = {}, []

    def __init__(self, ctx, op, shots):
        self.op, self.tile_shape, self.launch, self.dtype = op, S.TILE_32x64, S.LAUNCH_OVERLAP, None
        self.timed, self.exact = None, True
        FakePlan.made.append(self)

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        pass

    def set(self, *a):
        pass

    def set_exact(self, exact):
        self.exact = exact

    def set_snapshots(self, every, dtype):
        self.every, self.dtype = every, dtype

    def set_tile_shape(self, s):
        self.tile_shape = s

    def set_launch(self, f):
        self.launch = f

    def autotune(self, steps=10, force=False):
        key = self.op, self.dtype == S.SNAP_F16, self.exact
        if force:
            FakePlan.cache[key] = (S.TILE_16x128, S.LAUNCH_PER_TILE)
        elif key not in FakePlan.cache:
            FakePlan.cache[key] = (S.TILE_64x64, S.LAUNCH_OVERLAP)
        self.tile_shape, self.launch = FakePlan.cache[key]
        return self.tile_shape, [1.0] * len(S.TILE_SHAPES)

    def time_kernels(self, steps):
        self.timed = self.tile_shape, self.launch
        return [1.0, 2.0, 2.5], [1e6, 1e6]


class Survey:
    shots, vel0, dv = [0], None, None

    def wavelet(self):
        return np.zeros(1, np.float32)

    def sub(self, a, i):
        return None


@pytest.fixture
def rows(monkeypatch):
    spec = importlib.util.spec_from_file_location("bench_rows", os.path.join(ROOT, "bench.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    monkeypatch.setattr(S, "Plan", FakePlan)
    # the solver's own tuning, earlier in the process
    FakePlan.made = []
    FakePlan.cache = {(S.OP_BORN, False, False): (S.TILE_32x64, 3),
                      (S.OP_BORN_ADJOINT, True, False): (S.TILE_64x32, 2)}
    _, rows, tuning = b.kernel_roofline(None, Survey(), 10.0, {"born": 1, "adjoint": 1, "source": 1})
    return b, {r["kernel"]: r for r in rows}, tuning, {p.op: p for p in FakePlan.made}


def test_rows_are_timed_as_the_solver_runs(rows):
    b, r, tuning, plans = rows
    adj = plans[S.OP_BORN_ADJOINT]
    assert (adj.every, adj.dtype) == (b.SNAP_EVERY, S.SNAP_F16)
    assert plans[S.OP_BORN].timed == (S.TILE_32x64, 3)
    assert adj.timed == (S.TILE_64x32, 2)
    assert plans[S.OP_MODELING].timed == (S.TILE_64x32, 2)  # the adjoint's plan recomputes it
    assert tuning["born"]["chosen"] == "32x64" and tuning["adjoint"]["chosen"] == "64x32"
    assert [r[k]["shape"] for k in ("born_pad", "adjoint_step", "source_pad")] == \
        ["32x64", "64x32", "64x32"]


def test_traffic_only_at_the_captured_shape(rows):
    b, r, _, _ = rows
    for k, (shape, per_cell) in b.NCU_TRAFFIC_PER_CELL.items():
        assert r[k]["shape"] == shape and r[k]["traffic"] > 0
    b.NCU_TRAFFIC_PER_CELL["born_pad"] = ("32x32", 1.0)
    again = b.kernel_roofline(None, Survey(), 10.0, {"born": 1})[1]
    assert [x["traffic"] for x in again if x["kernel"] == "born_pad"] == [None]
