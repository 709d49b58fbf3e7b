"""bench.py's workloads beside the headline, on CPU with a fake engine: a serving
stream with a failed job is an error, and a leg that fails leaves the others and
the headline their figures."""
import os
import sys
from types import SimpleNamespace

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


class FakeEngine:
    bad, boom = (), ()

    def __init__(self, device):
        self.n = -1

    def __enter__(self):
        return self

    def __exit__(self, *a):
        pass

    def load(self, *a, **k):
        pass

    serve_start = serve_reset_stats = serve_stop = load

    def submit(self, *job):
        self.n += 1
        return self.n

    def wait(self, i, check=True):
        if i in self.boom:
            raise RuntimeError("gone")
        return {"state": 3 if i in self.bad else 2, "status": 7 if i in self.bad else 0}

    def release(self, i):
        pass

    def serve_stats(self):
        return {"completed": self.n - len(self.bad), "failed": len(self.bad)}


class FakeError(RuntimeError):
    def __init__(self, status):
        super().__init__(f"gi status {status}")
        self.status = status


def package(bad=(), boom=()):
    eng = type("E", (FakeEngine,), {"bad": bad, "boom": boom})
    return SimpleNamespace(Engine=eng, GI_JOB_DONE=2, GiError=FakeError, GI_ERR_CUDA=2,
                           GI_ERR_DEVICE=7)


ARGS = SimpleNamespace(slices=0, serve_slots=3, serve_budget_gb=1.0)


@pytest.mark.parametrize("bad,boom", [((3,), ()), ((), (4,)), ((1, 2), (5,))])
def test_failed_jobs_are_an_error(bad, boom):
    with pytest.raises(RuntimeError, match="serving jobs failed"):
        bench.serve_stream(package(bad, boom), None, [(1, 0, 1, 0)] * 8, [0.0] * 8, 0, 1, ARGS)


def test_a_stream_without_failures():
    st = bench.serve_stream(package(), None, [(1, 0, 1, 0)] * 8, [0.0] * 8, 0, 1, ARGS)
    assert st["failed"] == 0 and st["makespan_s"] > 0


def test_a_failed_leg_leaves_the_others():
    def fails(e):
        raise e
    leg = bench.Legs(package())
    assert leg("a", lambda x: {"value": x}, 3) == {"value": 3}
    assert "jobs failed" in leg("b", fails, RuntimeError("2 jobs failed"))["error"]
    assert leg("c", lambda: 4) == 4
    assert "gi status 1" in leg("d", fails, FakeError(1))["error"] and leg("e", lambda: 5) == 5
    # an error of the device: what follows would only fail too
    assert "gi status 2" in leg("f", fails, FakeError(2))["error"]
    assert leg("g", lambda: 6)["error"] == "not run: the device failed in f"
