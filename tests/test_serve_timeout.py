"""A design update that gave up on the device (-1 steps and a NaN change in its record) is reported with its step and
never committed; it is not redone in FP64, which helps uncertified solves only."""
import types

import numpy as np
import pytest

torch = pytest.importorskip("torch")


class _Event:
    def query(self):
        return True

    def elapsed_time(self, other):
        return 1.0


def _server(pkg, monkeypatch, gave_up, precision):
    """A server whose workers hold host records and whose solves certify."""
    sv = pkg.serve
    committed = []

    class Worker:
        def __init__(self, n, prec):
            self.n, self.precision, self.job, self.last_used, self.bytes = n, prec, None, 0.0, 1
            self.op, self.stream = types.SimpleNamespace(_ctx=None), types.SimpleNamespace(cuda_stream=0)
            self.Ch, self.sh = torch.zeros((6, 6), dtype=torch.float64), torch.zeros(4, dtype=torch.float64)

    class Lineage:
        step, bytes, pending_advance = 0, 1, False

    class Server(sv.Server):
        def _new_worker(self, n, prec):
            return Worker(n, prec)

        def _launch(self, w, job):
            w.job, job.admitted, job.start, job.end = job, 0.0, _Event(), _Event()
            job.lineage = job.lineage or Lineage()
            if job.lineage.pending_advance:
                committed.append(job.step - 1)
                job.lineage.pending_advance = False
            w.sh[1:3] = torch.tensor([-1.0, float("nan")] if job.step in gave_up else [40.0, 0.1])

        def _drain(self):
            pass

    monkeypatch.setattr(pkg._lib, "lib", lambda: types.SimpleNamespace(pgj_solve_wait=lambda *a: 0))
    monkeypatch.setattr(sv, "worker_bytes", lambda n, prec: 1)
    return Server(precision=precision), committed


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_design_update_that_gave_up_is_reported_and_not_committed(pkg, monkeypatch, precision):
    sv = pkg.serve
    server, committed = _server(pkg, monkeypatch, gave_up={1}, precision=precision)
    out = server.run([sv.Arrival(0.0, sv.Lineage(n=16, seed=0, steps=4))], realtime=False)
    assert [r.status for r in out] == [0, pkg._lib.PGJ_ERR_TIMEOUT, 0, 0]
    assert [r.oc_steps for r in out] == [40, -1, 40, 40] and np.isnan(out[1].change)
    assert committed == [0, 2] and server.fallbacks == 0
