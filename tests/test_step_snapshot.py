"""A call's steps are enqueued before the previous call's status is known: when that call
overflowed and runs again, the next one has to run again from (and keep) the new state."""
import torch

from nonnewton_b200 import _abi, sph


class FakeEngine:
    """Steps add 1 to x and v while the lists are large enough, 100 when they overflow."""

    def __init__(self, pd, overflow_at):
        self.pd, self.overflow_at, self.calls, self.max_neighbors, self.status, self.seen = pd, overflow_at, 0, 64, 0, 20
        self.starts = []

    def step(self, nsteps, sync=True, host_loop=False):
        self.starts.append(float(self.pd.x[0, 0]))
        bad = self.calls == self.overflow_at and self.max_neighbors == 64
        self.status = _abi.NN_ERR_NEIGHBOR_OVERFLOW if bad else 0
        self.seen = 70 if bad else 20
        self.calls += 0 if bad else 1
        self.pd.x += 100.0 if bad else float(nsteps)
        self.pd.v += 100.0 if bad else float(nsteps)

    def status_async(self, out):
        out[0], out[1] = self.status, self.seen

    def status_wait(self):
        pass

    def stats(self, scene):
        return {"status": self.status, "max_neighbors_seen": self.seen}

    def set_neighbor_cap(self, n):
        self.max_neighbors = n


def test_call_after_an_overflow_starts_from_the_rerun_state(monkeypatch):
    class PD:
        x, v = torch.zeros(4, 3), torch.zeros(4, 3)

    class Meta:
        pd, num_elastic_bodies = PD, 0

    monkeypatch.setattr(sph, "meta", Meta)
    s = sph.SPHBase.__new__(sph.SPHBase)
    s.host_loop, s.grow_neighbors = False, True
    s._snap = s._spare = s._status = s._pending = None
    s._last_max = 20
    s.engine = eng = FakeEngine(PD, overflow_at=1)
    for _ in range(4):
        s._advance(1)
    # the second call overflowed (101): the third ran ahead from there, then the second again
    # from 1, and the third from its new end
    assert eng.starts == [0.0, 1.0, 101.0, 1.0, 2.0, 3.0]
    assert float(PD.x[0, 0]) == 4.0 and float(PD.v[3, 2]) == 4.0
    assert float(s._snap[0][0, 0]) == 3.0 and float(s._snap[1][0, 0]) == 3.0
    assert not s._settle()
