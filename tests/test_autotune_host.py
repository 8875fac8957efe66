"""The autotuner's search and the serving loop's shapes on the CPU, with a stand-in
batch whose step time is a given function of the shapes it was set to: nothing is
pinned that the caller did not ask for, the library's own choice (0, 0) is timed
first and kept where nothing beats it, and the search reaches every shape that the
library itself may take (marches of 4 to 32 cells, 1 to 16 cells a thread)."""
import pytest

from gpluto_dev_b200 import api, autotune, serve
from gpluto_dev_b200.batch import TileShape
from test_serve_host import FakeBatch, FakeClock, job


class TimedBatch:
    """Each trial's time: cost(shapes by slot)."""

    def __init__(self, cost):
        self.cost, self.shapes, self.now, self.trials = cost, {}, 0.0, []

    def set_shape(self, slot, shape):
        self.shapes[slot] = (shape.seg, shape.cells_per_thread)

    def set_ctas(self, ctas):
        pass

    def advance(self, steps):
        self.trials.append(dict(self.shapes))
        self.now += steps * self.cost(self.shapes)

    def wait(self):
        pass


def tuned(monkeypatch, cost, table=None):
    b = TimedBatch(cost)
    monkeypatch.setattr(autotune.time, "perf_counter", lambda: b.now)
    info = {0: (2, 4096), 1: (2, 1 << 18), 2: (3, 1 << 14)}
    t = autotune.tune(b, info, table=table)
    return b, [tuple(t["shapes"][autotune.bin_of(t, *info[s])]) for s in info]


def test_library_choice_is_the_start_and_stays(monkeypatch):
    b, shapes = tuned(monkeypatch, lambda sh: 1.0 + sum(v != (0, 0) for v in sh.values()))
    assert b.trials[0] == {0: (0, 0), 1: (0, 0), 2: (0, 0)}
    assert shapes == [(0, 0)] * 3


@pytest.mark.parametrize("best", [(4, 16), (8, 4), (32, 16), (4, 1), (64, 8)])
def test_search_reaches_the_shapes_of_the_library(monkeypatch, best):
    miss = lambda v: (v[0] != best[0]) + (v[1] != best[1])
    _, shapes = tuned(monkeypatch, lambda sh: 1.0 + sum(map(miss, sh.values())))
    assert shapes == [best] * 3


def test_search_can_give_a_shape_back_to_the_library(monkeypatch):
    table = autotune.default_table()
    table["shapes"] = [[32, 2] for _ in table["shapes"]]
    _, shapes = tuned(monkeypatch, lambda sh: 1.0 + sum(v != (0, 0) for v in sh.values())
                      + 0.1 * sum(v[0] + v[1] for v in sh.values()), table)
    assert shapes == [(0, 0)] * 3


@pytest.mark.parametrize("table", [None, "given"])
def test_server_passes_shapes_only_from_a_table(table):
    if table:
        table = autotune.default_table()
        table["shapes"] = [[16, 4] for _ in table["shapes"]]
    seen = []

    class Batch(FakeBatch):
        def add(self, st, scheme, dt0, nsteps, shape=None):
            seen.append(shape)
            return super().add(st, scheme, dt0, nsteps, shape)

    clk = FakeClock()
    srv = serve.Server(pool_bytes=10 ** 9, max_slots=4, batch=Batch(4), table=table,
                       slot_bytes=lambda st, sch: st.ncells * 100, clock=clk)
    srv.serve([job(0, 0.0, 4096, 3), job(1, 0.0, 1 << 18, 3, ndim=3)], sleep=clk.sleep)
    assert seen == [TileShape(16, 4) if table else TileShape(0, 0)] * 2
