"""Which shapes of steps with prompt portions get one of the places for graphs: the rule alone, without a GPU."""
from collections import OrderedDict
from types import SimpleNamespace

import pytest
import torch

import cbis_b200      # noqa: F401
from cbis_b200.engine import runner as runner_module
from cbis_b200.engine.runner import ModelRunner, StepEntry


@pytest.fixture
def runner(monkeypatch):
    """A runner whose launches take 0.66 ms of a clock of its own and whose captures are counted."""
    r = object.__new__(ModelRunner)
    clock = [0.0]

    def forward(ctx):
        clock[0] += 0.66e-3
        return torch.zeros(1)
    monkeypatch.setattr(runner_module.time, "perf_counter", lambda: clock[0])
    monkeypatch.setattr(runner_module, "capture_graph", lambda fn: (SimpleNamespace(replay=lambda: None), torch.zeros(1)))
    r.use_graphs, r.small_step_graphs, r._small_ok, r.shape_graphs, r._small_pending = True, False, False, True, None
    r.max_shape_graphs, r.shape_graph_after, r.shape_graph_min_host_s, r.shape_graph_capture_s = 24, 8, 1e-3, 60e-3
    r._shape_seen, r._shape_graphs, r._shape_steps = {}, OrderedDict(), 0
    r.shape_captures = r.shape_replays = r.graph_replays = 0
    r.model = SimpleNamespace(forward=forward)
    r.build_context = lambda *a, **k: None
    r._pack = lambda *a: None

    def come(n):
        before = r.shape_captures
        r.step([StepEntry(0, 0, list(range(n)), [0])])
        return r.shape_captures - before
    r.come = come
    return r


@pytest.mark.parametrize("after,min_host_s", [(8, 1e-3), (8, 0.0)])
def test_more_shapes_than_places_in_rotation_do_not_capture_over_and_over(runner, after, min_host_s):
    """30 shapes for 24 places, 300 times round: cheap ones (the first rule) and, with no bound on the cost, dear ones."""
    runner.shape_graph_after, runner.shape_graph_min_host_s = after, min_host_s
    captures = {n: 0 for n in range(2, 32)}
    for _ in range(300):
        for n in captures:
            captures[n] += runner.come(n)
    assert len(runner._shape_graphs) == 24 and max(captures.values()) <= 2 and sum(captures.values()) <= 30
    assert runner.shape_replays >= 24 * 200


def test_traffic_that_moves_on_gets_the_places(runner):
    """After long use of 24 shapes another 24 come, and only those: all of them get a place, once each."""
    for _ in range(500):
        for n in range(2, 26):
            runner.come(n)
    moved = {n: 0 for n in range(100, 124)}
    for _ in range(200):
        for n in moved:
            moved[n] += runner.come(n)
    assert set(moved.values()) == {1}


def test_a_shape_that_comes_often_replaces_one_that_hardly_comes_and_that_one_is_counted_anew(runner):
    rare = list(range(2, 26))
    for _ in range(100):
        for n in rare:
            runner.come(n)
    for i in range(6000):      # the rare ones still come, each every 1,200th step
        if i % 50 == 0:
            runner.come(rare[i // 50 % 24])
        runner.come(1000)
    assert (runner.shape_captures, len(runner._shape_graphs)) == (25, 24)
    given_up = [n for n in rare if ((n, 1),) not in runner._shape_graphs]
    assert len(given_up) == 1
    assert runner.come(given_up[0]) == 0 and runner._shape_seen[((given_up[0], 1),)][0] <= 6000 // 1200 + 1
