"""When a layout of steps gets a captured step of its own, and which graph gives way."""
import random

import pytest

from railgun_b200.engine import runner
from railgun_b200.engine.runner import RepeatedLayouts


def run(layouts, keys):
    """The steps that were captured."""
    captured = []
    for i, key in enumerate(keys):
        if layouts.replay(key) is None and layouts.to_capture(key):
            layouts.keep(key, object())
            captured.append(i)
        assert len(layouts.graphs) <= layouts.kept and len(layouts.seen) <= layouts.counted + 1
    return captured


def short():
    return RepeatedLayouts(runner.SMALL_GRAPH_AT, runner.SMALL_GRAPHS_KEPT, runner.GIVES_WAY_AFTER[1], runner.LAYOUTS_COUNTED[1])


@pytest.mark.parametrize("n", [1, 9, 12, 16, 17, 24, 100, 1000])
def test_layouts_in_turn_are_captured_once(n):
    layouts = short()
    captured = run(layouts, [i % n for i in range(40 * n)])
    if n > runner.LAYOUTS_COUNTED[1]:                   # too many to count: launched one kernel at a time
        assert captured == []
    else:
        assert len(captured) == min(n, runner.SMALL_GRAPHS_KEPT) and captured[0] == (runner.SMALL_GRAPH_AT - 1) * n


@pytest.mark.parametrize("n", [20, 100, 2000])
def test_captures_of_layouts_in_any_order_are_bounded(n):
    rng = random.Random(n)
    steps = 20000
    captured = run(short(), [min(rng.randrange(n), rng.randrange(n)) for _ in range(steps)])
    assert len(captured) <= runner.SMALL_GRAPHS_KEPT * (1 + steps // runner.GIVES_WAY_AFTER[1])


def test_layouts_that_are_no_longer_used_give_way():
    layouts = short()
    run(layouts, list(range(16)) * 4)
    run(layouts, [100 + i % 4 for i in range(runner.GIVES_WAY_AFTER[1] + 4)])
    assert [k for k in layouts.graphs if k >= 100] == [100, 101, 102, 103]
    assert 0 not in layouts.seen and 4 in layouts.seen  # it counts anew: one step does not bring its graph back
    assert run(layouts, [0]) == [] and len(run(layouts, [0] * runner.GIVES_WAY_AFTER[1])) == 1


def test_the_graph_used_last_stays():
    layouts = RepeatedLayouts(2, 2, 0, 64)
    assert run(layouts, "aabba") == [1, 3]
    assert run(layouts, "cc") == [1] and list(layouts.graphs) == ["a", "c"]
    assert run(layouts, "bb") == [1] and list(layouts.graphs) == ["c", "b"]
