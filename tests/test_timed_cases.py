"""The timed cases call the device copies with raw addresses, whose extents nothing can check at
run time: the array that a copy reads or writes has extent dim + 2 (pad + ghost), and the grid
(dim + 2 ghost) / brick dims."""
import importlib.util
import math
import os
import types

from bricklib_gb300 import bricks as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def cases():
    spec = importlib.util.spec_from_file_location("timed_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_move_copies_stay_inside_their_arrays(monkeypatch):
    calls = []

    def copy(dims, pad, ghost, arr, grid, brick, stream=None):
        calls.append((arr, [d + 2 * (p + g) for d, p, g in zip(dims, pad, ghost)],
                      math.prod((d + 2 * g) // 8 for d, g in zip(dims, ghost))))

    monkeypatch.setattr(B, "copyToBrickDevice", copy)
    monkeypatch.setattr(B, "copyFromBrickDevice", copy)
    monkeypatch.setattr(B, "ghostFill", lambda *a: None)
    n, ghost = (16, 24, 40), (8, 8, 8)
    full = [a + 2 * g for a, g in zip(n, ghost)]
    array = lambda name: types.SimpleNamespace(data_ptr=lambda: name)  # noqa: E731
    cases().run_move({"n": n, "ghost": ghost, "arr": array("arr"), "back": array("back"), "a": None, "ta": None,
                      "plan": None, "grid_dev": types.SimpleNamespace(ptr=0)})
    bricks = math.prod(x // 8 for x in full)
    assert calls == [("arr", full[::-1], bricks), ("back", full[::-1], bricks)]
