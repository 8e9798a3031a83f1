"""The order in which kernels with waits are captured (``types.Nodes``): waits
that others imply are left out, chains stay together, and a capture sets a
kernel's waits only where it does not simply follow the one before it."""

from types import SimpleNamespace

import numpy as np
import pytest

from pyfr_gb300.backend.base import B200Backend
from pyfr_gb300.backend.types import Kernel, Nodes


class CountingCapture:
    def __init__(self):
        self.current, self.calls, self.waits = [], 0, {}

    def graph_capture_last(self, stream, buf, size, n):
        for i, h in enumerate(self.current):
            buf[i] = h
        n._obj.value = len(self.current)

    def graph_capture_after(self, stream, handles, n):
        self.current = [handles[i] for i in range(n)]
        self.calls += 1

    def kernel(self, handle):
        self.waits[handle] = list(self.current)
        self.current = [handle]


def _launch(deps):
    cap, nodes = CountingCapture(), Nodes()
    for i, d in enumerate(deps):
        nodes.add(Kernel(lambda s, h=i + 1: cap.kernel(h)), d)
    B200Backend.launcher(SimpleNamespace(lib=cap), nodes)(None)
    return cap, nodes


def test_interleaved_chains():
    """Three chains of four kernels, listed by turns: two of them have their
    waits set, and the end its own."""
    cap, _ = _launch([[]]*3 + [[i] for i in range(9)])
    assert cap.calls == 3
    assert all(cap.waits[i + 1] == ([i - 2] if i > 2 else [])
               for i in range(12))


def test_implied_waits():
    """A kernel that waits for another and for what that one waits for has
    one edge."""
    cap, nodes = _launch([[], [0], [0, 1], [0, 2], [1, 3]])
    assert [d for _, d in nodes.items] == [[], [0], [1], [2], [3]]
    assert cap.calls == 1


@pytest.mark.parametrize('seed', range(20))
def test_order_respects_the_waits(seed):
    rng = np.random.default_rng(seed)
    deps = [rng.integers(max(0, i - 6), i, rng.integers(0, 4)).tolist()
            if i else [] for i in range(50)]
    cap, nodes = _launch(deps)
    seen = set()
    for _, i, d in nodes.by_chains():
        assert seen.issuperset(d)
        seen.add(i)
    assert seen == set(range(50))

    def closure(waits):
        out = {}
        for i in sorted(waits):
            out[i] = set(waits[i]).union(*(out[d] for d in waits[i]))
        return out
    want = closure({i + 1: [d + 1 for d in ds] for i, ds in enumerate(deps)})
    assert closure(cap.waits) == want
