"""Kernels captured by what they wait for (``types.Nodes``, ``launcher``): the
captured graph orders exactly what the nodes' waits order, whatever the order
in which they were added; on a stand-in for the capture."""

from types import SimpleNamespace

import numpy as np
import pytest

from pyfr_gb300.backend.base import B200Backend
from pyfr_gb300.backend.types import Kernel, Nodes


class FakeCapture:
    """A captured stream: every kernel becomes a node that waits for the
    stream's current dependencies and replaces them."""

    def __init__(self, before):
        self.current = list(before)
        self.graph = {}

    def graph_capture_last(self, stream, buf, size, n):
        assert len(self.current) <= size
        for i, h in enumerate(self.current):
            buf[i] = h
        n._obj.value = len(self.current)

    def graph_capture_after(self, stream, handles, n):
        self.current = [handles[i] for i in range(n)]

    def kernel(self, handle):
        self.graph[handle] = list(self.current)
        self.current = [handle]


def _closure(waits):
    """All that comes before each node, in the order of ``waits``."""
    out = {}
    for i, deps in waits.items():
        out[i] = set(deps).union(*(out.get(d, set()) for d in deps))
    return out


@pytest.mark.parametrize('before', [[], [999]])
@pytest.mark.parametrize('seed', range(25))
def test_captured_order(before, seed):
    rng = np.random.default_rng(seed)
    cap, nodes = FakeCapture(before), Nodes()
    handle = lambda i: 1000 + int(i)
    for i in range(40):
        # (few dependents of each, as in a right-hand side; sometimes a
        # plain chain)
        lo = max(0, i - int(rng.integers(1, 7)))
        deps = rng.integers(lo, i, rng.integers(0, 4)).tolist() if i else []
        deps = [i - 1] if i and rng.random() < 0.3 else deps
        # one kernel of several launches in a row
        n = 2 if rng.random() < 0.2 else 1
        last = handle(i)
        hs = [handle(i) + 5000*j for j in range(1, n)] + [last]
        nodes.add(Kernel(lambda s, hs=hs: [cap.kernel(h) for h in hs]), deps)

    B200Backend.launcher(SimpleNamespace(lib=cap), nodes)(None)
    got = _closure(cap.graph)
    want = _closure({i: d for i, (_, d) in enumerate(nodes.items)})
    for i in want:
        assert {h for h in got[handle(i)] if 1000 <= h < 5000} == \
            {handle(d) for d in want[i]}
        assert not before or 999 in got[handle(i)]
    # what follows the graph's kernels waits for all of them
    end = set(cap.current).union(*(got[h] for h in cap.current))
    assert {handle(i) for i in want} <= end


def test_later_wait_refused():
    n = Nodes()
    n.add('a')
    with pytest.raises(ValueError):
        n.add('b', [1])
