"""The scratch buffers of one stream are listed for a capture while another thread's first call
adds its own (CPU: the insertion is made to happen between two entries)."""
from matpl_gb300 import ops

SIDE = 77


def test_workspaces_are_listed_while_other_threads_add_theirs(monkeypatch):
    """A capture lists its stream's workspaces while another thread's first call adds one."""
    cache = {("cuda:0", SIDE, k): k for k in range(4)}

    class Growing(int):
        def __eq__(self, other):               # what another thread does between two entries
            cache[("cuda:1", 5, len(cache))] = 0
            return int(self) == other
        __hash__ = int.__hash__

    cache[("cuda:0", Growing(SIDE + 1), 0)] = 9
    cache[("cuda:0", SIDE, 9)] = 8
    monkeypatch.setattr(ops, "_ws_cache", cache)
    assert ops.stream_workspaces(SIDE) == (0, 1, 2, 3, 8)
