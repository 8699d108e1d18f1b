"""Which steps that mix portions are recorded (CPU): what a shape is, when it is recorded, and which recordings go first.
The bits of recorded steps are compared on the device (test_replay_gpu.py)."""
from types import SimpleNamespace

import pytest
import torch

from lockstep_b200.engine import graphs as G
from lockstep_b200.engine.batch import StepEntry


@pytest.fixture
def graphs(monkeypatch):
    """The bookkeeping of recorded steps, with nothing recorded behind it."""
    runner = SimpleNamespace(model=SimpleNamespace(blocks=[]), dtype=torch.bfloat16, split_size=256, device=None, err=None,
                             cache=SimpleNamespace(max_live=64))
    monkeypatch.setattr(G, "StaticMixedContext", lambda *args: None)
    out = G.DecodeGraphs(runner)
    out._record = lambda ctx: ()
    return out


def key_of(graphs, lengths, want=1, start=0):
    return graphs.mixed_key_for([StepEntry(str(i), [0] * n, start, list(range(n - min(n, want), n))) for i, n in enumerate(lengths)])


def see(graphs, key):
    """A step of this shape that is not recorded yet; True where it then is."""
    if not graphs.mixed_seen_again(key):
        return False
    graphs.record_mixed(key, [], (0, 0, 0, 0))
    return True


def test_counts_of_long_steps_survive_many_short_ones(graphs):
    long, short = key_of(graphs, [2048]), key_of(graphs, [200])
    assert not see(graphs, long) and not see(graphs, long) and not see(graphs, short) and not see(graphs, short)
    for n in range(2, 2 + 70):                        # more shapes than are counted
        assert not see(graphs, key_of(graphs, [n]))
    assert see(graphs, long)
    assert not see(graphs, short)                     # its own class pushed it out
    for n in range(300, 300 + 70):
        assert not see(graphs, key_of(graphs, [n]))
    assert not see(graphs, short) and see(graphs, short)
