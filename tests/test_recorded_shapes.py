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


def test_what_makes_the_shape_of_a_step(graphs):
    assert key_of(graphs, [1, 1]) is None                              # decoded tokens alone
    assert key_of(graphs, [3] * 17) is None and key_of(graphs, [20] * 17) is None        # more portions than work lists hold
    assert key_of(graphs, [9] * 8, want=9) is None                     # more wanted rows than live requests
    assert [key_of(graphs, [2] * n)[3] for n in (1, 4, 5, 16)] == [4, 4, 16, 16]
    assert [key_of(graphs, [40], want=n)[1] for n in (0, 1, 8, 9)] == [8, 8, 8, 64]
    assert [key_of(graphs, [n], want=1)[1] for n in (255, 256)] == [8, 64]
    assert [key_of(graphs, [5, *[1] * n])[2] for n in (0, 1, 31)] == [0, 64, 64]
    assert key_of(graphs, [5, *[1] * 31], start=1000)[2] == 128       # four splits of 256 keys each
    assert key_of(graphs, [17]) != key_of(graphs, [18])


def test_the_recordings_of_a_class_do_not_push_out_the_other_class(graphs):
    long, short = ([key_of(graphs, [n]) for n in range(first, first + count)] for first, count in ((300, 5), (20, 30)))
    for key in long:
        graphs.record_mixed(key, [], (0, 0, 0, 0))
    for i, key in enumerate(short):
        graphs.record_mixed(key, [], (0, 0, 0, 0))
        if i == 20:
            graphs.mixed.move_to_end(short[10])       # replayed: kept longer
    kept = short[-15:] + [short[10]]
    assert len(kept) == G.SHORT_GRAPHS and set(graphs.mixed) == {*long, *kept} and graphs.dropped == 30 - G.SHORT_GRAPHS
    assert not graphs.mixed_ready(short[0]) and not see(graphs, short[0])          # it has to come three times again
    for n in range(400, 400 + G.MIXED_GRAPHS):
        graphs.record_mixed(key_of(graphs, [n]), [], (0, 0, 0, 0))
    assert not any(graphs.mixed_ready(key) for key in long) and all(graphs.mixed_ready(key) for key in kept)


def test_a_class_stops_recording_and_the_other_goes_on(graphs):
    recorded = 0
    for n in range(2, 2 + G.MIXED_RECORDINGS + 3):
        recorded += [see(graphs, key_of(graphs, [n])) for _ in range(3)][-1]
    assert recorded == G.MIXED_RECORDINGS
    assert not any(see(graphs, key_of(graphs, [200])) for _ in range(5))
    assert [see(graphs, key_of(graphs, [2048])) for _ in range(3)] == [False, False, True]


def test_steps_called_between_replays_look_their_portions_up_at_every_replay(graphs, monkeypatch):
    """A part that is not recorded (a norm of a user's own, say) takes the recurrent mixer behind it out of the recording with
    it: the list of portions that the mixer keeps on the context is then made for every step, also where a recorded run
    made one in its graph."""
    from lockstep_b200.parts import recurrent

    monkeypatch.setattr(recurrent.K, "find_portions", lambda token_slot, out, cap, err: out[:len(token_slot)].copy_(token_slot))
    seen = []

    def mixer(h, ctx):
        out, _ = recurrent.portion_list(ctx, torch.zeros(4, 1), SimpleNamespace(device="cpu", err=None))
        seen.append(out[:2].tolist())
        return h

    ctx = SimpleNamespace(token_slot=torch.zeros(2, dtype=torch.int32), wanted=2, _portion_list=(torch.full((7,), -1), 2))
    ctx.fill = lambda entries, slots: ctx.token_slot.copy_(torch.tensor(slots, dtype=torch.int32))
    recorded = SimpleNamespace(replay=lambda: None)
    logits = torch.zeros(2, 3)
    for table, replay in ((graphs.graphs, graphs.replay), (graphs.mixed, graphs.replay_mixed)):
        table["key"] = ([(recorded, None), (None, [mixer, mixer]), (recorded, None)], ctx, None, logits, 0)
        for slots in ([0, 1], [2, 3]):
            replay("key", [None, None], slots)
    assert seen == 2 * [[0, 1], [0, 1], [2, 3], [2, 3]]
