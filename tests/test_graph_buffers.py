"""The pinned buffers that a step's numbers go through outlive the copies out of them."""

from gtar_kimik3_public_b200.engine import graphs as module
from gtar_kimik3_public_b200.engine.graphs import StepGraphs


def test_buffers_are_kept_until_their_copies_have_run(monkeypatch):
    class Event:
        done = False

        def query(self):
            return self.done

    monkeypatch.setattr(module, "_retired", module.deque())
    events = [Event(), None, Event()]
    graphs = object.__new__(StepGraphs)
    graphs.events, graphs.host = events, ["buffers"]
    del graphs
    module._give_back_retired()
    events[0].done = True
    module._give_back_retired()
    assert [entry[0] for entry in module._retired] == [["buffers"]]
    events[2].done = True
    module._give_back_retired()
    assert not module._retired
    graphs = object.__new__(StepGraphs)  # one whose set-up failed
    del graphs
    graphs = object.__new__(StepGraphs)  # one that has run no step
    graphs.events, graphs.host = [None, None], []
    del graphs
    assert not module._retired
