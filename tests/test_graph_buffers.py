"""The pinned buffers that a step's numbers go through outlive the copies out of them."""

from gtar_kimik3_public_b200.engine.graphs import StepGraphs


def test_buffers_are_given_back_behind_the_copies():
    class Event:
        def synchronize(self):
            waited.append(self)

    waited, events = [], [Event(), None, Event()]
    graphs = object.__new__(StepGraphs)
    graphs.events = events
    del graphs
    assert waited == [events[0], events[2]]
    del events[:]
    graphs = object.__new__(StepGraphs)  # one whose set-up failed
    del graphs
