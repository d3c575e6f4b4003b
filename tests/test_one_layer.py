"""The mark on the kernels of one layer belongs to the call and to the thread that set it."""

import threading

import pytest

from gtar_kimik3_public_b200.ops.library import library, one_layer


def test_the_mark_ends_with_the_call_whatever_happens_in_it():
    chain = library().gk_chain
    seen = []

    @one_layer
    def fine(a, b=0):
        """what it does"""
        seen.append(chain(1))
        return a + b

    @one_layer
    def fails():
        raise ValueError("no")

    assert fine(2, b=3) == 5 and fine.__doc__ == "what it does" and seen == [1]
    assert chain(0) == 0
    with pytest.raises(ValueError, match="no"):
        fails()
    assert chain(0) == 0


def test_the_mark_is_the_threads_own():
    chain, other = library().gk_chain, []
    chain(1)
    thread = threading.Thread(target=lambda: other.append(chain(0)))
    thread.start()
    thread.join()
    assert other == [0] and chain(0) == 1


def test_a_layer_within_a_layer_leaves_the_mark_as_it_is():
    """2: the outer layer's first kernel has been launched."""
    chain, seen = library().gk_chain, []

    @one_layer
    def inner():
        seen.append(chain(2))

    @one_layer
    def outer():
        chain(2)
        inner()
        seen.append(chain(2))

    outer()
    assert seen == [2, 2] and chain(0) == 0
