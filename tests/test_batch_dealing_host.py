"""Dealing of shape groups to streams: which stream takes the next chunk, and the order of the groups."""
import numpy as np
import pytest


class _Event:
    def __init__(self, polls):
        self.polls = polls

    def query(self):
        self.polls -= 1
        return self.polls < 0


@pytest.mark.parametrize("polls,wanted,expect", [
    ([None, 0], [True, True], 0), ([3, None], [True, True], 1), ([3, 1], [True, True], 1), ([3, 1], [True, False], 0),
    ([2, 2], [True, True], 0), ([5], [True], 0)])
def test_next_stream(polls, wanted, expect):
    pytest.importorskip("torch")
    from khepri_gb300 import batch
    events = [None if p is None else _Event(p) for p in polls]
    assert batch._next_stream(events, wanted) == expect


def test_larger_groups_cost_more():
    pytest.importorskip("torch")
    from khepri_gb300 import batch
    key = lambda p: ((p, p), (1, 0), (0, 0), (None, 1.5))  # noqa: E731
    one = [np.arange(1)]
    assert batch._group_cost((key(13), one)) > batch._group_cost((key(11), one)) > batch._group_cost((key(3), one))
    assert batch._group_cost((key(5), [np.arange(64)] * 2)) > batch._group_cost((key(5), [np.arange(64)]))
