"""The Python call path keeps packed views per set of tensor addresses; what they say of a tensor is checked on every call."""
from collections import OrderedDict

import pytest
import torch

from aginfer_b200 import runtime as rt
from aginfer_b200.runner import MAX_BINDINGS, Runner


class RecordingSession:
    """Stands in for the native session: notes the shape, stride and byte size of every view it is handed."""
    bind = rt.Session.bind

    def __init__(self):
        self.seen = []

    def enqueue_packed(self, packed, stream=0, options=None):
        (ins, n, _), _ = packed
        self.seen.append([(tuple(v.shape[:v.rank]), tuple(v.stride[:v.rank]), v.byte_size) for v in ins[:n]])


@pytest.fixture
def runner():
    r = Runner.__new__(Runner)
    r.session, r._bindings, r._dtypes = RecordingSession(), OrderedDict(), {"x": "F32", "y": "F32"}
    r._side, r._replays, r._current_stream = None, True, lambda: 0
    return r


@pytest.mark.parametrize("change", [lambda x: x.t_(), lambda x: x.resize_(4, 6), lambda x: x.as_strided_((4, 3), (6, 2)),
                                    lambda x: x.unsqueeze_(0)], ids=["transposed", "resized", "strided", "unsqueezed"])
def test_a_tensor_changed_in_place_is_described_anew(runner, change):
    x, y = torch.zeros(6, 4), torch.zeros(3)
    address = x.data_ptr()
    runner.run({"x": x}, {"y": y})
    change(x)
    assert x.data_ptr() == address
    runner.run({"x": x}, {"y": y})
    assert runner.session.seen == [[((6, 4), (4, 1), 96)], [(tuple(x.shape), x.stride(), 96)]]


def test_another_tensor_at_the_same_address_is_described_anew(runner):
    base, y = torch.zeros(24), torch.zeros(3)
    for view in (base.view(6, 4), base.view(4, 6), base[:12].view(4, 3), base.view(6, 4)):
        runner.run({"x": view}, {"y": y})
        assert runner.session.seen[-1] == [(tuple(view.shape), view.stride(), 96)]


def test_kept_views_are_bounded(runner):
    tensors = [torch.zeros(2) for _ in range(3 * MAX_BINDINGS)]
    for x in tensors + tensors[:4]:
        runner.run({"x": x}, {"y": tensors[0]})
    assert len(runner._bindings) == MAX_BINDINGS and len(runner.session.seen) == len(tensors) + 4
