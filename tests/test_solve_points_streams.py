"""api.solve_points sets the context's group streams only when it is asked to: changing
them drops the captured group graphs, and a context's own setting (four streams at
first) holds otherwise."""
import numpy as np
import pytest


class Recorder:
    def __init__(self):
        self.calls = []

    def call(self, name, *args):
        self.calls.append((name, args))


@pytest.mark.parametrize("streams", [None, 1, 3])
def test_streams_are_set_only_when_given(streams):
    from tpsc_conductivity_b200 import api

    ctx = Recorder()
    api.solve_points(np.zeros((2, 8)), ctx=ctx, **({} if streams is None else {"streams": streams}))
    names = [c[0] for c in ctx.calls]
    assert names == ([] if streams is None else ["tpsc_set_group_streams"]) + ["tpsc_solve_points"]
    if streams is not None:
        assert ctx.calls[0][1] == (streams,)
