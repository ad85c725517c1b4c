"""An error on the way into a recorded call: nothing that the device may still read is let go before it has ended."""
import types

import pytest

from ngraph_python_b200 import lib, transformers


@pytest.mark.parametrize("failing", ["take", "executor", "read back"])
def test_device_is_waited_for_before_arguments_are_let_go(failing):
    events, arg = [], types.SimpleNamespace(src=None, in_place=0, inv_scale=1.0)

    def step(name):
        def run(*_):
            events.append(name)
            if name == failing:
                raise lib.B200Error(name)
        return run

    def synchronize():
        assert arg.src == 4096 and io.pageable[0] == 8192    # still there
        events.append("synchronize")
    t = types.SimpleNamespace(_clock=0, torch=types.SimpleNamespace(Tensor=int), _table_dirty=False,
                              _begin_call=lambda comp, io: setattr(io.block, "table_rows", 3),
                              _device_to_host_async=step("read back"), _end_call=step("end"),
                              stream=types.SimpleNamespace(synchronize=synchronize))
    io = transformers._CallIO.__new__(transformers._CallIO)
    io.t, io.block, io.pageable, io.flex_buffers = t, types.SimpleNamespace(table_rows=0), [8192], []
    io.comp = types.SimpleNamespace(executor=step("executor"), return_views=[None])
    io.results, io.taken = [None], False
    io.args = [(0, types.SimpleNamespace(version=0, flex=False), arg, False)]
    io._source = lambda k, value: (4096, value)
    io.take = step("take")
    with pytest.raises(lib.B200Error, match=failing):
        io.call([object()])
    assert events == ["take", "executor", "read back"][:1 + ["take", "executor", "read back"].index(failing)] + ["synchronize"]
    assert arg.src is None and io.pageable == [None] and io.block.table_rows == 0
    assert t._table_dirty                                    # the scale rows are sent again
