"""Host arrays as arguments: an array that is read-only goes to the device as directly as one that is not."""
import ctypes
import tracemalloc
import types

import numpy as np
import pytest
import torch

from ngraph_python_b200 import transformers

N = 2 << 20              # values: 8 MB, above what goes through a pinned buffer


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("writeable", [True, False])
def test_large_host_argument_is_not_copied_on_the_host(writeable, flex, recwarn):
    t = transformers.B200Transformer.__new__(transformers.B200Transformer)
    t.torch, t.device = torch, torch.device("cpu")           # (the "device" side of the copy)
    target = torch.zeros((N,))
    buf = types.SimpleNamespace(version=0, flex=flex, tensor=target, staging=target, size=N)
    view = types.SimpleNamespace(buffer=buf, axes=types.SimpleNamespace(lengths=[2, N // 2]), is_dense=lambda: True)
    io = transformers._CallIO.__new__(transformers._CallIO)
    io.t, io.views, io.lengths = t, [view], [(2, N // 2)]
    io.pinned, io.visible = [None], ctypes.c_void_p()
    value = np.arange(N, dtype=np.float32).reshape(2, N // 2)
    value.flags.writeable = writeable
    tracemalloc.start()
    try:
        address, keep = io._source(0, value)
        peak = tracemalloc.get_traced_memory()[1]
    finally:
        tracemalloc.stop()
    assert peak < value.nbytes // 8
    assert address == (target.data_ptr() if flex else 0) and keep is value
    assert torch.equal(target, torch.arange(N, dtype=torch.float32))
    assert not [w for w in recwarn.list if "writ" in str(w.message)]
