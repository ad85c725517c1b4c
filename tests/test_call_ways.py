"""Where a recorded call's arguments are taken in: by the step list's first node where they are few values, in front of
it elsewhere; and address words, which are written when they change."""
import ctypes as C

import numpy as np
import pytest

import ngraph_python_b200 as ng
from ngraph_python_b200 import lib, transformers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flex", [False, True])
@pytest.mark.parametrize("values", [1, 4096, (128 << 10) // 4 - 1, (128 << 10) // 4, (1 << 20) // 4 - 1, (1 << 20) // 4])
def test_arguments_of_every_kind(values, flex):
    import torch
    A = ng.make_axis(values, name="A")
    x, y = ng.placeholder([A]), ng.variable([A], initial_value=np.full(values, 0.5, np.float32))
    t = ng.transformers.make_transformer_factory("b200", flex=flex)()
    comp = t.computation([x + y, ng.max(x, reduction_axes=[A])], x)
    r = np.random.RandomState(3)
    arrays = [r.uniform(0.5, 1.0, values).astype(np.float32) for _ in range(3)]
    comp(arrays[0])
    comp.capture()
    assert comp._io.in_front == (4 * values >= transformers._CallIO.IN_FRONT_LEAST)
    pinned = torch.empty((values,)).pin_memory()
    for a in arrays + arrays:
        pinned.copy_(torch.from_numpy(a))
        device = torch.from_numpy(a).cuda()
        for given in (a, device, device, pinned.numpy(), torch.cat([device[:1], device])[1:], device.double()):
            got = comp(given)
            np.testing.assert_allclose(got[0], a + 0.5, atol=2.0 ** -12 if flex else 0)     # (15 bits of values below 2)
            np.testing.assert_allclose(got[1], a.max(), atol=2.0 ** -12 if flex else 0)
    t.close()


def test_words_are_written_when_they_change():
    import torch
    n, count = 8, 5                                           # (more words than the launch for words alone takes)
    out = torch.zeros((count, n), device="cuda")
    src = torch.arange(2.0 * count * n, device="cuda").reshape(2, count, n)
    words = torch.zeros((count,), dtype=torch.int64, device="cuda")
    held = (C.c_void_p * count)()
    ins, block, launches = (lib.CallInput * count)(), lib.CallBlock(), C.c_int32()

    def take(which, used, in_place=1):
        for k in range(count):
            ins[k].dst, ins[k].n, ins[k].flex_slot, ins[k].where = out[k].data_ptr(), n, -1, words[k:].data_ptr()
            ins[k].holds = C.addressof(held) + 8 * k
            block.arg[k].src = src[which, k].data_ptr() if k < used else None
            block.arg[k].in_place = in_place
        lib.check(lib.raw().b2_call_take(ins, count, C.addressof(block), None, None, None, C.byref(launches), 0,
                                         torch.cuda.current_stream().cuda_stream))
        want = [src[which, k].data_ptr() if k < used and in_place else out[k].data_ptr() for k in range(count)]
        assert words.tolist() == want and list(held) == want
        return launches.value
    assert take(0, 5) == 1 and take(0, 5) == 0                # all of them: nothing is known; nothing changes
    assert take(0, 1) == 1 and take(0, 1) == 0                # four go back to their own
    assert take(1, 3) == 1 and take(1, 3) == 0
    assert not out.any()
    assert take(1, 3, in_place=0) == 1 and torch.equal(out[:3], src[1, :3])
    held[1] = None                                            # not known: written again
    assert take(1, 0) == 1 and take(1, 0) == 0
