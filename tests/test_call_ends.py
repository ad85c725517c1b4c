"""The two ends of a recorded call through the C ABI: arguments taken in by a launch in front of the step list
(pageable memory in pieces) or by its first node, and results of any size stored by its last one."""
import ctypes as C

import numpy as np
import pytest

from ngraph_python_b200 import lib

pytestmark = pytest.mark.gpu

SIZES = [1, 4095, 49152, 73727, 73728, 98305, 300001]      # around one, two and four pieces of pageable memory


def quantised(x, inv):
    return np.trunc(np.clip(x * np.float32(inv), -32768, 32767)).astype(np.int16)


@pytest.mark.parametrize("first_node", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_arguments_of_both_types_from_host_and_device(n, first_node):
    import torch
    r = np.random.RandomState(n)
    host = r.randn(n).astype(np.float32)
    dev = torch.from_numpy(r.randn(n + 1).astype(np.float32)).cuda()[1:]      # (not 16-byte aligned)
    pinned = [torch.empty((n,)).pin_memory() for _ in range(2)]
    out = [torch.zeros((n + 8,), dtype=d, device="cuda") for d in (torch.int16, torch.float32, torch.float32)]
    table, rows = torch.zeros((3, 2), device="cuda"), torch.arange(6.0).reshape(3, 2).pin_memory()
    stats = torch.zeros((4,), dtype=torch.int32, device="cuda")
    words = torch.zeros((3,), dtype=torch.int64, device="cuda")
    ins = (lib.CallInput * 3)()
    for k, slot in enumerate((2, -1, -1)):
        ins[k].dst, ins[k].n, ins[k].flex_slot = out[k].data_ptr(), n, slot
        ins[k].where = words[k:].data_ptr()
    mem = torch.zeros((C.sizeof(lib.CallBlock),), dtype=torch.uint8).pin_memory()
    block = lib.CallBlock.from_address(mem.data_ptr())
    block.table, block.table_rows = rows.data_ptr(), 3
    block.arg[0].inv_scale = 4096.0
    sources = [pinned[0].data_ptr(), dev.data_ptr(), pinned[1].data_ptr()]
    for k in range(3):
        block.arg[k].src = sources[k]
    block.arg[2].in_place = 1
    stream = torch.cuda.current_stream().cuda_stream
    if first_node:
        pinned[0].numpy()[:] = host
        lib.check(lib.raw().b2_call_inputs(ins, 3, C.addressof(block), table.data_ptr(), stats.data_ptr(), stream))
    else:
        pageable = (C.c_void_p * 3)(host.ctypes.data, None, None)
        launches = C.c_int32()
        lib.check(lib.raw().b2_call_take(ins, 3, C.addressof(block), pageable, table.data_ptr(), stats.data_ptr(),
                                         C.byref(launches), 0, stream))
        assert launches.value == (1 if n < 73728 else 2 if n < 122880 else 4)
    torch.cuda.synchronize()
    want = quantised(host, 4096.0)
    assert np.array_equal(out[0].cpu().numpy(), np.concatenate([want, np.zeros(8, np.int16)]))
    assert np.array_equal(out[1].cpu().numpy()[:n], dev.cpu().numpy())
    assert not out[2].any()                                  # read in place by its reader
    assert words.tolist() == [out[0].data_ptr(), out[1].data_ptr(), sources[2]]
    assert stats.tolist() == [0, 0, int(np.abs(want.astype(np.int32)).max()), 0]
    assert torch.equal(table.cpu(), rows)


def test_nothing_to_take_in_launches_nothing():
    import torch
    ins, block, launches = (lib.CallInput * 1)(), lib.CallBlock(), C.c_int32(7)
    y = torch.zeros((8,), device="cuda")
    ins[0].dst, ins[0].n, ins[0].flex_slot = y.data_ptr(), 8, -1
    lib.check(lib.raw().b2_call_take(ins, 1, C.addressof(block), None, None, None, C.byref(launches), 0, None))
    assert launches.value == 0


@pytest.mark.parametrize("sizes", [[2], [4096, 4098, 2], [16, 14, 65536 + 6, 4094], [0, 1048576]])
def test_results_of_any_size(sizes):
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    src = [torch.randint(0, 256, (n + 16,), dtype=torch.uint8, device="cuda", generator=g) for n in sizes]
    dst = [torch.zeros((n + 16,), dtype=torch.uint8).pin_memory() for n in sizes]
    outs = (lib.CallOutput * len(sizes))(*[lib.CallOutput(s.data_ptr(), d.data_ptr(), n)
                                           for s, d, n in zip(src, dst, sizes)])
    stats = torch.arange(1, 301, dtype=torch.int32, device="cuda")
    status = torch.tensor([5], dtype=torch.int32, device="cuda")
    h_stats, h_status = torch.zeros((300,), dtype=torch.int32).pin_memory(), torch.zeros((1,), dtype=torch.int32).pin_memory()
    lib.check(lib.raw().b2_call_outputs(outs, len(sizes), stats.data_ptr(), 300, status.data_ptr(), h_stats.data_ptr(),
                                        h_status.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    for s, d, n in zip(src, dst, sizes):
        assert torch.equal(s[:n].cpu(), d[:n]) and not d[n:].any()
    assert h_stats.tolist() == list(range(1, 301)) and h_status.item() == 5 and not stats.any()
