"""ctypes binding of libb200ng.so (the C ABI declared in include/b200ng.h).

There is no fallback: if the shared library is missing, import fails with instructions to build
it; if a call fails, `B200Error` carries the library's message.
"""
import ctypes as C
import os

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "libb200ng.so")

EW_MAX_IN, EW_MAX_OUT, EW_MAX_CONST, EW_MAX_OPS = 12, 6, 16, 96
F32, FLEX16, FLEX16_PLANES, F32_AT, FLEX16_AT = 0, 1, 2, 3, 4
REDUCE_NONE, REDUCE_C, REDUCE_B = 0, 1, 2

OPCODES = {
    "assign": 0, "neg": 1, "abs": 2, "sqrt": 3, "sqr": 4, "exp": 5, "log": 6, "rcp": 7,
    "exp2": 8, "log2": 9, "sig": 10, "tanh": 11, "safelog": 12, "sgn": 13, "sin": 14, "cos": 15,
    "add": 32, "sub": 33, "mul": 34, "div": 35, "int_div": 36, "mod": 37, "eq": 38, "ne": 39,
    "lt": 40, "le": 41, "gt": 42, "ge": 43, "pow": 44, "minimum": 45, "maximum": 46, "onehot": 47,
    "requant": 48,      # (register, index of a flex16 result): the value as stored and read back
}
UNARY_OPS = frozenset(k for k, v in OPCODES.items() if v < 32) | {"onehot"}
REDOPS = {"sum": 0, "prod": 1, "max": 2, "min": 3, "argmax": 4, "argmin": 5}


class B200Error(RuntimeError):
    pass


class EwTensor(C.Structure):
    _fields_ = [("dtype", C.c_int32), ("flex_slot", C.c_int32),
                ("sa", C.c_int64), ("sb", C.c_int64), ("sc", C.c_int64),
                ("plane_bytes", C.c_int64)]


class EwLaunchJob(C.Structure):
    _fields_ = [("kernel", C.c_void_p), ("inputs", C.c_void_p), ("results", C.c_void_p),
                ("consts", C.c_void_p)]


class EwOp(C.Structure):
    _fields_ = [("opcode", C.c_int32), ("a", C.c_int32), ("b", C.c_int32)]


class EwResult(C.Structure):
    _fields_ = [("reg", C.c_int32), ("redop", C.c_int32), ("t", EwTensor)]


class ConvEpilogue(C.Structure):
    _fields_ = [("bias", C.c_void_p), ("slot_bias", C.c_int32),
                ("residual", C.c_void_p), ("slot_residual", C.c_int32),
                ("relu", C.c_int32), ("write_int16", C.c_int32),
                ("out_planes", C.c_void_p), ("plane_bytes", C.c_size_t), ("mask", C.c_void_p)]


class EwProgram(C.Structure):
    _fields_ = [("A", C.c_int64), ("B", C.c_int64), ("C", C.c_int64),
                ("reduce_mode", C.c_int32),
                ("n_in", C.c_int32), ("n_const", C.c_int32), ("n_ops", C.c_int32),
                ("n_out", C.c_int32), ("n_red", C.c_int32),
                ("inp", EwTensor * EW_MAX_IN),
                ("ops", EwOp * EW_MAX_OPS),
                ("out", EwResult * EW_MAX_OUT)]


class ConvDims(C.Structure):
    _fields_ = [(n, C.c_int32) for n in
                ("C", "D", "H", "W", "N", "K", "T", "R", "S", "M", "P", "Q", "pad_d", "pad_h",
                 "pad_w", "str_d", "str_h", "str_w", "dil_d", "dil_h", "dil_w")]


class ConvFilterJob(C.Structure):
    _fields_ = [("filters", C.c_void_p), ("planes", C.c_void_p), ("dims", ConvDims), ("conv_pass", C.c_int32)]


CHAIN_MAX = 32                 # B2_CONV_CHAIN_MAX
CHAIN_NONE = -2                # B2_CONV_CHAIN_NONE


class ConvChainLayer(C.Structure):
    _fields_ = [("dims", ConvDims), ("input", C.c_int32), ("residual", C.c_int32), ("relu", C.c_int32),
                ("slot_in", C.c_int32), ("slot_filters", C.c_int32), ("slot_out", C.c_int32),
                ("slot_bias", C.c_int32), ("slot_residual", C.c_int32),
                ("filters", C.c_void_p), ("bias", C.c_void_p), ("out", C.c_void_p)]


class FlexScale(C.Structure):
    _fields_ = [("scale", C.c_float), ("inv_scale", C.c_float)]


class GemmPlan(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("kernel", "tile_n", "slices", "waves")]


class ConvPlan(C.Structure):
    _fields_ = [(n, C.c_int32) for n in ("tile_h", "tile_w", "tile_n", "slices", "blocks", "in_one_sum")]


class ConvSums(C.Structure):
    _fields_ = ([(n, C.c_int32) for n in ("kernel", "large", "small", "reserved")] +
                [(n, C.c_double) for n in ("loss", "other_loss")])


CONV_DIRECT, CONV_GATHER = 1, 2
GEMM_DIRECT, GEMM_PAIRS, GEMM_TILES, GEMM_STREAM = 0, 1, 2, 3
CALL_MAX_INPUTS, CALL_MAX_OUTPUTS = 16, 16


class CallArg(C.Structure):
    _fields_ = [("src", C.c_void_p), ("inv_scale", C.c_float), ("in_place", C.c_int32)]


class CallBlock(C.Structure):
    _fields_ = [("table", C.c_void_p), ("table_rows", C.c_int32), ("reserved", C.c_int32),
                ("arg", CallArg * CALL_MAX_INPUTS)]


class CallInput(C.Structure):
    _fields_ = [("dst", C.c_void_p), ("n", C.c_int64), ("flex_slot", C.c_int32),
                ("reserved", C.c_int32), ("where", C.c_void_p), ("holds", C.c_void_p)]


class CallOutput(C.Structure):
    _fields_ = [("src", C.c_void_p), ("dst", C.c_void_p), ("bytes", C.c_int64)]


class FlexState(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in
                ("dec", "pending", "initialized", "overflows", "hist", "hist_len", "hist_pos",
                 "run_value", "run_length", "run_choice")]


def _load():
    if not os.path.exists(LIB_PATH):
        raise ImportError(
            "%s is missing: build it with `python ngraph_python_b200/build.py` "
            "(needs nvcc; there is no CPU fallback)" % LIB_PATH)
    lib = C.CDLL(LIB_PATH)
    vp, i32, i64, sz = C.c_void_p, C.c_int32, C.c_int64, C.c_size_t
    sigs = {
        "b2_last_error": (C.c_char_p, []),
        "b2_version": (C.c_int, []),
        "b2_device_count": (C.c_int, []),
        "b2_set_nvrtc_path": (C.c_int, [C.c_char_p]),
        "b2_ew_check": (C.c_int, [C.POINTER(EwProgram), C.c_int, C.c_int, C.c_char_p, sz]),
        "b2_ew_check_joint": (C.c_int, [C.POINTER(EwProgram), C.c_int, C.c_char_p, sz]),
        "b2_ew_compile": (C.c_int, [C.POINTER(EwProgram), C.POINTER(vp)]),
        "b2_ew_scratch_bytes": (C.c_int, [vp, C.POINTER(sz)]),
        "b2_ew_prepare": (C.c_int, [vp, C.POINTER(vp), C.POINTER(vp)]),
        "b2_ew_launch": (C.c_int, [vp, C.POINTER(vp), C.POINTER(vp), C.POINTER(C.c_float), vp, vp,
                                   vp, sz, vp, C.c_int, vp]),
        "b2_ew_joint_source": (C.c_int, [vp, C.POINTER(C.c_char_p)]),
        "b2_ew_joint_prepare": (C.c_int, [vp]),
        "b2_ew_launch_many": (C.c_int, [C.POINTER(EwLaunchJob), i32, vp, vp, vp, C.POINTER(i32), vp]),
        "b2_ew_launch_builtin_scratch": (C.c_int, [vp, C.POINTER(vp), C.POINTER(vp),
                                                   C.POINTER(C.c_float), vp, vp, vp, C.c_int, vp]),
        "b2_ew_source": (C.c_char_p, [vp]),
        "b2_ew_launch_count": (C.c_int, [vp]),
        "b2_gemm_scratch_bytes": (C.c_int, [i32, i32, i32, i32, C.POINTER(sz)]),
        "b2_gemm_launches": (C.c_int, [i32, i64, i64, i32, i32, i32, C.POINTER(i32)]),
        "b2_gemm_route": (C.c_int, [i32, i64, i64, i64, i64, i32, i32, i32, C.POINTER(GemmPlan), C.POINTER(i32)]),
        "b2_gemm_plan": (C.c_int, [i32, i64, i64, i32, i32, i32, C.POINTER(GemmPlan)]),
        "b2_gemm_f32": (C.c_int, [vp, i64, i64, vp, i64, i64, vp, i64, i32, i32, i32, vp, sz, vp,
                                  vp]),
        "b2_gemm_flex16": (C.c_int, [vp, i64, i64, vp, i64, i64, vp, i64, i32, i32, i32, vp, i32,
                                     i32, i32, vp, vp, sz, vp, vp, i32, vp]),
        "b2_conv_fprop_scratch_bytes": (C.c_int, [i32, C.POINTER(ConvDims), C.POINTER(sz)]),
        "b2_conv_launches": (C.c_int, [i32, C.POINTER(ConvDims), i32, C.POINTER(i32)]),
        "b2_conv_fprop_f32_fused": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, vp, i32, vp, vp]),
        "b2_conv_fprop_f32": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, sz, vp, vp]),
        "b2_conv_fprop_flex16": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, i32, i32, i32, vp,
                                           vp, sz, vp, vp, i32, vp]),
        "b2_conv_planes_info": (C.c_int, [C.POINTER(ConvDims), i32, C.POINTER(i32), C.POINTER(sz),
                                          C.POINTER(sz)]),
        "b2_conv_split_activations": (C.c_int, [vp, C.POINTER(ConvDims), i32, vp, vp]),
        "b2_conv_filter_planes_many": (C.c_int, [C.POINTER(ConvFilterJob), i32, C.POINTER(i32), vp]),
        "b2_conv_split_planes": (C.c_int, [vp, i32, i32, i32, i32, vp, vp]),
        "b2_conv_f32_plan": (C.c_int, [C.POINTER(ConvDims), i32, i32, C.POINTER(ConvPlan)]),
        "b2_conv_f32_sums": (C.c_int, [C.POINTER(ConvDims), i32, C.POINTER(ConvSums)]),
        "b2_conv_filter_tiles_info": (C.c_int, [C.POINTER(ConvDims), i32, C.POINTER(sz)]),
        "b2_conv_filter_tiles": (C.c_int, [C.POINTER(ConvFilterJob), i32, C.POINTER(i32), vp]),
        "b2_conv_f32_tiles": (C.c_int, [i32, vp, vp, vp, C.POINTER(ConvDims), vp, vp, i32, vp, vp, vp]),
        "b2_conv_filter_planes": (C.c_int, [vp, C.POINTER(ConvDims), i32, vp, vp]),
        "b2_conv_flex16_planes": (C.c_int, [i32, vp, vp, vp, C.POINTER(ConvDims), vp, i32, i32,
                                            i32, vp, vp, vp, i32, vp]),
        "b2_conv_flex16_planes_fused": (C.c_int, [i32, vp, vp, vp, C.POINTER(ConvDims), vp, i32, i32,
                                                  i32, C.POINTER(ConvEpilogue), vp, vp, vp, i32, vp]),
        "b2_conv_chain_info": (C.c_int, [C.POINTER(ConvChainLayer), i32, C.POINTER(i32), C.POINTER(sz)]),
        "b2_conv_chain_filters": (C.c_int, [C.POINTER(ConvChainLayer), i32, vp, C.POINTER(i32), vp]),
        "b2_conv_chain_flex16": (C.c_int, [C.POINTER(ConvChainLayer), i32, vp, vp, sz, vp, vp, vp, vp, vp, vp]),
        "b2_conv_bprop_scratch_bytes": (C.c_int, [i32, C.POINTER(ConvDims), C.POINTER(sz)]),
        "b2_conv_bprop_f32_fused": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, vp, vp, vp]),
        "b2_conv_bprop_f32": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, sz, vp, vp]),
        "b2_conv_bprop_flex16": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, i32, i32, i32, vp,
                                           vp, sz, vp, vp, i32, vp]),
        "b2_conv_update_scratch_bytes": (C.c_int, [i32, C.POINTER(ConvDims), C.POINTER(sz)]),
        "b2_conv_update_planes_info": (C.c_int, [C.POINTER(ConvDims), C.POINTER(i32), C.POINTER(sz)]),
        "b2_conv_update_flex16_planes": (C.c_int, [vp, vp, vp, vp, C.POINTER(ConvDims), vp, i32, i32, i32,
                                                   i32, vp, vp, vp, vp, i32, vp]),
        "b2_conv_update_f32": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, sz, vp, vp]),
        "b2_conv_update_flex16": (C.c_int, [vp, vp, vp, C.POINTER(ConvDims), vp, i32, i32, i32, vp,
                                            vp, sz, vp, vp, i32, vp]),
        "b2_pool_avg_fprop": (C.c_int, [vp, vp, i32, i32, i32, i32, i32, i32, i32, i32, i32, i32,
                                        i32, i32, i32, vp, vp]),
        "b2_pool_max_fprop": (C.c_int, [vp, vp, i32, i32, i32, i32, i32, i32, i32, i32, i32, i32,
                                        i32, i32, i32, vp, vp]),
        "b2_pool_bprop": (C.c_int, [vp, vp, vp, i32, i32, i32, i32, i32, i32, i32, i32, i32, i32,
                                    i32, i32, i32, i32, vp, i32, i32, vp, vp, i32, vp]),
        "b2_lut_fprop": (C.c_int, [vp, vp, vp, i32, i32, i32, i32, i32, vp, i32, vp]),
        "b2_lut_update": (C.c_int, [vp, vp, vp, i32, i32, i32, i32, i32, i32, vp, i32, i32, i32,
                                    vp, vp, i32, vp]),
        "b2_dimshuffle": (C.c_int, [vp, vp, i32, i32, C.POINTER(i64), C.POINTER(i64),
                                    C.POINTER(i64), vp]),
        "b2_rng_fill": (C.c_int, [vp, i32, i64, i32, C.c_float, C.c_float, C.c_uint64, C.c_uint64,
                                  vp, vp, i32, vp, vp, i32, vp]),
        "b2_selftest_bounded_wait": (C.c_int, [i32, vp, vp, vp]),
        "b2_set_nccl_path": (C.c_int, [C.c_char_p]),
        "b2_comm_version": (C.c_int, [C.POINTER(i32)]),
        "b2_comm_unique_id": (C.c_int, [vp]),
        "b2_comm_init": (C.c_int, [vp, i32, i32, i32, C.POINTER(vp)]),
        "b2_comm_allreduce_f32": (C.c_int, [vp, vp, i64, i32, vp]),
        "b2_comm_poll_error": (C.c_int, [vp]),
        "b2_comm_abort": (C.c_int, [vp]),
        "b2_comm_destroy": (C.c_int, [vp]),
        "b2_flex_host_quantize": (C.c_int, [vp, vp, i64, vp, i32, vp, vp]),
        "b2_flex_dequantize": (C.c_int, [vp, vp, i64, vp, i32, vp]),
        "b2_absmax_bits_f32": (C.c_int, [vp, i64, vp, vp]),
        "b2_flex_publish": (C.c_int, [vp, i32, vp, vp, vp, vp]),
        "b2_call_inputs": (C.c_int, [C.POINTER(CallInput), i32, vp, vp, vp, vp]),
        "b2_call_take": (C.c_int, [vp, i32, vp, vp, vp, vp, vp, i32, vp]),
        "b2_call_outputs": (C.c_int, [C.POINTER(CallOutput), i32, vp, i32, vp, vp, vp, vp]),
        "b2_call_wait": (C.c_int, [i32, vp]),
        "b2_call_stage": (C.c_int, [vp, sz, vp, C.POINTER(vp)]),
        "b2_flex_rows_written": (C.c_int, [C.POINTER(FlexState), i32, vp, vp, vp, vp, C.POINTER(i32)]),
        "b2_flex_begin_call": (C.c_int, [C.POINTER(FlexState), i32, vp, vp, vp, vp, vp,
                                         C.POINTER(i32)]),
        "b2_flex_end_call": (C.c_int, [C.POINTER(FlexState), i32, vp, vp, vp, vp, C.POINTER(i32),
                                       C.POINTER(i32)]),
    }
    for name, (res, args) in sigs.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    return lib, sigs


_lib, SIGNATURES = _load()


def check(rc):
    if rc < 0:
        raise B200Error("b200ng error %d: %s" % (rc, _lib.b2_last_error().decode(errors="replace")))
    return rc


def raw():
    return _lib


def _find_nvrtc_dir():
    try:
        import nvidia.cuda_nvrtc as m  # wheel bundled with torch
        d = os.path.join(os.path.dirname(m.__file__), "lib")
        if os.path.exists(os.path.join(d, "libnvrtc.so.12")):
            return d
    except Exception:
        pass
    return None


if not os.path.exists("/usr/local/cuda/lib64/libnvrtc.so.12"):
    _d = _find_nvrtc_dir()
    if _d:
        _lib.b2_set_nvrtc_path(_d.encode())


def _find_nccl_dir():
    try:
        import nvidia.nccl as m  # wheel bundled with torch
        d = os.path.join(list(m.__path__)[0], "lib")
        if os.path.exists(os.path.join(d, "libnccl.so.2")):
            return d
    except Exception:
        pass
    return None


_d = _find_nccl_dir()
if _d:
    _lib.b2_set_nccl_path(_d.encode())


def make_program(dims, inputs, consts, ops, outs, reds, reduce_mode):
    """dims=(A,B,C); inputs/outs/reds entries are dicts with dtype, slot, strides (sa,sb,sc);
    ops are (name, a, b); outs carry 'reg'; reds carry 'reg' and 'redop'."""
    p = EwProgram()
    p.A, p.B, p.C = [int(d) for d in dims]
    p.reduce_mode = reduce_mode
    if len(inputs) > EW_MAX_IN or len(ops) > EW_MAX_OPS or len(outs) + len(reds) > EW_MAX_OUT \
            or len(consts) > EW_MAX_CONST:
        raise B200Error("fused program exceeds the kernel limits")
    p.n_in, p.n_const, p.n_ops = len(inputs), len(consts), len(ops)
    p.n_out, p.n_red = len(outs), len(reds)

    def fill(t, d):
        t.dtype = d["dtype"]
        t.flex_slot = d.get("slot", -1)
        t.sa, t.sb, t.sc = [int(s) for s in d["strides"]]
        t.plane_bytes = int(d.get("plane_bytes", 0))
    for i, d in enumerate(inputs):
        fill(p.inp[i], d)
    for i, (name, a, b) in enumerate(ops):
        p.ops[i].opcode = OPCODES[name]
        p.ops[i].a = a
        p.ops[i].b = b if b is not None else 0
    for k, d in enumerate(list(outs) + list(reds)):
        p.out[k].reg = d["reg"]
        p.out[k].redop = REDOPS[d["redop"]] if "redop" in d else 0
        fill(p.out[k].t, d)
    return p


def ew_check(prog, vec=True, probe=False, want_source=False, joint=False):
    buf = C.create_string_buffer(1 << 18) if want_source else None
    size = len(buf) if buf else 0
    if joint:
        check(_lib.b2_ew_check_joint(C.byref(prog), int(vec), buf, size))
    else:
        check(_lib.b2_ew_check(C.byref(prog), int(vec), int(probe), buf, size))
    return buf.value.decode() if buf else None


def launch_many(jobs, flex_table=0, flex_stats=0, status=0, stream=0):
    """jobs: (EwKernel, input pointers, result pointers, constants) of one joint_source(); returns the
    number of launches."""
    arr, keep = (EwLaunchJob * len(jobs))(), []
    for a, (kernel, in_ptrs, out_ptrs, consts) in zip(arr, jobs):
        ins = (C.c_void_p * max(1, len(in_ptrs)))(*in_ptrs)
        outs = (C.c_void_p * max(1, len(out_ptrs)))(*out_ptrs)
        cs = (C.c_float * EW_MAX_CONST)(*consts)
        keep.append((ins, outs, cs))
        a.kernel, a.inputs, a.results, a.consts = kernel.handle, C.addressof(ins), C.addressof(outs), \
            C.addressof(cs)
    n = C.c_int32()
    check(_lib.b2_ew_launch_many(arr, len(jobs), flex_table, flex_stats, status, C.byref(n), stream))
    return n.value


class EwKernel(object):
    """A compiled fused kernel."""

    def __init__(self, prog):
        self.prog = prog
        h = C.c_void_p()
        check(_lib.b2_ew_compile(C.byref(prog), C.byref(h)))
        self.handle = h
        n = C.c_size_t()
        check(_lib.b2_ew_scratch_bytes(h, C.byref(n)))
        self.scratch_bytes = n.value
        self.launches = _lib.b2_ew_launch_count(h)
        self._consts = (C.c_float * EW_MAX_CONST)()

    def source(self):
        return _lib.b2_ew_source(self.handle).decode()

    def prepare_joint(self):
        check(_lib.b2_ew_joint_prepare(self.handle))

    def joint_source(self):
        """What kernels of one joint launch have in common; empty for one that is launched alone."""
        s = C.c_char_p()
        check(_lib.b2_ew_joint_source(self.handle, C.byref(s)))
        return s.value

    def prepare(self, in_ptrs, out_ptrs):
        """Compiles what a launch with these pointers needs (a recording must not)."""
        check(_lib.b2_ew_prepare(self.handle, (C.c_void_p * max(1, len(in_ptrs)))(*in_ptrs),
                                 (C.c_void_p * max(1, len(out_ptrs)))(*out_ptrs)))

    def launch(self, in_ptrs, out_ptrs, consts=(), flex_table=0, flex_stats=0, scratch=0,
               scratch_bytes=0, status=0, probe=False, stream=0):
        ins = (C.c_void_p * max(1, len(in_ptrs)))(*in_ptrs)
        outs = (C.c_void_p * max(1, len(out_ptrs)))(*out_ptrs)
        for i, c in enumerate(consts):
            self._consts[i] = c
        check(_lib.b2_ew_launch(self.handle, ins, outs, self._consts, flex_table, flex_stats,
                                scratch, scratch_bytes, status, int(probe), stream))

    def launch_builtin_scratch(self, in_ptrs, out_ptrs, consts=(), flex_table=0, flex_stats=0,
                               status=0, probe=False, stream=0):
        """Same launch through the entry point that allocates nothing: split reductions use the
        16 KiB scratch array that lives inside the library instead of a caller buffer."""
        ins = (C.c_void_p * max(1, len(in_ptrs)))(*in_ptrs)
        outs = (C.c_void_p * max(1, len(out_ptrs)))(*out_ptrs)
        for i, c in enumerate(consts):
            self._consts[i] = c
        check(_lib.b2_ew_launch_builtin_scratch(self.handle, ins, outs, self._consts, flex_table,
                                                flex_stats, status, int(probe), stream))


class PlannedKernel(object):
    """Generated and compiled for sm_100a, but not loaded (no device needed)."""

    def __init__(self, prog, flex=False):
        self.prog = prog
        self._source = ew_check(prog, vec=True, probe=False, want_source=True)
        if flex:
            ew_check(prog, vec=True, probe=True)
        self.scratch_bytes = 0
        self.launches = 2 if "b2_ew_finalize" in self._source else 1

    def source(self):
        return self._source

    def joint_source(self):
        return b""


def gemm_scratch_bytes(flex, M, N, K):
    n = C.c_size_t()
    check(_lib.b2_gemm_scratch_bytes(int(bool(flex)), M, N, K, C.byref(n)))
    return n.value


def gemm_launches(flex, a_k_stride, b_k_stride, M, N, K):
    n = C.c_int32()
    check(_lib.b2_gemm_launches(int(bool(flex)), a_k_stride, b_k_stride, M, N, K, C.byref(n)))
    return n.value


def gemm_plan(flex, a_k_stride, b_k_stride, M, N, K):
    """(kernel, columns of a tile, slices of K, waves of clusters) of a product."""
    p = GemmPlan()
    check(_lib.b2_gemm_plan(int(bool(flex)), a_k_stride, b_k_stride, M, N, K, C.byref(p)))
    return p.kernel, p.tile_n, p.slices, p.waves


def gemm_route(flex, a_strides, b_strides, M, N, K):
    """(kernel, columns of a tile, slices of K, waves of clusters, launches) of a product called with these strides:
    (row, K) of the first operand, (K, column) of the second."""
    p, n = GemmPlan(), C.c_int32()
    check(_lib.b2_gemm_route(int(bool(flex)), a_strides[0], a_strides[1], b_strides[0], b_strides[1], M, N, K, C.byref(p),
                             C.byref(n)))
    return p.kernel, p.tile_n, p.slices, p.waves, n.value


def conv_fprop_scratch_bytes(flex, dims):
    n = C.c_size_t()
    check(_lib.b2_conv_fprop_scratch_bytes(int(bool(flex)), C.byref(dims), C.byref(n)))
    return n.value


CONV_FPROP, CONV_BPROP, CONV_UPDATE = 0, 1, 2
RNG_UNIFORM, RNG_NORMAL = 0, 1


def conv_launches(flex, dims, conv_pass):
    n = C.c_int32()
    check(_lib.b2_conv_launches(int(bool(flex)), C.byref(dims), conv_pass, C.byref(n)))
    return n.value


def plane_bytes(lengths):
    """Offset of the low byte plane from the high one for a tensor of these extents (images last)."""
    size = (lengths[-1] + 15) // 16 * 16
    for n in lengths[:-1]:
        size *= n
    return (size + 1023) // 1024 * 1024


def conv_planes_info(dims, conv_pass=CONV_FPROP):
    """(supported, room for one plane of the streamed tensor, bytes of the filter planes)."""
    ok, a, f = C.c_int32(), C.c_size_t(), C.c_size_t()
    check(_lib.b2_conv_planes_info(C.byref(dims), conv_pass, C.byref(ok), C.byref(a), C.byref(f)))
    return bool(ok.value), a.value, f.value


def conv_f32_plan(dims, conv_pass, tiles):
    """ConvPlan of an fp32 pass, or None where it does not gather its operands (so)."""
    p = ConvPlan()
    check(_lib.b2_conv_f32_plan(C.byref(dims), conv_pass, int(tiles), C.byref(p)))
    return p if p.tile_n else None


def conv_f32_sums(dims, conv_pass):
    """ConvSums of an fp32 pass with its filters laid out, or None where it takes none."""
    s = ConvSums()
    check(_lib.b2_conv_f32_sums(C.byref(dims), conv_pass, C.byref(s)))
    return s if s.kernel else None


def conv_filter_tiles_info(dims, conv_pass):
    """Bytes of the filters as the fp32 kernel's stages hold them; 0 where it takes them as they lie."""
    n = C.c_size_t()
    check(_lib.b2_conv_filter_tiles_info(C.byref(dims), conv_pass, C.byref(n)))
    return n.value


def conv_chain_info(layers):
    """(whether the layers make a chain, bytes of their filter planes)."""
    ok, n = C.c_int32(), C.c_size_t()
    arr = (ConvChainLayer * len(layers))(*layers)
    check(_lib.b2_conv_chain_info(arr, len(layers), C.byref(ok), C.byref(n)))
    return bool(ok.value), n.value


def conv_update_planes_info(dims):
    """(supported, bytes of the workspace)."""
    ok, n = C.c_int32(), C.c_size_t()
    check(_lib.b2_conv_update_planes_info(C.byref(dims), C.byref(ok), C.byref(n)))
    return bool(ok.value), n.value


def conv_bprop_scratch_bytes(flex, dims):
    n = C.c_size_t()
    check(_lib.b2_conv_bprop_scratch_bytes(int(bool(flex)), C.byref(dims), C.byref(n)))
    return n.value


def conv_update_scratch_bytes(flex, dims):
    n = C.c_size_t()
    check(_lib.b2_conv_update_scratch_bytes(int(bool(flex)), C.byref(dims), C.byref(n)))
    return n.value


def dimshuffle(src_ptr, dst_ptr, elem_bytes, shape, src_strides, dst_strides, stream=0):
    """N-d strided copy (strides in elements)."""
    n = len(shape)
    arr = C.c_int64 * max(n, 1)
    check(_lib.b2_dimshuffle(src_ptr, dst_ptr, elem_bytes, n, arr(*shape), arr(*src_strides),
                             arr(*dst_strides), stream))
