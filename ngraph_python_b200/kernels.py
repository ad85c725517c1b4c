"""Executor steps for the dense contractions and pooling: each wraps one C-ABI entry point.

Takes the place of the reference's per-op kernel objects GEMMKernel (ngraph/transformers/gpu/
gemm.py:26-263), ConvFpropKernel / FlexConvFpropKernel (gpu/conv.py:24-100, gpu/flex_conv.py:
49-200) and PoolFpropKernel / FlexPoolFpropKernel (gpu/pool.py:27-220, gpu/flex_pool.py): bind
buffers once, then launch per call; in flex mode the first write of an output runs the measuring
("probe") variant so that the exponent fits the true range of the result.
"""
import ctypes as C

import numpy as np

from . import lib


def _merge(view, axes):
    """(extent, element stride) of `axes` walked as one dimension of `view`, or None."""
    axes = [a for a in axes if a.length != 1]
    if not axes:
        return 1, 0
    size, stride = 1, None
    for a in reversed(list(axes)):
        s = view.stride_of(a)
        if stride is None:
            stride = s
        elif s != stride * size:
            return None
        size *= a.length
    return size, stride


class _Step(object):
    launches = 0
    scratch_bytes = 0

    def __init__(self, index, op):
        self.index = index
        self.op = op
        self.out_views = []
        self.in_views = []

    def output_buffers(self):
        """The tensors whose exponents this step manages."""
        return [v.buffer for v in self.out_views]

    def writes(self):
        """Every tensor whose memory this step changes, with an exponent of its own or not."""
        return [v.buffer for v in self.out_views]

    def _ptr(self, v):
        return v.buffer.ptr() + v.offset * (2 if v.buffer.flex else 4)

    # flex first-write protocol shared by GEMM and conv -------------------------------------------
    def _flex_probe_then(self, t, out_buf, in_bufs, call):
        """call(probe) launches; on the first write of out_buf a probe launch measures the exact
        integer maximum, from which the output exponent is chosen."""
        e = out_buf.entry
        if not e.initialized:
            t._probe64.zero_()
            call(1)
            t.kernel_launches += self.launches
            imax = int(t._probe64[0].item())
            if getattr(self, "probe_is_float", False):
                # fused epilogue: the kernel leaves the bit pattern of max |fp32 result|
                real = float(np.array([imax & 0xffffffff], dtype=np.uint32).view(np.float32)[0])
            else:
                real = float(imax) * in_bufs[0].entry.scale * in_bufs[1].entry.scale
            dec = e.initialize_from_range(real)
            t._set_table_row(out_buf.slot_write, dec)
            t._stats[out_buf.slot_write:out_buf.slot_write + 1].zero_()
        call(0)
        t.kernel_launches += self.launches


class _PlaneUser(object):
    """flex16 convolution steps that can run on the implicit-GEMM tile kernels: the streamed
    tensors (activations, the error tensor) are read as two byte planes which their producer
    writes directly -- or else the first step that reads them -- and the filter planes are kept for
    as long as the filters do not change: one launch per convolution.  fp32: the filters as the
    kernel that gathers its operands holds them (`tiles`), kept likewise."""
    use_planes = False
    tiles = False
    plane_args = ()                 # indexes of the tensors read as planes in op.args / in_views
    splits = ()                     # those that this step splits unless their producer has
    filters_change = False          # the computation makes the filters, or takes them as an argument
    planes_built_first = False      # the first of the convolutions builds the filter planes of all
    joint_planes = None             # ... this one: the steps whose planes it builds
    filter_planes = None
    filter_version = None

    def _setup_planes(self, t, conv_pass, stream_arg, filter_arg):
        if self.flex:
            ok, _, filt_bytes = lib.conv_planes_info(self.dims, conv_pass)
        else:
            filt_bytes = lib.conv_filter_tiles_info(self.dims, conv_pass)
            ok = filt_bytes > 0
        if not ok:
            return
        self.conv_pass = conv_pass
        self.filter_arg = filter_arg
        self.filter_bytes = filt_bytes
        self.in_views[filter_arg].buffer.watched = True     # (what is kept follows its version)
        if self.flex:
            self.use_planes = True
            self._read_planes((stream_arg,))
        else:
            self.tiles = True

    def _read_planes(self, args):
        self.plane_args = self.splits = args
        for k in args:
            buf = self.in_views[k].buffer
            buf.plane_bytes = lib.plane_bytes(self.in_views[k].axes.lengths)
            buf.plane_images = self.in_views[k].axes.lengths[-1]
            # (planes whose rows of images are padded are written by the convolutions only)
            buf.plane_dense = self.dims.N % 16 == 0
            buf.plane_steps = getattr(buf, "plane_steps", []) + [self]
        self.launches = 1

    def _planes(self, t, k):
        """Address of the planes of argument k."""
        v = self.in_views[k]
        if k in self.splits and not v.buffer.planes_by_producer:
            d = self.dims
            lengths = (d.K, d.P, d.Q, d.N) if self.streams_errors(k) else (d.C, d.H, d.W, d.N)
            lib.check(lib.raw().b2_conv_split_planes(self._ptr(v), *lengths, v.buffer.planes_ptr,
                                                     t.stream.cuda_stream))
            t.kernel_launches += 1
        return v.buffer.planes_ptr

    def streams_errors(self, k):
        return False

    def allocate(self, t):
        if (self.use_planes or self.tiles) and self.filter_planes is None and not t.plan_only:
            self.filter_planes = t.torch.zeros((self.filter_bytes + 1024,), dtype=t.torch.uint8,
                                               device=t.device)
            self.filter_ptr = self.filter_planes.data_ptr() + (-self.filter_planes.data_ptr()) % 1024

    def _build_filter_planes(self, t):
        fv = self.in_views[self.filter_arg]
        if self.tiles:
            self._build_tiles(t, [self])
            self.filter_version = fv.buffer.version
            return
        lib.check(lib.raw().b2_conv_filter_planes(self._ptr(fv), C.byref(self.dims), self.conv_pass,
                                                  self.filter_ptr, t.stream.cuda_stream))
        t.kernel_launches += 1
        self.filter_version = fv.buffer.version

    @staticmethod
    def _build_tiles(t, users):
        jobs, n = _PlaneUser._filter_jobs(users), C.c_int32()
        lib.check(lib.raw().b2_conv_filter_tiles(jobs, len(users), C.byref(n), t.stream.cuda_stream))
        t.kernel_launches += n.value

    @staticmethod
    def _filter_jobs(users):
        jobs = (lib.ConvFilterJob * len(users))()
        for job, s in zip(jobs, users):
            job.filters, job.planes = s._ptr(s.in_views[s.filter_arg]), s.filter_ptr
            job.dims, job.conv_pass = s.dims, s.conv_pass
        return jobs

    def _build_joint_planes(self, t):
        users = self.joint_planes
        if self.tiles:
            self._build_tiles(t, users)
            return
        jobs, n = self._filter_jobs(users), C.c_int32()
        lib.check(lib.raw().b2_conv_filter_planes_many(jobs, len(users), C.byref(n), t.stream.cuda_stream))
        t.kernel_launches += n.value

    def kept_planes(self):
        """Whether `refresh` can have anything to do."""
        return (self.use_planes or self.tiles) and not self.planes_built_first and not self.filters_change

    def refresh(self, t):
        """Rebuilds the cached filter planes when the filters have changed since they were built
        (called before every launch, and before every replay of a captured step list)."""
        if not self.kept_planes():
            return
        fbuf = self.in_views[self.filter_arg].buffer
        if self.filter_version != fbuf.version:
            self._build_filter_planes(t)

    def _add_tail_views(self, t, epilogue):
        for key in ("bias", "residual", "mask"):
            if epilogue.get(key) is not None:
                v = t._view_of(epilogue[key])
                if not v.is_dense():
                    raise ValueError("fused convolution %s must be a dense tensor" % key)
                self.in_views.append(v)

    def _current_filter_planes(self, t):
        fbuf = self.in_views[self.filter_arg].buffer
        if self.joint_planes:
            self._build_joint_planes(t)
        elif self.planes_built_first:
            pass
        elif self.filters_change:
            self._build_filter_planes(t)
        else:
            self.refresh(t)

    def _launch_tiles(self, t):
        self._current_filter_planes(t)
        epi = getattr(self, "epi", None) or {}
        extra = [self._ptr(v) for v in self.in_views[2:]]
        tail = [extra.pop(0) if epi.get(k) is not None else None for k in ("bias", "residual", "mask")]
        lib.check(lib.raw().b2_conv_f32_tiles(
            self.conv_pass, self._ptr(self.in_views[1 - self.filter_arg]), self.filter_ptr,
            self._ptr(self.out_views[0]), C.byref(self.dims), tail[0], tail[1], int(bool(epi.get("relu"))),
            tail[2], t._status.data_ptr(), t.stream.cuda_stream))
        t.kernel_launches += self.launches

    def _launch_planes(self, t):
        xv, fv = self.in_views[self.plane_args[0]], self.in_views[self.filter_arg]
        ov = self.out_views[0]
        raw = lib.raw()
        st = t.stream.cuda_stream
        xbuf, fbuf = xv.buffer, fv.buffer
        planes_ptr = self._planes(t, self.plane_args[0])
        self._current_filter_planes(t)
        slots = (t._slot_for_read(xbuf, self), t._slot_for_read(fbuf, self), ov.buffer.slot_write)
        epi = getattr(self, "epi", None)
        if epi is None:
            def call(probe):
                lib.check(raw.b2_conv_flex16_planes(
                    self.conv_pass, planes_ptr, self.filter_ptr, self._ptr(ov),
                    C.byref(self.dims), t._table.data_ptr(), slots[0], slots[1], slots[2],
                    t._stats.data_ptr(), t._probe64.data_ptr(), t._status.data_ptr(), probe, st))
            self._flex_probe_then(t, ov.buffer, [xbuf, fbuf], call)
            return
        ce = lib.ConvEpilogue()
        extra = self.in_views[2:]
        k = 0
        ce.bias, ce.slot_bias, ce.residual, ce.slot_residual = None, -1, None, -1
        if epi.get("bias") is not None:
            ce.bias, ce.slot_bias = self._ptr(extra[k]), t._slot_for_read(extra[k].buffer, self)
            k += 1
        if epi.get("residual") is not None:
            ce.residual = self._ptr(extra[k])
            ce.slot_residual = t._slot_for_read(extra[k].buffer, self)
            k += 1
        if epi.get("mask") is not None:
            ce.mask = self._ptr(extra[k])
        ce.relu = int(bool(epi.get("relu")))
        obuf = ov.buffer
        ce.write_int16 = int(self.write_int16 or obuf.plane_bytes == 0)
        ce.out_planes, ce.plane_bytes = (obuf.planes_ptr, obuf.plane_bytes) if obuf.plane_bytes else (None, 0)

        def call(probe):
            lib.check(raw.b2_conv_flex16_planes_fused(
                self.conv_pass, planes_ptr, self.filter_ptr, self._ptr(ov),
                C.byref(self.dims), t._table.data_ptr(), slots[0], slots[1], slots[2],
                C.byref(ce), t._stats.data_ptr(), t._probe64.data_ptr(), t._status.data_ptr(),
                probe, st))
        self._flex_probe_then(t, obuf, [xbuf, fbuf], call)


def join_filter_planes(steps, arguments):
    """Which convolutions of a computation make their filter planes in every call: those whose filters it
    writes, computes or copies itself, or receives (`arguments`).  The filter planes of the convolutions
    whose filters this computation writes after reading them (a training step): the first of them builds
    all, one launch per 32 layers."""
    made = set(b for s in steps for b in s.writes())
    written, mine = set(), []
    for s in steps:
        if getattr(s, "filter_arg", None) is not None:
            buf = s.in_views[s.filter_arg].buffer
            s.filters_change = buf in made or buf in arguments
            if buf.last_write_step >= 0 and buf not in written:
                mine.append(s)
        written.update(s.writes())
    for s in mine:
        s.planes_built_first = True
    if mine:
        mine[0].joint_planes = mine


class ConvChainStep(_Step):
    """A run of convolution layers that a recorded call makes in one launch, with the activations between
    them in shared memory.  `layers` describes them, `members` are the steps it stands for: outside
    recorded calls (first writes, measuring launches) they run one by one, with the same bits."""
    kind = "conv_chain"
    launches = 1

    def __init__(self, members, layers, nbytes, kept, pool=None):
        """kept: results that somebody outside reads; pool: the averaging step behind the last layer,
        where it takes whole images and reads them alone."""
        super(ConvChainStep, self).__init__(members[0].index, members[0].op)
        self.members, self.layers, self.nbytes = members, layers, nbytes
        self.in_views = [v for s in members for v in s.in_views]
        self.out_views = [v for s in members for v in s.out_views]
        # results that only the run itself reads are not stored by it (as int16 tensors or byte planes,
        # which the members store when they run one by one)
        self.unstored = set(s.out_views[0].buffer for s in members) - kept
        self.kept, self.pool = kept, pool
        if pool is not None:
            self.out_views += pool.out_views
        self.planes = None
        self.filters = [s.in_views[s.filter_arg].buffer for s in members]
        self.versions = None
        # what a reader of unstored results has to know: tensors made by the run and before it, the rows of
        # the scale table that stand for them, and the state of all that at the end of the last call
        self.results = [s.out_views[0].buffer for s in members]
        self.reads = [b for b in dict.fromkeys(v.buffer for v in self.in_views) if b not in self.results]
        self.rows = sorted(set(r for b in self.reads + self.results for r in (b.slot, b.slot_write)))
        self.open = False            # the last call's results are not all stored
        self.clock = self.epoch = self.exponents = None

    def kept_planes(self):
        return True

    def refresh(self, t):
        """Filter planes as the chain reads them, made again when filters have changed."""
        versions = [b.version for b in self.filters]
        if versions == self.versions:
            return
        n = C.c_int32()
        if self.planes is None:
            self.planes = t.torch.zeros((self.nbytes,), dtype=t.torch.uint8, device=t.device)
        lib.check(lib.raw().b2_conv_chain_filters(self._layers(t), len(self.members), self.planes.data_ptr(),
                                                  C.byref(n), t.stream.cuda_stream))
        t.kernel_launches += n.value
        self.versions = versions

    def _layers(self, t):
        arr = (lib.ConvChainLayer * len(self.members))(*self.layers)
        for a, s in zip(arr, self.members):
            xv, fv, ov = s.in_views[0], s.in_views[1], s.out_views[0]
            a.filters = s._ptr(fv)
            a.slot_in, a.slot_filters = t._slot_for_read(xv.buffer, s), t._slot_for_read(fv.buffer, s)
            a.slot_out, a.slot_bias, a.slot_residual = ov.buffer.slot_write, -1, -1
            extra = list(s.in_views[2:])
            if s.epi.get("bias") is not None:
                v = extra.pop(0)
                a.bias, a.slot_bias = s._ptr(v), t._slot_for_read(v.buffer, s)
            if s.epi.get("residual") is not None:
                a.slot_residual = t._slot_for_read(extra.pop(0).buffer, s)
            a.out = s._ptr(ov) if ov.buffer in self.kept else None
        return arr

    def launch(self, t):
        x = self.members[0].in_views[0]
        planes = x.buffer.planes_ptr if x.buffer.planes_by_producer else None
        lib.check(lib.raw().b2_conv_chain_flex16(
            self._layers(t), len(self.members), None if planes else self._ptr(x), planes, x.buffer.plane_bytes,
            self.planes.data_ptr(), t._table.data_ptr(), t._stats.data_ptr(),
            self._ptr(self.pool.out_views[0]) if self.pool is not None else None, t._status.data_ptr(),
            t.stream.cuda_stream))
        t.kernel_launches += 1

    def called(self, t):
        """A recorded call has been launched."""
        self.open, self.clock = True, t._clock
        for b in self.kept:
            b.int16_at = b.version

    def keep_exponents(self, t):
        """... and its exponents are settled."""
        if self.epoch != t._flex_epoch:
            self.epoch, self.exponents = t._flex_epoch, t._dec_uploaded[self.rows]

    def store_result(self, t, buf):
        """For a reader from outside any call: `buf` as the last call made it, if that was a call of this
        run which did not store it."""
        if not self.open or buf not in self.unstored or buf.version > self.clock:
            return
        if t.closed:
            raise lib.B200Error("the transformer has been closed")
        changed = [b.name for b in self.reads if b.version > self.clock]
        if changed or (t._dec_uploaded[self.rows] != self.exponents).any():
            raise lib.B200Error(
                "the recorded call did not store %s, and %s changed since: read it before that, return it from "
                "the computation, or take its device_tensor before capture()"
                % (buf.name, ", ".join(changed) + (" have" if len(changed) > 1 else " has") if changed else
                   "the exponents of the tensors that it follows from have"))
        # the layers one by one write all their results: those that are stored, or that somebody else has
        # written since, stay as they are
        others = [b for b in self.results if b not in self.unstored or b.version > self.clock]
        for b in others:
            b.join_planes()
        saved = [(b, b.tensor.clone()) for b in others]
        for s in self.members:
            s.launch(t)
        for b, values in saved:
            b.tensor.copy_(values)
        self.open = False
        t._stats_clean = False           # (their statistics belong to the call that has been)


def chain_convolutions(steps, returned, t):
    """The step list with every run of convolution layers that fits one launch (b2_conv_chain_info)
    replaced by a ConvChainStep.  A run is made of neighbouring steps; what they stream comes from the
    run or, for its first layer's input, from int16 or byte planes that are complete before it; their
    filters do not change inside the computation, nor does anything else that they read behind them; and no
    step outside reads one of their results as byte planes.  `returned`: buffers whose contents are wanted
    after a call."""
    if not t.flex:
        return list(steps)

    def suits(s):
        return (isinstance(s, ConvStep) and s.use_planes and s.epi is not None and
                not s.planes_built_first and not s.joint_planes and s.splits in ((), (0,)) and
                not s.filters_change and s.epi.get("mask") is None and
                not s.out_views[0].buffer.persistent)

    def chain_of(run):
        made, layers = {}, []
        first = run[0].in_views[0].buffer
        for s in run:
            layer = lib.ConvChainLayer()
            layer.dims, layer.relu = s.dims, int(bool(s.epi.get("relu")))
            x = s.in_views[0].buffer
            layer.residual = lib.CHAIN_NONE
            if x is not first and x not in made:
                return None
            layer.input = made.get(x, -1)
            if s.epi.get("residual") is not None:
                r = s.in_views[3 if s.epi.get("bias") is not None else 2].buffer
                if r is not first and r not in made:
                    return None
                layer.residual = made.get(r, -1)
            made[s.out_views[0].buffer] = len(layers)
            layers.append(layer)
        mine = set(run)
        after = steps[steps.index(run[-1]) + 1] if steps.index(run[-1]) + 1 < len(steps) else None
        pool = after if isinstance(after, PoolStep) and after.averages_images() and \
            after.in_views[0].buffer is run[-1].out_views[0].buffer else None
        mine.add(pool)
        behind = set(b for s in steps[steps.index(run[-1]) + 1:] for b in s.writes())
        if any(v.buffer in behind for s in run for v in s.in_views):
            return None                      # (results that are not stored could not be made again)
        kept = set(b for b in made if b in returned)
        for s in steps:
            if s in mine:
                continue
            for k, v in enumerate(s.in_views):
                if v.buffer in made or v.buffer is first:
                    if k in getattr(s, "plane_args", ()):
                        return None
                    if v.buffer in made:
                        kept.add(v.buffer)
        for layer, s in zip(layers, run):
            if s.out_views[0].buffer in kept:
                layer.out = 16               # (an address follows when there is one)
        ok, nbytes = lib.conv_chain_info(layers)
        return ConvChainStep(list(run), layers, nbytes, kept, pool) if ok else None

    out, i = [], 0
    while i < len(steps):
        end = i
        while end < len(steps) and end - i < lib.CHAIN_MAX and suits(steps[end]):
            end += 1
        chain = None
        while end - i >= 2 and chain is None:
            chain = chain_of(steps[i:end])
            end -= chain is None
        if chain is None:
            out.append(steps[i])
            i += 1
        else:
            out.append(chain)
            i = end + (chain.pool is not None)
    return out


class GemmStep(_Step):
    """C[M,N] = op(A)[M,K] * op(B)[K,N] for a DotOp."""
    kind = "gemm"
    launches = 3

    def __init__(self, index, op, t):
        super(GemmStep, self).__init__(index, op)
        x, y = op.args
        xv, yv = t._view_of(x), t._view_of(y)
        red = [a for a in xv.axes if a in op.reduction_axes]
        am, ak = _merge(xv, op.x_out_axes), _merge(xv, red)
        bk, bn = _merge(yv, red), _merge(yv, op.y_out_axes)
        if None in (am, ak, bk, bn):
            raise ValueError("Unhandled op: dot operands must be 2-d collapsible: {}".format(op))
        self.M, self.K, self.N = am[0], ak[0], bn[0]
        if bk[0] != self.K:
            raise ValueError("Unhandled op: reduction axes of the dot operands disagree")
        # extents of 1 carry no stride of their own: describe them as row-major
        a_cs = ak[1] if self.K > 1 else 1
        a_rs = am[1] if self.M > 1 else (self.K if a_cs == 1 else 1)
        b_ns = bn[1] if self.N > 1 else 1
        b_ks = bk[1] if self.K > 1 else (self.N if b_ns == 1 else 1)
        self.a_str = (a_rs, a_cs)
        self.b_str = (b_ks, b_ns)
        if 1 not in self.a_str or 1 not in self.b_str:
            raise ValueError("Unhandled op: dot operand is not contiguous along M/K or K/N")
        self.in_views = [xv, yv]
        self.out_views = [t._view_of(op)]
        self.flex = t.flex
        self.scratch_bytes = lib.gemm_scratch_bytes(self.flex, self.M, self.N, self.K) + 1024
        self.launches = lib.gemm_route(self.flex, self.a_str, self.b_str, self.M, self.N, self.K)[-1]

    def launch(self, t):
        xv, yv = self.in_views
        ov = self.out_views[0]
        raw = lib.raw()
        sp, sb = t._scratch_aligned()
        st = t.stream.cuda_stream
        if not self.flex:
            lib.check(raw.b2_gemm_f32(self._ptr(xv), self.a_str[0], self.a_str[1], self._ptr(yv),
                                      self.b_str[0], self.b_str[1], self._ptr(ov), self.N, self.M,
                                      self.N, self.K, sp, sb, t._status.data_ptr(), st))
            t.kernel_launches += self.launches
            return
        slots = (t._slot_for_read(xv.buffer, self), t._slot_for_read(yv.buffer, self),
                 ov.buffer.slot_write)

        def call(probe):
            lib.check(raw.b2_gemm_flex16(
                self._ptr(xv), self.a_str[0], self.a_str[1], self._ptr(yv), self.b_str[0],
                self.b_str[1], self._ptr(ov), self.N, self.M, self.N, self.K, t._table.data_ptr(),
                slots[0], slots[1], slots[2], t._stats.data_ptr(), sp, sb, t._probe64.data_ptr(),
                t._status.data_ptr(), probe, st))
        self._flex_probe_then(t, ov.buffer, [xv.buffer, yv.buffer], call)


class ConvStep(_PlaneUser, _Step):
    """Convolution forward on C,D,H,W,N / C,T,R,S,K / K,M,P,Q,N tensors."""
    kind = "conv"
    launches = 3

    def __init__(self, index, op, t, epilogue=None):
        """epilogue (where takes_conv_tail): dict(out=<op whose tensor the step writes>,
        bias=<op or None>, residual=<op or None>, relu=bool) -- the elementwise tail of the layer,
        evaluated in the convolution kernel's epilogue."""
        super(ConvStep, self).__init__(index, op)
        inputs, filters = op.args
        self.epi = epilogue
        out_op = epilogue["out"] if epilogue else op
        iv, fv, ov = t._view_of(inputs), t._view_of(filters), t._view_of(out_op)
        if epilogue and not ov.is_dense():
            raise ValueError("fused convolution output must be a dense tensor")
        for v, what in ((iv, "input"), (fv, "filter")):
            if not v.is_dense():
                raise ValueError("Unhandled op: convolution %s must be a dense tensor" % what)
        cp = op.conv_params
        Cc, D, H, W, N = iv.axes.lengths
        C2, T, R, S, K = fv.axes.lengths
        K2, M, P, Q, N2 = op.axes.lengths          # (the tail's tensor may lack the unit axes)
        if K2 != K or N2 != N or ov.buffer.size != K2 * M * P * Q * N2:
            raise ValueError("convolution output axes do not match filter/input axes")
        d = lib.ConvDims()
        d.C, d.D, d.H, d.W, d.N = Cc, D, H, W, N
        d.K, d.T, d.R, d.S = K, T, R, S
        d.M, d.P, d.Q = M, P, Q
        for k in ("pad_d", "pad_h", "pad_w"):
            setattr(d, k, int(cp.get(k, 0)))
        for k in ("str_d", "str_h", "str_w", "dil_d", "dil_h", "dil_w"):
            setattr(d, k, int(cp.get(k, 1)))
        # the output extents must be what the parameters imply (reference: output_dim,
        # ngraph/frontends/neon/utils.py / conv_utils.py)
        for (x, f, pad, st, dil, o, nm) in ((D, T, d.pad_d, d.str_d, d.dil_d, M, "D"),
                                            (H, R, d.pad_h, d.str_h, d.dil_h, P, "H"),
                                            (W, S, d.pad_w, d.str_w, d.dil_w, Q, "W")):
            expect = (x + 2 * pad - dil * (f - 1) - 1) // st + 1
            if expect != o:
                raise ValueError("convolution output extent along %s is %d, parameters imply %d"
                                 % (nm, o, expect))
        self.dims = d
        self.in_views = [iv, fv]
        self.out_views = [ov]
        self.flex = t.flex
        self.scratch_bytes = lib.conv_fprop_scratch_bytes(self.flex, d) + 1024
        self.launches = lib.conv_launches(self.flex, d, lib.CONV_FPROP)
        self._setup_planes(t, lib.CONV_FPROP, 0, 1)
        if epilogue:
            if not (self.use_planes if self.flex else self.launches == 1):
                raise ValueError("a fused convolution epilogue needs a kernel that takes one")
            self.probe_is_float = True
            self.write_int16 = True          # the planner clears it when only planes are read
            self._add_tail_views(t, epilogue)

    def launch(self, t):
        if self.use_planes:
            return self._launch_planes(t)
        if self.tiles:
            return self._launch_tiles(t)
        iv, fv = self.in_views[:2]
        ov = self.out_views[0]
        raw = lib.raw()
        sp, sb = t._scratch_aligned()
        st = t.stream.cuda_stream
        if self.epi:
            extra = [self._ptr(v) for v in self.in_views[2:]]
            bias = extra.pop(0) if self.epi.get("bias") is not None else None
            residual = extra.pop(0) if self.epi.get("residual") is not None else None
            lib.check(raw.b2_conv_fprop_f32_fused(self._ptr(iv), self._ptr(fv), self._ptr(ov),
                                                  C.byref(self.dims), bias, residual,
                                                  int(bool(self.epi.get("relu"))),
                                                  t._status.data_ptr(), st))
            t.kernel_launches += self.launches
            return
        if not self.flex:
            lib.check(raw.b2_conv_fprop_f32(self._ptr(iv), self._ptr(fv), self._ptr(ov),
                                            C.byref(self.dims), sp, sb, t._status.data_ptr(), st))
            t.kernel_launches += self.launches
            return
        slots = (t._slot_for_read(iv.buffer, self), t._slot_for_read(fv.buffer, self),
                 ov.buffer.slot_write)

        def call(probe):
            lib.check(raw.b2_conv_fprop_flex16(
                self._ptr(iv), self._ptr(fv), self._ptr(ov), C.byref(self.dims),
                t._table.data_ptr(), slots[0], slots[1], slots[2], t._stats.data_ptr(), sp, sb,
                t._probe64.data_ptr(), t._status.data_ptr(), probe, st))
        self._flex_probe_then(t, ov.buffer, [iv.buffer, fv.buffer], call)


def takes_conv_tail(fprop, t, conv_pass=lib.CONV_FPROP):
    """Whether the convolution's kernel evaluates the elementwise tail behind it: the flex16 tile
    kernel, the fp32 kernel that gathers its operands."""
    d = _conv_dims_of(fprop, t)
    if t.flex:
        return lib.conv_planes_info(d, conv_pass)[0]
    return lib.conv_launches(False, d, conv_pass) == 1


def _conv_dims_of(fprop, t):
    """ConvDims of a forward ConvolutionOp (axes C,D,H,W,N / C,T,R,S,K / K,M,P,Q,N)."""
    cp = fprop.conv_params
    Cc, D, H, W, N = fprop.args[0].axes.lengths
    C2, T, R, S, K = fprop.args[1].axes.lengths
    K2, M, P, Q, N2 = fprop.axes.lengths
    d = lib.ConvDims()
    d.C, d.D, d.H, d.W, d.N = Cc, D, H, W, N
    d.K, d.T, d.R, d.S = K, T, R, S
    d.M, d.P, d.Q = M, P, Q
    for k in ("pad_d", "pad_h", "pad_w"):
        setattr(d, k, int(cp.get(k, 0)))
    for k in ("str_d", "str_h", "str_w", "dil_d", "dil_h", "dil_w"):
        setattr(d, k, int(cp.get(k, 1)))
    return d


class _ConvGradStep(_PlaneUser, _Step):
    """Shared part of the two convolution gradients: two dense operands, one dense result, the
    forward convolution's dimensions."""
    launches = 3
    what = None                     # "bprop" | "update"

    def __init__(self, index, op, t, epilogue=None):
        """epilogue (input gradient, where takes_conv_tail): dict(out, residual, mask) -- the sum
        with another gradient and the mask of a ReLU behind it."""
        super(_ConvGradStep, self).__init__(index, op)
        self.epi = epilogue
        av, bv = t._view_of(op.args[0]), t._view_of(op.args[1])
        ov = t._view_of(epilogue["out"] if epilogue else op)
        for v in (av, bv):
            if not v.is_dense():
                raise ValueError("Unhandled op: convolution %s operands must be dense tensors"
                                 % self.what)
        self.dims = _conv_dims_of(op.fprop, t)
        d = self.dims
        expect = {"bprop": ((d.K, d.M, d.P, d.Q, d.N), (d.C, d.T, d.R, d.S, d.K),
                            (d.C, d.D, d.H, d.W, d.N)),
                  "update": ((d.K, d.M, d.P, d.Q, d.N), (d.C, d.D, d.H, d.W, d.N),
                             (d.C, d.T, d.R, d.S, d.K))}[self.what]
        for v, shape in zip((av, bv, ov), expect):
            if v is ov and epilogue:
                same = ov.is_dense() and [n for n in v.axes.lengths if n != 1] == [n for n in shape if n != 1]
            else:
                same = tuple(v.axes.lengths) == shape
            if not same:
                raise ValueError("convolution %s: tensor of shape %s where %s is expected"
                                 % (self.what, tuple(v.axes.lengths), shape))
        self.in_views = [av, bv]
        self.out_views = [ov]
        self.flex = t.flex
        sizer = lib.conv_bprop_scratch_bytes if self.what == "bprop" else \
            lib.conv_update_scratch_bytes
        self.scratch_bytes = sizer(self.flex, d) + 1024
        self.launches = lib.conv_launches(
            self.flex, d, lib.CONV_BPROP if self.what == "bprop" else lib.CONV_UPDATE)
        if self.what == "bprop":
            self._setup_planes(t, lib.CONV_BPROP, 0, 1)      # streamed: delta; filters: args[1]
        if epilogue:
            if not (self.use_planes if self.flex else self.launches == 1):
                raise ValueError("a fused convolution epilogue needs a kernel that takes one")
            self.probe_is_float = True
            self.write_int16 = True          # the planner clears it when only planes are read
            self._add_tail_views(t, epilogue)

    def launch(self, t):
        if self.use_planes:
            return self._launch_planes(t)
        if self.tiles:
            return self._launch_tiles(t)
        av, bv = self.in_views[:2]       # (delta, filters) or (delta, inputs)
        ov = self.out_views[0]
        raw = lib.raw()
        sp, sb = t._scratch_aligned()
        st = t.stream.cuda_stream
        if self.what == "bprop":
            first, second = av, bv       # E, F
            f32, f16 = raw.b2_conv_bprop_f32, raw.b2_conv_bprop_flex16
        else:
            first, second = bv, av       # I, E
            f32, f16 = raw.b2_conv_update_f32, raw.b2_conv_update_flex16
        if self.epi:
            extra = [self._ptr(v) for v in self.in_views[2:]]
            residual = extra.pop(0) if self.epi.get("residual") is not None else None
            mask = extra.pop(0) if self.epi.get("mask") is not None else None
            lib.check(raw.b2_conv_bprop_f32_fused(self._ptr(first), self._ptr(second), self._ptr(ov),
                                                  C.byref(self.dims), residual, mask,
                                                  t._status.data_ptr(), st))
            t.kernel_launches += self.launches
            return
        if not self.flex:
            lib.check(f32(self._ptr(first), self._ptr(second), self._ptr(ov), C.byref(self.dims),
                          sp, sb, t._status.data_ptr(), st))
            t.kernel_launches += self.launches
            return
        slots = (t._slot_for_read(first.buffer, self), t._slot_for_read(second.buffer, self),
                 ov.buffer.slot_write)

        def call(probe):
            lib.check(f16(self._ptr(first), self._ptr(second), self._ptr(ov), C.byref(self.dims),
                          t._table.data_ptr(), slots[0], slots[1], slots[2], t._stats.data_ptr(),
                          sp, sb, t._probe64.data_ptr(), t._status.data_ptr(), probe, st))
        self._flex_probe_then(t, ov.buffer, [first.buffer, second.buffer], call)

    def streams_errors(self, k):
        return k == 0


class ConvBpropStep(_ConvGradStep):
    """Input gradient of a convolution: args (delta K,M,P,Q,N ; filters C,T,R,S,K)."""
    kind = "conv_bprop"
    what = "bprop"


class ConvUpdateStep(_ConvGradStep):
    """Filter gradient of a convolution: args (delta K,M,P,Q,N ; inputs C,D,H,W,N)."""
    kind = "conv_update"
    what = "update"
    workspace = None

    def __init__(self, index, op, t, bias_op=None):
        """bias_op (where the gradient reads planes): the reduction that sums the delta over all
        axes but the channels, evaluated in the same kernel."""
        super(ConvUpdateStep, self).__init__(index, op, t)
        self.reads_planes, self.workspace_bytes = False, 0
        if self.flex:
            self.reads_planes, self.workspace_bytes = lib.conv_update_planes_info(self.dims)
        if self.reads_planes:
            self.scratch_bytes = 0
            self._read_planes((0, 1))
        self.bias_op = bias_op
        if bias_op is not None:
            if not self.reads_planes:
                raise ValueError("a fused bias gradient needs the kernel that reads planes")
            self.out_views.append(t._view_of(bias_op))

    def allocate(self, t):
        if self.reads_planes and self.workspace is None and not t.plan_only:
            self.workspace = t.torch.zeros((self.workspace_bytes + 1024,), dtype=t.torch.uint8,
                                           device=t.device)
            self.workspace_ptr = self.workspace.data_ptr() + (-self.workspace.data_ptr()) % 1024

    def launch(self, t):
        if not self.reads_planes:
            return super(ConvUpdateStep, self).launch(t)
        ev, iv = self.in_views
        outs = [v.buffer for v in self.out_views]
        errors, acts = self._planes(t, 0), self._planes(t, 1)
        slot_i, slot_e = t._slot_for_read(iv.buffer, self), t._slot_for_read(ev.buffer, self)
        bias = self.out_views[1] if self.bias_op is not None else None

        def call(probe):
            lib.check(lib.raw().b2_conv_update_flex16_planes(
                acts, errors, self._ptr(self.out_views[0]), self._ptr(bias) if bias else None,
                C.byref(self.dims), t._table.data_ptr(), slot_i, slot_e, outs[0].slot_write,
                bias.buffer.slot_write if bias else -1, t._stats.data_ptr(), self.workspace_ptr,
                t._probe64.data_ptr(), t._status.data_ptr(), probe, t.stream.cuda_stream))
            t.kernel_launches += 1
        if not all(b.entry.initialized for b in outs):
            t._probe64.zero_()
            call(1)
            scales = (iv.buffer.entry.scale * ev.buffer.entry.scale, ev.buffer.entry.scale)
            for b, most, scale in zip(outs, t._probe64.tolist(), scales):
                if not b.entry.initialized:
                    t._set_table_row(b.slot_write, b.entry.initialize_from_range(float(most) * scale))
                    t._stats[b.slot_write:b.slot_write + 1].zero_()
        call(0)


class PoolStep(_Step):
    """Average or max pooling forward; a flex output keeps its input's exponent
    (ngraph/transformers/passes/flexpass.py:40-48)."""
    kind = "pool"
    launches = 1

    def __init__(self, index, op, t):
        super(PoolStep, self).__init__(index, op)
        pp = op.pool_params
        if pp["op"] not in ("avg", "max"):
            raise ValueError("Unhandled op: only average and max pooling are implemented: {}"
                             .format(op))
        self.pool_op = pp["op"]
        iv = t._view_of(op.args[0])
        if not iv.is_dense():
            raise ValueError("Unhandled op: pooling input must be a dense tensor")
        if int(pp.get("J", 1)) != 1 or int(pp.get("T", 1)) != 1:
            raise ValueError("Unhandled op: pooling over channels or depth")
        ov = t._view_of(op)
        if t.flex:
            t._share_entry(ov.buffer, iv.buffer)
        Cc, D, H, W, N = iv.axes.lengths
        K, M, P, Q, N2 = ov.axes.lengths
        self.args = (Cc, H, W, N, P, Q, int(pp["R"]), int(pp["S"]), int(pp.get("pad_h", 0)),
                     int(pp.get("pad_w", 0)), int(pp.get("str_h", 1)), int(pp.get("str_w", 1)))
        self.in_views = [iv]
        self.out_views = [ov]
        self.flex = t.flex

    def averages_images(self):
        """Whether a result is the average of a whole channel of an image (of at most 512 pixels)."""
        Cc, H, W, N, P, Q, R, S, pad_h, pad_w = self.args[:10]
        return (self.flex and self.pool_op == "avg" and P == Q == 1 and (R, S) == (H, W) and
                pad_h == pad_w == 0 and H * W <= 512)

    def output_buffers(self):
        return []          # no exponent of its own to manage

    def launch(self, t):
        iv, ov = self.in_views[0], self.out_views[0]
        stats = 0
        if self.flex:
            stats = t._stats.data_ptr() + 4 * (t._stats.numel() - 2)    # discarded
        fn = lib.raw().b2_pool_max_fprop if self.pool_op == "max" else lib.raw().b2_pool_avg_fprop
        lib.check(fn(self._ptr(iv), self._ptr(ov), int(self.flex),
                     *(self.args + (stats, t.stream.cuda_stream))))
        t.kernel_launches += 1


class PoolBpropStep(_Step):
    """Gradient of average or max pooling with respect to the pooled tensor."""
    kind = "pool_bprop"
    launches = 1
    probe_is_float = True

    def __init__(self, index, op, t):
        super(PoolBpropStep, self).__init__(index, op)
        pp = op.pool_params
        if pp["op"] not in ("avg", "max"):
            raise ValueError("Unhandled op: only average and max pooling are implemented: {}"
                             .format(op))
        if int(pp.get("J", 1)) != 1 or int(pp.get("T", 1)) != 1:
            raise ValueError("Unhandled op: pooling over channels or depth")
        ev, iv, ov = t._view_of(op.args[0]), t._view_of(op.args[1]), t._view_of(op)
        for v in (ev, iv):
            if not v.is_dense():
                raise ValueError("Unhandled op: pooling gradient operands must be dense tensors")
        Cc, D, H, W, N = iv.axes.lengths
        K, M, P, Q, N2 = ev.axes.lengths
        self.is_max = int(pp["op"] == "max")
        self.args = (Cc, H, W, N, P, Q, int(pp["R"]), int(pp["S"]), int(pp.get("pad_h", 0)),
                     int(pp.get("pad_w", 0)), int(pp.get("str_h", 1)), int(pp.get("str_w", 1)))
        self.in_views = [ev, iv]
        self.out_views = [ov]
        self.flex = t.flex

    def launch(self, t):
        ev, iv = self.in_views
        ov = self.out_views[0]
        raw = lib.raw()
        st = t.stream.cuda_stream
        if not self.flex:
            lib.check(raw.b2_pool_bprop(self._ptr(ev), self._ptr(iv), self._ptr(ov), 0, self.is_max,
                                        *(self.args + (None, -1, -1, None, None, 0, st))))
            t.kernel_launches += 1
            return
        t._slot_for_read(iv.buffer, self)
        slots = (t._slot_for_read(ev.buffer, self), ov.buffer.slot_write)

        def call(probe):
            lib.check(raw.b2_pool_bprop(self._ptr(ev), self._ptr(iv), self._ptr(ov), 1, self.is_max,
                                        *(self.args + (t._table.data_ptr(), slots[0], slots[1],
                                                       t._stats.data_ptr(), t._probe64.data_ptr(),
                                                       probe, st))))
        self._flex_probe_then(t, ov.buffer, [ev.buffer, iv.buffer], call)


class LutStep(_Step):
    """Embedding lookup; a flex output keeps the table's exponent (its mantissas are copied)."""
    kind = "lut"
    launches = 1

    def __init__(self, index, op, t):
        super(LutStep, self).__init__(index, op)
        lv, xv, ov = t._view_of(op.args[0]), t._view_of(op.args[1]), t._view_of(op)
        for v in (lv, xv):
            if not v.is_dense():
                raise ValueError("Unhandled op: lookup operands must be dense tensors")
        self.lut_axis = op.lut_axis
        self.V = lv.axes.lengths[op.lut_axis]
        self.F = lv.axes.lengths[1 - op.lut_axis]
        self.n = xv.axes.lengths[0]
        if t.flex:
            t._share_entry(ov.buffer, lv.buffer)
        self.in_views = [lv, xv]
        self.out_views = [ov]
        self.flex = t.flex

    def output_buffers(self):
        return []          # no exponent of its own to manage

    def launch(self, t):
        lv, xv = self.in_views
        ov = self.out_views[0]
        table, slot = (t._table.data_ptr(), t._slot_for_read(xv.buffer, self)) if self.flex else (None, -1)
        lib.check(lib.raw().b2_lut_fprop(self._ptr(lv), self._ptr(xv), self._ptr(ov), int(self.flex),
                                         self.lut_axis, self.V, self.F, self.n, table, slot,
                                         t.stream.cuda_stream))
        t.kernel_launches += 1


class LutUpdateStep(_Step):
    """Gradient of an embedding table: rows of delta added up per looked-up index."""
    kind = "lut_update"
    launches = 1
    probe_is_float = True

    def __init__(self, index, op, t):
        super(LutUpdateStep, self).__init__(index, op)
        dv, xv, ov = t._view_of(op.args[0]), t._view_of(op.args[1]), t._view_of(op)
        for v in (dv, xv):
            if not v.is_dense():
                raise ValueError("Unhandled op: lookup update operands must be dense tensors")
        self.lut_axis = op.lut_axis
        self.V = ov.axes.lengths[op.lut_axis]
        self.F = ov.axes.lengths[1 - op.lut_axis]
        self.n = xv.axes.lengths[0]
        self.pad_idx = -1 if op.pad_idx is None else int(op.pad_idx)
        self.in_views = [dv, xv]
        self.out_views = [ov]
        self.flex = t.flex

    def launch(self, t):
        dv, xv = self.in_views
        ov = self.out_views[0]
        raw = lib.raw()
        st = t.stream.cuda_stream
        head = (self._ptr(dv), self._ptr(xv), self._ptr(ov))
        dims = (self.lut_axis, self.V, self.F, self.n, self.pad_idx)
        if not self.flex:
            lib.check(raw.b2_lut_update(*(head + (0,) + dims + (None, -1, -1, -1, None, None, 0, st))))
            t.kernel_launches += 1
            return
        slots = (t._slot_for_read(dv.buffer, self), t._slot_for_read(xv.buffer, self),
                 ov.buffer.slot_write)

        def call(probe):
            lib.check(raw.b2_lut_update(*(head + (1,) + dims + (
                t._table.data_ptr(), slots[0], slots[1], slots[2], t._stats.data_ptr(),
                t._probe64.data_ptr(), probe, st))))
        self._flex_probe_then(t, ov.buffer, [dv.buffer, xv.buffer], call)


class RngStep(_Step):
    """Random fill (RngFillKernel / FlexRngFillKernel, ngraph/transformers/gpu/tensor_ops.py:
    621-661, 713-740).  The stream of numbers is fixed by the transformer's seed and the position
    of the op in its graph; a device-side counter moves it on after every execution, also under
    CUDA-graph replay."""
    kind = "rng"
    launches = 2           # the fill and the advance of its counter
    probe_is_float = True

    def __init__(self, index, op, t):
        super(RngStep, self).__init__(index, op)
        ov = t._view_of(op)
        self.out_views = [ov]
        self.in_views = []
        self.flex = t.flex
        p = op.params
        if op.distribution == "uniform":
            self.dist, self.a, self.b = lib.RNG_UNIFORM, float(p["low"]), float(p["high"])
        else:
            self.dist, self.a, self.b = lib.RNG_NORMAL, float(p["loc"]), float(p["scale"])
        self.seed = int(t.rng_seed)
        self.stream_id = t._next_rng_stream()
        self.counter = None

    def allocate(self, t):
        if self.counter is None and not t.plan_only:
            self.counter = t.torch.zeros((1,), dtype=t.torch.int64, device=t.device)

    def launch(self, t):
        ov = self.out_views[0]
        raw = lib.raw()
        st = t.stream.cuda_stream
        offset = self.stream_id << 40           # streams of different ops never meet
        head = (self._ptr(ov), int(self.flex), ov.buffer.size, self.dist, self.a, self.b, self.seed,
                offset, self.counter.data_ptr())
        if not self.flex:
            lib.check(raw.b2_rng_fill(*(head + (None, -1, None, None, 0, st))))
            t.kernel_launches += self.launches
            return
        slot = ov.buffer.slot_write

        def call(probe):
            lib.check(raw.b2_rng_fill(*(head + (t._table.data_ptr(), slot, t._stats.data_ptr(),
                                                t._probe64.data_ptr(), probe, st))))
        self._flex_probe_then(t, ov.buffer, [], call)


class DimshuffleStep(_Step):
    """A strided copy between two views with the same axes (DimShuffleKernel of the reference,
    ngraph/transformers/gpu/tensor_ops.py:119-204; it also carries AssignOp between differently
    laid-out tensors, gputransform.py:393-395).  A flex16 copy moves mantissas, so the destination
    shares the source's exponent (the reference propagates the FlexEntry through a dimshuffle the
    same way, ngraph/transformers/passes/flexpass.py:32-48)."""
    kind = "dimshuffle"
    launches = 1

    def __init__(self, index, op, t, src_view, dst_view, axes):
        super(DimshuffleStep, self).__init__(index, op)
        self.in_views = [src_view]
        self.out_views = [dst_view]
        self.lengths = [a.length for a in axes]
        self.src_strides = [src_view.stride_of(a) for a in axes]
        self.dst_strides = [dst_view.stride_of(a) for a in axes]
        if len(self.lengths) > 8:
            raise ValueError("Unhandled op: dimshuffle of more than 8 axes")
        if src_view.buffer.flex != dst_view.buffer.flex:
            raise ValueError("dimshuffle between tensors of different storage types")
        self.elem_bytes = 2 if src_view.buffer.flex else 4
        self.owns_version = True

    def output_buffers(self):
        return []          # no exponent of its own to manage

    def launch(self, t):
        sv, dv = self.in_views[0], self.out_views[0]
        lib.dimshuffle(self._ptr(sv), self._ptr(dv), self.elem_bytes, self.lengths,
                       self.src_strides, self.dst_strides, t.stream.cuda_stream)
        t.kernel_launches += 1


class CommStep(_Step):
    """One tensor's share of a bucketed allreduce (see comm.py).  The tensor lives inside the
    flat fp32 arena; when this step is the last of its bucket the collective for the whole bucket
    is started.  In flex mode the int16 gradient is first de-quantised into the arena."""
    kind = "comm"
    launches = 0

    def __init__(self, index, op, t, src_view, arena_buffer):
        super(CommStep, self).__init__(index, op)
        self.key = id(arena_buffer)
        self.src_view = src_view            # flex: the int16 tensor to de-quantise; else None
        self.arena_buffer = arena_buffer    # fp32 Buffer placed in the arena
        self.in_views = [src_view] if src_view is not None else []
        self.out_views = []
        self.closes_bucket = None           # set when the bucket plan is known
        self.launches = 1 if src_view is not None else 0

    def output_buffers(self):
        return []

    def writes(self):
        return [self.arena_buffer]

    def launch(self, t):
        if self.src_view is not None:
            v = self.src_view
            lib.check(lib.raw().b2_flex_dequantize(
                self._ptr(v), self.arena_buffer.ptr(), v.buffer.size, t._table.data_ptr(),
                t._slot_for_read(v.buffer, self), t.stream.cuda_stream))
            t.kernel_launches += 1
        if t._recording:
            return          # a graph is being recorded: the exchange is issued between replays
        t._allreduce.produced(self.key)
        if self.closes_bucket is not None:
            t._allreduce.bucket_ready(self.closes_bucket)
