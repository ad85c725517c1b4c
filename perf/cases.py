"""The workloads this backend is timed on: the benchmark configurations, through the calls a
user's program makes, over the range of sizes such programs use.

Five kinds of work:

  mlp    one SGD step of a three-layer perceptron with softmax cross-entropy (configuration 1),
         a captured computation fed with host arrays, as the examples feed it: a few dozen small
         kernels, so launches and the host side of a call count
  ew     y = tanh(a*x + b) * sigmoid(c), its row sums and row maxima of |y| (configuration 2),
         a captured computation; x arrives as a device tensor, a, b and c stay on the device
  gemm   C = A.B through the C ABI, fp32 or flex16 (configuration 3 and the dense layers)
  infer  ResNet inference (configuration 4), a captured computation fed from pinned host memory
         and read back, as a serving loop calls it
  train  one momentum-SGD step of the same network (configuration 5), a captured computation fed
         with device tensors

fp32 and flex16 (int16 mantissas with one exponent per tensor) are both in everyday use for all
of them.  Batches that are a multiple of 128 are the training sizes; serving and the last batch
of an epoch bring any size.
"""
import ctypes
import math

import numpy as np
import torch

import ngraph_python_b200 as ng
from ngraph_python_b200 import configs, lib


def listed():
    return [
        # configuration 1 as it stands
        dict(name="mlp_fp32_b128", kind="mlp", flex=False, n=128, hidden=512),
        # the same step in flex16 on an odd, small batch
        dict(name="mlp_flex16_b50", kind="mlp", flex=True, n=50, hidden=300),
        # configuration 2 at full size in both storage types, and a small odd-sized one
        dict(name="ew_fp32_8192x16384", kind="ew", flex=False, rows=8192, cols=16384),
        dict(name="ew_flex16_8192x16384", kind="ew", flex=True, rows=8192, cols=16384),
        dict(name="ew_flex16_333x1001", kind="ew", flex=True, rows=333, cols=1001),
        # configuration 3: its largest flex16 size, its middle fp32 size
        dict(name="gemm_flex16_8192", kind="gemm", flex=True, layout="nn", m=8192, n=8192, k=8192),
        dict(name="gemm_fp32_4096", kind="gemm", flex=False, layout="nn", m=4096, n=4096, k=4096),
        # a dense layer's products: the gradient of a weight matrix (transposed operand, odd sizes)
        # and the forward product of a 784-512 layer
        dict(name="gemm_fp32_1000x777x1500_nt", kind="gemm", flex=False, layout="nt",
             m=1000, n=777, k=1500),
        dict(name="gemm_flex16_512x128x784", kind="gemm", flex=True, layout="nn",
             m=512, n=128, k=784),
        # configuration 4 as it stands, and a ragged serving batch in fp32
        dict(name="infer_flex16_b256", kind="infer", flex=True, n=256, blocks=3),
        dict(name="infer_fp32_b100", kind="infer", flex=False, n=100, blocks=3),
        # configuration 5: the whole global batch on one GPU
        dict(name="train_flex16_b1024", kind="train", flex=True, n=1024, blocks=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "ew", "gemm", "infer", "train"])
    flex = rng.random() < 0.6
    if kind == "mlp":
        return dict(kind=kind, flex=flex, n=_log(rng, 16, 1024), hidden=_log(rng, 64, 1024))
    if kind == "ew":
        return dict(kind=kind, flex=flex, rows=_log(rng, 16, 8192), cols=_log(rng, 64, 16384))
    if kind == "gemm":
        top = 8192 if flex else 4096
        return dict(kind=kind, flex=flex, layout=rng.choice(["nn", "nt", "tn"]),
                    m=_log(rng, 16, top), n=_log(rng, 16, top), k=_log(rng, 16, top))
    if kind == "infer":
        # serving: any number of images up to the configuration's batch
        return dict(kind=kind, flex=flex, n=_log(rng, 1, 256), blocks=rng.choice([1, 2, 3]))
    # training: whole multiples of 128 images three times out of four
    n = 128 * rng.randint(1, 8) if rng.random() < 0.75 else _log(rng, 16, 256)
    if not flex:
        n = min(n, 512)
    return dict(kind=kind, flex=flex, n=n, blocks=rng.choice([1, 2, 3]))


# ---- the work and its tolerance -------------------------------------------------------------------
def _convolutions(blocks):
    """(C, input side, K, output side, R) of every convolution of the network."""
    out, size, cin = [(3, 32, 16, 32, 3)], 32, 16
    for s, width in enumerate((16, 32, 64)):
        for b in range(blocks):
            before = size
            if b == 0 and s > 0:
                size //= 2
            out.append((cin, before, width, size, 3))
            out.append((width, size, width, size, 3))
            if b == 0:
                out.append((cin, before, width, size, 1))
            cin = width
    return out


def work(case):
    """What a pass cannot do without.  Tensor-core products are counted at the 16-bit rate: a
    flex16 multiply-add is four int8 products at twice that rate (8 / 2), an fp32 one the three
    TF32 products that carry its precision at half of it (6 * 2)."""
    flex = case["flex"]
    size, mac = (2, 4) if flex else (4, 12)
    if case["kind"] == "mlp":
        n, h = case["n"], case["hidden"]
        weights = 784 * h + h * h + 10 * h + 2 * h + 10
        macs = n * (2 * 784 * h + 3 * h * h + 3 * 10 * h)
        return {"bytes": 794 * n * 4 + 2 * weights * size, "flops": mac * macs}
    if case["kind"] == "ew":
        elems = case["rows"] * case["cols"]
        return {"bytes": 4 * elems + (4 * elems + 2 * case["rows"]) * size, "flops": 12 * elems}
    if case["kind"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": (m * k + k * n + m * n) * size, "flops": mac * m * n * k}
    n = case["n"]
    convs = _convolutions(case["blocks"])
    acts = sum(c * i * i + k * o * o for c, i, k, o, r in convs) * n
    filters = sum(c * r * r * k for c, i, k, o, r in convs)
    macs = sum(c * r * r * k * o * o for c, i, k, o, r in convs) * n
    if case["kind"] == "infer":
        return {"bytes": (acts + filters) * size + (3 * 1024 + 20) * n * 4, "flops": mac * macs}
    # forward, input gradient, filter gradient: every layer's tensors three times; per weight
    # its gradient, itself, its velocity and the compensation term read and written
    return {"bytes": (3 * acts + 8 * filters) * size + (3 * 1024 + 10) * n * 4,
            "flops": 3 * mac * macs}


def tolerance(case):
    flex, kind = case["flex"], case["kind"]
    if kind == "gemm":
        # flex16 products are exact integers, rounded once; fp32 sums carry about 21 bits
        return "exact" if flex else {"rel": 1e-5, "max": 1e-4}
    if kind == "ew":
        # one mantissa step where the value lies on a rounding boundary
        return {"rel": 1e-4, "max": 1e-3, "differ": 2e-3} if flex else {"rel": 2e-6, "max": 1e-4}
    if kind == "mlp":
        return {"rel": 3e-4, "max": 1e-2, "differ": 1e-2} if flex else {"rel": 2e-5, "max": 1e-3}
    if kind == "infer":
        # twenty layers, each rounded to 16 bits
        return {"rel": 2e-3, "max": 2e-2} if flex else {"rel": 5e-5, "max": 2e-3}
    # activations close to zero change the side of their ReLU with the last bit of a sum
    return {"rel": 5e-4, "max": 2e-2, "differ": 1e-2} if flex else {"rel": 1e-4, "max": 1e-2}


# ---- what a program has in hand --------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _pinned(shape, values):
    p = torch.empty(shape, dtype=torch.float32).pin_memory()
    p.copy_(values.reshape(shape))
    return p.numpy()


def _transformer(flex):
    return ng.transformers.make_transformer_factory("b200", flex=flex)()


def _stored(t, op):
    """The device tensor an op's value is kept in."""
    return t.device_tensor(op).view.buffer.tensor


def _prepare_mlp(case, seed):
    n, h = case["n"], case["hidden"]
    r = np.random.RandomState(0)
    N, F, H1, H2, Y = [ng.make_axis(d, name=nm) for d, nm in
                       zip((n, 784, h, h, 10), ("N", "F", "H1", "H2", "Y"))]
    x, t = ng.placeholder([F, N]), ng.placeholder([Y, N])

    def layer(out_ax, in_ax):
        w = r.standard_normal((out_ax.length, in_ax.length)) * np.sqrt(2.0 / in_ax.length)
        return (ng.variable([out_ax, in_ax], initial_value=w.astype(np.float32)),
                ng.variable([out_ax], initial_value=np.zeros(out_ax.length, np.float32)))
    (w1, b1), (w2, b2), (w3, b3) = layer(H1, F), layer(H2, H1), layer(Y, H2)
    z1 = ng.dot(w1, x) + b1
    a1 = ng.maximum(z1, 0.0)
    z2 = ng.dot(w2, a1) + b2
    a2 = ng.maximum(z2, 0.0)
    z3 = ng.dot(w3, a2) + b3
    e = ng.exp(z3 - ng.max(z3, reduction_axes=[Y]))
    p = e / ng.sum(e, reduction_axes=[Y])
    loss = ng.sum(ng.negative(ng.sum(t * ng.safelog(p), reduction_axes=[Y])),
                  reduction_axes=[N]) * (1.0 / n)
    d3 = (p - t) * (1.0 / n)
    d2 = ng.dot(w3, d3) * ng.greater(z2, 0.0)
    d1 = ng.dot(w2, d2) * ng.greater(z1, 0.0)
    grads = [(w3, ng.dot(d3, a2)), (b3, ng.sum(d3, reduction_axes=[N])),
             (w2, ng.dot(d2, a1)), (b2, ng.sum(d2, reduction_axes=[N])),
             (w1, ng.dot(d1, x)), (b1, ng.sum(d1, reduction_axes=[N]))]
    step = ng.sequential([ng.assign(w, w - 0.01 * g) for w, g in grads] + [loss])
    tr = _transformer(case["flex"])
    comp = tr.computation([step, b1, b2, w3, b3], x, t)
    rs = np.random.RandomState(seed % (1 << 31))
    feed = [rs.uniform(0, 1, (784, n)).astype(np.float32),
            np.ascontiguousarray(np.eye(10, dtype=np.float32)[rs.randint(0, 10, n)].T)]
    comp(*feed)
    comp.capture()
    return dict(kind="call", comp=comp, feed=feed, keep=tr,
                stored=[_stored(tr, w1), _stored(tr, w2)])


def _prepare_ew(case, seed):
    R, C = ng.make_axis(case["rows"], name="R"), ng.make_axis(case["cols"], name="C")
    x = ng.placeholder([R, C])
    a, b, c = [ng.variable([R, C]) for _ in range(3)]
    yvar = ng.persistent_tensor([R, C])
    y = ng.tanh(a * x + b) * ng.sigmoid(c)
    out = ng.sequential([ng.assign(yvar, y), ng.sum(y, reduction_axes=[C])])
    tr = _transformer(case["flex"])
    comp = tr.computation([out, ng.max(ng.absolute(y), reduction_axes=[C])], x)
    tr.initialize()
    g = _generator(seed)
    make = lambda: torch.randn((case["rows"], case["cols"]), device="cuda", generator=g)  # noqa: E731
    for v in (a, b, c):
        tr.device_tensor(v)[...] = make()
    feed = [make()]
    comp(*feed)
    comp.capture()
    return dict(kind="call", comp=comp, feed=feed, keep=tr, stored=[_stored(tr, yvar)])


def _prepare_gemm(case, seed):
    m, n, k, flex = case["m"], case["n"], case["k"], case["flex"]
    g = _generator(seed)
    a_shape = (k, m) if case["layout"] == "tn" else (m, k)
    b_shape = (n, k) if case["layout"] == "nt" else (k, n)

    def make(shape):
        if flex:
            return torch.randint(-32767, 32768, shape, device="cuda", generator=g,
                                 dtype=torch.int16)
        return torch.randn(shape, device="cuda", generator=g)
    a, b = make(a_shape), make(b_shape)
    c = torch.zeros((m, n), dtype=torch.int16 if flex else torch.float32, device="cuda")
    nbytes = lib.gemm_scratch_bytes(flex, m, n, k)
    scratch = torch.empty((nbytes + 1024,), dtype=torch.uint8, device="cuda")
    aligned = scratch.data_ptr() + (-scratch.data_ptr()) % 1024
    status = torch.zeros((1,), dtype=torch.int32, device="cuda")
    strides = ((1, m) if case["layout"] == "tn" else (k, 1)) + \
        ((1, k) if case["layout"] == "nt" else (n, 1))
    keep = [a, b, c, scratch, status]
    if not flex:
        args = (a.data_ptr(), strides[0], strides[1], b.data_ptr(), strides[2], strides[3],
                c.data_ptr(), n, m, n, k, aligned, nbytes, status.data_ptr())
        return dict(kind="f32", call=lib.raw().b2_gemm_f32, args=args, keep=keep, out=[c])
    # exponents as configuration 3 has them; the result's holds sums of k random products
    # with five standard deviations to spare
    dec_c = 15 + 12 - max(0, math.ceil(math.log2(5 * math.sqrt(k) * 32767 ** 2 / 3 / 32767)))
    table = torch.tensor([[2.0 ** -d, 2.0 ** d] for d in (15, 12, dec_c)], dtype=torch.float32,
                         device="cuda")
    stats = torch.zeros((3,), dtype=torch.int32, device="cuda")
    probe = torch.zeros((1,), dtype=torch.int64, device="cuda")
    args = (a.data_ptr(), strides[0], strides[1], b.data_ptr(), strides[2], strides[3],
            c.data_ptr(), n, m, n, k, table.data_ptr(), 0, 1, 2, stats.data_ptr(), aligned,
            nbytes, probe.data_ptr(), status.data_ptr(), 0)
    return dict(kind="flex16", call=lib.raw().b2_gemm_flex16, args=args,
                keep=keep + [table, probe], out=[c, stats])


def _prepare_infer(case, seed):
    n = case["n"]
    outs, params, _ = configs.resnet20(ng, n=n, hw=32, blocks=case["blocks"])
    tr = _transformer(case["flex"])
    comp = tr.computation(outs, *params)
    images = torch.randn((3, 1, 32, 32, n), device="cuda", generator=_generator(seed))
    feed = [_pinned((3, 1, 32, 32, n), images)]
    comp(*feed)
    comp.capture()
    return dict(kind="call", comp=comp, feed=feed, keep=tr, stored=[])


def _trainable(op):
    seen, todo, found = set(), [op], []
    while todo:
        o = todo.pop()
        if id(o) in seen:
            continue
        seen.add(id(o))
        if getattr(o, "is_trainable", False):
            found.append(o)
        todo.extend(o.all_deps)
    return sorted(found, key=lambda v: v.uid)


def _prepare_train(case, seed):
    n = case["n"]
    # (untrained and without batch norm the network needs a rate at which it does not diverge)
    outs, params, vals = configs.resnet_train_step(ng, global_n=n, hw=32, blocks=case["blocks"],
                                                   lr=0.001)
    tr = _transformer(case["flex"])
    comp = tr.computation(outs, *params)      # the loss, first and last filters, linear weights
    g = _generator(seed)
    images = torch.randn(vals[0].shape, device="cuda", generator=g)
    classes = torch.randint(0, 10, (n,), device="cuda", generator=g)
    labels = torch.zeros((10, n), device="cuda").scatter_(0, classes[None], 1.0)
    feed = [images, labels]
    comp(*feed)
    comp.capture()
    # fp32: every weight as well.  In flex16 a weight near a rounding boundary moves a whole
    # mantissa step with the last bit of its gradient, which says nothing where a tensor has ten
    # values; what the computation returns are real values, and the next step's loss depends on
    # all weights.
    stored = [] if case["flex"] else [_stored(tr, w) for w in _trainable(outs[0])]
    return dict(kind="call", comp=comp, feed=feed, keep=tr, stored=stored)


def prepare(case, seed):
    return {"mlp": _prepare_mlp, "ew": _prepare_ew, "gemm": _prepare_gemm,
            "infer": _prepare_infer, "train": _prepare_train}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "call":
        got = state["comp"](*state["feed"])
        return list(got if isinstance(got, tuple) else (got,)) + state["stored"]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    lib.check(state["call"](*state["args"], stream))
    return state["out"]
