"""Which launches serve a call, as a captured graph shows them (kernels, cooperative or not, thread blocks of a cluster), and that
every form gives the same bits: cooperative launches switched off, refused, in a second context."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from cuda.bindings import runtime as rt  # noqa: E402

from niti_b200 import ops  # noqa: E402
from oracle import niti_oracle as O  # noqa: E402

DEV = "cuda:0"


def rnd8(rng, shape, lo=-127):
    return rng.integers(lo, 128, size=shape).astype(np.int8)


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def same(got, want):
    assert np.array_equal(got.cpu().numpy(), want)


def kernels(fn):
    """(cooperative, thread blocks of a cluster) of every kernel that fn() enqueues, and whatever else it does once."""
    fn()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1:]
    raw = rt.cudaGraph_t(graph.raw_cuda_graph())
    n = ok(rt.cudaGraphGetNodes(raw))[1]
    found = []
    for node in ok(rt.cudaGraphGetNodes(raw, n))[0]:
        if ok(rt.cudaGraphNodeGetType(node))[0] != rt.cudaGraphNodeType.cudaGraphNodeTypeKernel:
            continue
        value = lambda attr: ok(rt.cudaGraphKernelNodeGetAttribute(node, attr))[0]  # noqa: E731
        found.append((bool(value(rt.cudaLaunchAttributeID.cudaLaunchAttributeCooperative).cooperative),
                      max(1, value(rt.cudaLaunchAttributeID.cudaLaunchAttributeClusterDimension).clusterDim.x)))
    return found


class Layer:
    """One convolution layer's three calls, each with words of its own, and what they must give."""

    def __init__(self, N, H, W, C, K):
        rng = np.random.default_rng(N + H + W + C + K)
        self.x, self.w, self.err = rnd8(rng, (N, H, W, C), 0), rnd8(rng, (K, 3, 3, C)), rnd8(rng, (N, H, W, K))
        self.dx, self.dw, self.derr = cu(self.x), cu(self.w), cu(self.err)
        self.z = torch.zeros((), dtype=torch.int32, device=DEV)
        self.fwd, self.bwd, self.upd = ops.new_requant_state(DEV), ops.new_requant_state(DEV), ops.new_update_state(DEV)

    def forward(self):
        return ops.conv_fprop_fused(self.dx, self.dw, self.fwd, 1, 0, None, 0, 0, False, self.z, self.z)[0]

    def backward(self):
        return ops.conv_dgrad_fused(self.derr, self.dw, self.bwd, 1, 0, None, 0, 0, self.z, self.z)[0]

    def update(self):
        w = self.dw.clone()
        return ops.conv_wgrad_update(self.dx, self.derr, w, 1, 5, 2, None, 18, self.upd)[0], w

    def check(self):
        for _ in range(2):
            same(self.forward(), O.act_calc(O.conv_fprop(self.x, self.w), 0, 0)[0])
            same(self.backward(), O.err_calc(O.conv_dgrad(self.err, self.w), 0)[0])
            g, w = self.update()
            want = O.conv_wgrad(self.x, self.err, 3, 3, 1)
            same(g, want)
            same(w, O.weight_update(self.w, want, 5, 2)[0])
        ops.check_status(DEV)


@pytest.fixture
def no_cooperative_launches():
    old = ops.set_cooperative_launch(False)
    yield
    ops.set_cooperative_launch(old)


def test_without_cooperative_launches_only_the_parked_layers_meet_at_a_barrier(no_cooperative_launches):
    """NITI_OPT_COOPERATIVE_LAUNCH = 0: a layer whose tiles do not fit in tensor memory, a layer of few tiles and the weight gradient run
    without any thread block waiting for another: prediction and conditional second launch, one thread block to a tile, gradient
    and update apart."""
    large, few = Layer(75, 32, 32, 16, 128), Layer(1, 8, 8, 512, 512)
    assert kernels(large.forward) == [(False, 1)] * 2
    assert kernels(few.forward) == kernels(few.backward) == [(False, 1)]
    copy_and_update = kernels(few.update)  # the copy of the weights is a kernel or a copy node, as torch likes it
    assert copy_and_update[-2:] == [(False, 1)] * 2
    large.check()
    few.check()
    old = ops.set_accumulator_parking(False)
    try:
        assert kernels(few.forward) == [(False, 1)] * 2
        few.check()
    finally:
        ops.set_accumulator_parking(old)


CONTEXTS = """
import ctypes as C, sys
import numpy as np
from niti_b200._lib import lib
cu = C.CDLL("libcuda.so.1")
def ok(r):
    assert r == 0, r
ok(cu.cuInit(0))
dev, ctx = C.c_int(), C.c_void_p()
ok(cu.cuDeviceGet(C.byref(dev), 0))
rng = np.random.default_rng(3)
N, H, W, C_, K = 2, 8, 8, 144, 128
x, w, err = (rng.integers(-127, 128, n).astype(np.int8) for n in (N * H * W * C_, K * 9 * C_, N * H * W * K))
def put(a):
    p = C.c_uint64()
    ok(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(a.nbytes)))
    ok(cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes)))
    return p.value
def get(p, shape, type):
    a = np.empty(shape, type)
    ok(cu.cuCtxSynchronize())
    ok(cu.cuMemcpyDtoH_v2(a.ctypes.data_as(C.c_void_p), C.c_uint64(p), C.c_size_t(a.nbytes)))
    return a
def calls():
    dx, dw, de = put(x), put(w), put(err)
    y, g, c = (put(np.zeros(n, t)) for n, t in ((N * H * W * K, np.int8), (K * 9 * C_, np.int32), (K * K, np.int32)))
    words, status, mx = put(np.zeros(8, np.int32)), put(np.zeros(4, np.int32)), put(np.zeros(1, np.int32))
    assert lib.niti_conv_fprop_requant_i8(dx, dw, y, words, None, 0, N, H, W, C_, K, 3, 3, 1, 0, None, 0, 0, 0, None, None, None, None, status, None) == 0, lib.niti_last_cuda_error()
    assert lib.niti_conv_wgrad_accumulate_i8(dx, de, g, N, H, W, C_, K, 3, 3, 1, status, None) == 0, lib.niti_last_cuda_error()
    assert lib.niti_gemm_i8(de, de, c, mx, K, K, N * H * W, 1, 0, status, None) == 0, lib.niti_last_cuda_error()
    r = [get(y, N * H * W * K, np.int8), get(g, K * 9 * C_, np.int32), get(c, K * K, np.int32)]
    assert not get(status, 4, np.int32).any()
    return r
ok(cu.cuDevicePrimaryCtxRetain(C.byref(ctx), dev))
ok(cu.cuCtxSetCurrent(ctx))
first = calls()
assert all(a.any() for a in first)
def same(r):
    assert all(np.array_equal(a, b) for a, b in zip(first, r))
same(calls())
if sys.argv[1] == "second":
    other = C.c_void_p()
    ok(cu.cuCtxCreate_v2(C.byref(other), 0, dev))
    same(calls())
    ok(cu.cuCtxDestroy_v2(other))
else:
    ok(cu.cuDevicePrimaryCtxReset_v2(dev))
    ok(cu.cuDevicePrimaryCtxRetain(C.byref(ctx), dev))
ok(cu.cuCtxSetCurrent(ctx))
same(calls())
"""


@pytest.mark.parametrize("what", ["second", "reset"])
def test_contexts_after_the_first(what):
    """What a kernel is granted belongs to a context: the calls work in a second context of the device, and in the primary one after
    a reset.  In a process of its own, without torch."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CONTEXTS, what], cwd=root, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


SOME_SMS = """
import sys
from torch.cuda.green_contexts import GreenContext
import tests.test_gpu_launch_forms as T
large, few, one, ragged = T.Layer(75, 32, 32, 16, 128), T.Layer(32, 4, 4, 512, 512), T.Layer(1, 8, 8, 512, 512), T.Layer(37, 15, 13, 48, 80)
T.torch.cuda.synchronize()
part = GreenContext.create(32, 0)
part.set_context()
for _ in range(2):
    T.same(large.forward(), T.O.act_calc(T.O.conv_fprop(large.x, large.w), 0, 0)[0])
    T.same(large.backward(), T.O.err_calc(T.O.conv_dgrad(large.err, large.w), 0)[0])
    for l in (few, one):
        T.same(l.forward(), T.O.act_calc(T.O.conv_fprop(l.x, l.w), 0, 0)[0])
        T.same(l.backward(), T.O.err_calc(T.O.conv_dgrad(l.err, l.w), 0)[0])
    g, w = ragged.update()
    T.same(g, T.O.conv_wgrad(ragged.x, ragged.err, 3, 3, 1))
    T.same(w, T.O.weight_update(ragged.w, T.O.conv_wgrad(ragged.x, ragged.err, 3, 3, 1), 5, 2)[0])
T.torch.cuda.synchronize()
part.pop_context()
assert T.kernels(one.forward) == T.kernels(one.backward) == [(True, 8)], T.kernels(one.forward)
assert T.kernels(large.forward) == [(True, 1)]
large.check(), few.check()
"""


def test_calls_on_part_of_the_device():
    """A context of 32 SMs: a launch whose thread blocks have to be resident together and are too many is refused, and the layer goes
    through the form that takes any number of SMs; the whole device afterwards has its own forms.  In a process of its own."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SOME_SMS], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_the_library_counts_its_launches():
    """niti_launch_count against the kernels of a captured graph: gather and product of a thin layer, one launch of a parked, a
    streaming and a shared layer, the conditional second one on the way back, gradient and update in one and in two, an update of two
    layers, a head's step, the input."""
    def counted(fn, torch_kernels=0):
        n = len(kernels(fn)) - torch_kernels
        before = ops.lib.niti_launch_count()
        fn()
        assert ops.lib.niti_launch_count() - before == n, (fn, n)
        return n

    large, few, small = Layer(75, 32, 32, 16, 128), Layer(1, 8, 8, 512, 512), Layer(37, 15, 13, 48, 80)
    assert counted(large.forward) == 1 and counted(few.forward) == 1 and counted(small.forward) == 1
    wide = Layer(75, 32, 32, 128, 16)
    assert counted(wide.backward) == 2 and counted(few.backward) == 1
    g32 = [torch.zeros((n,), dtype=torch.int32, device=DEV) for n in (4096, 512)]
    ws = [torch.zeros((n,), dtype=torch.int8, device=DEV) for n in (4096, 512)]
    assert counted(lambda: ops.update_multi(ws, g32, [1, 2], 5)) == 2
    assert counted(lambda: ops.conv_wgrad_update(small.dx, small.derr, small.dw, 1, 5, 2, None, 18, small.upd)) == 1
    assert counted(lambda: ops.conv_wgrad_update(few.dx, few.derr, few.dw, 1, 5, 2, None, 18, few.upd)) == 2
    rng = np.random.default_rng(1)
    x, w = cu(rnd8(rng, (2, 32, 32, 3))), cu(rnd8(rng, (64, 3, 3, 3)))
    st = ops.new_requant_state(DEV)
    assert counted(lambda: ops.conv_fprop_fused(x, w, st, 1, 0, None, 0, 0, True, small.z, small.z)) == 2
    images = torch.randn(4, 3, 32, 32, device=DEV)
    assert counted(lambda: ops.quantize_input(images)) == 3
    a, b = cu(rnd8(rng, (64, 256))), cu(rnd8(rng, (256, 10)))
    assert counted(lambda: ops.gemm_acc(a, b)) == 1
    ops.check_status(DEV)


def test_the_smoke_step_holds_no_cluster_launch():
    """Its convolutions (128 channels, batch 4, 16x16 and 8x8 maps) keep one thread block to a tile, in every form the step uses."""
    for hw in (16, 8):
        l = Layer(4, hw, hw, 128, 128)
        assert ops.conv_fprop_pool_fused_supported(4, hw, hw, 128, 128, 3, 3, 1)
        pooled = kernels(lambda: ops.conv_fprop_pool_fused(l.dx, l.dw, l.fwd, 1, 0, None, 0, 0, True, l.z, l.z))
        back = kernels(lambda: ops.conv_dgrad_fused(l.derr, l.dw, l.bwd, 1, 0, None, 0, 0, l.z, l.z, relu_mask=l.dx))
        assert pooled + kernels(l.forward) + back == [(True, 1)] * 3
