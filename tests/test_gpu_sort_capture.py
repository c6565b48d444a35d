"""ypdq_sort_hits under stream capture: kernels alone, whatever the number of hits, so that the
graph can be instantiated twice, cloned and used as a child graph. Past 512 hits that is the
in-place sort, which also runs where its second buffer cannot be had."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNEL_NODE = 0  # cudaGraphNodeTypeKernel


@pytest.fixture(scope="module")
def rt(ctx):
    for line in open("/proc/self/maps"):
        if "libcudart.so" in line:
            return ctypes.CDLL(line.split()[-1])
    raise RuntimeError("libcudart not loaded")


def node_types(rt, graph):
    n = ctypes.c_size_t()
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    kind = ctypes.c_int()
    out = set()
    for node in nodes:
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        out.add(kind.value)
    return out


@pytest.mark.parametrize("n", [100, 500, 513, 1025, 2048, 2049, 3001, 8193, 100_001])
def test_captured_sort_is_a_plain_graph(ctx, yp, rt, n):
    rng = np.random.default_rng(n)
    h = np.zeros(n, yp.HIT_DTYPE)
    h["index"] = rng.integers(0, n // 2, n, dtype=np.uint64) << np.uint64(33)
    h["query"] = rng.permutation(n)
    h["distance"] = rng.integers(0, 257, n)
    want = h[np.lexsort((h["query"], h["index"]))]
    d = ctx.alloc((n + 2) * 16)
    guard = np.full(32, 0xCD, np.uint8)
    d.upload(guard, offset=16 * n)
    s = ctx.stream()
    graph, copy, parent = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(s, 1) == 0  # thread-local mode
    yp.core.sort_hits_device(ctx, d, n, stream=s)
    assert rt.cudaStreamEndCapture(s, ctypes.byref(graph)) == 0
    assert node_types(rt, graph) == {KERNEL_NODE}
    assert rt.cudaGraphClone(ctypes.byref(copy), graph) == 0
    assert rt.cudaGraphCreate(ctypes.byref(parent), 0) == 0
    node = ctypes.c_void_p()
    assert rt.cudaGraphAddChildGraphNode(ctypes.byref(node), parent, None, ctypes.c_size_t(0),
                                         graph) == 0
    execs = []
    for g in (graph, graph, copy, parent):
        e = ctypes.c_void_p()
        assert rt.cudaGraphInstantiate(ctypes.byref(e), g, ctypes.c_ulonglong(0)) == 0
        execs.append(e)
    for e in execs:
        d.upload(h)
        assert rt.cudaGraphLaunch(e, s) == 0
        ctx.sync(s)
        assert np.array_equal(d.download((n,), yp.HIT_DTYPE), want)
    assert np.array_equal(d.download((32,), np.uint8, offset=16 * n), guard)
    for e in execs:
        rt.cudaGraphExecDestroy(e)
    for g in (parent, copy, graph):
        rt.cudaGraphDestroy(g)
    ctx.lib.ypdq_stream_destroy(ctx.handle, s)
