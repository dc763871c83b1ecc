"""Worker of tests/test_gemm_split_gpu.py::test_first_product_of_a_process_is_captured: the process' first product is recorded into a
graph (arguments: dtype, columns, K, N), which is then looked at and run through the driver API, as a program does that has graphs of
its own.  Prints one JSON line with the worst NMSE and what the graph is made of."""
import ctypes as C
import json
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

from oracle import sgref  # noqa: E402
from scrapgpulibrary_b200 import capi  # noqa: E402
from tests import util as U  # noqa: E402


def main(dtype, m, k, n):
    capi.require_device()
    cu = C.CDLL("libcuda.so.1")

    def ok(status):
        assert status == 0, f"driver API: {status}"

    wq = U.quantize(dtype, U.seeded_weights(11 + dtype, n, k))
    xs = [U.seeded_acts(20 + i, m, k) for i in range(3)]
    want = [sgref.mul_mat(dtype, wq, k, x) for x in xs]
    stream = capi.Stream(0)
    wb, xb = U.to_device(capi, stream, capi.pack(dtype, k, wq)), U.to_device(capi, stream, xs[0])
    yb = [capi.Buffer(4 * n * m) for _ in range(2)]
    stream.sync()
    graph, copy, outer = C.c_void_p(), C.c_void_p(), C.c_void_p()
    ok(cu.cuStreamBeginCapture_v2(stream.handle, 1))   # thread-local, like sm100_graph_begin
    for y in yb:
        capi.mul_mat(stream, dtype, U.PACKED, wb, k, n, xb, m, y)
    ok(cu.cuStreamEndCapture(stream.handle, C.byref(graph)))
    count = C.c_size_t()
    ok(cu.cuGraphGetNodes(graph, None, C.byref(count)))
    nodes = (C.c_void_p * count.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, C.byref(count)))
    kinds = set()
    for node in nodes:
        kind = C.c_int()
        ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
        kinds.add(kind.value)
    # a copy, a graph that holds the graph, and two instances of the original; the originals go before they run
    ok(cu.cuGraphClone(C.byref(copy), graph))
    ok(cu.cuGraphCreate(C.byref(outer), 0))
    child = C.c_void_p()
    ok(cu.cuGraphAddChildGraphNode(C.byref(child), outer, None, C.c_size_t(0), graph))
    execs = []
    for g in (graph, graph, copy, outer):
        e = C.c_void_p()
        ok(cu.cuGraphInstantiateWithFlags(C.byref(e), g, C.c_ulonglong(0)))
        execs.append(e)
    for g in (graph, copy, outer):
        ok(cu.cuGraphDestroy(g))
    worst = 0.0

    def check(x):
        nonlocal worst
        stream.sync()
        for y in yb:
            got = y.download(stream, np.float32, n * m).reshape(m, n)
            worst = max(worst, float(sgref.nmse(got, x)) if np.isfinite(got).all() else float("inf"))
            y.fill(stream, 0xff)

    for i, x in enumerate(xs):
        for e in execs:
            xb.upload(stream, x)
            ok(cu.cuGraphLaunch(e, stream.handle))
            check(want[i])
    for e in execs:
        ok(cu.cuGraphExecDestroy(e))
    for i in range(2):   # and outside a capture, after the graphs are gone
        xb.upload(stream, xs[i])
        for y in yb:
            capi.mul_mat(stream, dtype, U.PACKED, wb, k, n, xb, m, y)
        check(want[i])
    g = capi.Graph(stream)
    with g:
        for y in yb:
            capi.mul_mat(stream, dtype, U.PACKED, wb, k, n, xb, m, y)
    g.launch()
    check(want[1])
    g.destroy()
    stream.close()
    print(json.dumps({"worst": worst, "kinds": sorted(kinds)}))


if __name__ == "__main__":
    main(*(int(a) for a in sys.argv[1:5]))
