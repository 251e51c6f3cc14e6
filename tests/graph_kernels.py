"""The kernels that a call puts into a stream, from a capture of the call:
names and grids, through the CUDA driver API (nothing runs)."""
from __future__ import annotations

import ctypes as C


class KernelParams(C.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


KERNEL_NODE = 0  # CU_GRAPH_NODE_TYPE_KERNEL
RELAXED = 2      # CU_STREAM_CAPTURE_MODE_RELAXED


def captured_kernels(stream, call):
    """[(mangled name, (grid x, y, z))] of the kernels that call() launches on
    `stream` (a torch stream, not the default one), in no particular order."""
    d = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, f"CUDA driver error {rc}"

    s, graph = C.c_void_p(stream.cuda_stream), C.c_void_p()
    ok(d.cuStreamBeginCapture_v2(s, C.c_int(RELAXED)))
    try:
        call()
    finally:
        rc = d.cuStreamEndCapture(s, C.byref(graph))
    ok(rc)
    try:
        count = C.c_size_t()
        ok(d.cuGraphGetNodes(graph, None, C.byref(count)))
        nodes = (C.c_void_p * count.value)()
        ok(d.cuGraphGetNodes(graph, nodes, C.byref(count)))
        found = []
        for raw in nodes:
            node, kind = C.c_void_p(raw), C.c_int()
            ok(d.cuGraphNodeGetType(node, C.byref(kind)))
            if kind.value != KERNEL_NODE:
                continue
            p, name = KernelParams(), C.c_char_p()
            ok(d.cuGraphKernelNodeGetParams_v2(node, C.byref(p)))
            if p.func:
                ok(d.cuFuncGetName(C.byref(name), C.c_void_p(p.func)))
            else:
                ok(d.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)))
            found.append((name.value.decode(), tuple(p.grid)))
        return found
    finally:
        d.cuGraphDestroy(graph)
