"""The kernels that a call enqueues, from a capture of the engine's stream into a CUDA graph
(driver API; nothing is executed)."""
import ctypes


class _Params(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("smem", ctypes.c_uint), ("kernelParams", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def captured_kernels(eng, call):
    """[(mangled name, grid, cooperative)] of the kernels that call() enqueues on eng's stream."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")

    def ck(rc):
        assert rc == 0, f"CUDA driver error {rc}"

    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    eng.set_stream(st.cuda_stream)
    graph = ctypes.c_void_p()
    ck(cu.cuStreamBeginCapture_v2(ctypes.c_void_p(st.cuda_stream), 2))  # relaxed
    try:
        call()
    finally:
        rc = cu.cuStreamEndCapture(ctypes.c_void_p(st.cuda_stream), ctypes.byref(graph))
        eng.set_stream(0)
    ck(rc)
    n = ctypes.c_size_t()
    ck(cu.cuGraphGetNodes(graph, None, ctypes.byref(n)))
    nodes = (ctypes.c_void_p * n.value)()
    ck(cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)))
    out = []
    for node in nodes:
        node = ctypes.c_void_p(node)
        kind = ctypes.c_int()
        ck(cu.cuGraphNodeGetType(node, ctypes.byref(kind)))
        if kind.value != 0:  # not a kernel
            continue
        p = _Params()
        ck(cu.cuGraphKernelNodeGetParams_v2(node, ctypes.byref(p)))
        name = ctypes.c_char_p()
        if p.func:
            ck(cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(p.func)))
        else:
            ck(cu.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(p.kern)))
        attr = (ctypes.c_char * 64)()
        ck(cu.cuGraphKernelNodeGetAttribute(node, 2, attr))  # CU_LAUNCH_ATTRIBUTE_COOPERATIVE
        out.append((name.value.decode(), tuple(p.grid), bool(ctypes.c_int.from_buffer(attr).value)))
    ck(cu.cuGraphDestroy(graph))
    return out
