"""Which kernels a call launches, read from a recording of it as a CUDA graph (nothing of the recording runs)."""
import ctypes
import re


class _KernelNode(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared_bytes", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kernel", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def launched(call):
    """[(mangled name, blocks)] of the kernels that call() launches on the current stream.  It is called once for
    itself first: one-time set-up must not happen inside a recording."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    handle, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cu.cuGraphGetNodes(handle, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(handle, nodes, ctypes.byref(count)) == 0
    out = []
    for n in nodes:
        kind, at, name = ctypes.c_int(-1), _KernelNode(), ctypes.c_char_p()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(n), ctypes.byref(kind)) == 0
        if kind.value != 0:
            continue
        assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(n), ctypes.byref(at)) == 0
        rc = cu.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(at.func)) if at.func else \
            cu.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(at.kernel))
        assert rc == 0
        out.append((name.value.decode(), at.grid[0] * at.grid[1] * at.grid[2]))
    return out


def qgemm_form(call, tiles_of_64=0):
    """(columns of a tile, "one" | "pair" | CTAs that share a tile's K) of the one tiled quant_dot that call() launches;
    tiles_of_64: the result's tiles of 128 x 64."""
    found = [(m, blocks) for name, blocks in launched(call)
             for m in [re.search(r"qgemm_kernelILi(\d+)ELb[01]E(?:i|f|6__half)Lb[01]ELb([01])ELb([01])E", name)] if m]
    assert len(found) == 1, found
    m, blocks = found[0]
    return int(m[1]), "pair" if m[2] == "1" else (blocks // tiles_of_64 if m[3] == "1" else "one")
