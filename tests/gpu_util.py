"""Helpers shared by the GPU parity tests (torch <-> numpy bit views, wire minting)."""
from __future__ import annotations

import numpy as np
import torch

import mlx_kquant_b200 as kq
from oracle import kq_oracle
from oracle.kq_oracle import GEOMETRY

# codecs with a host encoder in this package
HOST_ENCODED = {"q2_k", "q3_k", "q4_k", "q5_k", "q6_k", "q4_0", "q4_1", "q5_0", "q5_1", "q8_0", "iq4_nl", "iq4_xs",
                "iq2_xxs"}
TORCH_DT = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def t2np_bits(t: torch.Tensor) -> np.ndarray:
    """Device tensor -> numpy array of raw bit patterns (uint32 / uint16)."""
    t = t.detach().cpu().contiguous()
    if t.dtype == torch.float32:
        return t.view(torch.int32).numpy().view(np.uint32)
    return t.view(torch.int16).numpy().view(np.uint16)


def np_bits(a: np.ndarray) -> np.ndarray:
    return a.view(np.uint32) if a.dtype == np.float32 else a.view(np.uint16)


def x_to_torch(x_f32: np.ndarray, dt: str, device="cuda") -> tuple[torch.Tensor, np.ndarray]:
    """float32 numpy -> (torch tensor of dtype dt on device, the oracle-side storage array)."""
    t = torch.from_numpy(x_f32).to(TORCH_DT[dt])
    if dt == "f32":
        store = x_f32.copy()
    elif dt == "f16":
        store = t.numpy().copy()
    else:
        store = t.view(torch.int16).numpy().view(np.uint16).copy()
    return t.to(device), store


def y_to_f32(y: torch.Tensor) -> np.ndarray:
    return y.detach().float().cpu().numpy()


synthetic_wire = kq_oracle.synthetic_wire


def mint_wire(codec: str, W: np.ndarray, imatrix=None) -> np.ndarray:
    """Really-encoded wire bytes from the reference encoder when its library is
    present (and the codec has an encoder: mxfp4 / nvfp4 are decode-only in the
    reference, src/kquant_codec.cpp:33-34), else from this package's host encoder (byte-identical with it,
    tests/test_quantize.py), else synthetic valid bytes of the same shape."""
    if kq_oracle.Ref.available() and codec not in kq_oracle.DECODE_ONLY:
        if imatrix is None and GEOMETRY[codec][3]:
            imatrix = np.ones(W.shape[-1], np.float32)
        return kq_oracle.Ref().quantize(W, codec, imatrix)
    if codec in HOST_ENCODED:
        im = torch.from_numpy(imatrix) if imatrix is not None else (torch.ones(W.shape[-1]) if GEOMETRY[codec][3] else None)
        return kq.quantize(torch.from_numpy(np.ascontiguousarray(W, np.float32)), codec, im)[0].numpy()
    return synthetic_wire(codec, W.shape[0], W.shape[1], seed=int(abs(W[0, 0]) * 1e6) % 9973)


def kernels(call) -> list[str]:
    """Mangled names of the kernels that `call` launches, in some order: it is captured into a graph, which is not run."""
    import ctypes as C

    call()   # (what is set up once is no part of a capture)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call()
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, f"driver call: {rc}"

    raw, count = C.c_void_p(int(graph.raw_cuda_graph())), C.c_size_t(0)
    ok(cu.cuGraphGetNodes(raw, None, C.byref(count)))
    nodes = (C.c_void_p * count.value)()
    ok(cu.cuGraphGetNodes(raw, nodes, C.byref(count)))

    class Params(C.Structure):   # CUDA_KERNEL_NODE_PARAMS of version 2
        _fields_ = [("func", C.c_void_p), ("shape", C.c_uint * 7), ("params", C.c_void_p), ("extra", C.c_void_p),
                    ("kern", C.c_void_p), ("ctx", C.c_void_p), ("room", C.c_uint64 * 8)]
    names = []
    for node in nodes:
        kind = C.c_int()
        ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
        if kind.value != 0:   # CU_GRAPH_NODE_TYPE_KERNEL
            continue
        p, name = Params(), C.c_char_p()
        ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)))
        ok(cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)) if p.func else cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)))
        names.append(name.value.decode())
    return names


def product_kernels(codec: str, m: int, n: int, k: int, dt: str) -> str:
    """The kernels that x [m, k] . w [n, k]^T launches, one string."""
    wpb, bpb = GEOMETRY[codec][0], GEOMETRY[codec][1]
    x = torch.zeros(m, k, dtype=TORCH_DT[dt], device="cuda")
    w = torch.zeros(n, k // wpb * bpb, dtype=torch.uint8, device="cuda")
    return " ".join(kernels(lambda: kq.quantized_matmul(x, w, None, codec)))
