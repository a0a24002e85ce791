"""More than sixteen rows on matrices that are dequantized to fp16 once and multiplied tile by tile (kq_gemm.cu)."""
import numpy as np
import pytest
import torch

from gpu_util import x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu

# (codec, m, n, k): the smallest matrices of the rule with ragged rows and columns, K not a whole number of K-steps,
# K split over a cluster, two row blocks, and an fp16 copy made in two parts (128 MiB)
CASES = [("q5_k", 17, 4099, 1024), ("q8_0", 130, 2051, 2080), ("iq4_xs", 300, 1025, 4096), ("q4_0", 64, 1024, 8192),
         ("q3_k", 513, 4100, 1280), ("q6_k", 40, 2051, 2304), ("q6_k", 1027, 1056, 4096), ("q2_k", 33, 9000, 8192),
         # either side of the shortest K with few rows, and of 256 rows
         ("iq4_xs", 256, 4104, 1024), ("iq4_xs", 257, 4104, 1024), ("q4_0", 100, 8200, 512), ("q4_0", 40, 4100, 1024)]


@pytest.mark.parametrize("codec,m,n,k", CASES)
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_half_copy_against_float64(codec, m, n, k, dt):
    import mlx_kquant_b200 as kq

    rng = np.random.default_rng(m * 31 + n + k)
    some = kq.quantize(torch.from_numpy(rng.standard_normal((64, k)).astype(np.float32) * 0.05), codec)[0].numpy()
    pick = rng.integers(0, 64, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), dt)
    xr = (x.bfloat16() if dt == "f32" else x).double().cpu().numpy()
    ref = (xr @ Oracle().dequantize(some, codec, "f32").astype(np.float64).T)[:, pick]
    w = torch.from_numpy(some[pick]).cuda()
    y = y_to_f32(kq.quantized_matmul(x, w, None, codec)).astype(np.float64)
    # one rounding of a weight to fp16 is at most 2^-11 of it: over K random terms at most that of the product's root
    # mean square, six of them for the largest of many outputs; then half a unit of the output type
    off = np.abs(y - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off.max() < 6 * 2.0 ** -11 * np.sqrt(np.mean(ref ** 2))


@pytest.mark.parametrize("codec,m,n,k", [("q5_k", 17, 4099, 1024), ("q8_0", 130, 2051, 2080), ("q6_k", 300, 1056, 4096),
                                         ("q3_k", 64, 4100, 1280), ("iq4_xs", 40, 1025, 4096)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_without_room_for_the_copy(codec, m, n, k, dt):
    """A call with the smaller workspace (none for fp16 rows) takes the fused kernel, to the same bound."""
    import mlx_kquant_b200 as kq

    lib = kq._lib.lib()
    rng = np.random.default_rng(m + n)
    some = kq.quantize(torch.from_numpy(rng.standard_normal((64, k)).astype(np.float32) * 0.05), codec)[0].numpy()
    pick = rng.integers(0, 64, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), dt)
    code = kq.ops._DT[x.dtype]
    need = lib.kq_quantized_matmul_workspace_bytes(code, m, k)
    assert lib.kq_quantized_matmul_workspace_bytes_for(codec.encode(), code, m, n, k) > need
    ref = (x.double().cpu().numpy() @ Oracle().dequantize(some, codec, "f32").astype(np.float64).T)[:, pick]
    w, y = torch.from_numpy(some[pick]).cuda(), torch.empty(m, n, dtype=x.dtype, device="cuda")
    ws = torch.empty(need, dtype=torch.uint8, device="cuda") if need else None
    kq._lib.check(lib.kq_quantized_matmul(
        x.data_ptr(), code, m, k, k, w.data_ptr(), w.shape[1], n, codec.encode(), 1, y.data_ptr(), n,
        ws.data_ptr() if need else None, need, torch.cuda.current_stream().cuda_stream))
    off = np.abs(y_to_f32(y).astype(np.float64) - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off.max() < 6 * 2.0 ** -11 * np.sqrt(np.mean(ref ** 2))


def test_unaligned_workspace_of_fp16_rows():
    """fp16 rows need no workspace: a large one off the 256-byte grid is no error, the call does without the copy."""
    import mlx_kquant_b200 as kq

    lib = kq._lib.lib()
    m, n, k = 24, 1024, 4096
    rng = np.random.default_rng(3)
    wire = kq.quantize(torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32) * 0.05), "q8_0")[0]
    x = torch.from_numpy(rng.standard_normal((m, k))).half().cuda()
    want = kq.quantized_matmul(x, wire.cuda(), None, "q8_0")
    room = lib.kq_quantized_matmul_workspace_bytes_for(b"q8_0", kq.ops._DT[torch.float16], m, n, k)
    assert room > 0
    ws = torch.empty(room + 256, dtype=torch.uint8, device="cuda")
    y, w = torch.empty_like(want), wire.cuda()
    for shift in (0, 8):
        y.zero_()
        kq._lib.check(lib.kq_quantized_matmul(
            x.data_ptr(), kq.ops._DT[torch.float16], m, k, k, w.data_ptr(), w.shape[1], n, b"q8_0", 1, y.data_ptr(), n,
            ws.data_ptr() + shift, room, torch.cuda.current_stream().cuda_stream))
        # both kernels multiply the same fp16 weights; sums in another order, one rounding to fp16
        ref = want.double()
        assert ((y.double() - ref).abs() <= 2.0 ** -10 * ref.abs() + 1e-5 * ref.square().mean().sqrt()).all()
