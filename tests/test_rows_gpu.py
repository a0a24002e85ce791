"""Two to sixteen rows of q4_k, q5_k, q6_k and iq4_xs (kq_rows.cu) against float64 products of the oracle's weights."""
import numpy as np
import pytest
import torch

from gpu_util import x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu

# (m, n, k): row tiles and row blocks with remainders, one superblock, stages with remainders, rows of q6_k that do
# not start on 16-byte boundaries and a matrix whose last byte does not end on one (k = 512 * odd, odd n), more rows
# than one pass of the SMs holds, both column tiles
SHAPES = [(2, 8, 512), (3, 333, 512), (8, 2049, 1536), (9, 257, 1024), (16, 40, 4096), (5, 4099, 2560), (12, 3000, 512),
          (2, 38000, 512), (4, 301, 768), (16, 38000, 256)]


def _close(y, ref, out_eps):
    """Every output within half a unit of the output type (out_eps, relative; at least the 2^-25 of fp16 subnormals)
    plus the sums in float32: 2e-5 of the outputs' root mean square, some hundred units of float32."""
    off = np.abs(y - ref) - np.maximum(out_eps * np.abs(ref), 2.0 ** -25)
    assert off.max() < 2e-5 * np.sqrt(np.mean(ref ** 2)), off.max()


@pytest.mark.parametrize("codec", ["q4_k", "q5_k", "q6_k", "iq4_xs"])
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_rows_against_float64(codec, dt, m, n, k):
    import mlx_kquant_b200 as kq

    if codec == "iq4_xs" and n * k > 4 << 20:
        pytest.skip("another kernel's range")
    rng = np.random.default_rng(m * 1000003 + n * 101 + k)
    some = rng.standard_normal((min(n, 64), k)).astype(np.float32) * 0.05
    wire = kq.quantize(torch.from_numpy(some), codec)[0].numpy()
    wire = wire[rng.integers(0, len(wire), n)]
    x_f32 = rng.standard_normal((m, k)).astype(np.float32)
    x_f32[0] *= 1e-3
    x_f32[-1] *= 300.0
    x, _ = x_to_torch(x_f32, dt)
    xr = (x.bfloat16() if dt == "f32" else x).double().cpu().numpy()
    ref = xr @ Oracle().dequantize(wire, codec, "f32").astype(np.float64).T
    w = torch.from_numpy(wire).cuda()
    y = y_to_f32(kq.quantized_matmul(x, w, None, codec)).astype(np.float64)
    for r in range(m):  # rows of very different magnitude
        _close(y[r], ref[r], 2.0 ** -11 if dt == "f16" else 2.0 ** -8)


def test_rows_largest_finite_bf16():
    """Rows near the largest bf16 number: the operands' power of two keeps every partial sum finite."""
    import mlx_kquant_b200 as kq

    rng = np.random.default_rng(5)
    for codec in ("q4_k", "q6_k"):
        w = kq.quantize(torch.from_numpy(rng.standard_normal((64, 512)).astype(np.float32) * 1e-3), codec)[0]
        x = (torch.from_numpy(rng.standard_normal((4, 512))).clamp(-3, 3) * 1e38).bfloat16()
        ref = x.double().numpy() @ Oracle().dequantize(w.numpy(), codec, "f32").astype(np.float64).T
        y = kq.quantized_matmul(x.cuda(), w.cuda(), None, codec).double().cpu().numpy()
        _close(y, ref, 2.0 ** -8)


@pytest.mark.parametrize("codec", ["q4_k", "q5_k", "q6_k", "iq4_xs"])
@pytest.mark.parametrize("m", [3, 13])
def test_rows_of_small_bf16(codec, m):
    """Rows of 5e-35 (2^-114), whose products with the weights are normal float32 numbers still."""
    import mlx_kquant_b200 as kq

    rng = np.random.default_rng(7)
    w = kq.quantize(torch.from_numpy(rng.standard_normal((64, 512)).astype(np.float32) * 0.5), codec)[0]
    x = (torch.from_numpy(rng.standard_normal((m, 512))) * 2.0 ** -114).bfloat16()
    ref = x.double().numpy() @ Oracle().dequantize(w.numpy(), codec, "f32").astype(np.float64).T
    y = kq.quantized_matmul(x.cuda(), w.cuda(), None, codec).double().cpu().numpy()
    _close(y * 2.0 ** 114, ref * 2.0 ** 114, 2.0 ** -8)


def _gathered(x, w, codec):
    """The same product as a gather of one row per entry from a stack of one matrix."""
    import mlx_kquant_b200 as kq

    at = torch.arange(x.shape[0], dtype=torch.int32, device="cuda")
    return kq.gather_qmm(x[:, None], w[None], None, codec, lhs_indices=at, rhs_indices=torch.zeros_like(at))[:, 0]


@pytest.mark.parametrize("codec", ["q4_k", "q5_k", "q6_k", "iq4_xs"])
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("m,k", [(5, 1024), (12, 768)])
@pytest.mark.parametrize("gather", [False, True])
def test_rows_not_finite(codec, dt, m, k, gather):
    """Infinite activations give signed infinities (NaN where the weight is zero), NaN gives NaN, and the rows beside
    them are as ever."""
    import mlx_kquant_b200 as kq

    if gather and dt == "f32":
        pytest.skip("another kernel's range")
    rng = np.random.default_rng(m * 7 + k)
    wire = kq.quantize(torch.from_numpy(rng.standard_normal((40, k)).astype(np.float32) * 0.05), codec)[0]
    x_f32 = rng.standard_normal((m, k)).astype(np.float32)
    x_f32[0, 37], x_f32[1, k - 1], x_f32[2, 300] = np.inf, -np.inf, np.nan
    x, _ = x_to_torch(x_f32, dt)
    xr = (x.bfloat16() if dt == "f32" else x).double().cpu().numpy()
    with np.errstate(invalid="ignore"):
        ref = xr @ Oracle().dequantize(wire.numpy(), codec, "f32").astype(np.float64).T
    y = _gathered(x, wire.cuda(), codec) if gather else kq.quantized_matmul(x, wire.cuda(), None, codec)
    y = y_to_f32(y).astype(np.float64)
    np.testing.assert_array_equal(y[:3], ref[:3])
    for r in range(3, m):
        _close(y[r], ref[r], 2.0 ** -11 if dt == "f16" else 2.0 ** -8)


@pytest.mark.parametrize("codec", ["q4_k", "q5_k", "q6_k", "iq4_xs"])
@pytest.mark.parametrize("gather", [False, True])
def test_rows_of_one_sign_near_the_largest_bf16(codec, gather):
    """Sums of offset integers overflow long before the products of weights and activations do."""
    import mlx_kquant_b200 as kq

    rng = np.random.default_rng(6)
    w = kq.quantize(torch.from_numpy(rng.standard_normal((64, 512)).astype(np.float32) * 1e-3), codec)[0]
    x = (torch.from_numpy(rng.standard_normal((4, 512))).abs().clamp(max=3) * 1e38).bfloat16()
    ref = x.double().numpy() @ Oracle().dequantize(w.numpy(), codec, "f32").astype(np.float64).T
    y = _gathered(x.cuda(), w.cuda(), codec) if gather else kq.quantized_matmul(x.cuda(), w.cuda(), None, codec)
    _close(y.double().cpu().numpy(), ref, 2.0 ** -8)


@pytest.mark.parametrize("codec,m", [("q4_k", 8), ("q6_k", 2), ("q5_k", 16)])
def test_weights_written_just_before(codec, m):
    """The weights may come from the kernel before: nothing of them is read ahead of its end."""
    import mlx_kquant_b200 as kq

    n, k = 4096, 1024
    rows = torch.randn(2, 256, k, generator=torch.Generator().manual_seed(2)) * 0.05
    pair = [kq.quantize(r, codec)[0].repeat(n // 256, 1).cuda() for r in rows]
    x = torch.randn(m, k, dtype=torch.bfloat16, device="cuda")
    want = [kq.quantized_matmul(x, w, None, codec) for w in pair]
    buf, got = torch.empty_like(pair[0]), []
    for i in range(64):
        buf.copy_(pair[i % 2])
        got.append(kq.quantized_matmul(x, buf, None, codec))
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2])


def test_strided_weights_of_one_row():
    """A copy made for the call is written before the one-row kernel, which reads ahead, can see it."""
    import mlx_kquant_b200 as kq

    n, k = 2048, 4096
    rows = torch.randn(2, 64, k, generator=torch.Generator().manual_seed(4)) * 0.05
    pair = [kq.quantize(r, "q4_k")[0].repeat(n // 64, 1).cuda() for r in rows]
    wide = torch.stack(pair, 1)   # [n, 2, bytes]: either matrix with the other between its rows
    x = torch.randn(1, k, dtype=torch.float16, device="cuda")
    want = [kq.quantized_matmul(x, w, None, "q4_k") for w in pair]
    got = [kq.quantized_matmul(x, wide[:, i % 2], None, "q4_k") for i in range(64)]
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2])
