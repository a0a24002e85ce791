"""One dense row: the TMA kernel of q4_k, q5_k, q6_k (kq_gemv_one.cu), and the integer dot-product kernels with rows that are
not whole sixteens (kq_gemv_dp4a.cuh)."""
import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from gpu_util import product_kernels, x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu


def product(codec, m, n, k, dt, seed):
    rng = np.random.default_rng(seed)
    rows = torch.from_numpy(rng.standard_normal((48, k)).astype(np.float32) * 0.05)
    some = kq.quantize(rows, codec, torch.ones(k) if codec == "iq2_xxs" else None)[0].numpy()
    pick = rng.integers(0, 48, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), dt)
    xr = (x.bfloat16() if dt == "f32" else x).double().cpu().numpy()
    ref = (xr @ Oracle().dequantize(some, codec, "f32").astype(np.float64).T)[:, pick]
    return x, torch.from_numpy(some[pick]).cuda(), ref


def check(y, ref, dt):
    # An activation as an integer is off by at most 2^-16 of the largest of its 32 (below 3 here), evenly spread: 2.6e-5 root
    # mean square. The quants of q4_k and q5_k have a mean of half their range, twice the weights they stand for. Six of that
    # for the largest of many outputs: 3.2e-4 < 2^-11 of the outputs' root mean square; then half a unit of the output type.
    off = np.abs(y_to_f32(y).astype(np.float64) - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off.max() < 2.0 ** -11 * np.sqrt(np.mean(ref ** 2))


# one block and several a CTA, rows that leave the last one short, fewer rows than SMs; superblocks fewer and more than warps
# x slots, and the longest row; q6_k's K are multiples of 2048 here (whole sixteens)
CASES = [("q4_k", 12300, 2048), ("q4_k", 33, 8192), ("q4_k", 1537, 16384), ("q4_k", 20001, 4096),
                                       ("q5_k", 1024, 2048), ("q5_k", 5001, 768), ("q5_k", 90, 8448), ("q5_k", 14336, 256),
                                       ("q6_k", 1025, 2048), ("q6_k", 4800, 4096), ("q6_k", 77, 14336), ("q6_k", 9999, 2048)]


@pytest.mark.parametrize("codec,n,k", CASES)
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_one_row(codec, n, k, dt):
    x, w, ref = product(codec, 1, n, k, dt, n + k)
    check(kq.quantized_matmul(x, w, None, codec), ref, dt)


@pytest.mark.parametrize("codec", ["q4_k", "q5_k", "q6_k"])
def test_not_finite(codec):
    """An infinity or a NaN among the activations reaches every output; the largest bf16 numbers stay finite."""
    x, w, ref = product(codec, 1, 1500, 8192, "bf16", 9)
    for bad in (float("inf"), float("-inf"), float("nan")):
        xb = x.clone()
        xb[0, 4100] = bad
        assert not torch.isfinite(kq.quantized_matmul(xb, w, None, codec)).any()
    big = torch.zeros_like(x)
    big[0, 7] = 1e38
    assert torch.isfinite(kq.quantized_matmul(big, w, None, codec)).all()


# rows of 2, 4 and 8 bytes past a sixteen: one to four of them, odd numbers of rows (a last block of one parity alone)
RAGGED = [("q6_k", 1, 1001, 2304), ("q6_k", 1, 63, 5120), ("q3_k", 1, 1000, 1280), ("q3_k", 2, 31, 768),
          ("q3_k", 4, 515, 1536), ("q2_k", 1, 400, 1536), ("q2_k", 3, 97, 256), ("iq4_xs", 1, 333, 2304),
          ("iq2_xxs", 1, 20000, 2816), ("q6_k", 3, 129, 1280), ("q3_k", 1, 4100, 256)]


@pytest.mark.parametrize("codec,m,n,k", RAGGED)
@pytest.mark.parametrize("dt", ["f16", "f32"])
def test_ragged_rows(codec, m, n, k, dt):
    x, w, ref = product(codec, m, n, k, dt, n + k)
    check(kq.quantized_matmul(x, w, None, codec), ref, dt)


def test_ragged_rows_end_at_the_matrix():
    """The last row's window runs past the matrix, which here is followed by nothing of its own: poisoned bytes do not matter."""
    x, w, ref = product("q6_k", 1, 65, 1280, "f16", 4)
    pad = torch.full((w.numel() + 4096,), 0xff, dtype=torch.uint8, device="cuda")
    inside = pad[:w.numel()].view(w.shape)
    inside.copy_(w)
    check(kq.quantized_matmul(x, inside, None, "q6_k"), ref, "f16")


@pytest.mark.parametrize("codec,n,k", [("q6_k", 3001, 2304), ("q6_k", 1500, 5120), ("q3_k", 4000, 1280), ("iq4_xs", 1500, 2304)])
def test_ragged_rows_of_bf16_are_hardly_rounded(codec, n, k):
    """bf16 activations within 2^-7 of the largest of their 32 are exact as integers, one in seventy of normal ones is not: by
    half a unit of 2^-14 of the largest at most, evenly spread. 2^-14 / sqrt(12) x sqrt(1 / 70) x 2.4 = 5e-6 of an activation's
    size, and as much of an output's. An output y is then another bf16 number than the exact one's with a probability of
    0.8 x 5e-6 over the distance of two bf16 numbers there, 2^-8 |y| to 2^-7 |y|, and the mean of 1 / |y| over normal outputs
    between a hundredth of their size and twice it is 3.8: 0.2 to 0.4 %. Half a percent of 4800 (three deviations more than
    0.37 %). (All rounded to 2^-15 of the largest: four times as many; 1.3 to 2 % counted.)"""
    x, w, ref = product(codec, 1, n, k, "bf16", n + k)
    distinct = np.unique(ref, return_index=True)[1]
    other = total = 0
    for seed in range(100):
        x = torch.randn(1, k, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)).bfloat16()
        y = kq.quantized_matmul(x, w, None, codec)[0]
        near = (x.double() @ kq.dequantize(w, None, codec, torch.float32).double().T).bfloat16()[0]
        at = torch.from_numpy(distinct).cuda()
        other += int((y[at] != near[at]).sum())
        total += len(distinct)
    assert other < 0.005 * total


@pytest.mark.parametrize("n,k", [(8192, 8192), (15400, 4096)])
def test_fp16_rows_of_large_q4_k(n, k):
    """An activation as an integer is off by 2^-16 of the largest of its 32 (2.4 of their size), evenly spread, 2.1e-5 of their size
    root mean square; with quants less their middle the weights that it is multiplied by are hardly larger than the real ones,
    so that outputs are off by as much of theirs. (With the quants themselves: above 4e-5.)"""
    beyond = size = 0.0
    for seed in range(8):
        x, w, ref = product("q4_k", 1, n, k, "f16", seed)
        ref = torch.from_numpy(ref)
        y = kq.quantized_matmul(x, w, None, "q4_k").double().cpu()
        beyond += float((y - ref).square().sum() - (ref.half().double() - ref).square().sum())
        size += float(ref.square().sum())
    assert beyond < 3e-5 ** 2 * size


@pytest.mark.parametrize("codec,n,k", CASES + [("q4_k", 8192, 8192), ("q4_k", 15400, 4096)])
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_which_kernel(codec, n, k, dt):
    assert "gemv_one_kernel" in product_kernels(codec, 1, n, k, dt)


# (three rows of q6_k: the rows kernel takes them, ragged or not)
@pytest.mark.parametrize("codec,m,n,k", RAGGED)
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_which_kernel_has_ragged_rows(codec, m, n, k, dt):
    assert ("rows_kernel" if (codec, m) == ("q6_k", 3) else "gemv_dp4a_kernel") in product_kernels(codec, m, n, k, dt)
