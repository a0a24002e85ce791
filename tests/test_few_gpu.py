"""Two to sixteen dense rows (kq_few.cu): q4_k, q5_k, q6_k, and iq4_xs from one row on."""
import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from gpu_util import product_kernels, x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu


def product(codec, m, n, k, dt, seed):
    rng = np.random.default_rng(seed)
    some = kq.quantize(torch.from_numpy(rng.standard_normal((48, k)).astype(np.float32) * 0.05), codec, None)[0].numpy()
    pick = rng.integers(0, 48, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), dt)
    ref = (x.double().cpu().numpy() @ Oracle().dequantize(some, codec, "f32").astype(np.float64).T)[:, pick]
    return x, torch.from_numpy(some[pick]).cuda(), ref


def check(y, ref, dt):
    # Products of integers and 16-bit activations are exact; K of them are added in float32, with offsets up to three times
    # the weights, in blocks whose sums are K / 16 apart at most: below 2^-12 of the outputs' root mean square for K up to
    # 16384 (half of it measured on the CPU with float32 sums). Then half a unit of the output type.
    off = np.abs(y_to_f32(y).astype(np.float64) - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off.max() < 2.0 ** -11 * np.sqrt(np.mean(ref ** 2))


# the edges: fewer rows than a tile; a last row block of a few rows; row blocks of several tiles, shares that end inside one;
# several row blocks a CTA; one and two column tiles, odd columns; activations that need a pair of CTAs, with an odd number of
# superblocks too; iq4_xs in rows that are no whole sixteens
CASES = [
    ("q4_k", 2, 8, 4096), ("q4_k", 3, 1200, 4096), ("q4_k", 8, 2367, 4352), ("q4_k", 9, 4099, 4096), ("q4_k", 16, 2368, 4096),
    ("q4_k", 5, 40001, 1024), ("q4_k", 6, 300, 14336), ("q4_k", 16, 999, 8448), ("q5_k", 7, 2000, 5120), ("q5_k", 13, 150, 4096),
    ("q5_k", 8, 777, 8192), ("q6_k", 2, 4097, 4096), ("q6_k", 4, 1111, 8192), ("q6_k", 8, 9000, 6144), ("q6_k", 2, 500, 14336),
    ("iq4_xs", 1, 100, 4096), ("iq4_xs", 1, 20000, 256), ("iq4_xs", 4, 4001, 2304), ("iq4_xs", 16, 2500, 2304),
    ("iq4_xs", 15, 1300, 5376), ("iq4_xs", 8, 700, 8448), ("iq4_xs", 2, 60, 16384), ("iq4_xs", 8, 77, 4352)]


@pytest.mark.parametrize("codec,m,n,k", CASES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_few_rows(codec, m, n, k, dt):
    x, w, ref = product(codec, m, n, k, dt, n + k)
    check(kq.quantized_matmul(x, w, None, codec), ref, dt)


@pytest.mark.parametrize("codec", ["q4_k", "q6_k", "iq4_xs"])
def test_not_finite(codec):
    """An infinity or a NaN stays in its row; the largest bf16 numbers stay finite."""
    x, w, ref = product(codec, 4, 1200, 4096, "bf16", 9)
    for bad in (float("inf"), float("nan")):
        xb = x.clone()
        xb[2, 1300] = bad
        y = kq.quantized_matmul(xb, w, None, codec)
        assert not torch.isfinite(y[2]).any()
        check(y[[0, 1, 3]], ref[[0, 1, 3]], "bf16")
    big = torch.zeros_like(x)
    big[0, 7] = 1e38
    assert torch.isfinite(kq.quantized_matmul(big, w, None, codec)).all()


@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_rows_too_long_to_count_in_int(dt):
    """Sixteen rows of 2^26 are 2^31 bytes: more than any shared memory, and the table kernel has them."""
    k, n, m = 1 << 26, 8, 16
    g = torch.Generator().manual_seed(1)
    pool = kq.quantize(torch.randn(256, 256, generator=g) * k ** -0.5, "iq4_xs", None)[0].cuda()
    w = pool[torch.randint(0, 256, (n, k // 256), generator=g).cuda()].reshape(n, -1)
    x = torch.randn(m, k, device="cuda", dtype=torch.float16 if dt == "f16" else torch.bfloat16)
    y = kq.quantized_matmul(x, w, None, "iq4_xs").double()
    ref = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    step = 1 << 22
    for k0 in range(0, k, step):
        d = kq.dequantize(w[:, k0 // 256 * 136:(k0 + step) // 256 * 136].contiguous(), None, "iq4_xs", torch.float32)
        ref += x[:, k0:k0 + step].double() @ d.double().T
    # half a unit of the output, and float32 sums of 2^26 terms in eight or more parts: 2^-24 sqrt(2^26) of their size at most
    assert float((y - ref).norm() / ref.norm()) < (2.0 ** -11 if dt == "f16" else 2.0 ** -8) + 2.0 ** -11


# the longest sixteen rows of q4_k that a pair of CTAs has room for, and fifteen with an odd number of superblocks; one
# superblock more with sixteen and the rows kernel has them
@pytest.mark.parametrize("codec,m,n,k,few", [c + (c != ("q4_k", 16, 999, 8448),) for c in CASES] + [("q4_k", 16, 999, 8192, True),
                                                                                                 ("q4_k", 15, 999, 8448, True)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_which_kernel(codec, m, n, k, few, dt):
    assert ("few_kernel" if few else "rows_kernel") in product_kernels(codec, m, n, k, dt)


@pytest.mark.parametrize("m,k", [(16, 8192), (15, 8448)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_pairs_of_two_column_tiles(m, k, dt):
    x, w, ref = product("q4_k", m, 999, k, dt, m + k)
    check(kq.quantized_matmul(x, w, None, "q4_k"), ref, dt)
