"""The tile kernel with the weights on the M side (kq_tile.cu): its shapes, rings and row classes at their edges."""
import ctypes as C

import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from gpu_util import product_kernels, x_to_torch, y_to_f32
from mlx_kquant_b200 import _lib
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu


def some_rows(codec, k, seed):
    rng = np.random.default_rng(seed)
    rows = torch.from_numpy(rng.standard_normal((64, k)).astype(np.float32) * 0.05)
    return rng, kq.quantize(rows, codec)[0].numpy()


def check(y, ref, dt):
    # one rounding of a weight to fp16 is at most 2^-11 of it (twice that where scale and product are rounded): over K random
    # terms at most that of the product's root mean square, six of them for the largest of many outputs; then half a unit of
    # the output type
    off = np.abs(y_to_f32(y).astype(np.float64) - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off.max() < 6 * 2.0 ** -10 * np.sqrt(np.mean(ref ** 2))
    flags = C.c_int(-1)
    _lib.check(_lib.lib().kq_device_error_flags(C.byref(flags), 1))
    assert flags.value == 0


# rows around the token blocks (16, 64, 112, 128, 160, 256) and several tiles a CTA; columns short of a tile, of a pair, and
# of many tiles; K of one superblock, an odd number of them (the wire ring crosses tiles at an odd place), split in 2, 4, 8.
# q6_k: K of 256 (2048 j + 256, 512, 1024, 2048) has wire rows in groups of eight, four, two, one on sixteen bytes.
SHAPES = [(17, 136, 256), (64, 1000, 512), (65, 264, 768), (112, 4104, 1024), (113, 256, 2048), (129, 2056, 1280),
          (161, 520, 4096), (256, 1032, 3328), (257, 14344, 512), (509, 392, 8192), (700, 3080, 1792), (1500, 2312, 256),
          (40, 4096, 4096), (30, 1024, 8192)]


@pytest.mark.parametrize("codec", ["q4_k", "q6_k"])
@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_shapes(codec, m, n, k, dt):
    rng, some = some_rows(codec, k, m * 31 + n + k)
    pick = rng.integers(0, 64, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), dt)
    ref = (x.double().cpu().numpy() @ Oracle().dequantize(some, codec, "f32").astype(np.float64).T)[:, pick]
    check(kq.quantized_matmul(x, torch.from_numpy(some[pick]).cuda(), None, codec), ref, dt)


# rows in groups of eight, four and two: with producers (few rows) and by the fp16 copy (many)
CLASSES = [(70, 6000, 768), (300, 6000, 768), (620, 8200, 512), (130, 8200, 512), (300, 4100, 1536), (700, 4098, 1024)]


@pytest.mark.parametrize("m,n,k", CLASSES)
def test_q6k_rows_in_classes(m, n, k):
    rng, some = some_rows("q6_k", k, m + n + k)
    pick = rng.integers(0, 64, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), "bf16")
    ref = (x.double().cpu().numpy() @ Oracle().dequantize(some, "q6_k", "f32").astype(np.float64).T)[:, pick]
    check(kq.quantized_matmul(x, torch.from_numpy(some[pick]).cuda(), None, "q6_k"), ref, "bf16")


@pytest.mark.parametrize("n", [1001, 1002, 1004])
def test_q6k_rows_that_do_not_fill_a_class(n):
    """Wire rows in groups of eight, and a number of rows that is no multiple: another kernel, the same result."""
    rng, some = some_rows("q6_k", 1280, n)
    pick = rng.integers(0, 64, n)
    x, _ = x_to_torch(rng.standard_normal((33, 1280)).astype(np.float32), "bf16")
    ref = (x.double().cpu().numpy() @ Oracle().dequantize(some, "q6_k", "f32").astype(np.float64).T)[:, pick]
    check(kq.quantized_matmul(x, torch.from_numpy(some[pick]).cuda(), None, "q6_k"), ref, "bf16")


def test_strided_rows_and_unaligned_weights():
    """Activation rows with a stride; weights one byte off the 16-byte grid take the general kernel: the same bits."""
    rng, some = some_rows("q4_k", 1024, 5)
    w = torch.from_numpy(some[rng.integers(0, 64, 300)]).cuda()
    x = torch.randn(70, 2048, device="cuda").half()[:, 512:1536]
    want = kq.quantized_matmul(x.contiguous(), w, None, "q4_k")
    assert torch.equal(kq.quantized_matmul(x, w, None, "q4_k"), want)
    raw = torch.empty(w.numel() + 16, dtype=torch.uint8, device="cuda")
    off = raw[1:1 + w.numel()].view(w.shape)
    off.copy_(w)
    got = kq.quantized_matmul(x.contiguous(), off, None, "q4_k").double()
    # both round a weight to fp16: q4_k's once more here (the min), then sums in another order
    assert ((got - want.double()).abs() <= 2.0 ** -9 * want.double().abs() + 6 * 2.0 ** -10 * want.double().square().mean().sqrt()).all()


# rows per expert from none to several tiles; averages that take tiles of 64, 128 and 256 rows
@pytest.mark.parametrize("codec,k", [("q4_k", 768), ("q6_k", 1024), ("q6_k", 256)])
@pytest.mark.parametrize("counts", [[0, 1, 64, 65, 16, 30, 128, 208], [300, 20, 0, 129, 128, 3, 30, 70],
                                    [256, 257, 0, 1500, 7, 255, 512, 513]])
def test_grouped(codec, k, counts):
    n, e = 264, len(counts)
    rng, some = some_rows(codec, k, sum(counts) + k)
    pick = rng.integers(0, 64, (e, n))
    rhs = np.repeat(np.arange(e), counts)
    rng.shuffle(rhs)
    lhs = rng.integers(0, 100, rhs.size)
    x, _ = x_to_torch(rng.standard_normal((100, 1, k)).astype(np.float32), "bf16")
    y = kq.gather_qmm(x, torch.from_numpy(some[pick]).cuda(), None, codec, lhs_indices=torch.from_numpy(lhs).cuda(),
                      rhs_indices=torch.from_numpy(rhs).cuda())
    full = x[:, 0].double().cpu().numpy() @ Oracle().dequantize(some, codec, "f32").astype(np.float64).T   # [100, 64]
    ref = np.stack([full[a, pick[b]] for a, b in zip(lhs, rhs)])
    check(y.reshape(rhs.size, n), ref, "bf16")


@pytest.mark.parametrize("rows", [64, 600])
def test_q6k_weights_are_rounded_once(rows):
    """One-hot activations show the producers' weights: those of dequantize to fp16, but for the last bit of a few where the
    scale's second part (2^-11 of the first, itself in fp16) decides a tie."""
    g = torch.Generator().manual_seed(6)
    w = kq.quantize(torch.randn(512, 2048, generator=g) * 0.05, "q6_k", None)[0].cuda()
    k = torch.randperm(2048, generator=g)[:rows].cuda()
    x = torch.zeros(rows, 2048, dtype=torch.float16, device="cuda")
    x[torch.arange(rows, device="cuda"), k] = 1
    y = kq.quantized_matmul(x, w, None, "q6_k")
    ref = kq.dequantize(w, None, "q6_k", torch.float16)[:, k].T.contiguous()
    bits = lambda v: (v + 0.0).view(torch.int16).int()  # (a weight of zero has the scale's sign or none)
    off = (bits(y) - bits(ref)).abs()
    assert int(off.max()) <= 1 and float((off > 0).float().mean()) < 0.02


@pytest.mark.parametrize("codec", ["q4_k", "q6_k"])
@pytest.mark.parametrize("m,n,k", SHAPES + CLASSES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_which_kernel(codec, m, n, k, dt):
    names = product_kernels(codec, m, n, k, dt)
    assert "tile_kernel" in names and (codec != "q4_k" or "dequant_kernel" not in names)
    if codec == "q6_k" and (m, n, k) in CLASSES:   # few rows: producers, many: the copy
        assert ("dequant_kernel" in names) == (m > 600)


@pytest.mark.parametrize("n", [1001, 1002, 1004])
def test_which_kernel_has_rows_that_do_not_fill_a_class(n):
    names = product_kernels("q6_k", 33, n, 1280, "bf16")
    assert "dequant_kernel" in names and "tile_kernel" in names


@pytest.mark.parametrize("m,n,k", [(17, 9, 256), (53, 763, 1024), (300, 259, 768), (130, 3001, 1280), (65, 1178, 512)])
@pytest.mark.parametrize("room", [True, False])
def test_small_q6k_rows_that_do_not_fill_a_class(m, n, k, room):
    """By the copy, and with the room for the converted activations alone by the general kernel."""
    rng, some = some_rows("q6_k", k, m + n + k)
    pick = rng.integers(0, 64, n)
    x, _ = x_to_torch(rng.standard_normal((m, k)).astype(np.float32), "bf16")
    ref = (x.double().cpu().numpy() @ Oracle().dequantize(some, "q6_k", "f32").astype(np.float64).T)[:, pick]
    w = torch.from_numpy(some[pick]).cuda()
    if room:
        y = kq.quantized_matmul(x, w, None, "q6_k")
    else:
        lib, dt = kq._lib.lib(), kq.ops._DT[x.dtype]
        ws = torch.empty(lib.kq_quantized_matmul_workspace_bytes(dt, m, k), dtype=torch.uint8, device="cuda")
        y = torch.empty(m, n, dtype=x.dtype, device="cuda")
        kq._lib.check(lib.kq_quantized_matmul(x.data_ptr(), dt, m, k, k, w.data_ptr(), w.shape[1], n, b"q6_k", 1, y.data_ptr(), n,
                                              ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    check(y, ref, "bf16")
