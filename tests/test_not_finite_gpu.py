"""Activations that the integer kernels' 16-bit integers cannot carry: infinities, NaN, the smallest and the largest bf16
numbers. The outputs are those of the sum of activation x weight in plain arithmetic."""
import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from gpu_util import product_kernels, x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu

ROWS = 24   # distinct rows of weights


def problem(codec, m, n, k, seed):
    """(activations in float32, wire bytes on the GPU, the weights of their distinct rows, which one each row is)"""
    rng = np.random.default_rng(seed)
    some = kq.quantize(torch.from_numpy(rng.standard_normal((ROWS, k)).astype(np.float32) * 0.01), codec,
                       torch.ones(k) if codec == "iq2_xxs" else None)[0].numpy()
    pick = rng.integers(0, ROWS, n)
    return rng.standard_normal((m, k)).astype(np.float32), torch.from_numpy(some[pick]).cuda(), \
        Oracle().dequantize(some, codec, "f32").astype(np.float64), pick


def stored(xf, dt):
    x, _ = x_to_torch(xf, dt)
    return x, (x.bfloat16() if dt == "f32" else x).double().cpu().numpy()


def products(x, w):
    with np.errstate(invalid="ignore", over="ignore"):
        return np.stack([(r[None] * w).sum(1) for r in x])   # (no BLAS: it may leave out products with zeros)


def check_not_finite(call, xf, w, pick, dt):
    """One infinity or NaN in the last row: that row's outputs have their kind and sign, the other rows do not see it."""
    for bad in (np.inf, -np.inf, np.nan):
        xb = xf.copy()
        xb[-1, 77] = bad
        x, xs = stored(xb, dt)
        y, ref = y_to_f32(call(x)), products(xs, w)[:, pick]
        assert np.array_equal(np.isnan(y[-1]), np.isnan(ref[-1]))
        inf = np.isinf(ref[-1])
        assert (inf.any() or np.isnan(bad)) and np.array_equal(y[-1][inf], ref[-1][inf])
        assert np.isfinite(y[:-1]).all()


def check_range(call, xf, w, pick, dt):
    """The integers of a group are off by 2^-15 of its largest at most, for the smallest groups by 2^-128 instead; sums of the
    largest numbers may not overflow before the block's scale does its part. Half a unit of the output beside."""
    for scale in (1e-36, 1e-35, 3e34):
        x, xs = stored((xf * scale).astype(np.float32), dt)
        y, ref = y_to_f32(call(x)).astype(np.float64), products(xs, w)[:, pick]
        root = np.sqrt((w ** 2).sum(1))[pick]   # of a row's weights: errors of the activations are independent
        off = np.maximum(2.0 ** -15 * np.abs(xs).max(), 2.0 ** -128)
        assert (np.abs(y - ref) <= 2.0 ** -8 * np.abs(ref) + 6 * off * root[None] + 2.0 ** -133).all(), scale
    for signs in (1, -1):   # the group's own sum leaves float32, half-way or for good
        big = xf.copy()
        big[-1, 64:68], big[-1, 68:72] = 2e38, signs * 2e38
        x, xs = stored(big, dt)
        y, ref = y_to_f32(call(x))[-1].astype(np.float64), products(xs, w)[-1][pick]
        size = (np.abs(xs[-1]) * np.abs(w)).sum(1)[pick]   # nothing on the way to the output is larger
        assert (size < 3e38).all() and np.isfinite(y).all()
        assert (np.abs(y - ref) <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -13 * size).all()


def check(codec, m, n, k, dt):
    xf, wire, w, pick = problem(codec, m, n, k, n + k)
    call = lambda x: kq.quantized_matmul(x, wire, None, codec)
    check_not_finite(call, xf, w, pick, dt)
    if dt != "f16":
        check_range(call, xf, w, pick, dt)


# kq_gemv_dp4a.cuh: rows that are no whole sixteens of bytes, and rows that are
RAGGED = [("q6_k", 1, 1001, 2304), ("q6_k", 1, 70, 5120), ("q3_k", 1, 100, 1280), ("q3_k", 2, 31, 768), ("q3_k", 4, 65, 1536),
          ("q2_k", 1, 400, 1536), ("q2_k", 3, 97, 256), ("q2_k", 4, 33, 512), ("iq4_xs", 1, 333, 2304), ("iq2_xxs", 1, 20000, 2816)]
WHOLE = [("q2_k", 1, 90, 1024), ("q3_k", 1, 90, 2048), ("q3_k", 4, 90, 2048), ("q6_k", 1, 90, 2048), ("q5_k", 1, 90, 512),
         ("q8_0", 1, 90, 768), ("q8_0", 4, 33, 512), ("q4_0", 2, 90, 1024), ("q4_1", 1, 90, 512), ("q5_0", 3, 90, 512),
         ("q5_1", 1, 90, 512), ("iq4_nl", 1, 90, 1024)]


@pytest.mark.parametrize("codec,m,n,k", RAGGED + WHOLE)
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_dot_product_kernels(codec, m, n, k, dt):
    check(codec, m, n, k, dt)


# kq_gemv_one.cu
ONE = [("q4_k", 70, 8192), ("q4_k", 6200, 4096), ("q5_k", 1030, 2048), ("q5_k", 40, 8448),
       ("q6_k", 1030, 2048), ("q6_k", 90, 14336)]


@pytest.mark.parametrize("codec,n,k", ONE)
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_one_row(codec, n, k, dt):
    check(codec, 1, n, k, dt)


@pytest.mark.parametrize("codec", ["q2_k", "q3_k", "q8_0", "q4_0"])
def test_task_lists(codec):
    """gather_qmm of a few rows an expert: the same kernels over task lists."""
    e, n, k, b, at = 6, 96, 2048, 20, 17
    experts = [problem(codec, 1, n, k, 5 + i) for i in range(e)]
    rng = np.random.default_rng(5)
    xf, rhs = rng.standard_normal((b, k)).astype(np.float32), rng.integers(0, e, b)
    wd, rd = torch.stack([p[1] for p in experts]), torch.from_numpy(rhs).cuda()
    for bad in (np.inf, -np.inf, np.nan):
        xb = xf.copy()
        xb[at, 77] = bad
        x, xs = stored(xb, "bf16")
        y = y_to_f32(kq.gather_qmm(x[:, None], wd, None, codec, rhs_indices=rd))[:, 0]
        _, _, w, pick = experts[rhs[at]]
        ref = products(xs[at:at + 1], w)[0][pick]
        inf = np.isinf(ref)
        assert np.array_equal(np.isnan(y[at]), np.isnan(ref)) and np.array_equal(y[at][inf], ref[inf])
        assert np.isfinite(np.delete(y, at, 0)).all()


@pytest.mark.parametrize("codec,m,n,k,name", [c + ("gemv_dp4a_kernel",) for c in RAGGED + WHOLE] +
                         [(c, 1, n, k, "gemv_one_kernel") for c, n, k in ONE])
@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
def test_which_kernel(codec, m, n, k, name, dt):
    assert name in product_kernels(codec, m, n, k, dt)
