"""Mixture-of-experts products grouped by expert (csrc/kq_moe_decode.cu): tasks of eight and of sixteen entries, even parts of
all tasks' tiles per CTA, shares of units per warp."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from gpu_util import mint_wire, x_to_torch, y_to_f32
from mlx_kquant_b200 import _lib
from mlx_kquant_b200.moe import gather_qmv_mix_ns_kq
from oracle.kq_oracle import to_f32

pytestmark = pytest.mark.gpu


def stack(E, n, k, seed):
    return np.stack([mint_wire("q4_k", np.random.default_rng(seed + e).normal(0, 0.02, (n, k)).astype(np.float32)) for e in range(E)])


def glu(x, wg, wu, ids, dt, ws=None):
    T, K = x.shape
    E, F, R = wg.shape[0], wg.shape[1], ids.shape[1]
    L = _lib.lib()
    y = torch.full((T, R, F), 3.0, dtype=x.dtype, device="cuda")
    if ws is None:
        ws = torch.empty(L.kq_moe_decode_workspace_bytes(T * R, E, 0), dtype=torch.uint8, device="cuda")
    idx = ids if isinstance(ids, torch.Tensor) else torch.from_numpy(ids.astype(np.int32)).cuda()
    _lib.check(L.kq_moe_glu_gather(x.data_ptr(), _lib.KQ_F16 if dt == "f16" else _lib.KQ_BF16, T, K, wg.data_ptr(), wg.stride(0),
                                   wu.data_ptr(), wu.stride(0), wg.shape[2], F, E, b"q4_k", idx.data_ptr(), R, b"silu", 0.0,
                                   y.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    return y


# experts, features, K, tokens, experts a token, share of the entries in one expert. At most five entries an expert: tasks of
# eight; more: of sixteen (with eight and fewer in some). The longest rows, one superblock, fewer tiles than SMs, odd rows
CASES = [(40, 17, 2048, 50, 4, 0.0), (64, 200, 512, 80, 4, 0.3), (128, 33, 256, 77, 2, 0.0), (32, 128, 768, 40, 4, 1.0),
         (5, 520, 2048, 40, 4, 0.0), (24, 96, 1024, 60, 4, 0.2), (3, 16, 256, 200, 1, 0.0)]


def routing(E, T, R, busy, seed):
    rng = np.random.default_rng(seed)
    ids = rng.integers(0, E, (T, R))
    return np.where(rng.random((T, R)) < busy, 1, ids)


@pytest.mark.parametrize("E,F,K,T,R,busy", CASES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_gate_up(oracle, E, F, K, T, R, busy, dt):
    wg, wu = stack(E, F, K, 1), stack(E, F, K, 500)
    x, store = x_to_torch(np.random.default_rng(2).normal(0, 1, (T, K)).astype(np.float32), dt)
    ids = routing(E, T, R, busy, 3)
    y = y_to_f32(glu(x, torch.from_numpy(wg).cuda(), torch.from_numpy(wu).cuda(), ids, dt))
    xs = to_f32(store, dt).astype(np.float64)
    dg, du = (oracle.dequantize(w, "q4_k", "f32").astype(np.float64) for w in (wg, wu))
    g, u = np.einsum("tk,trfk->trf", xs, dg[ids]), np.einsum("tk,trfk->trf", xs, du[ids])
    assert_close(y.reshape(T * R, F), (g / (1 + np.exp(-g)) * u).reshape(T * R, F), dt, 2e-3)


@pytest.mark.parametrize("E,N,K,T,R,busy", [(40, 24, 1280, 50, 4, 0.0), (64, 2000, 256, 80, 4, 0.3), (5, 136, 768, 40, 4, 0.0)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_down(oracle, E, N, K, T, R, busy, dt):
    w = stack(E, N, K, 1)
    x, store = x_to_torch(np.random.default_rng(2).normal(0, 1, (T, R, K)).astype(np.float32), dt)
    ids = routing(E, T, R, busy, 3)
    scores = np.random.default_rng(4).uniform(0.1, 0.5, (T, R)).astype(np.float32)
    y = gather_qmv_mix_ns_kq(x, torch.from_numpy(w).cuda(), "q4_k", torch.from_numpy(ids).cuda(), torch.from_numpy(scores).cuda())
    d = oracle.dequantize(w, "q4_k", "f32").astype(np.float64)
    ref = np.einsum("tr,trk,trnk->tn", scores, to_f32(store, dt).astype(np.float64), d[ids])
    assert np.linalg.norm(y_to_f32(y) - ref) / np.linalg.norm(ref) < 4e-3  # every product is rounded once before the sum


def test_not_finite():
    """An infinity or a NaN stays with its token's entries; the largest bf16 numbers stay finite in both products."""
    E, F, K, T, R = 40, 64, 512, 50, 4
    wg, wu = torch.from_numpy(stack(E, F, K, 1)).cuda(), torch.from_numpy(stack(E, F, K, 500)).cuda()
    x = torch.randn(T, K, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    ids = routing(E, T, R, 0.0, 3)
    y = glu(x, wg, wu, ids, "bf16")
    xb = x.clone()
    xb[7, 300], xb[9, 1] = float("nan"), float("inf")
    yb = glu(xb, wg, wu, ids, "bf16")
    others = [t for t in range(T) if t not in (7, 9)]
    assert torch.equal(yb[others], y[others])
    assert torch.isnan(yb[7]).all() and not torch.isfinite(yb[9]).all()
    xb = torch.zeros_like(x)
    xb[3, 5] = 1e18
    assert torch.isfinite(glu(xb, wg, wu, ids, "bf16")).all()


def test_replayed_with_other_routing():
    """The products start beside the grouping in a captured graph, and take the task list only once it is there."""
    E, F, K, T, R = 40, 64, 512, 50, 4
    wg, wu = torch.from_numpy(stack(E, F, K, 1)).cuda(), torch.from_numpy(stack(E, F, K, 500)).cuda()
    x = torch.randn(T, K, generator=torch.Generator().manual_seed(1)).bfloat16().cuda()
    ws = torch.zeros(_lib.lib().kq_moe_decode_workspace_bytes(T * R, E, 0), dtype=torch.uint8, device="cuda")
    idx = torch.zeros((T, R), dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = glu(x, wg, wu, idx, "bf16", ws)
    for seed in range(3):
        ids = torch.from_numpy(routing(E, T, R, 0.3 * seed, seed).astype(np.int32)).cuda()
        want = glu(x, wg, wu, ids, "bf16")
        torch.cuda.synchronize()
        idx.copy_(ids)
        ws.zero_()
        g.replay()
        assert torch.equal(y, want)
