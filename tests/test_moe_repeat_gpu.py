"""The grouped decode products of a mixture-of-experts block give the same bits call after call: which entries of an expert
share a task, and with it the order of a product's sums, may not hang on the order in which the grouping's counters are
reached."""
import ctypes

import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from mlx_kquant_b200 import _lib, moe

pytestmark = pytest.mark.gpu


def experts(n, k, e, seed):
    g = torch.Generator().manual_seed(seed)
    pool = kq.quantize(torch.randn(256, 256, generator=g) * k ** -0.5, "q4_k", None)[0]
    return pool[torch.randint(0, 256, (e, n, k // 256), generator=g)].reshape(e, n, -1).cuda()


# tasks of eight and of sixteen entries; every expert with several tasks, a busy one, one that has nearly all
@pytest.mark.parametrize("tokens,e,top_k,skew", [(64, 128, 8, 0.), (64, 128, 8, 3.), (40, 16, 8, 1.), (128, 60, 4, 3.), (64, 16, 4, 1.),
                                                 (200, 200, 2, 5.)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_same_bits_again(tokens, e, top_k, skew, dt):
    k, f = 1024, 512
    gate_up, down = experts(2 * f, k, e, 1), experts(k, f, e, 2)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(tokens, k, device="cuda", generator=g).to(dt)
    logits = torch.randn(tokens, e, device="cuda", generator=g) + skew * torch.randn(1, e, device="cuda", generator=g)
    ids, probs = moe.route_topk(logits, top_k)
    call = lambda: moe.moe_glu(x, None, None, down, "q4_k", ids, probs, w_gate_up=gate_up)
    first = call()
    for _ in range(60):
        assert torch.equal(call(), first)


# one CTA and several of the grouping, and its long form (more than 1024 experts)
@pytest.mark.parametrize("entries,e,busy", [(300, 4, 0), (512, 40, 0), (2048, 9, 900), (4096, 130, 700), (3000, 3, 0), (600, 1100, 40)])
def test_tasks(entries, e, busy):
    k, f = 1024, 64
    w = experts(2 * f, k, e, 5)
    rng = np.random.default_rng(entries)
    idx = rng.integers(0, e, entries)
    idx[:busy] = 1
    idx = torch.from_numpy(rng.permutation(idx).astype(np.int32)).cuda().reshape(-1, 1)
    x = torch.randn(entries, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).bfloat16()
    call = lambda: moe.moe_glu_gather_kq(x, w[:, :f], w[:, f:], "q4_k", idx)
    first = call()
    for _ in range(20):
        assert torch.equal(call(), first)
    ref = []
    for xs, i in zip(x.split(256), idx[:, 0].long().split(256)):
        h = torch.einsum("bk,bnk->bn", xs.double(), kq.dequantize(w[i], None, "q4_k", torch.float32).double())
        ref.append(torch.nn.functional.silu(h[:, :f]) * h[:, f:])
    ref = torch.cat(ref)
    # one rounding to bf16, 2^-9 of a value on average at most; sums in float32 beside
    assert float((first[:, 0].double() - ref).norm() / ref.norm()) < 2.0 ** -8
    flags = ctypes.c_int()
    _lib.check(_lib.lib().kq_device_error_flags(ctypes.byref(flags), 0))
    assert flags.value == 0
