"""Entries by expert in one launch (csrc/kq_gather.cu): one CTA, a cluster, and the long form beyond both."""
import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from conftest import assert_close
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu


# the last size of one CTA and the first of a cluster, a cluster's last and the first beyond; up to 1024 experts, one, more
@pytest.mark.parametrize("rows,experts", [(1, 1), (2048, 1024), (2049, 7), (65536, 300), (65537, 5), (4000, 1025), (30000, 1024)])
def test_tile_map(rows, experts):
    ids = np.sort(np.random.default_rng(rows).integers(0, experts, rows))
    m, count = kq.expert_tile_map(torch.from_numpy(ids.astype(np.int32)).cuda(), experts)
    want, at = [], 0
    for e, c in enumerate(np.bincount(ids, minlength=experts)):
        want += [(e, at + j, min(64, c - j)) for j in range(0, c, 64)]
        at += c
    assert int(count[0]) == len(want)
    assert np.array_equal(m.cpu().numpy().reshape(-1, 3)[:len(want)], np.array(want))


# entries by sixteen, in tiles (an expert's last one ragged) and in tasks; a busy expert, experts without any, indices out of range
@pytest.mark.parametrize("entries,experts,codec", [(130, 6, "q8_0"), (2100, 20, "q8_0"), (3000, 8, "q4_k"), (700, 40, "q8_0"), (66000, 3, "q4_0")])
def test_gather(entries, experts, codec):
    k, n = 256, 24
    rng = np.random.default_rng(entries)
    wire = kq.quantize(torch.from_numpy(rng.standard_normal((experts * n, k)).astype(np.float32) * 0.05), codec, None)[0]
    x = torch.from_numpy(rng.standard_normal((50, 1, k)).astype(np.float32)).half().cuda()
    rhs = np.where(rng.random(entries) < 0.3, 1, rng.integers(0, experts - 1, entries))
    lhs = rng.integers(0, 50, entries)
    rhs[5] = experts
    y = kq.gather_qmm(x, wire.reshape(experts, n, -1).cuda(), None, codec, lhs_indices=torch.from_numpy(lhs).cuda(),
                      rhs_indices=torch.from_numpy(rhs).cuda())[:, 0].double().cpu().numpy()
    d = Oracle().dequantize(wire.numpy(), codec, "f32").astype(np.float64).reshape(experts, n, k)
    table = np.einsum("bk,enk->ebn", x[:, 0].double().cpu().numpy(), d)
    ok = rhs < experts
    ref = table[rhs[ok], lhs[ok]]
    # the bound of the other tests of these kernels (weights in fp16); a wrong place is off by the outputs themselves
    assert_close(y[ok], ref, "f16", 2e-3)
