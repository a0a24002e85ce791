"""gather_qmm(transpose=False) where entries share matrices: the weights of 256 rows at a time in shared memory."""
import numpy as np
import pytest
import torch

import mlx_kquant_b200 as kq
from gpu_util import mint_wire, x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu


# less than a chunk of 256 rows, an odd number, several; columns of one CTA and several, the last one short; one pass of eight
# entries and several (chunks are staged again), matrices without any; rows that are and are not whole sixteens; an odd base
@pytest.mark.parametrize("codec,experts,k,n,entries,off", [
    ("q6_k", 8, 128, 512, 64, 0), ("q6_k", 3, 257, 256, 70, 0), ("q4_k", 5, 31, 768, 9, 0), ("q8_0", 4, 600, 160, 100, 0),
    ("q8_0", 6, 255, 32, 12, 2), ("q6_k", 4, 300, 1280, 40, 1), ("iq4_xs", 3, 256, 256, 60, 0), ("q3_k", 7, 513, 256, 20, 0),
    ("q4_0", 2, 64, 96, 40, 0), ("iq4_nl", 9, 130, 416, 30, 1), ("nvfp4", 4, 140, 192, 33, 0)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_shared_matrices(codec, experts, k, n, entries, off, dt):
    rng = np.random.default_rng(k + n)
    wire = torch.from_numpy(mint_wire(codec, rng.standard_normal((experts * k, n)).astype(np.float32) * 0.05))
    wire = wire.reshape(experts, k, -1)
    room = torch.zeros(wire.numel() + 16, dtype=torch.uint8, device="cuda")
    w = room[off:off + wire.numel()].view(wire.shape)
    w.copy_(wire)
    x, _ = x_to_torch(rng.standard_normal((entries, k)).astype(np.float32), dt)
    rhs = rng.integers(0, experts, entries)
    rhs[rhs == 1] = 0  # (a matrix without entries)
    lhs = rng.permutation(entries)
    y = kq.gather_qmm(x.unsqueeze(1), w, None, codec, lhs_indices=torch.from_numpy(lhs.astype(np.int32)).cuda(),
                      rhs_indices=torch.from_numpy(rhs.astype(np.int32)).cuda(), transpose=False)
    d = Oracle().dequantize(wire.reshape(experts * k, -1).numpy(), codec, "f32").astype(np.float64).reshape(experts, k, n)
    ref = np.einsum("ek,ekn->en", x.double().cpu().numpy()[lhs], d[rhs])
    # float32 sums of at most 600 products, each within 2^-23 of its terms: K 2^-24 of the sum of magnitudes, below
    # 2^-14 of its root mean square scale here; then half a unit of the output type
    off_by = np.abs(y_to_f32(y).reshape(entries, n) - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off_by.max() < 2.0 ** -12 * np.sqrt(np.mean(ref ** 2))
