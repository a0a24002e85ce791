"""gather_qmm of one row per entry in one launch: the row kernel's gather form ([N, K] weights, kq_rows.cu) and the
shared decode of [K, N] weights (kq_qvm.cu), against float64 products of the oracle's weights."""
import numpy as np
import pytest
import torch

from gpu_util import x_to_torch, y_to_f32
from oracle.kq_oracle import Oracle

pytestmark = pytest.mark.gpu

# (matrices, n, k, entries, routing): fewer entries than matrices, one matrix with most entries (several passes, shared
# by CTAs), as many as the kernels take, one more (the general path), ragged rows and stages, odd superblock counts
CASES = [(40, 136, 512, 7, "any"), (16, 72, 256, 200, "one"), (5, 1000, 768, 33, "any"), (64, 128, 512, 512, "even"),
         (8, 40, 1280, 513, "any"), (3, 264, 2048, 1024, "any"), (3, 264, 256, 1025, "one"),
         # a busy matrix's passes in groups of one and of two, among more matrices than 32 and than entries
         (70, 136, 1536, 300, "one"), (2000, 24, 512, 900, "one"), (33, 200, 512, 1024, "one"),
         # [K, N]: one entry a matrix on either side of the rule, few matrices with few and with many entries
         (64, 128, 512, 64, "even"), (1, 512, 512, 3, "even"), (2, 512, 256, 300, "even"), (5, 136, 1280, 5, "even")]


@pytest.mark.parametrize("codec", ["q4_k", "q5_k", "q6_k", "iq4_xs", "q8_0"])
@pytest.mark.parametrize("transpose", [True, False])
@pytest.mark.parametrize("E,n,k,entries,routing", CASES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_gather_rows_against_float64(codec, transpose, E, n, k, entries, routing, dt):
    import mlx_kquant_b200 as kq

    rng = np.random.default_rng(E * 7919 + n + k + entries)
    some = kq.quantize(torch.from_numpy(rng.standard_normal((32, k)).astype(np.float32) * 0.05), codec)[0].numpy()
    pick = rng.integers(0, 32, (E, n))
    dense = Oracle().dequantize(some, codec, "f32").astype(np.float64)
    rhs = rng.integers(0, E, entries)
    if routing == "one":
        rhs[rng.random(entries) < 0.8] = E - 1
    elif routing == "even":
        rhs = np.arange(entries) % E
    lhs = rng.permutation(entries)
    x, _ = x_to_torch(rng.standard_normal((entries, 1, k if transpose else n)).astype(np.float32), dt)
    xr = x.double().cpu().numpy()[lhs, 0]
    y = kq.gather_qmm(x, torch.from_numpy(some[pick]).cuda(), None, codec, lhs_indices=torch.from_numpy(lhs).cuda(),
                      rhs_indices=torch.from_numpy(rhs).cuda(), transpose=transpose)
    y = y_to_f32(y)[:, 0].astype(np.float64)
    ref = np.stack([dense[pick[r]] @ xr[i] if transpose else xr[i] @ dense[pick[r]] for i, r in enumerate(rhs)])
    # half a unit of the output type, and a weight rounded to fp16 where the general path does that (six of its rms)
    off = np.abs(y - ref) - (2.0 ** -11 if dt == "f16" else 2.0 ** -8) * np.abs(ref)
    assert off.max() < 6 * 2.0 ** -11 * np.sqrt(np.mean(ref ** 2))


@pytest.mark.parametrize("transpose", [True, False])
def test_entries_out_of_range_stay_unwritten(transpose):
    import mlx_kquant_b200 as kq

    lib = kq._lib.lib()
    E, n, k, entries = 4, 64, 256, 12
    w = kq.quantize(torch.randn(E * n, k) * 0.05, "q6_k")[0].reshape(E, n, -1).cuda()
    x = torch.randn(entries, 1, k if transpose else n, dtype=torch.float16, device="cuda")
    lhs = torch.arange(entries, dtype=torch.int32, device="cuda")
    rhs = torch.arange(entries, dtype=torch.int32, device="cuda") % E
    good = kq.gather_qmm(x, w, None, "q6_k", lhs_indices=lhs, rhs_indices=rhs, transpose=transpose)
    lhs[3], rhs[5] = entries, E   # a row and a matrix that do not exist
    y = torch.full_like(good, 7.0)
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    kq._lib.check(lib.kq_gather_qmm(x.data_ptr(), 1, entries, 1, x.shape[-1], w.data_ptr(), E, w.stride(0), w.shape[2],
                                    n if transpose else k, b"q6_k", lhs.data_ptr(), rhs.data_ptr(), entries,
                                    int(transpose), 0, y.data_ptr(), ws.data_ptr(), ws.numel(),
                                    torch.cuda.current_stream().cuda_stream))
    keep = torch.ones(entries, dtype=torch.bool, device="cuda")
    keep[3] = keep[5] = False
    assert torch.equal(y[keep], good[keep]) and (y[~keep] == 7.0).all()


def test_last_slice_of_a_long_call():
    """[K, N] weights take at most 65535 entries a launch: the entries of the second one are its own."""
    import mlx_kquant_b200 as kq

    rng = np.random.default_rng(11)
    E, k, n, tail = 4, 32, 32, 9   # the second slice fits the shared decode: at least E entries, at most 512
    wire = kq.quantize(torch.from_numpy(rng.standard_normal((E * k, n)).astype(np.float32)), "q8_0")[0]
    dense = Oracle().dequantize(wire.numpy(), "q8_0", "f32").astype(np.float64).reshape(E, k, n)
    entries = 65535 + tail
    x = torch.from_numpy(rng.standard_normal((64, 1, k))).half()
    lhs, rhs = rng.integers(0, 64, entries), rng.integers(0, E, entries)
    y = kq.gather_qmm(x.cuda(), wire.reshape(E, k, -1).cuda(), None, "q8_0", lhs_indices=torch.from_numpy(lhs).cuda(),
                      rhs_indices=torch.from_numpy(rhs).cuda(), transpose=False)[:, 0].double().cpu().numpy()
    ref = np.einsum("ek,ekn->en", x[:, 0].double().numpy()[lhs], dense[rhs])
    # half a unit of fp16, and float32 sums of 32 terms
    assert (np.abs(y - ref) <= 2.0 ** -11 * np.abs(ref) + 2.0 ** -18 * np.sqrt(np.mean(ref ** 2))).all()
