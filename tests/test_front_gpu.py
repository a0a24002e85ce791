"""quantized_matmul's native front (csrc/kq_torch.cpp) against the Python form of the same call."""
import threading

import pytest
import torch

import mlx_kquant_b200 as kq
from mlx_kquant_b200 import _lib, ops

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wire():
    g = torch.Generator().manual_seed(3)
    return {c: kq.quantize(torch.randn(96, 512, generator=g) * 0.05, c, None)[0].cuda() for c in ("q4_k", "q6_k", "q8_0")}


def both(monkeypatch, call):
    """The call as it is, and with the front out of the way; an exception counts as an outcome."""
    def outcome():
        try:
            return call()
        except Exception as e:
            return type(e), str(e)
    here = outcome()
    with monkeypatch.context() as m:
        m.setattr(ops, "_front_qmm", lambda *args: None)
        return here, outcome()


def same(a, b):
    if not isinstance(a, torch.Tensor):
        return a == b
    return (type(a) is type(b) and a.shape == b.shape and a.stride() == b.stride() and a.dtype == b.dtype and a.device == b.device
            and a.requires_grad == b.requires_grad and torch.equal(a.view(torch.int16), b.view(torch.int16)))


def test_it_is_there(wire):
    front = _lib.torch_front()
    x = torch.randn(1, 512, device="cuda").half()
    assert isinstance(front.qmm(x, wire["q4_k"], "q4_k", True), torch.Tensor)
    assert front.qmm(x, wire["q4_k"], "no_codec", True) is None and front.qmm(x.cpu(), wire["q4_k"], "q4_k", True) is None
    assert front.qmm(x, wire["q4_k"], "q4_k", False) is None and front.qmm(x, wire["q4_k"][:, 144:], "q4_k", True) is None


@pytest.mark.parametrize("codec", ["q4_k", "q6_k", "q8_0"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32, torch.float64])
def test_forms(monkeypatch, wire, codec, dtype):
    w = wire[codec]
    x = torch.randn(24, 1024, device="cuda", dtype=dtype)
    forms = [x[:1, :512].contiguous(), x[0, :512], x[:5, :512], x[:16, 512:], x[:17, :512].contiguous(), x[:1, 1:513],
             x[:4, :1024:2], x[:12, :512].contiguous().view(3, 4, 512), x[:12, :512].view(3, 4, 512), x[:0, :512], x[:2, :256],
             torch.nn.Parameter(x[:2, :512].contiguous()), x[:3, :512].contiguous().requires_grad_(), x[:1, :512].contiguous().cpu(),
             x[:2, :512].contiguous().expand(2, 512), x[:1, :512].expand(3, 512)]
    for f in forms:
        a, b = both(monkeypatch, lambda: kq.quantized_matmul(f, w, None, codec))
        assert same(a, b), (tuple(f.shape), f.stride(), a, b)
    one = forms[0]
    others = [lambda: kq.quantized_matmul(one, w[:, :-1], None, codec), lambda: kq.quantized_matmul(one, w[::2], None, codec),
              lambda: kq.quantized_matmul(one, w.cpu(), None, codec), lambda: kq.quantized_matmul(one, w.int(), None, codec),
              lambda: kq.quantized_matmul(one, w, None, "q9_k"), lambda: kq.quantized_matmul(one, w[None], None, codec),
              lambda: kq.quantized_matmul(one, torch.nn.Parameter(w, requires_grad=False), None, codec),
              lambda: kq.quantized_matmul(x[:2, :96], w, None, codec, transpose=False),
              lambda: torch.vmap(lambda v: kq.quantized_matmul(v, w, None, codec))(forms[2]),
              lambda: kq.quantized_matmul(one, w, None, codec, stream=torch.cuda.current_stream())]
    for call in others:
        a, b = both(monkeypatch, call)
        assert same(a, b), (a, b)


def test_capture_inference_and_threads(wire):
    w, x = wire["q4_k"], torch.randn(1, 512, device="cuda").bfloat16()
    ref = kq.quantized_matmul(x, w, None, "q4_k")
    g, out = torch.cuda.CUDAGraph(), None
    with torch.cuda.graph(g):
        out = kq.quantized_matmul(x, w, None, "q4_k")
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
    with torch.inference_mode():
        assert kq.quantized_matmul(x, w, None, "q4_k").is_inference()
    results = {}

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            xi = torch.full_like(x, float(i))
            results[i] = [kq.quantized_matmul(xi, w, None, "q4_k") for _ in range(50)][-1]
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for i, y in results.items():
        assert torch.equal(y, kq.quantized_matmul(torch.full_like(x, float(i)), w, None, "q4_k"))
