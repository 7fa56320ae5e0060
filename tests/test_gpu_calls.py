"""The native host path of module calls (csrc/py_calls.cpp) against the general path of linear.py, over the forms an input can have:
the same bits, shapes and types where both take it, the same errors where neither does."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


class _General:
    """stands in for the native module: takes nothing, so every call goes the general way"""
    linear = linear_list = staticmethod(lambda *a: None)


def _layers(Ms, N, bias=False):
    from statetree_b200 import TreeLinear
    g = torch.Generator(DEV).manual_seed(sum(Ms) + N)
    out = []
    for M in Ms:
        W = (torch.randn(M, N, device=DEV, generator=g) * 0.05).to(torch.bfloat16)
        b = torch.randn(M, device=DEV, generator=g).to(torch.bfloat16) if bias else None
        out.append(TreeLinear.from_weight(W, b))
    return out


def _forms(N):
    """name -> input of width N"""
    g = torch.Generator(DEV).manual_seed(N)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)                                     # noqa: E731
    bf = lambda *s: r(*s).to(torch.bfloat16)                                                    # noqa: E731
    wide = bf(6, 2 * N)
    flat = bf(5 * N + 8)
    return {"one": bf(1, N), "vector": bf(N), "three": bf(3, N), "lead": bf(2, 1, 3, N), "gemv_last": bf(16, N), "gemm_first": bf(17, N),
            "gemm": bf(2, 65, N), "pairs": bf(331, N), "scratch": bf(600, N), "no_rows": bf(0, N), "no_rows_lead": bf(2, 0, N),
            "float": r(3, N), "half": r(3, N).half(), "strided": wide[:, :N], "columns": bf(N, 4).t(), "expanded": bf(1, N).expand(4, N),
            "offset_2": flat[1:1 + 5 * N].view(5, N), "offset_16": flat[8:8 + 5 * N].view(5, N), "cpu": bf(3, N).cpu(),
            "grad": bf(3, N).requires_grad_()}


# what needs a conversion, and inputs without rows: these go the general way, and nothing is fetched for the other way first
GENERAL = {"no_rows", "no_rows_lead", "float", "half", "strided", "columns", "expanded", "offset_2", "cpu"}
GEMM = {"gemm_first", "gemm", "pairs", "scratch"}


class _Counting:
    """the native module, counting the calls that it is given and those it answers"""

    def __init__(self, module):
        self.module, self.asked, self.answered = module, 0, 0

    def _one(self, name, *args):
        self.asked += 1
        result = getattr(self.module, name)(*args)
        self.answered += result is not None
        return result

    def linear(self, *args):
        return self._one("linear", *args)

    def linear_list(self, *args):
        return self._one("linear_list", *args)


def _both(monkeypatch, call, native, launches):
    """call() with the native module and without it.  native: is the first way served by one native call; launches: products
    that go out otherwise"""
    import statetree_b200.linear as L
    from statetree_b200 import ops
    module, library = ops.calls()
    counting, state, states = _Counting(module), L._state, []
    with monkeypatch.context() as m:
        m.setattr(L, "calls", lambda: (counting, library))
        m.setattr(L, "_state", lambda device: (states.append(device), state(device))[1])
        got = call()
    assert (counting.asked, counting.answered) == ((1, 1) if native else (0, 0))
    assert len(states) == (1 if native else launches)
    with monkeypatch.context() as m:
        m.setattr(L, "calls", lambda: (_General, None))
        want = call()
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.device == b.device and a.shape == b.shape and a.stride() == b.stride()
        assert not a.requires_grad and torch.equal(a, b)


@pytest.mark.parametrize("Ms,N,bias", [((128,), 64, False), ((256,), 512, False), ((256,), 512, True), ((48,), 128, False)])
def test_layer_calls(Ms, N, bias, monkeypatch):
    from statetree_b200 import ops
    tl, = _layers(Ms, N, bias)
    for name, x in _forms(N).items():
        native = not bias and name not in GENERAL and name != "scratch" and not (name in GEMM and Ms[0] % 128)
        _both(monkeypatch, lambda: [tl(x)], native, 1 if x.numel() else 0)
    for bad in (torch.zeros(4, 2 * N), torch.zeros(2 * N), torch.zeros(4, N // 2)):
        with pytest.raises(RuntimeError):
            tl(bad.to(DEV, torch.bfloat16))
    assert ops.device_status() == 0


@pytest.mark.parametrize("Ms,N,bias", [((128, 128), 64, False), ((256, 128, 384), 512, False), ((256, 128), 512, True),
                                       ((48, 16, 32, 64), 128, False)])
def test_list_calls(Ms, N, bias, monkeypatch):
    from statetree_b200 import ops
    from statetree_b200.linear import forward_list
    tls = _layers(Ms, N, bias)
    for name, x in _forms(N).items():
        if x.dim() > 1:
            one_by_one = name in GEMM and any(M % 128 for M in Ms)
            _both(monkeypatch, lambda: forward_list(tls, x), not bias and name not in GENERAL and not one_by_one,
                  (len(Ms) if one_by_one else 1) if x.numel() else 0)
    with pytest.raises(RuntimeError):
        forward_list(tls, torch.zeros(4, 2 * N, dtype=torch.bfloat16, device=DEV))
    assert ops.device_status() == 0


def test_calls_in_a_graph_and_on_another_stream(monkeypatch):
    """outputs come from the capture's pool and the kernels go to the current stream"""
    from statetree_b200.linear import forward_list
    tls = _layers((256, 128), 512)
    x = torch.empty(3, 512, dtype=torch.bfloat16, device=DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call = lambda: forward_list(tls, x) + [tls[0](x)]                                       # noqa: E731
        x.normal_()
        call()
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = call()
        for _ in range(3):
            x.normal_()
            graph.replay()
            side.synchronize()
            for a, b in zip(out, call()):
                assert torch.equal(a, b)
        side.synchronize()


@pytest.mark.parametrize("M,N", [(256, 512), (48, 640), (128, 64)])
def test_library_alone(M, N, monkeypatch):
    """without the native module: conversion with its check, products and lists by the same kernels, the same bits"""
    from statetree_b200 import TreeLinear, format as F, ops
    from statetree_b200.linear import forward_list
    g = torch.Generator(DEV).manual_seed(M + N)
    Ws = [(torch.randn(M, N, device=DEV, generator=g) * 0.05).to(torch.bfloat16), torch.ones(M, N, dtype=torch.bfloat16, device=DEV)]
    Ws[0][:, 5] *= 4096                                         # escapes in one, none in the other
    x = torch.randn(3, N, device=DEV, generator=g).to(torch.bfloat16)

    def work():
        tls = [TreeLinear.from_weight(W) for W in Ws]
        out = [t for tl in tls for t in (tl(x), tl.dequantize(), *tl.tables(), *(tl._buffers[n] for n in ("tree", "esc_rows", "esc_cols", "esc_bits")))]
        enc = F.encode(Ws[0])
        other = Ws[0].clone()
        other[M - 1, N - 1] += 1
        eo, el, _ = tls[0].tables()
        out += forward_list(tls, x) + [enc[k] for k in sorted(enc)]
        return out + [torch.tensor(ops.ext().dec_check(tls[0].tree, eo, el, W)) for W in (Ws[0], other)]

    want = work()
    monkeypatch.setattr(ops, "CALLS_PATH", "/nonexistent/_calls.so")
    monkeypatch.setattr(ops, "_CALLS", None)
    got = work()
    assert [bool(t) for t in got[-2:]] == [True, False]
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    assert ops.device_status() == 0


@pytest.mark.parametrize("same_stream", [False, True])
def test_calls_from_two_threads(same_stream):
    """the native call lets other threads run: layers and inputs shared by two threads, on one stream and on a stream each, give the
    products of a single thread (which are checked against fp64: BF16 results, half an ulp each)"""
    import threading
    from statetree_b200 import ops
    from statetree_b200.linear import forward_list
    N = 1088
    tls = _layers((256, 128, 384), N)
    Ws = [tl.dequantize().double() for tl in tls]
    xs = [torch.randn(B, N, device=DEV).to(torch.bfloat16) for B in (1, 3, 16, 70, 330)]
    work = lambda x: forward_list(tls, x) + [tls[0](x)]                                         # noqa: E731
    want = [work(x) for x in xs]
    for x, ys in zip(xs, want):
        for y, W in zip(ys, Ws + Ws[:1]):
            exact = x.double() @ W.t()
            assert float((y.double() - exact).norm() / exact.norm()) < 2.0 ** -9 * 1.1
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream()] * 2 if same_stream else [torch.cuda.Stream() for _ in range(2)]
    start, got, failed = threading.Barrier(2), [None, None], []

    def thread(i):
        try:
            with torch.cuda.stream(streams[i]), torch.no_grad():
                start.wait()
                got[i] = [[work(x) for x in xs[::1 - 2 * i]] for _ in range(20)]
                streams[i].synchronize()
        except Exception as e:                                  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=thread, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for i in range(2):
        for lap in got[i]:
            for ys, right in zip(lap, want[::1 - 2 * i]):
                assert all(torch.equal(a, b) for a, b in zip(ys, right))
    assert ops.device_status() == 0
