"""The tcgen05 GEMM on CTA pairs (more than 320 activation rows, and fewer where it is the faster one) at the sizes where it can
go wrong, against fp64 products over the exact weights.

fp32 accumulators: a k range of N products is summed in fp32, so an element's error is at most N * 2^-24 of the sum of the
products' magnitudes (the worst case; |x| |W|^T below).  BF16 output: the rounded accumulator, bit for bit.
"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _weight(M, N, seed):
    g = torch.Generator(DEV).manual_seed(seed)
    W = (torch.randn(M, N, device=DEV, generator=g) * 0.05).to(torch.bfloat16)
    W[:, 5] *= 4096                                             # escapes in every row's first record
    W[M // 2] *= torch.where(torch.rand(N, device=DEV, generator=g) < 0.5, 2.0 ** -30, 1.0).to(torch.bfloat16)   # a crowded row
    return W


def _check(y, yf, W, x):
    want, size = x.double() @ W.double().t(), x.double().abs() @ W.double().abs().t()
    if yf is not None:
        assert torch.equal(y, yf.to(torch.bfloat16))
        assert float(((yf.double() - want).abs() / size).max()) <= W.shape[1] * 2.0 ** -24
    assert float(((y.double() - want).abs() - W.shape[1] * 2.0 ** -24 * size - 2.0 ** -8 * want.abs()).max()) <= 0.0


# token tiles: one MMA of 32 to 256 tokens, two of equal and of different widths (288 = 160 + 128, 352 = 192 + 160, 384), ragged
# last tiles, two and more tiles; row blocks: one (the pair's second CTA has none), odd, even; k-tiles: one (half of a pair), odd,
# a split k range; more units than the SMs hold at once (persistent clusters)
@pytest.mark.parametrize("M,N,Bs", [(128, 64, (321, 384, 385)), (384, 320, (321, 352, 353, 384, 641)), (256, 2048, (330, 384, 770)),
                                    (2048, 2048, (129, 200, 300, 500)), (128 * 149, 64, (129, 352, 700)), (128 * 75, 640, (257, 769, 1153)),
                                    (128 * 192, 192, (160, 289, 384))])
def test_pairs_match_fp64(M, N, Bs, monkeypatch):
    import statetree_b200.linear as L
    from statetree_b200 import TreeLinear, ops
    monkeypatch.setattr(L, "PREFILL_MIN", 0)
    W = _weight(M, N, M + N)
    tl = TreeLinear.from_weight(W)
    for B in Bs:
        x = torch.randn(B, N, device=DEV, generator=torch.Generator(DEV).manual_seed(B)).to(torch.bfloat16)
        guard = torch.full((B + 8, M), 7.0, dtype=torch.bfloat16, device=DEV)     # rows behind the output stay as they are
        yf = torch.full((B, M), float("nan"), device=DEV)
        tl._run(x, guard[:B], yf)
        _check(guard[:B], yf, W, x)
        assert bool((guard[B:] == 7.0).all())
        assert torch.equal(tl(x), guard[:B])                                    # without the fp32 output, and again
    assert ops.device_status() == 0


@pytest.mark.parametrize("Ms,N,B", [((128, 128), 256, 321), ((128, 256, 384), 320, 400), ((128 * 147, 128, 128 * 2), 128, 385),
                                    ((256, 128, 128, 640), 1024, 700)])
def test_lists_on_pairs(Ms, N, B):
    """members that begin and end inside a CTA pair's 256 rows"""
    from statetree_b200 import TreeLinear, ops
    from statetree_b200.linear import forward_list
    Ws = [_weight(M, N, M + i) for i, M in enumerate(Ms)]
    x = torch.randn(B, N, device=DEV, generator=torch.Generator(DEV).manual_seed(B)).to(torch.bfloat16)
    for W, y in zip(Ws, forward_list([TreeLinear.from_weight(W) for W in Ws], x)):
        _check(y, None, W, x)
    assert ops.device_status() == 0


class _Node(ctypes.Structure):
    """CUDA_KERNEL_NODE_PARAMS of cuda.h"""
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def _kernels(fn):
    """[(name of the kernel, CTAs of a cluster)] that fn launches, read from a captured graph, and what fn returns, replayed"""
    cu, side = ctypes.CDLL("libcuda.so.1"), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
        side.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph, stream=side):
            out = fn()
        handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
        assert cu.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
        nodes = (ctypes.c_void_p * n.value)()
        assert cu.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
        found = []
        for node in nodes:
            p, name, cluster = _Node(), ctypes.c_char_p(), (ctypes.c_uint * 16)()          # (an attribute's value: 64 bytes)
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            ask, which = (cu.cuFuncGetName, p.func) if p.func else (cu.cuKernelGetName, p.kern)
            assert ask(ctypes.byref(name), ctypes.c_void_p(which)) == 0
            assert cu.cuGraphKernelNodeGetAttribute(ctypes.c_void_p(node), 4, cluster) == 0    # 4: the cluster's dimensions
            found.append(("pair" if b"pair_kernel" in name.value else "one" if b"gemm_kernel" in name.value else name.value.decode(),
                          max(1, cluster[0])))
        graph.replay()
        side.synchronize()
        return found, [t.clone() for t in out]


def _on_148_sms():
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the splits are those of 148 SMs")


@pytest.mark.parametrize("M,tiles,B,split", [(2048, 65, 700, 2), (128, 41, 257, 3), (384, 41, 512, 3), (128, 85, 257, 4), (384, 85, 257, 4),
                                             (2048, 64, 700, 2)])
def test_split_with_an_odd_last_tile(M, tiles, B, split):
    """a k range split over pairs whose last one ends with half a pair of k-tiles (and an even number of tiles beside it)"""
    from statetree_b200 import TreeLinear, ops
    _on_148_sms()
    W = _weight(M, tiles * 64, M + tiles)
    tl = TreeLinear.from_weight(W)
    tl.allow_dec = False
    x = torch.randn(B, tiles * 64, device=DEV, generator=torch.Generator(DEV).manual_seed(B)).to(torch.bfloat16)
    guard, yf = torch.full((B + 8, M), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((B, M), float("nan"), device=DEV)
    tl._run(x, guard[:B], yf)
    _check(guard[:B], yf, W, x)
    assert bool((guard[B:] == 7.0).all())
    kernels, (y,) = _kernels(lambda: [tl(x)])
    assert kernels == [("pair", 2 * split)] and torch.equal(y, guard[:B])
    assert ops.device_status() == 0


# tiles of one CTA beyond 320 rows: two (176 and 192 wide, the last one ragged or with a single row), three, five; a k range split
# and not, odd numbers of k-tiles; lists
@pytest.mark.parametrize("Ms,tiles,B", [((128,), 33, 321), ((128,), 97, 1300), ((384,), 47, 641), ((1152,), 65, 700), ((4608,), 56, 384),
                                        ((128, 256), 33, 353), ((128 * 9, 128 * 27), 56, 384)])
def test_one_cta_per_tile_beyond_320_rows(Ms, tiles, B):
    from statetree_b200 import TreeLinear, ops
    from statetree_b200.linear import forward_list
    _on_148_sms()
    N = tiles * 64
    Ws = [_weight(M, N, M + i) for i, M in enumerate(Ms)]
    tls = [TreeLinear.from_weight(W) for W in Ws]
    for tl in tls:
        tl.allow_dec = False
    x = torch.randn(B, N, device=DEV, generator=torch.Generator(DEV).manual_seed(B)).to(torch.bfloat16)
    if len(tls) == 1:
        guard, yf = torch.full((B + 8, Ms[0]), 7.0, dtype=torch.bfloat16, device=DEV), torch.full((B, Ms[0]), float("nan"), device=DEV)
        tls[0]._run(x, guard[:B], yf)
        _check(guard[:B], yf, Ws[0], x)
        assert bool((guard[B:] == 7.0).all())
    kernels, ys = _kernels(lambda: forward_list(tls, x))
    assert [k for k, _ in kernels] == ["one"]
    for W, y in zip(Ws, ys):
        _check(y, None, W, x)
    assert ops.device_status() == 0


# measured, us, one CTA per tile / pairs, from the second: 11.2 / 10.1, 11.1 / 12.7, 18.2 / 22.3, 28.2 / 24.8, 32.4 / 29.7, 17.5 / 20.2
@pytest.mark.parametrize("M,N,B,kernel", [(2048, 2048, 128, "one"), (2048, 2048, 300, "pair"), (2048, 2048, 321, "one"), (4608, 3584, 321, "one"),
                                          (6144, 4096, 321, "pair"), (4608, 3584, 1000, "pair"), (4096, 4096, 300, "one")])
def test_kernel_of_a_batch(M, N, B, kernel):
    """beyond 128 rows the kernel that is estimated to be the faster: where the two differ by a tenth, it is"""
    from statetree_b200 import TreeLinear, ops
    _on_148_sms()
    W = _weight(M, N, M + B)
    tl = TreeLinear.from_weight(W)
    tl.allow_dec = False
    x = torch.randn(B, N, device=DEV, generator=torch.Generator(DEV).manual_seed(B)).to(torch.bfloat16)
    kernels, (y,) = _kernels(lambda: [tl(x)])
    assert {k for k, _ in kernels} == {kernel}
    _check(y, None, W, x)
    assert ops.device_status() == 0


@pytest.mark.parametrize("M,N,B", [(128 * 149, 1024, 321), (128 * 224, 2048, 330)])
def test_one_launch_where_it_is_the_faster(M, N, B):
    """between one and two waves of CTA pairs: one launch, whose clusters take a second unit, instead of a full wave and a rest with a
    split of its own (measured, us, two launches / one: 28672 x 2048 at 330 rows 45.8 / 39.2)"""
    from statetree_b200 import TreeLinear, ops
    _on_148_sms()
    W = _weight(M, N, M + B)
    tl = TreeLinear.from_weight(W)
    tl.allow_dec = False
    x = torch.randn(B, N, device=DEV, generator=torch.Generator(DEV).manual_seed(B)).to(torch.bfloat16)
    kernels, (y,) = _kernels(lambda: [tl(x)])
    assert kernels == [("pair", 2)]
    _check(y, None, W, x)
    assert ops.device_status() == 0
