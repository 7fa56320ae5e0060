"""The tcgen05 GEMM on CTA pairs (more than 320 activation rows, and fewer where it is the faster one) at the sizes where it can
go wrong, against fp64 products over the exact weights.

fp32 accumulators: a k range of N products is summed in fp32, so an element's error is at most N * 2^-24 of the sum of the
products' magnitudes (the worst case; |x| |W|^T below).  BF16 output: the rounded accumulator, bit for bit.
"""
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
