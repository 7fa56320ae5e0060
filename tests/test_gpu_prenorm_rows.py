"""The GEMV that forms RMSNorm(x + delta) * w itself, at row lengths and batches where the batches of loads end unevenly."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows of one 16-byte vector per thread and fewer, of two with a ragged second, of exactly two, of three (beyond the norm weights kept
# in registers); the vectors of 1 to 8 rows in batches of four: whole batches, one left over, a row that ends inside a batch
@pytest.mark.parametrize("N", [64, 2048, 2112, 4096, 4160, 6144])
@pytest.mark.parametrize("B", [1, 2, 3, 5, 8])
def test_prenorm_rows(N, B):
    """residual stream bit for bit; the product against fp64 over the rows as the kernel rounds them (BF16 after the norm and after
    the weights: two half ulps of 2^-9, and half an ulp of the BF16 result)"""
    from statetree_b200 import ops, TreeLinear
    from statetree_b200.linear import _state
    E, M = ops.ext(), 256
    if not E.gemv_prenorm_supported(M, N, B, False):
        pytest.skip("rows do not fit in shared memory")
    g = torch.Generator(device=DEV).manual_seed(N + B)
    W = (torch.randn(M, N, device=DEV, generator=g) * 0.05).to(torch.bfloat16)
    tl = TreeLinear.from_weight(W)
    eo, el, eb = tl.tables()
    x, d = (torch.randn(B, N, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    nw = (1 + 0.1 * torch.randn(N, device=DEV, generator=g)).to(torch.bfloat16)
    ws = _state(torch.device(DEV)).get_ws(E.gemv_workspace_bytes(M, N, B))
    for delta in (d, None):
        stream = x if delta is None else (x.float() + d.float()).to(torch.bfloat16)
        x_out, y = torch.full_like(x, 7.0), torch.empty(B, M, dtype=torch.bfloat16, device=DEV)
        E.gemv_prenorm(tl.tree, eo, eb, el, x, delta, nw, 1e-6, x_out, y, ws, False)
        torch.cuda.synchronize()
        assert torch.equal(x_out, stream)
        s = stream.double()
        h = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()
        want, size = h @ W.double().t(), h.abs() @ W.double().abs().t()
        assert float(((y.double() - want).abs() - (2 * 2.0 ** -9 + N * 2.0 ** -24 + 2.0 ** -16) * size - 2.0 ** -9 * 1.02 * want.abs()).max()) <= 0.0
        again = torch.empty_like(y)
        E.gemv_prenorm(tl.tree, eo, eb, el, x, delta, nw, 1e-6, x_out, again, ws, False)
        assert torch.equal(y, again)
    assert ops.device_status() == 0
