"""Conversion of matrices and of whole KV pages: the forms of a block's loads, and the prefix sums between the two passes."""
import pytest
import torch

import gen_inputs as G
from util import bits_to_torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("offset,extra", [(0, 0), (2, 0), (8, 0), (0, 2), (6, 10), (8, 8)])
@pytest.mark.parametrize("n", [16, 40, 1040])
def test_whole_pages_from_rows_of_any_alignment(offset, extra, n):
    """keys and values at a 4-byte offset, or with a token stride, that rules 16-byte loads out (or not): the same page bytes,
    pool and counters as from a contiguous copy"""
    from statetree_b200.kvcache import PageStore
    H = 3
    K, V = (bits_to_torch(t, DEV) for t in G.kv_tokens(n, H, seed=offset + extra + n, tiny=0.02))
    slots = torch.arange(n, device=DEV)
    stores = []
    for strided in (False, True):
        if strided:
            views = []
            for t in (K, V):
                flat = torch.zeros(offset + n * (H * 128 + extra), dtype=torch.bfloat16, device=DEV)
                view = flat[offset:].view(n, H * 128 + extra)[:, :H * 128].unflatten(1, (H, 128))
                view.copy_(t)
                views.append(view)
        else:
            views = [K, V]
        st = PageStore(-(-n // 16), H, DEV, pool_blocks=4096)
        st.append(*views, slots)
        torch.cuda.synchronize()
        st.check()
        stores.append(st)
    a, b = stores
    assert torch.equal(a.pages[..., :1552], b.pages[..., :1552])
    assert torch.equal(a.dense()[0], b.dense()[0]) and torch.equal(a.dense()[1], b.dense()[1])
    assert torch.equal(b.dense()[0].reshape(-1, H, 128)[:n], K) and torch.equal(b.dense()[1].reshape(-1, H, 128)[:n], V)
    assert int(a.pcnt[0]) == int(b.pcnt[0])


@pytest.mark.parametrize("M,N", [(16, 64), (256, 1024), (256, 1088), (272, 1024), (4096, 64), (16, 64 * 4097), (4096, 4096)])
def test_offsets_are_the_prefix_sums(M, N):
    """chunks of 4096 counts: fewer than one, exactly one, one more, many; byte arrays whose length is no multiple of 16 of them"""
    from statetree_b200.ops import lib
    NG, L = N // 64, lib()
    g = torch.Generator(DEV).manual_seed(M + N)
    rowcnt = torch.randint(0, 65, (M * NG,), device=DEV, generator=g).to(torch.uint8)
    reccnt = torch.randint(0, 1025, (M // 16 * NG + 1,), device=DEV, generator=g).to(torch.int32)
    roff, eo = (torch.full((t.numel() + 8,), -7, dtype=torch.int32, device=DEV) for t in (rowcnt, reccnt))
    need = L.st_encode_offsets_workspace_bytes(M, N)
    ws = torch.empty(need, dtype=torch.uint8, device=DEV)
    stream = torch.cuda.current_stream().cuda_stream
    args = (rowcnt.data_ptr(), reccnt.data_ptr(), M, N, roff.data_ptr(), eo.data_ptr(), ws.data_ptr())
    assert L.st_encode_offsets(*args, need - 1, stream) != 0                    # (refused: nothing runs)
    assert L.st_encode_offsets(*args, need, stream) == 0
    for out, counts in ((roff, rowcnt), (eo, reccnt)):
        n = counts.numel()
        assert torch.equal(out[:n], counts.to(torch.int64).cumsum(0).to(torch.int32)) and bool((out[n:] == -7).all())


@pytest.mark.parametrize("how", ["whole", "shifted", "holes", "outside", "reversed_pages"])
def test_long_appends_equal_short_ones(how):
    """a call of 1024 tokens and more (a warp per sixteen tokens, rows requested before their slots are looked up) against the same
    tokens one call each: groups that are whole pages, start inside one, have dropped or foreign tokens"""
    from statetree_b200.kvcache import PageStore
    H, n = 2, 1061
    K, V = (bits_to_torch(t, DEV) for t in G.kv_tokens(n, H, seed=n, tiny=0.02))
    slots, pages = torch.arange(n, device=DEV), n // 16 + 3
    if how == "shifted":
        slots = slots + 5
    elif how == "holes":
        slots[torch.arange(0, n, 37, device=DEV)] = -1
    elif how == "outside":
        slots[160:176] += pages * 16
        slots[200:205] = -1
    elif how == "reversed_pages":
        slots = (n // 16 - slots // 16) * 16 + slots % 16
    stores = []
    for step in (n, 1):
        st = PageStore(pages, H, DEV, pool_blocks=4096)
        for reuse in (False, True):                             # (the second time over pages that have chains)
            for a in range(0, n, step):
                st.append(K[a:a + step], V[a:a + step], slots[a:a + step].contiguous(), reuse)
        torch.cuda.synchronize()
        st.check()
        stores.append(st)
    for x, y in zip(stores[0].dense(), stores[1].dense()):
        assert torch.equal(x, y)
    ok = (slots >= 0) & (slots < pages * 16)
    assert torch.equal(stores[0].dense()[0].view(-1, H, 128)[slots[ok]], K[ok])
