"""Rows appended behind the first of a page that was never written (the page's memory holds anything): its header names escape slots
and a pool block that do not exist, which must not be followed."""
import pytest
import torch

import gen_inputs as G
from util import bits_to_torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("fill", [0xFF, 0x1F])
@pytest.mark.parametrize("n", [6, 1040])
def test_rows_behind_a_header_that_names_no_block(fill, n):
    from statetree_b200 import ops
    from statetree_b200.kvcache import PageStore
    H, P = 2, 1 << 12
    K, V = (bits_to_torch(t, DEV) for t in G.kv_tokens(n, H, seed=n + fill, tiny=0.02))
    st = PageStore(-(-(n + 5) // 16), H, DEV, pool_blocks=P)
    st.pages.fill_(fill)                                        # header 0xFFFFFFFF: block 2^24 - 1; 0x1F1F1F1F: block 2039583
    st.append(K, V, torch.arange(n, device=DEV) + 5)
    torch.cuda.synchronize()
    st.check()
    for dense, want in zip(st.dense(), (K, V)):
        got = dense.reshape(-1, H, 128)[5:5 + n]
        # what the page held before stays in its eleven slots: row 15, column 63 of each half (0xFFFF...) or row 12, column 31
        wild = torch.zeros_like(want, dtype=torch.bool)
        row, col = (15, 63) if fill == 0xFF else (0x1F1F1F1F >> 6 & 15, 0x1F1F1F1F & 63)
        for half in (0, 64):
            if row - 5 < min(n, 11):
                wild[row - 5, :, half + col] = True
        assert torch.equal(got[~wild].view(torch.int16), want[~wild].view(torch.int16))
    assert ops.device_status() == 0
