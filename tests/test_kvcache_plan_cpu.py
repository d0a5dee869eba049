"""Which kernel attends a KV-cache call with num_splits = 0, and the scratch memory it asks for: host-side rules, asked of the library
without a GPU."""
import ctypes

import pytest

from flash_attention_turing_b200 import capi

pytestmark = pytest.mark.skipif(not capi.LIB_PATH.exists(), reason="libfa_b200.so not built")


def _params(b, capacity, hk, rows, d=128, new=0, splits=0):
    p = capi.FaKvcacheParams()
    p.b, p.seqlen_q, p.seqlen_new, p.h, p.h_k, p.d = b, 1, new, rows * hk, hk, d
    p.cache_batch, p.seqlen_cache, p.num_splits = b, capacity, splits
    return p


def _chunks(b, capacity, hk, new=0):
    """Split count of the chunk plan: fixed chunks of at least 8 tiles of 64 tokens, about 1184 CTAs at full capacity."""
    tiles = -(-(capacity + new) // 64)
    chunk = max(8, -(-tiles // min(256, -(-1184 // (b * hk)))))
    return -(-tiles // chunk)


# (sequences, capacity, KV heads, rows per KV head, head size 128 unless it follows)
CHUNKS = [
    (2, 9200, 2, 4), (2, 9200, 2, 1), (9, 4738, 1, 1), (4, 3200, 4, 1),   # 75 to 148 chunks, all at once
    (2, 9200, 2, 8), (4, 3200, 4, 5), (4, 9200, 4, 8), (1, 9200, 8, 8),   # two rows a warp
    (33, 389, 12, 1), (4, 400, 8, 1), (150, 450, 8, 8),                  # one chunk a sequence
    (16384, 160, 1, 2), (4096, 200, 1, 4), (512, 1000, 4, 2),            # the tiles of many sequences are counted by every CTA
    (16, 1600, 149, 1), (16, 1600, 99, 1), (2, 1600, 300, 1),            # heads that leave CTAs over
    (4, 9200, 1, 16),                                                    # sixteen rows
    (97, 3842, 32, 1, 64), (97, 1000, 32, 1), (60, 10240, 16, 1), (34, 22344, 16, 1, 64),  # large batches
]
SHARES = [
    (1, 4096, 8, 4), (1, 30200, 8, 4), (1, 3200, 2, 8),                   # one sequence
    (2, 30200, 8, 4), (64, 33024, 8, 4), (2, 30200, 8, 8), (16, 9200, 4, 8), (4, 20000, 1, 1),
    (128, 164, 32, 1), (2048, 110, 8, 2), (1024, 110, 4, 2),              # short ones, several rounds of chunks
    (23, 600, 12, 1), (4, 700, 8, 8),                                    # never cut
    (16, 1600, 64, 1), (16, 1600, 130, 1, 64), (2, 3200, 2, 4), (2, 3200, 4, 1), (97, 1000, 32, 1, 64), (60, 5000, 16, 1),
]


@pytest.mark.parametrize("case", CHUNKS)
def test_chunks_where_they_are_faster(case):
    b, capacity, hk, rows, d = (*case, 128)[:5]
    p = _params(*case)
    splits = _chunks(b, capacity, hk)
    assert capi.lib().fa_kvcache_num_splits(ctypes.byref(p)) == splits
    need = 0 if splits == 1 else sum(-(-splits * b * hk * rows * n * 4 // 256) * 256 for n in (d, 1))
    assert capi.lib().fa_kvcache_workspace_bytes(ctypes.byref(p)) == need


@pytest.mark.parametrize("case", SHARES)
def test_even_shares_elsewhere(case):
    b, capacity, hk = case[:3]
    p = _params(*case)
    tiles, shares = -(-capacity // 64), max(1, min(296 // hk, -(-capacity // 64) * b))
    cut = shares > 1 and not (tiles <= 12 and b <= shares)
    want = min(shares, tiles) if cut else 1
    assert capi.lib().fa_kvcache_num_splits(ctypes.byref(p)) == want
    if (b, hk) == (1, 8) or want > 1:
        assert want != _chunks(b, capacity, hk)  # the case tells the two apart
    assert (capi.lib().fa_kvcache_workspace_bytes(ctypes.byref(p)) > 0) == cut
