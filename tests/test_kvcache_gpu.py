"""GPU parity of flash_attn_with_kvcache (append + attend + split merge) against the CPU oracle.
Mirrors the functional groups of the reference's KV-cache tests (test_flash_attn.py:1104-1964 of
Cy-47/flash-attention-turing): read, append with cache-content check, explicit splits, paged read and
append, shuffled block tables, page sizes 256/512/768/1024, cache_batch_idx, scale, LSE, int lengths,
MHA, and query chunks of several tokens (decode kernel up to 16 rows per KV head, tiled kernel above)."""
import pytest
import torch

from helpers import LSE_TOL, err_stats, load_golden, randn_half, t
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
O_TOL = 2e-3  # fp16 output rounding of O(1) values; the reference's own bound is atol = rtol = 1e-2


def _run(b, sq, h, hk, d, cap, lens, s_new, paged=False, page=256, splits=0, causal=True, batch_idx=False,
         scale=None, seed=7, poison_tail=False):
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    gen = torch.Generator().manual_seed(seed)
    q = randn_half(gen, b, sq, h, d)
    kn = randn_half(gen, b, s_new, hk, d) if s_new else None
    vn = randn_half(gen, b, s_new, hk, d) if s_new else None
    lens_t = torch.tensor(lens, dtype=torch.int32)
    table = idx = None
    if paged:
        per = (cap + page - 1) // page
        n_pages = b * per + 3
        kc, vc = randn_half(gen, n_pages, page, hk, d), randn_half(gen, n_pages, page, hk, d)
        table = torch.randperm(n_pages, generator=gen)[: b * per].to(torch.int32).view(b, per).contiguous()
    else:
        rows = b + 2 if batch_idx else b
        kc, vc = randn_half(gen, rows, cap, hk, d), randn_half(gen, rows, cap, hk, d)
        if batch_idx:
            idx = torch.randperm(rows, generator=gen)[:b].to(torch.int32)
    if poison_tail and not paged:
        # cache memory past the used length is uninitialised in real use: make it NaN
        for i, n in enumerate(lens):
            row = i if idx is None else int(idx[i])
            kc[row, n + s_new:] = float("nan")
            vc[row, n + s_new:] = float("nan")
    kc_ref, vc_ref = kc.clone(), vc.clone()
    o_ref, lse_ref = orc.kvcache_forward(q, kc_ref, vc_ref, kn, vn, lens_t, idx, table,
                                         d ** -0.5 if scale is None else scale, causal)
    kcd, vcd = kc.to(DEV), vc.to(DEV)
    out, lse = flash_attn_with_kvcache(
        q.to(DEV), kcd, vcd, kn.to(DEV) if s_new else None, vn.to(DEV) if s_new else None,
        cache_seqlens=lens_t.to(DEV), cache_batch_idx=None if idx is None else idx.to(DEV),
        block_table=None if table is None else table.to(DEV), softmax_scale=scale, causal=causal,
        num_splits=splits, return_softmax_lse=True)
    assert not torch.isnan(out).any()
    assert err_stats(out, o_ref)[0] <= O_TOL
    assert err_stats(lse, lse_ref)[0] <= LSE_TOL
    # the appended cache is an observable output: bit-exact copies, nothing else touched
    assert torch.equal(torch.nan_to_num(kcd.cpu()), torch.nan_to_num(kc_ref))
    assert torch.equal(torch.nan_to_num(vcd.cpu()), torch.nan_to_num(vc_ref))
    return out, lse


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("h,hk", [(6, 1), (4, 2), (4, 4)])
@pytest.mark.parametrize("splits", [0, 1, 2, 3, 8])
def test_contiguous_decode(ext, d, h, hk, splits):
    _run(3, 1, h, hk, d, 1024, [1, 511, 1000], 0, splits=splits)
    _run(3, 1, h, hk, d, 1024, [0, 511, 1000], 1, splits=splits)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("page", [256, 512, 768, 1024])
@pytest.mark.parametrize("splits", [0, 1, 4, 16])
def test_paged_decode_append(ext, d, page, splits):
    _run(3, 1, 8, 2, d, 4096, [5, 3000, 4095], 1, paged=True, page=page, splits=splits)


@pytest.mark.parametrize("sq,s_new", [(2, 2), (3, 1), (4, 4), (7, 7), (16, 16), (16, 0), (200, 200), (130, 5)])
@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("causal", [False, True])
def test_query_chunks(ext, sq, s_new, paged, causal):
    # (sq * group) <= 16 rows -> split-KV decode kernel; above -> tiled tcgen05 kernel over the cache
    _run(2, sq, 4, 2, 128, 2048, [300, 1500], s_new, paged=paged, splits=0, causal=causal)
    _run(2, sq, 6, 3, 64, 2048, [0, 1800], s_new, paged=paged, splits=2, causal=causal)


def test_cache_batch_idx_and_scale(ext):
    _run(3, 1, 6, 1, 64, 1024, [1, 511, 1000], 1, splits=2, batch_idx=True, scale=0.3)
    _run(2, 7, 6, 3, 64, 1024, [10, 1000], 7, splits=1, batch_idx=True)
    _run(2, 40, 4, 2, 128, 1024, [10, 900], 40, splits=0, batch_idx=True)


def test_uninitialised_cache_tail_is_never_used(ext):
    _run(2, 1, 4, 2, 128, 1024, [100, 777], 1, splits=1, poison_tail=True)
    _run(2, 1, 4, 2, 64, 1024, [100, 777], 1, splits=4, poison_tail=True)
    # query chunks that go through the tiled tcgen05 kernel (more than 16 rows per KV head)
    _run(2, 40, 4, 2, 128, 1024, [100, 777], 40, splits=0, poison_tail=True)
    _run(2, 130, 4, 4, 64, 1024, [3, 500], 130, splits=0, poison_tail=True, causal=False)


def test_int_and_default_cache_seqlens(ext):
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    gen = torch.Generator().manual_seed(1)
    q, kc, vc = randn_half(gen, 2, 1, 4, 64), randn_half(gen, 2, 320, 2, 64), randn_half(gen, 2, 320, 2, 64)
    o_ref, _ = orc.kvcache_forward(q, kc.clone(), vc.clone(), None, None, [200, 200], None, None, None, True)
    out = flash_attn_with_kvcache(q.to(DEV), kc.to(DEV), vc.to(DEV), cache_seqlens=200, causal=True)
    assert isinstance(out, torch.Tensor) and err_stats(out, o_ref)[0] <= O_TOL
    o_ref, _ = orc.kvcache_forward(q, kc.clone(), vc.clone(), None, None, [320, 320], None, None, None, True)
    out = flash_attn_with_kvcache(q.to(DEV), kc.to(DEV), vc.to(DEV), causal=True)  # whole cache
    assert err_stats(out, o_ref)[0] <= O_TOL


def test_split_counts_agree(ext):
    # the merged result does not depend on the split count beyond fp32 rounding
    outs = [_run(2, 1, 8, 2, 128, 8192, [8000, 4099], 1, paged=True, splits=s)[0] for s in (1, 2, 4, 16, 0)]
    for o in outs[1:]:
        assert err_stats(o, outs[0])[0] <= 1e-3


def test_long_paged_decode(ext):
    # 16k-token paged decode (the reference's largest functional case, test_flash_attn.py:1491-1569)
    _run(2, 1, 8, 2, 128, 16384, [16000, 12345], 1, paged=True, splits=0)


@pytest.mark.parametrize("name", ["fwd_d64_split3", "fwd_d128_decode_split4"])
def test_golden_split_fixtures(ext, name):
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    g = load_golden(name)
    q, k, v = t(g["q"]), t(g["k"]), t(g["v"])
    out, lse = flash_attn_with_kvcache(q.to(DEV), k.to(DEV), v.to(DEV), cache_seqlens=t(g["lens"]).to(DEV),
                                       softmax_scale=float(g["scale"]), causal=bool(g["causal"]),
                                       num_splits=int(g["splits"]), return_softmax_lse=True)
    assert err_stats(out, t(g["out"]))[0] <= O_TOL
    assert err_stats(lse, t(g["lse"]))[0] <= LSE_TOL


@pytest.mark.parametrize("name,paged", [("cache_contiguous", False), ("cache_paged", True)])
def test_golden_cache_append(ext, name, paged):
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    g = load_golden(name)
    kc, vc = t(g["k_cache_before"]).to(DEV), t(g["v_cache_before"]).to(DEV)
    b, hk, d = g["k_new"].shape[0], g["k_new"].shape[2], g["k_new"].shape[3]
    q = torch.zeros(b, 1, hk, d, dtype=torch.half, device=DEV)
    flash_attn_with_kvcache(q, kc, vc, t(g["k_new"]).to(DEV), t(g["v_new"]).to(DEV), cache_seqlens=t(g["lens"]).to(DEV),
                            cache_batch_idx=None if paged else t(g["cache_batch_idx"]).to(DEV),
                            block_table=t(g["block_table"]).to(DEV) if paged else None)
    assert torch.equal(kc.cpu(), t(g["k_cache_after"])) and torch.equal(vc.cpu(), t(g["v_cache_after"]))


def test_cache_batch_idx_out_of_range_is_rejected_on_the_host(ext):
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    q = torch.zeros(1, 1, 2, 64, dtype=torch.half, device=DEV)
    kc = torch.zeros(2, 256, 2, 64, dtype=torch.half, device=DEV)
    with pytest.raises(RuntimeError, match="within cache batch bounds"):
        flash_attn_with_kvcache(q, kc, kc.clone(), cache_seqlens=torch.tensor([4], dtype=torch.int32, device=DEV),
                                cache_batch_idx=torch.tensor([2], dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("splits", [1, 4, 16])
def test_c4_paged_decode_full_size(ext, splits):
    # C4 of the benchmark configs: batch 64, one query token, Hq32 Hkv8 D128, cache_seqlens U[1024, 32768],
    # page 256, 16384-page pool, shuffled block table, in-place append.  Four sequences are checked against
    # the oracle (gathering their pages on the CPU); the appended rows of the pool must hold k/v exactly.
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    b, h, hk, d, page, pages, max_pages = 64, 32, 8, 128, 256, 16384, 129
    gen_c = torch.Generator().manual_seed(1004)
    lens = torch.randint(1024, 32768, (b,), generator=gen_c, dtype=torch.int32)
    perm = torch.randperm(pages, generator=gen_c).to(torch.int32)
    table = torch.zeros(b, max_pages, dtype=torch.int32)
    off = 0
    for i in range(b):
        n = (int(lens[i]) + 1 + page - 1) // page
        table[i, :n] = perm[off:off + n]
        off += n
    gen = torch.Generator(device=DEV).manual_seed(1004)
    kc = torch.randn(pages, page, hk, d, device=DEV, dtype=torch.half, generator=gen)
    vc = torch.randn(pages, page, hk, d, device=DEV, dtype=torch.half, generator=gen)
    q = torch.randn(b, 1, h, d, device=DEV, dtype=torch.half, generator=gen)
    kn = torch.randn(b, 1, hk, d, device=DEV, dtype=torch.half, generator=gen)
    vn = torch.randn(b, 1, hk, d, device=DEV, dtype=torch.half, generator=gen)
    out, lse = flash_attn_with_kvcache(q, kc, vc, kn, vn, cache_seqlens=lens.to(DEV), block_table=table.to(DEV),
                                       causal=True, num_splits=splits, return_softmax_lse=True)
    for i in (0, 17, 40, 63):
        n_tok = int(lens[i]) + 1
        ids = table[i, : (n_tok + page - 1) // page].to(DEV).long()
        ks = kc[ids].reshape(-1, hk, d)[:n_tok].cpu()
        vs = vc[ids].reshape(-1, hk, d)[:n_tok].cpu()
        assert torch.equal(ks[-1], kn[i, 0].cpu()) and torch.equal(vs[-1], vn[i, 0].cpu())  # appended in place
        o_ref, lse_ref = orc.attention_forward_one(q[i].cpu(), ks, vs, d ** -0.5, True)
        assert err_stats(out[i], o_ref)[0] <= O_TOL
        assert err_stats(lse[i], lse_ref)[0] <= LSE_TOL


def test_device_side_capacity_clamp_without_host_check(ext):
    # With the host-side capacity check switched off (no device synchronisation per call) an oversized
    # length must neither read nor write out of bounds: it is clamped to the capacity on the device, the
    # result equals the one for the clamped length, and bit 1 of the status word reports the clamp.
    from flash_attention_turing_b200 import flash_attention_interface as iface

    gen = torch.Generator().manual_seed(4)
    b, h, hk, d, page, per = 2, 4, 2, 128, 256, 2
    kc, vc = randn_half(gen, b * per, page, hk, d), randn_half(gen, b * per, page, hk, d)
    table = torch.arange(b * per, dtype=torch.int32).view(b, per)
    q = randn_half(gen, b, 1, h, d)
    lens_bad = torch.tensor([300, 9999], dtype=torch.int32)       # capacity is 512 tokens per sequence
    lens_ok = torch.tensor([300, 512], dtype=torch.int32)
    o_ref, _ = orc.kvcache_forward(q, kc.clone(), vc.clone(), None, None, lens_ok, None, table, None, True)
    iface.HOST_CAPACITY_CHECK = False
    try:
        out = iface.flash_attn_with_kvcache(q.to(DEV), kc.to(DEV), vc.to(DEV), cache_seqlens=lens_bad.to(DEV),
                                            block_table=table.to(DEV), causal=True, num_splits=2)
        status = ext.device_status(True)
    finally:
        iface.HOST_CAPACITY_CHECK = True
    assert status == 2
    assert err_stats(out, o_ref)[0] <= O_TOL
    with pytest.raises(ValueError, match="cache capacity is insufficient"):
        iface.flash_attn_with_kvcache(q.to(DEV), kc.to(DEV), vc.to(DEV), cache_seqlens=lens_bad.to(DEV),
                                      block_table=table.to(DEV), causal=True)


@pytest.mark.parametrize("b,new,h,hk,d,length,capacity,page,splits", [
    (1, 1, 8, 2, 128, 700, 1024, 0, 0),     # append, attend and merge overlap
    (1, 1, 4, 4, 64, 63, 512, 256, 1),      # no merge; the appended token starts a tile
    (3, 4, 8, 2, 64, 250, 512, 256, 4),     # the new tokens straddle a page
    (2, 64, 4, 2, 128, 190, 512, 256, 0),   # tiled path
])
def test_overlapped_steps_see_the_appended_rows(ext, b, new, h, hk, d, length, capacity, page, splits):
    """The attend kernel starts under the append kernel and the merge under the attend kernel.  The rows that are appended
    hold NaN before every call, so a kernel that did not wait would not return the same bits; also replayed from a graph."""
    torch.manual_seed(0)
    half = lambda *s: torch.randn(*s, device=DEV, dtype=torch.float16)  # noqa: E731
    q, kn, vn = half(b, new, h, d), half(b, new, hk, d), half(b, new, hk, d)
    rows = (b * (capacity // page), page) if page else (b, capacity)
    kc, vc = half(*rows, hk, d), half(*rows, hk, d)
    table = torch.arange(rows[0], dtype=torch.int32, device=DEV).view(b, -1) if page else None
    lens = torch.full((b,), length, dtype=torch.int32, device=DEV)
    flat_k, flat_v = kc.view(b, -1, hk, d), vc.view(b, -1, hk, d)

    def step():
        flat_k[:, length:] = float("nan")
        flat_v[:, length:] = float("nan")
        return ext.fwd_kvcache(q, kc, vc, kn, vn, lens, None, None, None, None, table, None, None, d ** -0.5, True, -1, -1,
                               0.0, True, splits)

    want, want_lse = step()
    torch.cuda.synchronize()
    assert torch.isfinite(want).all() and torch.equal(flat_k[:, length:length + new], kn)
    got = [step() for _ in range(20)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(5):
        graph.replay()
        got.append([x.clone() for x in captured])
    torch.cuda.synchronize()
    for out, lse in got:
        assert torch.equal(out, want) and torch.equal(lse, want_lse)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("splits", [1, 3, 4, 5, 31, 32, 33, 64, 67])
def test_merge_at_the_edges_of_its_batches(ext, d, splits):
    """Partials are fetched four at a time and weights held for 32 splits; empty splits (LSE = -inf, NaN rows) lie between."""
    gen = torch.Generator().manual_seed(splits)
    b, h, sq = 2, 3, 3
    rows = b * h * sq
    o_acc, l_acc = torch.randn(splits, rows, d, generator=gen), torch.randn(splits, rows, generator=gen) * 3
    dead = torch.rand(splits, rows, generator=gen) < 0.4
    dead[:, 0], dead[:, 1] = False, True
    l_acc[dead], o_acc[dead] = float("-inf"), float("nan")
    out, lse = ext.combine(o_acc.to(DEV), l_acc.to(DEV), b, sq, h)
    want = torch.logsumexp(l_acc.double(), 0)
    weight = torch.where(dead, 0.0, torch.exp(l_acc.double() - want))
    o_ref = (weight[..., None] * torch.nan_to_num(o_acc).double()).sum(0)
    want[dead.all(0)] = 0  # nothing to attend to
    got = out.float().cpu().permute(0, 2, 1, 3).reshape(rows, d)
    # half an fp16 ulp of the result, and 1e-5 for the exponentials and the fp32 sums
    assert ((got - o_ref).abs() <= o_ref.abs() * 2 ** -11 + 1e-5).all()
    assert err_stats(lse.view(-1), want)[0] <= 1e-5


def _more_tiles_than_sms(b, sq, h):
    return b * h * -(-sq // 128) > torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("layout", ["contiguous", "paged", "batch_idx"])
def test_chunks_of_more_tiles_than_sms(ext, d, causal, layout):
    """What a serving batch uses: items of two 128-row tiles over a cache (smaller chunks, as in the tests above, get an item per
    tile).  A ragged second tile, an odd number of tiles, an empty cache, and NaN behind the used part of a contiguous one."""
    b, sq, h, hk = 4, 300, 16, 4
    assert _more_tiles_than_sms(b, sq, h)
    _run(b, sq, h, hk, d, 1280, [0, 129, 700, 955], sq, paged=layout == "paged", batch_idx=layout == "batch_idx",
         causal=causal, poison_tail=True)
    _run(b, sq, h, hk, d, 1280, [300, 1, 700, 1280], 0, paged=layout == "paged", batch_idx=layout == "batch_idx",
         causal=causal, poison_tail=True)


@pytest.mark.parametrize("b,sq,h", [(2, 100, 4), (4, 300, 16)])  # an item per tile, items of two tiles
def test_tiled_path_clamps_lengths_to_the_capacity_and_reports_it(ext, b, sq, h):
    from flash_attention_turing_b200 import flash_attention_interface as iface

    assert _more_tiles_than_sms(b, sq, h) == (b == 4)
    gen = torch.Generator().manual_seed(4)
    hk, d, page, per = 2, 64, 256, 2
    kc, vc = randn_half(gen, b * per, page, hk, d), randn_half(gen, b * per, page, hk, d)
    table = torch.randperm(b * per, generator=gen).to(torch.int32).view(b, per)
    q = randn_half(gen, b, sq, h, d)
    lens_bad = torch.tensor([9999, 300, 512, 1][:b], dtype=torch.int32)
    o_ref, _ = orc.kvcache_forward(q, kc.clone(), vc.clone(), None, None, lens_bad.clamp(max=page * per), None, table, None, True)
    iface.HOST_CAPACITY_CHECK = False
    try:
        out = iface.flash_attn_with_kvcache(q.to(DEV), kc.to(DEV), vc.to(DEV), cache_seqlens=lens_bad.to(DEV),
                                            block_table=table.to(DEV), causal=True)
        status = ext.device_status(True)
    finally:
        iface.HOST_CAPACITY_CHECK = True
    assert status == 2
    assert err_stats(out, o_ref)[0] <= O_TOL


@pytest.mark.parametrize("b,sq,new,d,capacity,page", [
    (1, 1, 1, 128, 512, 0),      # append kernel of one block
    (300, 1, 1, 64, 256, 256),   # more lengths than threads of a block
    (3, 2, 0, 128, 512, 0),      # nothing to append: a kernel of its own looks at the lengths
    (2, 64, 64, 64, 512, 256),   # tiled path
])
def test_lengths_beyond_the_capacity_write_nothing(ext, b, sq, new, d, capacity, page):
    """The device finds out whether the lengths fit, under kernels that are already launched: one token too many in the last
    sequence leaves the cache and the status word as they were, and the calls before and after it are not affected."""
    from concurrent.futures import ThreadPoolExecutor

    from flash_attention_turing_b200 import flash_attn_with_kvcache

    torch.manual_seed(b)
    h, hk = 4, 2
    half = lambda *s: torch.randn(*s, device=DEV, dtype=torch.float16)  # noqa: E731
    rows = (b * (capacity // page), page) if page else (b, capacity)
    q, kn, vn, kc, vc = half(b, sq, h, d), half(b, new, hk, d), half(b, new, hk, d), half(*rows, hk, d), half(*rows, hk, d)
    kwargs = dict(k=kn if new else None, v=vn if new else None, causal=True, return_softmax_lse=True,
                  block_table=torch.arange(rows[0], dtype=torch.int32, device=DEV).view(b, -1) if page else None)
    full = torch.full((b,), capacity - new, dtype=torch.int32, device=DEV)  # the last token fits exactly
    over = full.clone()
    over[-1] += 1
    kw, vw = kc.clone(), vc.clone()
    want = flash_attn_with_kvcache(q, kw, vw, cache_seqlens=full, **kwargs)
    k0, v0 = kc.clone(), vc.clone()
    for _ in range(3):
        with pytest.raises(ValueError, match="cache capacity is insufficient"):
            flash_attn_with_kvcache(q, kc, vc, cache_seqlens=over, **kwargs)
    assert torch.equal(kc, k0) and torch.equal(vc, v0)
    assert ext.device_status(False) == 0

    def step(i):
        k, v = kc.clone(), vc.clone()
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
            if i % 2:
                with pytest.raises(ValueError, match="cache capacity is insufficient"):
                    flash_attn_with_kvcache(q, k, v, cache_seqlens=over, **kwargs)
                out = None
            else:
                out = flash_attn_with_kvcache(q, k, v, cache_seqlens=full, **kwargs)
            torch.cuda.current_stream().synchronize()
        return out, k, v

    with ThreadPoolExecutor(4) as pool:  # every thread waits for an answer of its own
        for i, (out, k, v) in enumerate(pool.map(step, range(16))):
            assert torch.equal(k, k0 if i % 2 else kw) and torch.equal(v, v0 if i % 2 else vw)
            assert out is None or (torch.equal(out[0], want[0]) and torch.equal(out[1], want[1]))


@pytest.mark.parametrize("sq,new", [(1, 1), (2, 2), (64, 64)])  # decode kernel, tiled kernel
def test_lengths_near_the_largest_int_do_not_wrap_around(ext, sq, new):
    """cache_seqlens + seqlen_new past 2^31 is beyond the capacity, not negative: refused without a mark in the status word, or
    with HOST_CAPACITY_CHECK off clamped to the capacity like any other length."""
    from flash_attention_turing_b200 import flash_attention_interface as iface

    gen = torch.Generator().manual_seed(sq)
    b, h, hk, d, cap = 2, 4, 2, 64, 256
    q, kn, vn = (randn_half(gen, b, n, x, d).to(DEV) for n, x in ((sq, h), (new, hk), (new, hk)))
    kc, vc = randn_half(gen, b, cap, hk, d).to(DEV), randn_half(gen, b, cap, hk, d).to(DEV)
    k0, v0 = kc.clone(), vc.clone()
    lens = torch.tensor([100, 2 ** 31 - 1], dtype=torch.int32, device=DEV)
    with pytest.raises(ValueError, match="cache capacity is insufficient"):
        iface.flash_attn_with_kvcache(q, kc, vc, kn, vn, cache_seqlens=lens, causal=True)
    assert ext.device_status(False) == 0
    assert torch.equal(kc, k0) and torch.equal(vc, v0)
    want = iface.flash_attn_with_kvcache(q[1:], k0[1:], v0[1:], cache_seqlens=cap, causal=True)
    iface.HOST_CAPACITY_CHECK = False
    try:
        out = iface.flash_attn_with_kvcache(q, kc, vc, kn, vn, cache_seqlens=lens, causal=True)
        status = ext.device_status(True)
    finally:
        iface.HOST_CAPACITY_CHECK = True
    assert status == 2
    assert torch.equal(kc[1], k0[1]) and torch.equal(vc[1], v0[1])
    assert torch.equal(out[1:], want)


def test_errors_of_the_library_become_exceptions(ext):
    """What only the library refuses (an address that is not a multiple of 16 bytes) comes back as RuntimeError with its code and
    message, from each of the bindings."""
    q = torch.randn(2 * 16 * 4 * 64 + 1, device=DEV, dtype=torch.float16)[1:].view(2, 16, 4, 64)
    kv = torch.randn(2, 256, 4, 64, device=DEV, dtype=torch.float16)
    lens = torch.tensor([16, 100], dtype=torch.int32, device=DEV)
    cu = torch.tensor([0, 16, 32], dtype=torch.int32, device=DEV)
    lse = torch.zeros(2, 4, 16, device=DEV)
    flat = q.flatten(0, 1)
    for call in (lambda: ext.fwd(q, kv, kv, 0.125, True),
                 lambda: ext.bwd(q, kv, kv, q, lse, q, 0.125, True),
                 lambda: ext.varlen_fwd(flat, flat, flat, cu, cu, 16, 16, 0.125, True),
                 lambda: ext.fwd_kvcache(q, kv, kv, None, None, lens, None, None, None, None, None, None, None, 0.125, True, -1, -1,
                                         0.0, True, 0)):
        with pytest.raises(RuntimeError, match=r"failed \(-1\): .*16-byte aligned"):
            call()


def test_refused_arguments_cost_no_answer_word(ext):
    """Each thread has one word for the device's answer.  A call that is refused for its arguments, before or after the append kernel
    was launched, keeps it, and it goes with its thread."""
    import time
    from concurrent.futures import ThreadPoolExecutor

    from flash_attention_turing_b200 import flash_attn_with_kvcache

    torch.manual_seed(0)
    b, h, hk, d, cap = 2, 4, 2, 64, 256
    half = lambda *s: torch.randn(*s, device=DEV, dtype=torch.float16)  # noqa: E731
    q, kn, vn, kc, vc = half(b, 1, h, d), half(b, 1, hk, d), half(b, 1, hk, d), half(b, cap, hk, d), half(b, cap, hk, d)
    fits = torch.tensor([100, cap - 1], dtype=torch.int32, device=DEV)
    over = fits + 1

    def call(query=q, cache=kc, lens=fits):
        return flash_attn_with_kvcache(query, cache, vc, kn, vn, cache_seqlens=lens, causal=True)

    want = call()
    unaligned = half(b * h * d + 1)[1:].view(b, 1, h, d)  # refused before anything is launched
    one_head = half(b, cap, 1, d).expand(b, cap, hk, d)   # refused by the attend step, behind the append kernel
    words = ext.kvcache_answer_words()
    for _ in range(20):
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            call(query=unaligned)
        with pytest.raises(RuntimeError, match="strides must be positive"):
            call(cache=one_head)
        for wrong in (dict(query=unaligned), dict(cache=one_head), dict(query=q.float()), {}):
            with pytest.raises(ValueError, match="cache capacity is insufficient"):  # told of first, whatever else is wrong
                call(lens=over, **wrong)
        assert torch.equal(call(), want)
    assert ext.kvcache_answer_words() == words

    with ThreadPoolExecutor(4) as pool:
        for out in pool.map(lambda _: call(), range(32)):
            assert torch.equal(out, want)
    deadline = time.monotonic() + 10
    while ext.kvcache_answer_words() != words and time.monotonic() < deadline:
        time.sleep(0.01)
    assert ext.kvcache_answer_words() == words


def test_an_error_behind_the_launch_is_not_hidden_by_a_second_try(ext, monkeypatch):
    """A failed launch or an answer that never comes is an error of the call: repeating the step on the path that checks beforehand
    would append and attend again and report nothing."""
    from flash_attention_turing_b200 import flash_attention_interface as iface

    class NoAnswer:
        def __getattr__(self, name):
            return getattr(ext, name)

        def fwd_kvcache_checked(self, *args):
            raise RuntimeError("fa_kvcache_checked gave no answer")

    q, kv = torch.zeros(1, 1, 2, 64, device=DEV, dtype=torch.float16), torch.zeros(1, 256, 2, 64, device=DEV, dtype=torch.float16)
    lens = torch.tensor([5], dtype=torch.int32, device=DEV)
    monkeypatch.setattr(iface, "_gpu", NoAnswer)
    with pytest.raises(RuntimeError, match="gave no answer"):
        iface.flash_attn_with_kvcache(q, kv, kv.clone(), cache_seqlens=lens)


@pytest.mark.parametrize("d,h,hk,new,page,cap,lens", [
    (128, 6, 3, 1, 0, 5120, (5000,)),                                        # one sequence over many shares
    (64, 2, 1, 1, 256, 20480, (0, 8000, 1, 64)),                             # parts of several CTAs, empty and one-tile sequences
    (128, 32, 4, 1, 0, 30208, (30000,)),                                     # eight rows, 37 parts: two rounds of rows, two of weights
    (64, 8, 2, 2, 256, 12800, (700, 63, 64, 12000, 2100)),                   # eight rows at two positions, several sequences cut
    (128, 5, 1, 1, 0, 20480, (6000, 10, 15000, 64)),                         # five rows: one warp has two
    (64, 5, 5, 3, 0, 512, tuple((37 * i) % 450 for i in range(70))),         # three rounds of lengths, shares of several sequences
    (128, 32, 32, 1, 0, 256, tuple(1 + (53 * i) % 130 for i in range(40))),  # nine shares per head
    (64, 300, 300, 1, 0, 768, (700,)),                                       # more heads than CTAs: a share per head
])
def test_even_shares_equal_single_splits(ext, d, h, hk, new, page, cap, lens):
    """num_splits = 0 against 1.  P is rounded to fp16 against another reference maximum and O once more: 2^-11 (2 max|V| + max|O|)."""
    import ctypes
    from flash_attention_turing_b200 import capi, flash_attn_with_kvcache

    gen = torch.Generator(device=DEV).manual_seed(9)
    r = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.half)  # noqa: E731
    b = len(lens)
    q, k, v = r(b, new, h, d), r(b, new, hk, d), r(b, new, hk, d)
    rows = (b * cap // page, page) if page else (b, cap)
    kc, vc = r(*rows, hk, d), r(*rows, hk, d)
    table = torch.randperm(rows[0], generator=gen, device=DEV).int().view(b, -1) if page else None
    seqlens = torch.tensor(lens, dtype=torch.int32, device=DEV)
    # the most parts of the even shares: the call does not go to the chunks
    p = capi.kvcache_params(q, kc, vc, k, v, torch.empty_like(q), torch.empty(b, h, new, device=DEV), seqlens, table, d ** -0.5, True, 0)
    assert capi.lib().fa_kvcache_num_splits(ctypes.byref(p)) == max(1, min(296 // hk, -(-(cap + new) // 64)))

    def run(splits):
        return flash_attn_with_kvcache(q, kc, vc, k, v, cache_seqlens=seqlens, block_table=table, causal=True, num_splits=splits,
                                       return_softmax_lse=True)

    (out, lse), (want, want_lse) = run(0), run(1)
    assert (out - want).abs().max() <= 2.0 ** -11 * (2 * vc.abs().max() + want.abs().max())
    assert (lse - want_lse).abs().max() <= 1e-4
    for _ in range(20):  # whoever merges, and whatever the scratch memory held before
        torch.full((1 << 20,), -1, dtype=torch.int32, device=DEV)
        again, again_lse = run(0)
        assert torch.equal(again, out) and torch.equal(again_lse, lse)


def test_even_shares_without_scratch_memory(ext):
    """The calls that needed no scratch memory when num_splits = 0 meant a split count from the shape still need none; others are refused."""
    import ctypes
    from flash_attention_turing_b200 import capi, flash_attn_with_kvcache

    lib, stream = capi.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    r = lambda *s: torch.randn(*s, device=DEV, dtype=torch.half)  # noqa: E731
    for cap, ok in ((512, True), (1024, False)):
        q, kc, vc = r(2, 1, 4, 64), r(2, cap, 2, 64), r(2, cap, 2, 64)
        out, lse = torch.empty_like(q), torch.empty(2, 4, 1, device=DEV)
        lens = torch.tensor([cap, 100], dtype=torch.int32, device=DEV)
        p = capi.kvcache_params(q, kc, vc, None, None, out, lse, lens, None, 0.125, True, 0)
        rc = lib.fa_kvcache(ctypes.byref(p), stream)
        assert rc == (0 if ok else -3)  # FA_ERR_WORKSPACE
        if ok:
            want = flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, num_splits=1)
            assert torch.equal(out, want)


def test_captured_decode_beside_eager_decode(ext, monkeypatch):
    """Sequences over many shares: replays of two graphs, captured more than 1024 launches apart, beside each other and beside eager
    calls on a third stream.  Every result is that of a call by itself, bit for bit."""
    import flash_attention_turing_b200.flash_attention_interface as iface

    monkeypatch.setattr(iface, "HOST_CAPACITY_CHECK", False)
    gen = torch.Generator(device=DEV).manual_seed(12)
    r = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.half)  # noqa: E731

    def inputs(lens, new):
        return r(len(lens), 1, 8, 128), r(len(lens), 20480, 2, 128), r(len(lens), 20480, 2, 128), *(
            (r(len(lens), 1, 2, 128), r(len(lens), 1, 2, 128)) if new else (None, None)), torch.tensor(lens, dtype=torch.int32, device=DEV)

    def call(q, kc, vc, k, v, lens):
        return iface.flash_attn_with_kvcache(q, kc, vc, k, v, cache_seqlens=lens, causal=True, return_softmax_lse=True)

    sets = [inputs((8000, 3000), True), inputs((5000, 7000, 600), False), inputs((100, 6500), True)]
    want = [[x.clone() for x in call(*s)] for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    graphs = []
    for s, stream in zip(sets[:2], streams):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            out = call(*s)
        graphs.append((g, out))
        for _ in range(1023):  # a pool of 1024 counters would come round to the same one
            call(*sets[2])
    torch.cuda.synchronize()
    for _ in range(20):
        eager = []
        for _ in range(20):
            for (g, _), stream in zip(graphs, streams):
                with torch.cuda.stream(stream):
                    g.replay()
            with torch.cuda.stream(streams[2]):
                eager.append(call(*sets[2]))
        torch.cuda.synchronize()
        for got, expected in [(graphs[0][1], want[0]), (graphs[1][1], want[1]), *((e, want[2]) for e in eager)]:
            assert all(torch.equal(x, y) for x, y in zip(got, expected))


def _share_begins(tiles, rows):
    """First tiles of the even shares of sequences of `tiles` 64-token tiles laid end to end, one KV head (csrc/kvcache_sm100.cu)."""
    total, least = sum(tiles), max(2, int((0.05 * max(tiles) * max(rows, 4)) ** 0.5))
    n = min(296, -(-total // least))
    return [i * (total // n) + min(i, total % n) for i in range(n)]


def test_hidden_values_of_a_part_without_visible_keys_stay_out(ext):
    """V that is not finite, causally hidden from a query row and in a part (or a sequence) in which that row sees no key at all: the row
    is that of a cache with finite values there, bit for bit; a row without any visible key is zero."""
    from flash_attention_turing_b200 import flash_attn_with_kvcache

    gen = torch.Generator(device=DEV).manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.half)  # noqa: E731
    d, cap, first = 64, 400 * 64, 40  # tiles of sequence 0; its last one holds a single key
    second = next(n for n in range(20, 200) if first - 1 in _share_begins((first, n, 30, 1), 2))
    lens = torch.tensor([(first - 1) * 64 + 1, second * 64, 30 * 64, 1], dtype=torch.int32, device=DEV)
    q, kc, vc = r(4, 2, 1, d), r(4, cap, 1, d), r(4, cap, 1, d)
    want, want_lse = flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, return_softmax_lse=True)
    for i in (0, 3):
        vc[i, lens[i] - 1] = float("nan")
    out, lse = flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, return_softmax_lse=True)
    assert torch.equal(out[:, 0], want[:, 0]) and torch.equal(out[1:3], want[1:3]) and torch.equal(lse, want_lse)
    assert (out[3, 0] == 0).all() and lse[3, 0, 0] == 0
    assert out[0, 1].isnan().all() and out[3, 1].isnan().all()


@pytest.mark.parametrize("b,hk,cap,new,given,ok", [
    (160, 8, 512, 0, "none", True), (160, 8, 512, 0, "few", True), (160, 8, 512, 0, "odd", True),  # even shares with scratch
    (160, 8, 1024, 1, "few", True),
    (200, 4, 511, 1, "none", True), (200, 4, 512, 1, "none", False), (200, 4, 512, 1, "few", False),
])
def test_scratch_memory_that_does_not_suffice(ext, b, hk, cap, new, given, ok):
    """Calls whose chunk plan is one split a sequence (capacity + new tokens <= 512, or 1184 pairs) never look at a workspace that is
    missing, too small or not aligned; others are refused without it, and then nothing has been appended."""
    import ctypes
    from flash_attention_turing_b200 import capi, flash_attn_with_kvcache

    lib, stream = capi.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    r = lambda *s: torch.randn(*s, device=DEV, dtype=torch.half)  # noqa: E731
    q, kc, vc = r(b, 1, hk, 64), r(b, cap, hk, 64), r(b, cap, hk, 64)
    k, v = (r(b, 1, hk, 64), r(b, 1, hk, 64)) if new else (None, None)
    out, lse = torch.empty_like(q), torch.empty(b, hk, 1, device=DEV)
    lens = (torch.arange(b, device=DEV, dtype=torch.int32) * 37) % (cap - new)
    want = flash_attn_with_kvcache(q, kc.clone(), vc.clone(), k, v, cache_seqlens=lens, causal=True, num_splits=1)
    p = capi.kvcache_params(q, kc, vc, k, v, out, lse, lens, None, 0.125, True, 0)
    need = lib.fa_kvcache_workspace_bytes(ctypes.byref(p))
    room = torch.empty(need + 64, dtype=torch.uint8, device=DEV)
    if given == "few":
        p.workspace, p.workspace_bytes = room.data_ptr(), max(0, need - 1)
    elif given == "odd":
        p.workspace, p.workspace_bytes = room.data_ptr() + 8, need
    before = kc.clone()
    rc = lib.fa_kvcache(ctypes.byref(p), stream)
    assert rc == (0 if ok else -3)  # FA_ERR_WORKSPACE
    assert torch.equal(out, want) if ok else torch.equal(kc, before)
