"""GPU parity of the forward and backward kernels against the CPU fp32 oracle, through the torch
binding (which calls the C ABI).  Shapes follow the reference's grid (test_flash_attn.py:51-140 of
Cy-47/flash-attention-turing: odd lengths, Sq != Sk both ways, GQA/MQA head pairs, both head dims,
causal on/off, explicit scale) plus MHA cases for the packed variants, which the reference's grid
never reaches (all of its head pairs have Hq != Hk)."""
import ctypes

import pytest
import torch

from helpers import (LSE_TOL, assert_reference_suite_bounds, assert_within_twice_reference_kernel,
                     emulate_reference_kernel, emulate_reference_kernel_one, emulate_reference_kernel_varlen,
                     err_stats, load_golden, randn_half, t)
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"

SEQ_PAIRS = [(1, 1), (2, 2), (63, 65), (65, 63), (127, 129), (128, 128), (129, 257), (257, 129), (113, 203),
             (256, 512), (512, 256), (384, 384), (897, 1024), (1025, 1023), (1, 239), (239, 1), (799, 3), (3, 799)]
HEAD_PAIRS = [(2, 1), (4, 2), (6, 3), (6, 1), (4, 4)]


def _inputs(seed, b, sq, sk, h, hk, d):
    gen = torch.Generator().manual_seed(seed)
    return (randn_half(gen, b, sq, h, d), randn_half(gen, b, sk, hk, d), randn_half(gen, b, sk, hk, d),
            randn_half(gen, b, sq, h, d))


def _check(name, got, want, emul, absolute=True):
    """The stated tolerance: error against the fp32 oracle within twice the error of the reference's CUDA
    kernel on the same inputs (emulated rounding points, helpers.py).  ``absolute`` adds the reference
    suite's own bounds (max 9e-3, mean 2e-4), which are meant for its grid of short sequences: at the
    benchmark sizes |dK|, |dV| reach 16 and more, where half an fp16 ulp of the result alone is 8e-3."""
    assert_within_twice_reference_kernel(name, got, want, emul)
    if absolute:
        assert_reference_suite_bounds(name, got, want, emul)


@pytest.fixture
def single_kernel_backward(ext):
    """Runs the test body with the single-kernel backward selected, and puts the default back afterwards."""
    ext.set_single_kernel_backward(True)
    yield
    ext.set_single_kernel_backward(False)


@pytest.mark.parametrize("path", ["single_kernel", "two_kernels"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("sq,sk", SEQ_PAIRS)
def test_dense_forward_backward_grid(ext, request, d, causal, sq, sk, path):
    from flash_attention_turing_b200 import flash_attn_func

    if path == "single_kernel":
        request.getfixturevalue("single_kernel_backward")

    idx = SEQ_PAIRS.index((sq, sk))
    h, hk = HEAD_PAIRS[idx % len(HEAD_PAIRS)]
    b = 1 + idx % 3
    scale = None if idx % 2 == 0 else 0.3
    q, k, v, dout = _inputs(100 + idx, b, sq, sk, h, hk, d)
    qd, kd, vd = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    out = flash_attn_func(qd, kd, vd, softmax_scale=scale, causal=causal)
    dq, dk, dv = torch.autograd.grad(out, (qd, kd, vd), dout.to(DEV))
    s = d ** -0.5 if scale is None else scale
    o_ref, _ = orc.attention_forward(q, k, v, s, causal)
    rq, rk, rv = orc.attention_backward(q, k, v, dout, s, causal)
    em = emulate_reference_kernel(q, k, v, dout, s, causal)
    _check("O", out, o_ref, em.out)
    _check("dQ", dq, rq, em.dq)
    _check("dK", dk, rk, em.dk)
    _check("dV", dv, rv, em.dv)


def test_c1_forward_full_size(ext):
    # C1 of the benchmark configs: forward, non-causal, B2 S512 H8 D64, scale 1/sqrt(64); O and LSE of
    # every (batch, head) against the oracle.
    b, s, h, d = 2, 512, 8, 64
    q, k, v, _ = _inputs(1001, b, s, s, h, h, d)
    out, lse = ext.fwd(q.to(DEV), k.to(DEV), v.to(DEV), d ** -0.5, False)
    o_ref, lse_ref = orc.attention_forward(q, k, v, None, False)
    em = emulate_reference_kernel(q, k, v, None, d ** -0.5, False)
    _check("O", out, o_ref, em.out)
    assert err_stats(lse, lse_ref)[0] <= LSE_TOL


@pytest.mark.parametrize("name", ["fwd_d64_noncausal", "fwd_d64_causal", "fwd_d128_causal_gqa", "fwd_d128_sq_gt_sk"])
def test_golden_fixtures(ext, name):
    # fixtures hold outputs of the reference's own Python math; keys beyond lens[b] are cut per sequence
    g = load_golden(name)
    q, k, v, dout = (t(g[x]) for x in ("q", "k", "v", "dout"))
    lens = g["lens"].tolist()
    scale, causal = float(g["scale"]), bool(g["causal"])
    for b in range(q.shape[0]):
        qb, kb, vb = q[b:b + 1].to(DEV), k[b:b + 1, : lens[b]].contiguous().to(DEV), v[b:b + 1, : lens[b]].contiguous().to(DEV)
        out, lse = ext.fwd(qb, kb, vb, scale, causal)
        dq, dk, dv = ext.bwd(qb, kb, vb, out, lse, dout[b:b + 1].to(DEV), scale, causal)
        want_out = torch.nan_to_num(t(g["out"])[b:b + 1], nan=0.0)
        want_lse = t(g["lse"])[b:b + 1]
        want_lse = torch.where(torch.isfinite(want_lse), want_lse, torch.zeros_like(want_lse))
        em = emulate_reference_kernel(q[b:b + 1], k[b:b + 1, : lens[b]], v[b:b + 1, : lens[b]], dout[b:b + 1], scale, causal)
        _check("O", out, want_out, em.out)
        assert err_stats(lse, want_lse)[0] <= LSE_TOL
        _check("dQ", dq, t(g["dq"])[b:b + 1], em.dq)
        _check("dK", dk, t(g["dk"])[b:b + 1, : lens[b]], em.dk)
        _check("dV", dv, t(g["dv"])[b:b + 1, : lens[b]], em.dv)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_packed_variants_match_unpacked(ext, d, causal):
    from flash_attention_turing_b200 import flash_attn_func, flash_attn_kvpacked_func, flash_attn_qkvpacked_func

    b, s, h = 2, 200, 4
    gen = torch.Generator().manual_seed(7 + d)
    qkv = randn_half(gen, b, s, 3, h, d).to(DEV).requires_grad_(True)
    dout = randn_half(gen, b, s, h, d).to(DEV)
    out_p = flash_attn_qkvpacked_func(qkv, causal=causal)
    (dqkv,) = torch.autograd.grad(out_p, qkv, dout)
    q, k, v = (qkv.detach()[:, :, i].contiguous().requires_grad_(True) for i in range(3))
    out = flash_attn_func(q, k, v, causal=causal)
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), dout)
    assert torch.equal(out_p, out)  # same kernel, same data, strided vs contiguous: bit-identical
    assert torch.equal(dqkv[:, :, 0], dq) and torch.equal(dqkv[:, :, 1], dk) and torch.equal(dqkv[:, :, 2], dv)
    o_ref, _ = orc.attention_forward(q.detach().cpu(), k.detach().cpu(), v.detach().cpu(), None, causal)
    em = emulate_reference_kernel(q.detach().cpu(), k.detach().cpu(), v.detach().cpu(), None, d ** -0.5, causal)
    _check("O", out_p, o_ref, em.out)

    hk = 2
    kv = randn_half(gen, b, s, 2, hk, d).to(DEV).requires_grad_(True)
    q2 = q.detach().clone().requires_grad_(True)
    out_kv = flash_attn_kvpacked_func(q2, kv, causal=causal)
    dq2, dkv = torch.autograd.grad(out_kv, (q2, kv), dout)
    k2, v2 = (kv.detach()[:, :, i].contiguous().requires_grad_(True) for i in range(2))
    q3 = q.detach().clone().requires_grad_(True)
    out3 = flash_attn_func(q3, k2, v2, causal=causal)
    dq3, dk3, dv3 = torch.autograd.grad(out3, (q3, k2, v2), dout)
    assert torch.equal(out_kv, out3) and torch.equal(dq2, dq3)
    assert torch.equal(dkv[:, :, 0], dk3) and torch.equal(dkv[:, :, 1], dv3)


def test_bwd_binding_writes_into_given_strided_gradients(ext):
    b, s, h, d = 1, 130, 2, 64
    gen = torch.Generator().manual_seed(21)
    q, k, v, dout = (randn_half(gen, b, s, h, d).to(DEV) for _ in range(4))
    out, lse = ext.fwd(q, k, v, d ** -0.5, True)
    dq, dk, dv = ext.bwd(q, k, v, out, lse, dout, d ** -0.5, True)  # the reference's eight arguments
    packed = torch.full((b, s, 3, h, d), float("nan"), dtype=torch.half, device=DEV)
    views = packed.unbind(2)
    got = ext.bwd(q, k, v, out, lse, dout, d ** -0.5, True, *views)
    assert all(g.data_ptr() == w.data_ptr() for g, w in zip(got, views))  # written in place, nothing new
    assert torch.equal(packed[:, :, 0], dq) and torch.equal(packed[:, :, 1], dk) and torch.equal(packed[:, :, 2], dv)
    with pytest.raises(RuntimeError, match="shape"):
        ext.bwd(q, k, v, out, lse, dout, d ** -0.5, True, packed[:, :-1, 0], views[1], views[2])
    with pytest.raises(RuntimeError, match="float16"):
        ext.bwd(q, k, v, out, lse, dout, d ** -0.5, True, views[0].float(), views[1], views[2])


def _varlen_case(seed, lens_q, lens_k, h, hk, d):
    gen = torch.Generator().manual_seed(seed)
    cq = torch.tensor([0] + torch.tensor(lens_q).cumsum(0).tolist(), dtype=torch.int32)
    ck = torch.tensor([0] + torch.tensor(lens_k).cumsum(0).tolist(), dtype=torch.int32)
    tq, tk = int(cq[-1]), int(ck[-1])
    return (randn_half(gen, tq, h, d), randn_half(gen, tk, hk, d), randn_half(gen, tk, hk, d),
            randn_half(gen, tq, h, d), cq, ck)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lens_q,lens_k,h,hk", [
    ([100, 300, 57], [100, 300, 57], 4, 2),
    ([128, 1, 513, 64], [200, 64, 513, 1], 2, 1),
    ([1, 2, 3, 129, 255], [7, 2, 300, 129, 1], 6, 3),
    ([640], [640], 4, 4),
])
@pytest.mark.parametrize("path", ["single_kernel", "two_kernels"])
def test_varlen_forward_backward(ext, request, d, causal, lens_q, lens_k, h, hk, path):
    from flash_attention_turing_b200 import flash_attn_varlen_func

    if path == "single_kernel":
        request.getfixturevalue("single_kernel_backward")

    q, k, v, dout, cq, ck = _varlen_case(31 + d, lens_q, lens_k, h, hk, d)
    qd, kd, vd = (x.to(DEV).requires_grad_(True) for x in (q, k, v))
    out = flash_attn_varlen_func(qd, kd, vd, cq.to(DEV), ck.to(DEV), max(lens_q), max(lens_k), causal=causal)
    dq, dk, dv = torch.autograd.grad(out, (qd, kd, vd), dout.to(DEV))
    o_ref, lses = orc.varlen_forward(q, k, v, cq, ck, None, causal)
    rq, rk, rv = orc.varlen_backward(q, k, v, dout, cq, ck, None, causal)
    em = emulate_reference_kernel_varlen(q, k, v, dout, cq, ck, d ** -0.5, causal)
    _check("O", out, o_ref, em.out)
    _check("dQ", dq, rq, em.dq)
    _check("dK", dk, rk, em.dk)
    _check("dV", dv, rv, em.dv)
    # padded LSE (b, h, max_seqlen_q): valid part matches, padding stays zero
    _, lse = ext.varlen_fwd(qd.detach(), kd.detach(), vd.detach(), cq.to(DEV), ck.to(DEV), max(lens_q), max(lens_k),
                            d ** -0.5, causal)
    for i, l in enumerate(lses):
        assert err_stats(lse[i, :, : lens_q[i]], l)[0] <= LSE_TOL
        assert lse[i, :, lens_q[i]:].abs().max().item() == 0 if lens_q[i] < max(lens_q) else True


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_varlen_backward_of_many_short_sequences(ext, d, causal):
    # Items of one to four key blocks, nearly all with a ragged last block, several per CTA: the loads of an item run
    # under the products of the one before it.  Every launch bit for bit equal to dense launches per sequence.
    h, hk = 8, 4
    lens = [(37 * i + 11) % 511 + 1 for i in range(96)]
    q, k, v, dout, cq, _ = _varlen_case(77 + d, lens, lens, h, hk, d)
    q, k, v, dout, cu = (x.to(DEV) for x in (q, k, v, dout, cq))
    args = (cu, cu, max(lens), max(lens), d ** -0.5, causal)
    out, lse = ext.varlen_fwd(q, k, v, *args)
    grads = ext.varlen_bwd(q, k, v, out, lse, dout, *args)
    for _ in range(30):
        for got, want in zip(ext.varlen_bwd(q, k, v, out, lse, dout, *args), grads):
            assert torch.equal(got, want)
    for i in range(0, len(lens), 7):
        a, b = int(cq[i]), int(cq[i + 1])
        one = [x[None, a:b] for x in (q, k, v)]
        o, l = ext.fwd(*one, d ** -0.5, causal)
        for got, want in zip(grads, ext.bwd(*one, o, l, dout[None, a:b], d ** -0.5, causal)):
            assert torch.equal(got[a:b], want[0])


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("d,h,hk", [(64, 6, 6), (64, 6, 2), (128, 6, 6), (128, 6, 2)])
def test_packed_key_gradients_equal_dense_ones(ext, d, h, hk, causal):
    # Key tiles and Q tiles of one row, whole ones and one row more, more queries than keys and the reverse, several key tiles
    # per CTA: both dK/dV kernels of packed batches against the one of dense batches, bit for bit.
    lens_q = [1, 128, 129, 500, 127, 257, 40, 256, 300] * 6
    lens_k = [300, 129, 128, 1, 127, 640, 256, 40, 300] * 6
    q, k, v, dout, cq, ck = _varlen_case(91 + d, lens_q, lens_k, h, hk, d)
    q, k, v, dout, cq_d, ck_d = (x.to(DEV) for x in (q, k, v, dout, cq, ck))
    args = (cq_d, ck_d, max(lens_q), max(lens_k), d ** -0.5, causal)
    out, lse = ext.varlen_fwd(q, k, v, *args)
    grads = ext.varlen_bwd(q, k, v, out, lse, dout, *args)
    for i in list(range(9)) + [30, 49, 53]:
        rq, rk = slice(int(cq[i]), int(cq[i + 1])), slice(int(ck[i]), int(ck[i + 1]))
        o, l = ext.fwd(q[None, rq], k[None, rk], v[None, rk], d ** -0.5, causal)
        dense = ext.bwd(q[None, rq], k[None, rk], v[None, rk], o, l, dout[None, rq], d ** -0.5, causal)
        for got, want, rows in zip(grads, dense, (rq, rk, rk)):
            assert torch.equal(got[rows], want[0])


def test_varlen_packed_variants(ext):
    from flash_attention_turing_b200 import (flash_attn_varlen_func, flash_attn_varlen_kvpacked_func,
                                             flash_attn_varlen_qkvpacked_func)

    lens = [90, 257, 33]
    d, h = 128, 4
    gen = torch.Generator().manual_seed(5)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32).to(DEV)
    total = sum(lens)
    qkv = randn_half(gen, total, 3, h, d).to(DEV).requires_grad_(True)
    dout = randn_half(gen, total, h, d).to(DEV)
    out_p = flash_attn_varlen_qkvpacked_func(qkv, cu, max(lens), causal=True)
    (dqkv,) = torch.autograd.grad(out_p, qkv, dout)
    q, k, v = (qkv.detach()[:, i].contiguous().requires_grad_(True) for i in range(3))
    out = flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), causal=True)
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), dout)
    assert torch.equal(out_p, out)
    assert torch.equal(dqkv[:, 0], dq) and torch.equal(dqkv[:, 1], dk) and torch.equal(dqkv[:, 2], dv)
    kv = torch.stack((k.detach(), v.detach()), dim=1).requires_grad_(True)
    q2 = q.detach().clone().requires_grad_(True)
    out_kv = flash_attn_varlen_kvpacked_func(q2, kv, cu, cu, max(lens), max(lens), causal=True)
    dq2, dkv = torch.autograd.grad(out_kv, (q2, kv), dout)
    assert torch.equal(out_kv, out) and torch.equal(dq2, dq) and torch.equal(dkv[:, 0], dk) and torch.equal(dkv[:, 1], dv)


def test_run_to_run_determinism(ext):
    # Two-kernel backward (the default): every accumulation order is fixed (no atomics), so repeated launches are
    # bit-identical, which also catches races on shared memory / TMEM.  Single-kernel backward: O, LSE, dK, dV
    # are bit-identical as well; dQ is summed with global fp32 reductions in scheduling order, so it is only
    # held to agree within one fp16 ulp of its largest value from run to run.
    q, k, v, dout = _inputs(77, 2, 700, 700, 4, 2, 128)
    qd, kd, vd, dd = (x.to(DEV) for x in (q, k, v, dout))
    for single in (False, True):
        ext.set_single_kernel_backward(single)
        try:
            first = None
            for _ in range(3):
                out, lse = ext.fwd(qd, kd, vd, 128 ** -0.5, True)
                dq, dk, dv = ext.bwd(qd, kd, vd, out, lse, dd, 128 ** -0.5, True)
                cur = [out, lse, dk, dv, dq]
                if first is None:
                    first = [x.clone() for x in cur]
                    continue
                assert all(torch.equal(a, b) for a, b in zip(first[:4], cur[:4]))
                if not single:
                    assert torch.equal(first[4], dq)
                else:
                    ulp = 2.0 ** -10 * first[4].float().abs().max().item()
                    assert (first[4].float() - dq.float()).abs().max().item() <= ulp
        finally:
            ext.set_single_kernel_backward(False)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,sq,sk,h,hk,causal", [
    (2, 897, 1024, 4, 4, False),   # items of eight whole key blocks, a ragged last Q tile
    (1, 2048, 2048, 16, 4, True),  # items of one block up to sixteen
    (3, 197, 197, 12, 12, False),  # fewer items than SMs
    (40, 130, 260, 8, 2, True),    # several items per SM, each of three blocks or fewer
])
def test_repeated_launches_are_bit_identical(ext, d, b, sq, sk, h, hk, causal):
    # No accumulation order depends on timing, so a hand-over that does (a product issued before its operand is whole) shows as a
    # difference between launches: rarely in one of them, hence 200, back to back.
    q, k, v, dout = _inputs(511 + sq, b, sq, sk, h, hk, d)
    qd, kd, vd, dd = (x.to(DEV) for x in (q, k, v, dout))
    scale = d ** -0.5
    out, lse = ext.fwd(qd, kd, vd, scale, causal)
    first = [out, lse, *ext.bwd(qd, kd, vd, out, lse, dd, scale, causal)]
    differ = torch.zeros(5, dtype=torch.int64, device=DEV)
    for _ in range(200):
        o, l = ext.fwd(qd, kd, vd, scale, causal)
        again = [o, l, *ext.bwd(qd, kd, vd, out, lse, dd, scale, causal)]
        differ += torch.stack([(x != y).any() for x, y in zip(again, first)])
    assert differ.tolist() == [0] * 5
    refs = (orc.attention_forward(q, k, v, scale, causal)[0], *orc.attention_backward(q, k, v, dout, scale, causal))
    em = emulate_reference_kernel(q, k, v, dout, scale, causal)
    for name, got, want, emul in zip(("O", "dQ", "dK", "dV"), [first[0], *first[2:]], refs, (em.out, em.dq, em.dk, em.dv)):
        _check(name, got, want, emul)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("h,hk,causal", [(8, 8, True), (8, 2, True), (8, 2, False)])
def test_repeated_packed_launches_are_bit_identical(ext, d, h, hk, causal):
    lens_q = [130, 1, 640, 257, 129, 40, 1500, 384] * 3
    lens_k = [130, 300, 640, 129, 257, 1, 1500, 300] * 3
    q, k, v, dout, cq, ck = (x.to(DEV) for x in _varlen_case(17 + d, lens_q, lens_k, h, hk, d))
    args = (cq, ck, max(lens_q), max(lens_k), d ** -0.5, causal)
    out, lse = ext.varlen_fwd(q, k, v, *args)
    first = [out, *ext.varlen_bwd(q, k, v, out, lse, dout, *args)]
    differ = torch.zeros(4, dtype=torch.int64, device=DEV)
    for _ in range(200):
        again = [ext.varlen_fwd(q, k, v, *args)[0], *ext.varlen_bwd(q, k, v, out, lse, dout, *args)]
        differ += torch.stack([(x != y).any() for x, y in zip(again, first)])
    assert differ.tolist() == [0] * 4


@pytest.mark.parametrize("d", [64, 128])
def test_both_backward_paths_agree(ext, d):
    # the single-kernel and the two-kernel backward compute the same sums with the same rounding points:
    # dK and dV agree bit for bit or within an ulp (different accumulation chunks), dQ within an ulp
    q, k, v, dout = _inputs(78, 2, 600, 900, 6, 2, d)
    qd, kd, vd, dd = (x.to(DEV) for x in (q, k, v, dout))
    out, lse = ext.fwd(qd, kd, vd, d ** -0.5, True)
    a = ext.bwd(qd, kd, vd, out, lse, dd, d ** -0.5, True)
    ext.set_single_kernel_backward(True)
    try:
        b = ext.bwd(qd, kd, vd, out, lse, dd, d ** -0.5, True)
    finally:
        ext.set_single_kernel_backward(False)
    for x, y in zip(a, b):
        assert (x.float() - y.float()).abs().max().item() <= 2.0 ** -9 * max(1.0, y.float().abs().max().item())


def test_no_grad_and_requires_grad_flags(ext):
    from flash_attention_turing_b200 import flash_attn_func

    q, k, v, _ = _inputs(3, 1, 64, 64, 2, 2, 64)
    with torch.no_grad():
        out = flash_attn_func(q.to(DEV), k.to(DEV), v.to(DEV))
    assert not out.requires_grad
    qd = q.to(DEV).requires_grad_(True)
    out = flash_attn_func(qd, k.to(DEV), v.to(DEV), causal=True)
    (dq,) = torch.autograd.grad(out.float().sum(), qd)
    assert dq.shape == qd.shape and dq.dtype == torch.float16


def test_binding_errors(ext):
    q = torch.randn(1, 8, 4, 96, device=DEV, dtype=torch.half)
    with pytest.raises(RuntimeError, match="head_dim 64 or 128"):
        ext.fwd(q, q, q, 1.0, False)
    q = torch.randn(1, 8, 4, 64, device=DEV, dtype=torch.half)
    k = torch.randn(1, 8, 3, 64, device=DEV, dtype=torch.half)
    with pytest.raises(RuntimeError, match="divisible by num_heads_k"):
        ext.fwd(q, k, k, 1.0, False)
    with pytest.raises(RuntimeError, match="rank-4"):
        ext.fwd(q[0], k[0], k[0], 1.0, False)


def _sampled_slices_check(q, k, v, dout, out, lse, dq, dk, dv, slices, causal=True):
    """Attention is independent per (batch, head): a slice of a full-size launch must match the oracle of
    that slice, within twice the reference kernel's error (emulated on the same slice)."""
    d = q.shape[-1]
    for bi, hi in slices:
        sl = lambda x: x[bi:bi + 1, :, hi:hi + 1].cpu()  # noqa: E731
        o_ref, lse_ref = orc.attention_forward(sl(q), sl(k), sl(v), None, causal)
        rq, rk, rv = orc.attention_backward(sl(q), sl(k), sl(v), sl(dout), None, causal)
        em = emulate_reference_kernel(sl(q), sl(k), sl(v), sl(dout), d ** -0.5, causal)
        _check("O", sl(out), o_ref, em.out, absolute=False)
        assert err_stats(lse[bi:bi + 1, hi:hi + 1], lse_ref)[0] <= LSE_TOL
        _check("dQ", sl(dq), rq, em.dq, absolute=False)
        _check("dK", sl(dk), rk, em.dk, absolute=False)
        _check("dV", sl(dv), rv, em.dv, absolute=False)


@pytest.mark.parametrize("s", [4096, 8192])
def test_full_size_causal_config_by_sampling(ext, s):
    # S = 4096: C2 of the benchmark configs (B4 S4096 H32 D128 causal, forward + backward).  S = 8192: the
    # shape the headline metric is quoted on.  Full-size launches; the oracle is evaluated on two
    # (batch, head) slices.
    b, h, d = 4, 32, 128
    gen = torch.Generator(device=DEV).manual_seed(1002)
    q, k, v, dout = (torch.randn(b, s, h, d, device=DEV, dtype=torch.half, generator=gen) for _ in range(4))
    out, lse = ext.fwd(q, k, v, d ** -0.5, True)
    dq, dk, dv = ext.bwd(q, k, v, out, lse, dout, d ** -0.5, True)
    _sampled_slices_check(q, k, v, dout, out, lse, dq, dk, dv, [(0, 0), (3, 17)])
    # size-independent property: every softmax row sums to one => with V = 1, O = 1 exactly
    ones = torch.ones_like(v)
    o1, _ = ext.fwd(q, k, ones, d ** -0.5, True)
    assert (o1.float() - 1).abs().max().item() <= 2e-3


def _c3_lengths():
    """C3 of the benchmark configs: 16 sequences, lengths U[256, 4096] (seeded), capped at 32768 tokens."""
    gen = torch.Generator().manual_seed(1003)
    lens = torch.randint(256, 4097, (16,), generator=gen)
    total = int(lens.sum())
    if total > 32768:
        lens = torch.clamp(lens * 32768 // total, min=256)
    return [int(x) for x in lens]


def test_c3_gqa_varlen_full_size(ext):
    # C3: GQA varlen forward + backward, causal, Hq32 Hkv8 D128, 16 sequences.  The full-size launch is
    # checked on two whole sequences (all heads of one KV group each) against the oracle.
    from flash_attention_turing_b200 import flash_attn_varlen_func

    lens = _c3_lengths()
    assert sum(lens) <= 32768
    h, hk, d = 32, 8, 128
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    total = int(cu[-1])
    gen = torch.Generator(device=DEV).manual_seed(1003)
    q = torch.randn(total, h, d, device=DEV, dtype=torch.half, generator=gen).requires_grad_(True)
    k = torch.randn(total, hk, d, device=DEV, dtype=torch.half, generator=gen).requires_grad_(True)
    v = torch.randn(total, hk, d, device=DEV, dtype=torch.half, generator=gen).requires_grad_(True)
    dout = torch.randn(total, h, d, device=DEV, dtype=torch.half, generator=gen)
    out = flash_attn_varlen_func(q, k, v, cu.to(DEV), cu.to(DEV), max(lens), max(lens), causal=True)
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), dout)
    order = sorted(range(16), key=lambda i: lens[i])
    for seq, kv_head in ((order[0], 0), (order[8], 5)):
        a, b = int(cu[seq]), int(cu[seq + 1])
        hs = slice(kv_head * 4, kv_head * 4 + 4)
        qs, ks, vs, ds = (x.detach()[a:b].cpu() for x in (q[:, hs], k[:, kv_head:kv_head + 1], v[:, kv_head:kv_head + 1], dout[:, hs]))
        o_ref, _ = orc.attention_forward_one(qs, ks, vs, d ** -0.5, True)
        rq, rk, rv = orc.attention_backward_one(qs, ks, vs, ds, d ** -0.5, True)
        em = emulate_reference_kernel_one(qs, ks, vs, ds, d ** -0.5, True)
        _check("O", out[a:b, hs], o_ref, em.out, absolute=False)
        _check("dQ", dq[a:b, hs], rq, em.dq, absolute=False)
        _check("dK", dk[a:b, kv_head:kv_head + 1], rk, em.dk, absolute=False)
        _check("dV", dv[a:b, kv_head:kv_head + 1], rv, em.dv, absolute=False)


@pytest.mark.parametrize("d", [64, 128])
def test_c5_long_context_by_sampling(ext, d):
    # C5: B1 S65536 H16 causal, forward + backward at full size on a head shard (2 of 16 heads, as one rank
    # of an 8-GPU head-sharded run).  Causality makes exact value checks of the 65536-token launch cheap:
    #   * rows [0, 8192) of O, LSE and dQ depend only on the first 8192 tokens: they must equal the oracle of
    #     that prefix;
    #   * dK, dV of the keys [61440, 65536) receive contributions from the query rows >= 61440 only: they must
    #     equal the oracle evaluated on those 4096 query rows against all keys.
    # Both within twice the reference kernel's (emulated) error; sampled rows and two identities on top.
    b, s, h = 1, 65536, 2
    scale = d ** -0.5
    gen = torch.Generator(device=DEV).manual_seed(1005)
    q, k, v, dout = (torch.randn(b, s, h, d, device=DEV, dtype=torch.half, generator=gen) for _ in range(4))
    out, lse = ext.fwd(q, k, v, scale, True)
    rows = [0, 1, 127, 128, 4095, 30000, 65535]
    for r in rows:
        qs = q[:, r:r + 1, :1].cpu()
        o_ref, lse_ref = orc.attention_forward(qs, k[:, : r + 1, :1].cpu(), v[:, : r + 1, :1].cpu(), None, False)
        assert err_stats(out[:, r:r + 1, :1], o_ref)[0] <= 2e-3
        assert err_stats(lse[:, :1, r:r + 1], lse_ref)[0] <= LSE_TOL
    o1, _ = ext.fwd(q, k, torch.ones_like(v), scale, True)
    assert (o1.float() - 1).abs().max().item() <= 2e-3
    dq, dk, dv = ext.bwd(q, k, v, out, lse, dout, scale, True)
    assert not any(torch.isnan(x).any().item() for x in (dq, dk, dv))
    hd = 1  # the head that is compared value by value
    one = lambda x, a, e: x[0, a:e, hd:hd + 1].cpu()  # noqa: E731
    # prefix: the first 8192 tokens
    n = 8192
    qp, kp, vp, dp = (one(x, 0, n) for x in (q, k, v, dout))
    o_ref, lse_ref = orc.attention_forward_one(qp, kp, vp, scale, True)
    rq, _, _ = orc.attention_backward_one(qp, kp, vp, dp, scale, True)
    em = emulate_reference_kernel_one(qp, kp, vp, dp, scale, True)
    _check("O[:8192]", one(out, 0, n), o_ref, em.out, absolute=False)
    assert err_stats(lse[0, hd:hd + 1, :n], lse_ref)[0] <= LSE_TOL
    _check("dQ[:8192]", one(dq, 0, n), rq, em.dq, absolute=False)
    # tail: the last 4096 query rows against all keys
    r0 = s - 4096
    qa, ka, va, da = (one(x, 0, s) for x in (q, k, v, dout))
    rq, rk, rv = orc.attention_backward_one(qa, ka, va, da, scale, True, row_chunk=1024, row_start=r0)
    em = emulate_reference_kernel_one(qa, ka, va, da, scale, True, row_chunk=1024, row_start=r0)
    _check("dQ[-4096:]", one(dq, r0, s), rq[r0:], em.dq[r0:], absolute=False)
    _check("dK[-4096:]", one(dk, r0, s), rk[r0:], em.dk[r0:], absolute=False)
    _check("dV[-4096:]", one(dv, r0, s), rv[r0:], em.dv[r0:], absolute=False)
    # identities over the whole launch: sum(dQ * Q) = sum(dK * K) (the scores depend on Q K^T only) ...
    lhs = (dq.float() * q.float()).sum().item()
    rhs = (dk.float() * k.float()).sum().item()
    assert abs(lhs - rhs) <= 2e-3 * max(abs(lhs), abs(rhs), (dq.float().abs() * q.float().abs()).sum().item() * 1e-3)
    # ... and dV of the last key row is exactly P[last query, last key] * dO[last query]
    p_last = torch.exp((q[0, -1].float() * k[0, -1].float()).sum(-1) * scale - lse[0, :, -1])
    want = p_last[:, None] * dout[0, -1].float()
    assert (dv[0, -1].float() - want).abs().max().item() <= 1e-3


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("lens,h,hk,d,poison", [([100, 300, 57], 4, 2, 128, 1), ([200, 64, 513], 2, 1, 64, 2),
                                                ([130, 130, 130], 2, 2, 128, 0)])
def test_varlen_gradients_ignore_nan_in_a_neighbouring_sequence(ext, lens, h, hk, d, poison, causal):
    """The sequences of a packed batch are independent: NaN in every tensor of one sequence must not reach the
    outputs or gradients of the others (rows of the next sequence share 128-row tiles with this one)."""
    from flash_attention_turing_b200 import flash_attn_varlen_func

    gen = torch.Generator().manual_seed(5)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    total = int(cu[-1])
    q, do = randn_half(gen, total, h, d), randn_half(gen, total, h, d)
    k, v = randn_half(gen, total, hk, d), randn_half(gen, total, hk, d)
    ro, _ = orc.varlen_forward(q, k, v, cu, cu, None, causal)
    rq, rk, rv = orc.varlen_backward(q, k, v, do, cu, cu, None, causal)
    em = emulate_reference_kernel_varlen(q, k, v, do, cu, cu, d ** -0.5, causal)
    lo, hi = int(cu[poison]), int(cu[poison + 1])
    for t in (q, k, v, do):
        t[lo:hi] = float("nan")
    qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
    out = flash_attn_varlen_func(qd, kd, vd, cu.to(DEV), cu.to(DEV), max(lens), max(lens), causal=causal)
    dq, dk, dv = torch.autograd.grad(out, (qd, kd, vd), do.to(DEV))
    keep = torch.ones(total, dtype=torch.bool)
    keep[lo:hi] = False
    for name, got, want, emu in (("O", out, ro, em.out), ("dQ", dq, rq, em.dq), ("dK", dk, rk, em.dk), ("dV", dv, rv, em.dv)):
        got = got.detach().float().cpu()[keep]
        assert not torch.isnan(got).any(), name
        _check(name, got, want[keep], emu[keep])


CANARY = 0x7BCD  # an fp16 bit pattern (finite, 6.2e4) that no kernel result takes by accident


def _canary_view(shape, pad_elems=4096, dtype=torch.half):
    """A tensor of `shape` cut out of a larger canary-filled buffer: `pad_elems` untouched elements before and
    after, and a row pitch one head wider than needed, so that every (row) has a gap after its last head.
    Returns (view, buffer, mask of the elements the view covers)."""
    b, s, h, d = shape
    pitch = (h + 1) * d
    n = b * s * pitch
    buf = torch.empty(n + 2 * pad_elems, dtype=dtype, device=DEV)
    if dtype == torch.half:
        buf.view(torch.int16).fill_(CANARY)
    else:
        buf.view(torch.int32).fill_(0x7BCD7BCD)
    view = buf[pad_elems:pad_elems + n].view(b, s, h + 1, d)[:, :, :h]
    mask = torch.zeros_like(buf, dtype=torch.bool)
    mask[pad_elems:pad_elems + n].view(b, s, h + 1, d)[:, :, :h] = True
    return view, buf, mask


def _canaries_intact(buf, mask):
    raw = buf.view(torch.int16) if buf.dtype == torch.half else buf.view(torch.int32)
    want = CANARY if buf.dtype == torch.half else 0x7BCD7BCD
    return bool((raw[~mask] == want).all().item())


@pytest.mark.parametrize("flags", [0, 1])  # 0: two-kernel backward, 1: FA_BWD_SINGLE_KERNEL
@pytest.mark.parametrize("b,sq,sk,h,hk,d,causal", [(2, 129, 257, 4, 2, 64, True), (1, 385, 131, 3, 1, 128, False),
                                                   (2, 1, 300, 2, 2, 128, True), (1, 700, 700, 6, 3, 64, True)])
def test_guard_bands_around_outputs_and_scratch(b, sq, sk, h, hk, d, causal, flags):
    """Nothing is written outside the tensors the caller handed over: O, LSE, dQ, dK, dV and the backward
    scratch are cut out of canary-filled buffers (pads before and after, a gap after every row) through the
    C ABI's strides, and the canaries are intact after forward and backward at odd sizes.  (The memory
    checker of the CUDA toolkit is not available on the test machines.)"""
    import ctypes

    from flash_attention_turing_b200 import capi

    lib = capi.lib()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    q, k, v, dout = (x.to(DEV) for x in _inputs(5 + sq, b, sq, sk, h, hk, d))
    o, o_buf, o_mask = _canary_view((b, sq, h, d))
    dq, dq_buf, dq_mask = _canary_view((b, sq, h, d))
    dk, dk_buf, dk_mask = _canary_view((b, sk, hk, d))
    dv, dv_buf, dv_mask = _canary_view((b, sk, hk, d))
    lse_buf = torch.empty(b * h * sq + 2048, dtype=torch.float32, device=DEV)
    lse_buf.view(torch.int32).fill_(0x7BCD7BCD)
    lse = lse_buf[1024:1024 + b * h * sq].view(b, h, sq)
    scale = d ** -0.5
    capi.check(lib.fa_fwd(ctypes.byref(capi.fwd_params(q, k, v, o, lse, scale, causal)), stream))
    bp = capi.bwd_params(q, k, v, o, dout, lse, dq, dk, dv, None, scale, causal)
    bp.flags = flags
    need = lib.fa_bwd_workspace_bytes(ctypes.byref(bp))
    ws_buf = torch.empty(need + 8192, dtype=torch.uint8, device=DEV)
    ws_buf.fill_(0xA5)
    bp.workspace, bp.workspace_bytes = ws_buf.data_ptr() + 4096, need
    capi.check(lib.fa_bwd(ctypes.byref(bp), stream))
    torch.cuda.synchronize()
    for name, buf, mask in (("O", o_buf, o_mask), ("dQ", dq_buf, dq_mask), ("dK", dk_buf, dk_mask), ("dV", dv_buf, dv_mask)):
        assert _canaries_intact(buf, mask), f"{name}: a write outside the tensor"
    raw = lse_buf.view(torch.int32)
    assert bool((raw[:1024] == 0x7BCD7BCD).all()) and bool((raw[1024 + b * h * sq:] == 0x7BCD7BCD).all()), "LSE"
    assert bool((ws_buf[:4096] == 0xA5).all()) and bool((ws_buf[4096 + need:] == 0xA5).all()), "backward scratch"
    # and the results inside are the right ones
    qc, kc, vc, dc = (x.cpu() for x in (q, k, v, dout))
    o_ref, lse_ref = orc.attention_forward(qc, kc, vc, None, causal)
    rq, rk, rv = orc.attention_backward(qc, kc, vc, dc, None, causal)
    em = emulate_reference_kernel(qc, kc, vc, dc, scale, causal)
    for name, got, want, emu in (("O", o, o_ref, em.out), ("dQ", dq, rq, em.dq), ("dK", dk, rk, em.dk), ("dV", dv, rv, em.dv)):
        _check(name, got, want, emu)
    assert err_stats(lse, lse_ref)[0] <= LSE_TOL
    assert lib.fa_device_status(1) == 0


def _multi_wave_case(seed, causal=True, d=128):
    """More work items than SMs, so that the forward takes its items from the global work counter."""
    gen = torch.Generator().manual_seed(seed)
    b, s, h, hk = 2, 2048, 12, 4   # 2 x 12 x 8 = 192 items of 256 rows
    q, k, v = randn_half(gen, b, s, h, d), randn_half(gen, b, s, hk, d), randn_half(gen, b, s, hk, d)
    return q.to(DEV), k.to(DEV), v.to(DEV), d ** -0.5, causal


def test_forward_work_counters_are_left_clean_over_many_launches(ext):
    """The persistent forward takes a {next item, finished CTAs} pair from a pool of 16384 and its last CTA puts
    the pair back to zero.  33000 launches go round the pool twice: a pair left dirty by an earlier launch would
    make a later one skip items, i.e. leave rows of O unwritten."""
    q, k, v, scale, causal = _multi_wave_case(31)
    want, want_lse = ext.fwd(q, k, v, scale, causal)
    out, lse = torch.empty_like(want), torch.empty_like(want_lse)
    for i in range(33000):
        if i % 550 == 0:
            out.fill_(float("nan"))
        ext.fwd(q, k, v, scale, causal, out=out, lse=lse)
        if i % 550 == 549:
            assert torch.equal(out, want) and torch.equal(lse, want_lse), i
    assert ext.device_status(True) == 0


def test_forward_launches_on_two_streams_do_not_share_work_counters(ext):
    q, k, v, scale, causal = _multi_wave_case(32)
    q2, k2, v2, _, _ = _multi_wave_case(33, causal=False)
    want, _ = ext.fwd(q, k, v, scale, causal)
    want2, _ = ext.fwd(q2, k2, v2, scale, False)
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    outs = []
    for _ in range(20):  # launches of the two streams overlap on the GPU (each fills it for ~30 us)
        with torch.cuda.stream(s1):
            o1, _ = ext.fwd(q, k, v, scale, causal)
        with torch.cuda.stream(s2):
            o2, _ = ext.fwd(q2, k2, v2, scale, False)
        outs.append((o1, o2))
    torch.cuda.synchronize()
    for o1, o2 in outs:
        assert torch.equal(o1, want) and torch.equal(o2, want2)
    assert ext.device_status(True) == 0


def test_forward_in_a_cuda_graph_replays(ext):
    """A captured launch keeps the counter pair it was given; it is clean again whenever a replay ends, so the
    graph can be replayed any number of times (new inputs written into the captured tensors)."""
    q, k, v, scale, causal = _multi_wave_case(34)
    out = torch.empty_like(q)
    lse = torch.empty(q.shape[0], q.shape[2], q.shape[1], dtype=torch.float32, device=DEV)
    ext.fwd(q, k, v, scale, causal, out=out, lse=lse)  # first launch on this device outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ext.fwd(q, k, v, scale, causal, out=out, lse=lse)
    gen = torch.Generator().manual_seed(35)
    for _ in range(5):
        q.copy_(randn_half(gen, *q.shape))
        graph.replay()
        got = out.clone()
        want, _ = ext.fwd(q, k, v, scale, causal)
        assert torch.equal(got, want)
    assert ext.device_status(True) == 0


def _kernel_arguments(graph):
    """The argument bytes of the kernels of a captured graph, in order."""
    from cuda.bindings import driver

    def ok(result):
        assert int(result[0]) == 0, result
        return result[1:] if len(result) != 2 else result[1]

    n = ok(driver.cuGraphGetNodes(graph.raw_cuda_graph()))[1]
    found = []
    for node in ok(driver.cuGraphGetNodes(graph.raw_cuda_graph(), n))[0]:
        if ok(driver.cuGraphNodeGetType(node)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ok(driver.cuGraphKernelNodeGetParams(node))
            _, size = (ok(driver.cuFuncGetParamInfo(params.func, 0)) if int(params.func)
                       else ok(driver.cuKernelGetParamInfo(params.kern, 0)))
            found.append(ctypes.string_at(ctypes.cast(params.kernelParams, ctypes.POINTER(ctypes.c_void_p))[0], size))
    return found


def test_graphs_captured_many_launches_apart_have_work_counters_of_their_own(ext):
    """The same calls captured twice, 1024 launches apart: the arguments of the three persistent kernels differ, and only in the
    pointer to the work counters (a pool that eager and captured launches shared came round after 1024)."""
    from flash_attention_turing_b200 import capi

    q, k, v, scale, causal = _multi_wave_case(36)
    dout, (dq, dk, dv) = torch.randn_like(q), (torch.empty_like(x) for x in (q, k, v))
    out, lse = ext.fwd(q, k, v, scale, causal)
    fwd = capi.fwd_params(q, k, v, out, lse, scale, causal)
    room = torch.empty(1 << 20, dtype=torch.uint8, device=DEV)
    bwd = capi.bwd_params(q, k, v, out, dout, lse, dq, dk, dv, room, scale, causal)

    def capture(what):
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
            for call, params in what:
                capi.check(call(ctypes.byref(params), stream))
        return graph

    both = [(capi.lib().fa_fwd, fwd), (capi.lib().fa_bwd, bwd)]  # three pairs of counters
    first = capture(both)
    between = capture([both[0]] * 1021)
    second = capture(both)
    words = [[(x, y) for x, y in zip(memoryview(a[:len(a) // 8 * 8]).cast("Q"), memoryview(b[:len(b) // 8 * 8]).cast("Q")) if x != y]
             for a, b in zip(_kernel_arguments(first), _kernel_arguments(second))]
    assert [len(w) for w in words if w] == [1, 1, 1]
    assert all(abs(y - x) == 1024 * 8 for w in words for x, y in w)
    del between


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("h,hk,d", [(3, 1, 128), (4, 4, 64)])
def test_varlen_forward_many_ragged_sequences(ext, h, hk, d, causal):
    """The forward's work-item mapping for packed sequences (slots from cu_seqlens_q / 256) over 70 sequences with
    the lengths that matter to it: empty ones, single rows, exact multiples of 256 and of 128, one row more or
    less, and long ones -- more items than SMs, so that the counter path runs.  Every sequence must equal the
    dense launch on that sequence alone (same kernel, same rounding: bit for bit), which is compared with the
    oracle elsewhere; LSE padding stays zero."""
    gen = torch.Generator().manual_seed(77 + d)
    lens = [0, 1, 255, 256, 257, 511, 512, 513, 128, 127, 129, 0, 0, 3, 1024, 2047, 2048, 2049, 5, 640]
    lens += [int(x) for x in torch.randint(1, 700, (50,), generator=gen)]
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    total = int(cu[-1])
    q, k, v = randn_half(gen, total, h, d).to(DEV), randn_half(gen, total, hk, d).to(DEV), randn_half(gen, total, hk, d).to(DEV)
    scale = d ** -0.5
    out, lse = ext.varlen_fwd(q, k, v, cu.to(DEV), cu.to(DEV), max(lens), max(lens), scale, causal)
    assert not torch.isnan(out).any()
    for i, n in enumerate(lens):
        a, b = int(cu[i]), int(cu[i + 1])
        if n == 0:
            assert lse[i].abs().max().item() == 0
            continue
        o1, l1 = ext.fwd(q[a:b].unsqueeze(0), k[a:b].unsqueeze(0), v[a:b].unsqueeze(0), scale, causal)
        assert torch.equal(out[a:b], o1[0]), (i, n)
        assert torch.equal(lse[i, :, :n], l1[0]), (i, n)
        assert lse[i, :, n:].abs().max().item() == 0 if n < max(lens) else True
    assert ext.device_status(True) == 0


def test_package_reports_the_device_status_word(ext):
    import flash_attention_turing_b200 as fa

    assert fa.device_status() == 0
    assert fa.device_status(reset=True) == 0


def _bwd_params_for(ext, b, s, h, hk, d, causal, lens):
    """Inputs, outputs and filled FaBwdParams of a dense batch, or of packed sequences of the given lengths."""
    from flash_attention_turing_b200 import capi

    torch.manual_seed(0)
    rows = (sum(lens),) if lens else (b, s)
    q, k, v, dout = (torch.randn(*rows, n, d, device=DEV, dtype=torch.float16) for n in (h, hk, hk, h))
    cu = torch.tensor([0] + list(lens), dtype=torch.int32, device=DEV).cumsum(0, dtype=torch.int32) if lens else None
    extra = () if cu is None else (cu, cu, s, s)
    scale = d ** -0.5
    out, lse = ext.fwd(q, k, v, scale, causal) if cu is None else ext.varlen_fwd(q, k, v, *extra, scale, causal)
    grads = [torch.empty_like(x) for x in (q, k, v)]
    four_d = [x if cu is None else x.unsqueeze(0) for x in (q, k, v, out, dout, *grads)]
    p = capi.bwd_params(*four_d[:5], lse, *four_d[5:], None, scale, causal)
    p.b, p.seqlen_q, p.seqlen_k = b, s, s
    if cu is not None:
        p.cu_seqlens_q = p.cu_seqlens_k = cu.data_ptr()
        p.total_q = p.total_k = sum(lens)
    ws = torch.empty(capi.lib().fa_bwd_workspace_bytes(ctypes.byref(p)), dtype=torch.uint8, device=DEV)
    p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    return p, grads, ws, (q, k, v, out, dout, lse, cu)  # the last: kept alive by the caller


@pytest.mark.parametrize("b,s,h,hk,d,causal,lens", [
    (1, 1, 1, 1, 64, False, ()),          # one item in every kernel
    (3, 197, 12, 12, 64, False, ()),      # fewer items than SMs: the dK/dV kernel runs beside the dQ kernel
    (2, 640, 16, 4, 128, True, ()),       # a few more items than SMs in the dQ kernel
    (1, 4096, 8, 8, 128, True, ()),
    (3, 300, 4, 2, 128, True, (300, 1, 129)),
    (2, 700, 24, 24, 64, True, (700, 256)),
])
def test_overlapped_backward_launches_equal_separate_ones(ext, b, s, h, hk, d, causal, lens):
    """dQ starts under the preprocess kernel and dK/dV under dQ; a kernel that did not wait for the row statistics would
    read the NaN pattern that the workspace is filled with before every call.  Bit for bit, also replayed from a graph."""
    from flash_attention_turing_b200 import capi

    lib = capi.lib()
    p, grads, ws, keep = _bwd_params_for(ext, b, s, h, hk, d, causal, lens)

    def stream():
        return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    for stage in (1, 2, 4):
        capi.check(lib.fa_bwd_stages(ctypes.byref(p), stage, stream()))
        torch.cuda.synchronize()
    want = [g.clone() for g in grads]
    assert all(torch.isfinite(g).all() for g in want)
    got = []
    for _ in range(20):
        ws.fill_(255)
        for g in grads:
            g.fill_(float("nan"))
        capi.check(lib.fa_bwd(ctypes.byref(p), stream()))
        got.append([g.clone() for g in grads])  # on the stream, right behind the last kernel
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ws.fill_(255)
        capi.check(lib.fa_bwd(ctypes.byref(p), stream()))
        copies = [g.clone() for g in grads]
    for _ in range(5):
        for g in grads:
            g.fill_(float("nan"))
        graph.replay()
        got.append([c.clone() for c in copies])
    torch.cuda.synchronize()
    assert lib.fa_device_status(0) == 0
    for run in got:
        assert all(torch.equal(a, w) for a, w in zip(run, want))


@pytest.mark.parametrize("before", [127, 128, 255, 256, 700])
def test_packed_sequences_that_start_past_the_first_tiles(ext, before):
    """cu_seqlens[0] > 0: the work indices below the first sequence's are spare ones.  Bit for bit what the sequences give
    when they start at row 0."""
    gen = torch.Generator().manual_seed(6)
    lens, h, hk, d = (300, 1, 70), 4, 2, 64
    used, scale = sum(lens), d ** -0.5
    q, k, v, dout = (randn_half(gen, before + used, n, d).to(DEV) for n in (h, hk, hk, h))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)

    def run(q, k, v, dout, cu):
        out, lse = ext.varlen_fwd(q, k, v, cu, cu, max(lens), max(lens), scale, True)
        return (out, *ext.varlen_bwd(q, k, v, out, lse, dout, cu, cu, max(lens), max(lens), scale, True))

    got = run(q, k, v, dout, cu + before)
    want = run(*(x[before:].contiguous() for x in (q, k, v, dout)), cu)
    for a, b in zip(got, want):
        assert torch.equal(a[before:], b) and a[:before].abs().sum() == 0
    assert ext.device_status(True) == 0


@pytest.mark.parametrize("path", ["default", "single_kernel"])
@pytest.mark.parametrize("d,before,after,lens,max_k", [
    (64, 0, 0, (5, 300, 128), 300),      # nothing to clear
    (64, 3, 0, (130,), 130),
    (128, 0, 1, (1, 257), 600),
    (128, 140, 77, (64, 0, 200), 256),   # an empty sequence in between
])
def test_rows_outside_every_packed_sequence_are_zero(ext, request, path, d, before, after, lens, max_k):
    """cu_seqlens may start above 0 and end below the last row: O, dQ, dK, dV are zero there, whatever the memory held, and
    the sequences come out as they do without the extra rows, bit for bit."""
    if path == "single_kernel":
        request.getfixturevalue("single_kernel_backward")
    gen = torch.Generator().manual_seed(5)
    h, hk, used = 4, 2, sum(lens)
    total = before + used + after
    q, k, v, dout = (randn_half(gen, total, n, d).to(DEV) for n in (h, hk, hk, h))
    inner = slice(before, before + used)
    cu0 = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)
    cu = cu0 + before
    max_q, scale = max(lens), d ** -0.5
    torch.cuda.empty_cache()
    junk = [torch.full_like(x, float("nan")) for x in (q, q, k, v)]
    grads = [torch.full_like(x, float("nan")) for x in (q, k, v)]
    del junk  # the allocator hands this memory out for O
    out, lse = ext.varlen_fwd(q, k, v, cu, cu, max_q, max_k, scale, True)
    ext.varlen_bwd(q, k, v, out, lse, dout, cu, cu, max_q, max_k, scale, True, *grads)
    qi, ki, vi, di = (x[inner].contiguous() for x in (q, k, v, dout))
    want, want_lse = ext.varlen_fwd(qi, ki, vi, cu0, cu0, max_q, max_k, scale, True)
    want_grads = ext.varlen_bwd(qi, ki, vi, want, want_lse, di, cu0, cu0, max_q, max_k, scale, True)
    assert torch.equal(out[inner], want) and torch.equal(lse, want_lse)
    for i, (got, ref) in enumerate(zip(grads, want_grads)):
        if i == 0 and path == "single_kernel":  # summed in no fixed order: an fp16 ulp, and fp32 noise where it cancels
            torch.testing.assert_close(got[inner], ref, rtol=2 ** -10, atol=1e-4)
        else:
            assert torch.equal(got[inner], ref)
    for x in (out, *grads):
        assert x[:before].abs().sum() == 0 and x[before + used:].abs().sum() == 0
    assert ext.device_status(True) == 0


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("b,sq,sk,h,hk,causal", [
    (1, 1, 1, 1, 1, False),
    (1, 129, 300, 4, 2, True),       # a second tile of one row
    (1, 128 * 37, 700, 4, 4, True),  # 148 tiles: one item per SM, rows past sk without a visible key on the way
    (1, 128 * 37 + 1, 257, 4, 4, False),  # 152 tiles: pairs again
    (2, 500, 90, 3, 1, True),        # rows that see no key
])
def test_forward_items_of_one_tile(ext, d, b, sq, sk, h, hk, causal):
    """A small dense batch gets a work item per 128-row tile.  A row does not depend on how rows are grouped, so the result
    equals, bit for bit, that of the same batch among copies of itself (more tiles than SMs: items of two tiles)."""
    q, k, v, _ = (x.to(DEV) for x in _inputs(11, b, sq, sk, h, hk, d))
    out, lse = torch.full_like(q, float("nan")), torch.full((b, h, sq), float("nan"), device=DEV)
    ext.fwd(q, k, v, d ** -0.5, causal, out=out, lse=lse)
    n = 149
    many = [x[:1].repeat(n, 1, 1, 1) for x in (q, k, v)]
    want, want_lse = ext.fwd(*many, d ** -0.5, causal)
    assert torch.equal(out[0], want[0]) and torch.equal(lse[0], want_lse[0])
    o_ref, lse_ref = orc.attention_forward(*(x.cpu() for x in (q, k, v)), None, causal)
    assert err_stats(out, o_ref)[0] <= 2e-3 and err_stats(lse, lse_ref)[0] <= LSE_TOL
    assert ext.device_status(True) == 0


def _shortest_us(fn, runs=9, calls=4):
    best = float("inf")
    for _ in range(runs + 1):  # the first is a warm-up
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        for _ in range(calls):
            fn()
        end.record()
        end.synchronize()
        best = min(best, start.elapsed_time(end) * 1e3 / calls)
    return best


@pytest.mark.parametrize("h,d,lens", [(16, 64, (64,) * 64), (1, 64, (64,) * 64), (8, 128, (100,))])
def test_rows_without_a_sequence_cost_no_more_than_a_full_clear(ext, h, d, lens):
    """A buffer of fixed capacity, mostly unused (normal under CUDA graphs).  Bound: what the used rows take in a buffer of their
    own, and clearing whole tensors, with half as much again and 20 us for the spread of the timings."""
    torch.manual_seed(0)
    used, rows, scale = sum(lens), 32768, d ** -0.5
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)
    args = (cu, cu, max(lens), max(lens), scale, True)

    def times(rows):
        q, k, v, dout = (torch.randn(rows, h, d, device=DEV, dtype=torch.float16) for _ in range(4))
        grads = [torch.empty_like(x) for x in (q, k, v)]
        out, lse = ext.varlen_fwd(q, k, v, *args)
        return (_shortest_us(lambda: ext.varlen_fwd(q, k, v, *args)),
                _shortest_us(lambda: ext.varlen_bwd(q, k, v, out, lse, dout, *args, *grads)),
                _shortest_us(lambda: [g.zero_() for g in grads]))

    fwd, bwd, _ = times(used)
    fwd_spare, bwd_spare, clear = times(rows)
    assert fwd_spare <= 1.5 * (fwd + clear / 3) + 20, (fwd_spare, fwd, clear)
    assert bwd_spare <= 1.5 * (bwd + clear) + 20, (bwd_spare, bwd, clear)


@pytest.mark.parametrize("h,hk,d", [(1, 1, 64), (3, 1, 64), (5, 5, 128), (16, 4, 128)])
@pytest.mark.parametrize("before,after", [(0, 9001), (4097, 3), (2500, 2500)])
def test_thousands_of_unused_rows_in_strided_gradients_are_zero(ext, h, hk, d, before, after):
    """More unused rows than threads that clear, in gradients that are slices of a wider tensor; the rest of that tensor stays."""
    gen = torch.Generator().manual_seed(9)
    lens, scale = (70, 129), d ** -0.5
    total = before + sum(lens) + after
    q, k, v, dout = (randn_half(gen, total, n, d).to(DEV) for n in (h, hk, hk, h))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV) + before
    args = (cu, cu, max(lens), max(lens), scale, True)
    out, lse = ext.varlen_fwd(q, k, v, *args)
    wide = torch.full((total, h + 2 * hk + 1, d), float("nan"), device=DEV, dtype=torch.float16)
    grads = [wide[:, :h], wide[:, h:h + hk], wide[:, h + hk:h + 2 * hk]]
    ext.varlen_bwd(q, k, v, out, lse, dout, *args, *grads)
    for x in (out, *grads):
        assert x[:before].abs().sum() == 0 and x[before + sum(lens):].abs().sum() == 0
        assert torch.isfinite(x).all() and x.abs().sum() > 0
    assert torch.isnan(wide[:, h + 2 * hk]).all()


def test_row_statistics_are_read_at_the_rate_of_a_copy(ext):
    """The first stage of a dense backward reads O and dO once.  Bound: a copy that moves as many bytes on the same GPU, and 10 %
    (with two blocks per SM in place of three it took 18 % more)."""
    from flash_attention_turing_b200 import capi

    p, _, ws, keep = _bwd_params_for(ext, 4, 8192, 32, 32, 128, True, ())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    stage = _shortest_us(lambda: capi.check(capi.lib().fa_bwd_stages(ctypes.byref(p), 1, stream)))
    out, dst = keep[3], torch.empty_like(keep[3])
    copy = _shortest_us(lambda: dst.copy_(out))  # reads one tensor and writes one, where the stage reads two
    assert stage <= 1.1 * copy, (stage, copy)


@pytest.mark.parametrize("b,s,h,hk,d,causal,lens", [
    (2, 197, 12, 12, 64, False, ()),    # fewer items than SMs: the dK/dV kernel could start at once
    (1, 4096, 8, 2, 128, True, ()),
    (3, 300, 4, 2, 128, True, (300, 1, 129)),
])
@pytest.mark.parametrize("swapped", [False, True])
def test_gradients_may_be_written_over_keys_and_values(ext, b, s, h, hk, d, causal, lens, swapped):
    """dK and dV in the memory of K and V (or of V and K): bit for bit the gradients in memory of their own."""
    from flash_attention_turing_b200 import capi

    lib = capi.lib()
    p, grads, ws, keep = _bwd_params_for(ext, b, s, h, hk, d, causal, lens)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    capi.check(lib.fa_bwd(ctypes.byref(p), stream))
    k, v = keep[1], keep[2]
    k0, v0 = k.clone(), v.clone()
    dk, dv = (v, k) if swapped else (k, v)
    p.dk, p.dv = dk.data_ptr(), dv.data_ptr()
    for _ in range(10):
        k.copy_(k0), v.copy_(v0)
        capi.check(lib.fa_bwd(ctypes.byref(p), stream))
        assert torch.equal(dk, grads[1]) and torch.equal(dv, grads[2])


def test_packed_outputs_after_a_time_out_are_zero(ext):
    """While the time-out bit of the status word is set the kernels return at once.  The outputs of a packed call are zero then,
    not what the memory held before."""
    from flash_attention_turing_b200 import capi

    gen = torch.Generator().manual_seed(8)
    lens, h, hk, d = (300, 1, 129), 4, 2, 64
    total, scale = sum(lens) + 40, d ** -0.5
    q, k, v, dout = (randn_half(gen, total, n, d).to(DEV) for n in (h, hk, hk, h))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV) + 9
    args = (cu, cu, max(lens), max(lens), scale, True)
    want, want_lse = ext.varlen_fwd(q, k, v, *args)
    grads = [torch.full_like(x, float("nan")) for x in (q, k, v)]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    capi.check(capi.lib().fa_selftest_wait_timeout(1000, stream))
    torch.cuda.synchronize()
    try:
        junk = torch.full_like(q, float("nan"))
        torch.cuda.synchronize()
        del junk  # the allocator hands this memory out for O
        out, _ = ext.varlen_fwd(q, k, v, *args)
        ext.varlen_bwd(q, k, v, want, want_lse, dout, *args, *grads)
        torch.cuda.synchronize()
    finally:
        assert ext.device_status(True) & 1
    for x in (out, *grads):
        assert (x == 0).all()
    assert torch.equal(ext.varlen_fwd(q, k, v, *args)[0], want)


@pytest.mark.parametrize("flags", [0, 2, 3, -1, 0x7fffffff])
def test_forward_flags_of_no_meaning_leave_unused_rows_alone(ext, flags):
    """The field was a reserved one before: whatever a host of that time left in it clears nothing."""
    from flash_attention_turing_b200 import capi

    gen = torch.Generator().manual_seed(3)
    lens, h, d, spare = (70, 129), 2, 64, 11
    q, k, v = (randn_half(gen, sum(lens) + spare, h, d).to(DEV) for _ in range(3))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)
    out = torch.full_like(q, 7.0)
    lse = torch.zeros(len(lens), h, max(lens), device=DEV)
    p = capi.fwd_params(*(x[None] for x in (q, k, v, out)), lse, d ** -0.5, False)
    p.b, p.seqlen_q, p.seqlen_k, p.lse_row_stride = len(lens), max(lens), max(lens), max(lens)
    p.cu_seqlens_q = p.cu_seqlens_k = cu.data_ptr()
    p.total_q = p.total_k = q.shape[0]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for value in (flags, capi.FA_FWD_ZERO_UNUSED_ROWS):
        p.flags = value
        capi.check(capi.lib().fa_fwd(ctypes.byref(p), stream))
        assert (out[sum(lens):] == (0 if value == capi.FA_FWD_ZERO_UNUSED_ROWS else 7)).all()
        assert torch.equal(out[:sum(lens)], ext.varlen_fwd(q, k, v, cu, cu, max(lens), max(lens), d ** -0.5, False)[0][:sum(lens)])


@pytest.mark.parametrize("d", [64, 128])
def test_compiler_keeps_the_hand_back_of_the_dq_kernel_ahead_of_its_arithmetic(ext, d):
    """The block boundary behind the hand-back (schedule_barrier) is one that a compiler might remove.  The dQ kernel takes 0.69
    (D = 128) and 0.76 (D = 64) of the time of the dK/dV kernel with it, 0.97 to 1.0 without; the bound lies between."""
    from flash_attention_turing_b200 import capi

    lib = capi.lib()
    p, _, ws, keep = _bwd_params_for(ext, 2, 2048, 16, 16, d, False, ())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    capi.check(lib.fa_bwd_stages(ctypes.byref(p), 1, stream))
    dq, dkdv = (_shortest_us(lambda: capi.check(lib.fa_bwd_stages(ctypes.byref(p), stage, stream))) for stage in (2, 4))
    assert dq <= 0.87 * dkdv, (dq, dkdv)


@pytest.mark.parametrize("max_k", [128, 130, 384])
@pytest.mark.parametrize("d,lens", [(64, (300, 520)), (128, (520, 300, 1)), (128, (700,))])
def test_key_gradients_past_the_given_maximum_are_zero(ext, d, lens, max_k):
    """A max_seqlen_k below a sequence's length: dK and dV are written for the whole tiles within it and zero from there on, in
    a sequence in between as in the last one, whatever the memory held.  O and dQ do not depend on it."""
    gen = torch.Generator().manual_seed(12)
    h, hk, scale = 4, 2, d ** -0.5
    q, k, v, dout = (randn_half(gen, sum(lens), n, d).to(DEV) for n in (h, hk, hk, h))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)

    def run(max_k):
        args = (cu, cu, max(lens), max_k, scale, True)
        out, lse = ext.varlen_fwd(q, k, v, *args)
        grads = [torch.full_like(x, float("nan")) for x in (q, k, v)]
        ext.varlen_bwd(q, k, v, out, lse, dout, *args, *grads)
        return out, *grads

    out, dq, dk, dv = run(max_k)
    want_out, want_dq, want_dk, want_dv = run(max(lens))
    assert torch.equal(out, want_out) and torch.equal(dq, want_dq)
    written = -(-max_k // 128) * 128
    for got, want in ((dk, want_dk), (dv, want_dv)):
        first = 0
        for n in lens:
            assert torch.equal(got[first:first + min(n, written)], want[first:first + min(n, written)])
            assert (got[first + min(n, written):first + n] == 0).all()
            first += n


@pytest.mark.parametrize("d,lens,h,hk", [(128, (2048,) * 5, 7, 7), (128, (4096,) * 3, 18, 9), (64, (4096,) * 5, 14, 14),
                                         (128, (300, 8192, 5000), 18, 9), (64, (16384, 129), 9, 9)])
def test_heads_of_several_sections_equal_heads_by_themselves(ext, d, lens, h, hk):
    """More heads than one section of the work order holds, and a last section that is not full: every item runs once and its
    result does not depend on the others (bitwise)."""
    gen = torch.Generator(device=DEV).manual_seed(21)
    total, group, scale = sum(lens), h // hk, d ** -0.5
    q, k, v, dout = (torch.randn(total, n, d, generator=gen, device=DEV, dtype=torch.half) for n in (h, hk, hk, h))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)

    def run(kv_heads):
        heads = slice(kv_heads.start * group, kv_heads.stop * group)
        qq, kk, vv, dd = q[:, heads], k[:, kv_heads], v[:, kv_heads], dout[:, heads]
        if len(set(lens)) > 1:
            args = (cu, cu, max(lens), max(lens), scale, True)
            out, lse = ext.varlen_fwd(qq, kk, vv, *args)
            return out, *ext.varlen_bwd(qq, kk, vv, out, lse, dd, *args)
        qq, kk, vv, dd = (x.unflatten(0, (len(lens), -1)) for x in (qq, kk, vv, dd))
        out, lse = ext.fwd(qq, kk, vv, scale, True)
        return tuple(x.flatten(0, 1) for x in (out, *ext.bwd(qq, kk, vv, out, lse, dd, scale, True)))

    got = run(slice(0, hk))
    for i in range(hk):
        for x, want in zip(got, run(slice(i, i + 1))):
            n = want.shape[1]
            assert torch.equal(x[:, i * n:(i + 1) * n], want)


def _public_calls(d, grad):
    """(name, native function, class, inputs, further arguments) of the six public functions with an autograd class."""
    import flash_attention_turing_b200.flash_attention_interface as fi

    gen = torch.Generator().manual_seed(5)
    r = lambda *s: randn_half(gen, *s).to(DEV).requires_grad_(grad)  # noqa: E731
    cu = torch.tensor([0, 70, 199], dtype=torch.int32, device=DEV)
    dense, var = (None, True), (129, 129, None, True)
    return [
        ("dense", fi.flash_attn_func, fi.FlashAttnFunc, [r(2, 130, 4, d), r(2, 150, 2, d), r(2, 150, 2, d)], (), dense),
        ("qkv", fi.flash_attn_qkvpacked_func, fi.FlashAttnQKVPackedFunc, [r(2, 130, 3, 4, d)], (), dense),
        ("kv", fi.flash_attn_kvpacked_func, fi.FlashAttnKVPackedFunc, [r(2, 130, 4, d), r(2, 150, 2, 2, d)], (), dense),
        ("varlen", fi.flash_attn_varlen_func, fi.FlashAttnVarlenFunc, [r(199, 4, d), r(199, 2, d), r(199, 2, d)], (cu, cu), var),
        ("varlen qkv", fi.flash_attn_varlen_qkvpacked_func, fi.FlashAttnVarlenQKVPackedFunc, [r(199, 3, 4, d)], (cu,), var[1:]),
        ("varlen kv", fi.flash_attn_varlen_kvpacked_func, fi.FlashAttnVarlenKVPackedFunc, [r(199, 4, d), r(199, 2, 2, d)], (cu, cu), var),
    ]


@pytest.mark.parametrize("which", range(6))
@pytest.mark.parametrize("d", [64, 128])
def test_native_autograd_node_equals_the_class(ext, d, which):
    """Outputs, gradients, what is saved (as saved-tensor hooks see it), no gradients, a second backward, a transposed dout."""
    _, fn, cls, inputs, extra, rest = _public_calls(d, True)[which]

    def run(call, *tail):
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append((t.shape, t.stride(), t.dtype)) or t, lambda t: t):
            out = call(*inputs, *extra, *rest, *tail)
        dout = torch.linspace(-1, 1, out.numel(), device=DEV).half().view(out.mT.shape).mT  # last dimension not contiguous
        first = torch.autograd.grad(out, inputs, dout, retain_graph=True)
        again = torch.autograd.grad(out, inputs, dout)
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(out, inputs, dout)
        assert all(torch.equal(x, y) for x, y in zip(first, again))
        return seen, (out.detach(), *first)

    saved, got = run(fn)
    saved_class, want = run(cls.apply, True)
    assert saved == saved_class
    assert all(torch.equal(x, y) and x.stride() == y.stride() for x, y in zip(got, want))
    with torch.no_grad():
        out = fn(*inputs, *extra, *rest)
    assert not out.requires_grad and torch.equal(out, want[0])
    # a gradient of some inputs only, and a mutated input
    inputs[-1].requires_grad_(False)
    if len(inputs) > 1:
        out = fn(*inputs, *extra, *rest)
        g = torch.autograd.grad(out, inputs[0], torch.ones_like(out), retain_graph=True)[0]
        assert g.shape == inputs[0].shape
        inputs[-1].add_(1)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            torch.autograd.grad(out, inputs[0], torch.ones_like(out))


@pytest.mark.parametrize("which", range(6))
def test_transforms_and_modes_still_go_to_the_class(ext, which):
    """What the native node does not know: functorch transforms and forward-mode AD are refused as by the class, a traced call is
    recorded, a tensor subclass and a mode reach the class."""
    from torch.overrides import TorchFunctionMode

    name, fn, cls, inputs, extra, rest = _public_calls(64, False)[which]
    call = lambda *x: fn(*x, *extra, *rest)  # noqa: E731
    with pytest.raises(RuntimeError, match="functorch transforms"):
        torch.func.vmap(call)(*(x[None] for x in inputs))
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(inputs[0], torch.ones_like(inputs[0]))
        with pytest.raises((RuntimeError, NotImplementedError)):
            call(dual, *inputs[1:])
    traced = torch.jit.trace(call, tuple(inputs), check_trace=False)
    other = [x.flip(0).contiguous() for x in inputs]
    assert torch.equal(traced(*other), call(*other))
    applied = []
    real = cls.apply
    try:
        cls.apply = classmethod(lambda c, *a: applied.append(1) or real(*a))

        class Mode(TorchFunctionMode):
            def __torch_function__(self, func, types, args=(), kwargs=None):
                return func(*args, **(kwargs or {}))

        with Mode():
            call(*inputs)
        call(inputs[0].as_subclass(type("Sub", (torch.Tensor,), {})), *inputs[1:])
        assert len(applied) == 2
        call(*inputs)
        assert len(applied) == 2
    finally:
        del cls.apply
    assert torch.equal(call(*inputs), cls.apply(*inputs, *extra, *rest, False))


@pytest.mark.parametrize("lens", [(1, 1023, 1024), (1025, 0, 3), (2100, 700), (5,) * 300])
def test_lse_past_the_end_of_a_sequence_is_zero(ext, lens):
    """Whatever the memory held before, by the binding and by the flag of the C entry; without the flag it is left alone."""
    from flash_attention_turing_b200 import capi

    gen = torch.Generator().manual_seed(4)
    h, d, longest = 3, 64, max(lens) + 1
    q, k, v = (randn_half(gen, sum(lens), h, d).to(DEV) for _ in range(3))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).to(DEV)
    inside = torch.arange(longest, device=DEV)[None, None] < torch.tensor(lens, device=DEV)[:, None, None].expand(-1, h, 1)
    for _ in range(3):
        junk = [torch.full((len(lens), h, longest), float("nan"), device=DEV) for _ in range(4)]
        torch.cuda.synchronize()
        del junk  # the allocator hands this memory out for the LSE
        _, lse = ext.varlen_fwd(q, k, v, cu, cu, longest, longest, d ** -0.5, True)
        assert torch.isfinite(lse).all() and (lse[~inside] == 0).all()
    for flags in (0, capi.FA_FWD_ZERO_UNUSED_ROWS):
        out, got = torch.empty_like(q), torch.full_like(lse, 7.0)
        p = capi.fwd_params(*(x[None] for x in (q, k, v, out)), got, d ** -0.5, True)
        p.b, p.seqlen_q, p.seqlen_k, p.lse_row_stride = len(lens), longest, longest, longest
        p.cu_seqlens_q = p.cu_seqlens_k = cu.data_ptr()
        p.total_q, p.total_k, p.flags = q.shape[0], k.shape[0], flags
        capi.check(capi.lib().fa_fwd(ctypes.byref(p), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert torch.equal(got[inside], lse[inside]) and (got[~inside] == (0 if flags else 7)).all()
