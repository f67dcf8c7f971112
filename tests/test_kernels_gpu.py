"""sm_100a kernels vs the PyTorch fp32 oracle (runs on the B200 box: `pytest -m gpu`)."""
import contextlib
import math
import os
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from gllm_b200.ops import ref


def _dev():
    return torch.device("cuda:0")


def _rel_err(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / (b.norm() + 1e-12)).item()


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (1, 512, 128), (37, 384, 192), (256, 6144, 4096),
                                   (1000, 4096, 4096), (2048, 24576, 4096), (5, 151936, 1024),
                                   (130, 72, 320)])
@pytest.mark.parametrize("bn", [0, 32, 64, 128, 256])
def test_gemm_bf16(m, n, k, bn, monkeypatch):
    from gllm_b200.ops import sm100
    if bn and m * n * k > 2e10:
        pytest.skip("big shape only with auto tile")
    monkeypatch.setattr(sm100, "_FORCE_BN", bn)
    torch.manual_seed(0)
    x = (torch.randn(m, k, device=_dev()) * 0.5).bfloat16()
    w = (torch.randn(n, k, device=_dev()) * 0.05).bfloat16()
    y = sm100.linear(x, w)
    torch.cuda.synchronize()
    yr = x.float() @ w.float().t()
    assert _rel_err(y, yr) < 6e-3, _rel_err(y, yr)
    assert torch.isfinite(y.float()).all()


def test_gemm_bias_and_strided():
    from gllm_b200.ops import sm100
    torch.manual_seed(1)
    m, n, k = 300, 1024, 512
    big = (torch.randn(m, k * 2, device=_dev()) * 0.5).bfloat16()
    x = big[:, :k]  # row stride 2k
    w = (torch.randn(n, k, device=_dev()) * 0.05).bfloat16()
    b = torch.randn(n, device=_dev()).bfloat16()
    y = sm100.linear(x, w, b)
    yr = x.float() @ w.float().t() + b.float()
    assert _rel_err(y, yr) < 6e-3


def test_gemm_silu_mul():
    from gllm_b200.ops import sm100
    torch.manual_seed(2)
    m, i, k = 200, 1024, 512
    x = (torch.randn(m, k, device=_dev()) * 0.5).bfloat16()
    w = (torch.randn(2 * i, k, device=_dev()) * 0.05).bfloat16()
    wi = ref.interleave_gate_up(w, 128)
    y = sm100.linear_silu_mul(x, wi)
    h = x.float() @ w.float().t()
    yr = torch.nn.functional.silu(h[:, :i]) * h[:, i:]
    assert _rel_err(y, yr) < 1e-2
    # and the oracle's own interleaved path agrees
    assert _rel_err(ref.linear_silu_mul(x, wi, 128), yr) < 1e-2


@pytest.mark.parametrize("t,h", [(1, 4096), (7, 1024), (300, 4096), (64, 8192), (3, 7168), (2, 16384)])
@pytest.mark.parametrize("add", [False, True])
def test_rmsnorm(t, h, add):
    from gllm_b200.ops import sm100
    torch.manual_seed(3)
    x = torch.randn(t, h, device=_dev()).bfloat16()
    w = (1 + 0.1 * torch.randn(h, device=_dev())).bfloat16()
    r = torch.randn(t, h, device=_dev()).bfloat16() if add else None
    o_ref, r_ref = ref.rmsnorm(x, w, 1e-6, r.clone() if add else None)
    o, r_out = sm100.rmsnorm(x, w, 1e-6, r.clone() if add else None)
    assert _rel_err(o, o_ref) < 5e-3
    if add:
        assert _rel_err(r_out, r_ref) < 1e-3


def test_silu_and_mul():
    from gllm_b200.ops import sm100
    x = torch.randn(77, 2 * 1536, device=_dev()).bfloat16()
    assert _rel_err(sm100.silu_and_mul(x), ref.silu_and_mul(x)) < 5e-3


def test_embedding_and_gather():
    from gllm_b200.ops import sm100
    table = torch.randn(1000, 512, device=_dev()).bfloat16()
    ids = torch.randint(0, 2000, (333,), device=_dev(), dtype=torch.int32)
    o = sm100.embedding(ids, table, 500, 1500)
    o_ref = ref.embedding(ids, table, 500, 1500)
    assert torch.equal(o, o_ref)
    idx = torch.randint(0, 1000, (50,), device=_dev(), dtype=torch.int32)
    assert torch.equal(sm100.gather_rows(table, idx), table[idx.long()])


@pytest.mark.parametrize("d,rot,neox,qk_norm", [(128, 128, True, True), (128, 128, True, False),
                                                (64, 64, True, False), (128, 64, False, False),
                                                (256, 256, True, True)])
def test_rope_kv_write(d, rot, neox, qk_norm):
    from gllm_b200.ops import sm100
    torch.manual_seed(4)
    t, hq, hkv, page, pages = 83, 8, 2, 16, 32
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device=_dev()).bfloat16()
    qkv_ref = qkv.clone()
    pos = torch.randint(0, 500, (t,), device=_dev(), dtype=torch.int32)
    slots = torch.randperm(pages * page, device=_dev())[:t].to(torch.int32)
    slots[5] = -1
    cs = ref.build_cos_sin_cache(rot, 512, 10000.0).to(_dev())
    qn = (1 + 0.1 * torch.randn(d, device=_dev())).bfloat16() if qk_norm else None
    kn = (1 + 0.1 * torch.randn(d, device=_dev())).bfloat16() if qk_norm else None
    shape = ref.kv_cache_shape(pages, hkv, d, page)
    kc, vc = torch.zeros(shape, device=_dev(), dtype=torch.bfloat16), torch.zeros(shape, device=_dev(), dtype=torch.bfloat16)
    kc_r, vc_r = kc.clone(), vc.clone()

    def views(buf):
        q = buf[:, : hq * d].view(t, hq, d)
        k = buf[:, hq * d: (hq + hkv) * d].view(t, hkv, d)
        v = buf[:, (hq + hkv) * d:].view(t, hkv, d)
        return q, k, v

    q, k, v = views(qkv)
    sm100.rope_kv_write(q, k, v, pos, cs, rot, neox, qn, kn, 1e-6, kc, vc, slots)
    qr, kr, vr = views(qkv_ref)
    ref.rope_kv_write(qr, kr, vr, pos, cs, rot, neox, qn, kn, 1e-6, kc_r, vc_r, slots)
    assert _rel_err(qkv, qkv_ref) < 8e-3
    assert _rel_err(kc, kc_r) < 8e-3
    assert torch.equal(vc, vc_r)


@pytest.mark.parametrize("t,hq,hkv", [(1, 5, 1), (3, 32, 8), (700, 19, 3), (2100, 32, 8)])   # one head per lane, or four
@pytest.mark.parametrize("d,rot,neox", [(64, 32, True), (64, 0, True), (128, 96, True), (128, 24, False), (256, 256, True)])
@pytest.mark.parametrize("shift", [0, 1])     # 1: rows off the 16-byte boundary (the 4-byte kernel)
def test_rope_kv_write_edges(t, hq, hkv, d, rot, neox, shift):
    """Head counts that leave lane groups empty, partly rotated heads, skipped slots, both access widths; against fp32
    formulas at bf16 rounding (2^-9 relative per step, two steps)."""
    from gllm_b200.ops import sm100
    if (rot // 2) % (d // 32):
        pytest.skip("rotated halves must hold whole lanes")
    torch.manual_seed(t + d)
    page, pages = 16, (t + 15) // 16 + 2
    width = (hq + 2 * hkv) * d
    buf = torch.randn(t, width + 8, device=_dev()).bfloat16()
    ref_buf = buf.clone()
    pos = torch.randint(0, 4000, (t,), device=_dev(), dtype=torch.int32)
    slots = torch.randperm(pages * page, device=_dev())[:t].to(torch.int32)
    slots[t // 2] = -1
    cs = ref.build_cos_sin_cache(rot, 4096, 10000.0).to(_dev()) if rot else None
    qn = (1 + 0.1 * torch.randn(d, device=_dev())).bfloat16()
    kn = (1 + 0.1 * torch.randn(d, device=_dev())).bfloat16()
    shape = ref.kv_cache_shape(pages, hkv, d, page)
    caches = [torch.zeros(shape, device=_dev(), dtype=torch.bfloat16) for _ in range(4)]

    def views(b):
        b = b[:, 2 * shift:2 * shift + width]
        return (b[:, : hq * d].unflatten(1, (hq, d)), b[:, hq * d: (hq + hkv) * d].unflatten(1, (hkv, d)),
                b[:, (hq + hkv) * d:].unflatten(1, (hkv, d)))

    sm100.rope_kv_write(*views(buf), pos, cs, rot, neox, qn, kn, 1e-6, caches[0], caches[1], slots)
    ref.rope_kv_write(*views(ref_buf), pos, cs, rot, neox, qn, kn, 1e-6, caches[2], caches[3], slots)
    assert _rel_err(buf, ref_buf) < 8e-3 and _rel_err(caches[0], caches[2]) < 8e-3
    assert torch.equal(caches[1], caches[3])


@pytest.mark.parametrize("t,hq,hkv", [(1, 5, 1), (3, 33, 8), (700, 19, 3), (2100, 32, 8)])   # one head per lane group, or two
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("norms,cached", [("qk", True), ("q", True), ("", True), ("k", False)])
def test_rope_kv_write_whole_heads(t, hq, hkv, d, norms, cached):
    """NeoX rotation of whole heads, both halves of a pair in one lane: lane groups without a head, one norm of the two, no cache;
    tolerance as above (two roundings to bf16)."""
    from gllm_b200.ops import sm100
    torch.manual_seed(t + d)
    page, pages = 16, (t + 15) // 16 + 2
    buf = torch.randn(t, (hq + 2 * hkv) * d, device=_dev()).bfloat16()
    ref_buf = buf.clone()
    pos = torch.randint(0, 4000, (t,), device=_dev(), dtype=torch.int32)
    slots = torch.randperm(pages * page, device=_dev())[:t].to(torch.int32)
    slots[t // 2] = -1
    cs = ref.build_cos_sin_cache(d, 4096, 10000.0).to(_dev())
    qn, kn = ((1 + 0.1 * torch.randn(d, device=_dev())).bfloat16() if n in norms else None for n in "qk")
    shape = ref.kv_cache_shape(pages, hkv, d, page)
    caches = [torch.zeros(shape, device=_dev(), dtype=torch.bfloat16) if cached else None for _ in range(4)]

    def views(b):
        q, k, v = b.split([hq * d, hkv * d, hkv * d], 1)
        return q.unflatten(1, (hq, d)), k.unflatten(1, (hkv, d)), v.unflatten(1, (hkv, d)) if cached else None

    sm100.rope_kv_write(*views(buf), pos, cs, d, True, qn, kn, 1e-6, caches[0], caches[1], slots if cached else None)
    ref.rope_kv_write(*views(ref_buf), pos, cs, d, True, qn, kn, 1e-6, caches[2], caches[3], slots if cached else None)
    assert _rel_err(buf, ref_buf) < 8e-3
    if cached:
        assert _rel_err(caches[0], caches[2]) < 8e-3
        assert torch.equal(caches[1], caches[3])


@pytest.mark.parametrize("d,sec", [(64, [8, 12, 12]), (128, [16, 24, 24])])
@pytest.mark.parametrize("t", [300, 4099])                          # one head per lane group, or two
def test_rope_kv_write_both_forms_give_the_same_bits(d, sec, t):
    """Three equal rows of positions take the form with a lane per eight elements, one row the one with both halves of a pair in a lane:
    sums, roundings and rotations are the same, and so is every bit."""
    from gllm_b200.ops import sm100
    torch.manual_seed(d)
    hq, hkv = 24, 8
    pos = torch.randint(0, 4000, (t,), device=_dev(), dtype=torch.int32)
    slots = torch.randperm(t + 16, device=_dev())[:t].to(torch.int32)
    cs = ref.build_cos_sin_cache(d, 4096, 10000.0).to(_dev())
    qn, kn = ((1 + 0.1 * torch.randn(d, device=_dev())).bfloat16() for _ in range(2))
    src, got = torch.randn(t, (hq + 2 * hkv) * d, device=_dev()).bfloat16(), []
    for p, section in ((pos, None), (pos.repeat(3, 1), sec)):
        buf = src.clone()
        q, k, v = buf.split([hq * d, hkv * d, hkv * d], 1)
        caches = [torch.zeros(ref.kv_cache_shape(t // 16 + 2, hkv, d, 16), device=_dev(), dtype=torch.bfloat16) for _ in range(2)]
        sm100.rope_kv_write(q.unflatten(1, (hq, d)), k.unflatten(1, (hkv, d)), v.unflatten(1, (hkv, d)), p, cs, d, True, qn, kn, 1e-6,
                            *caches, slots, section)
        got.append((buf, *caches))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("sec", [[16, 24, 24], [24, 20, 20, 1]])   # chunked (Qwen2.5-VL) / interleaved (Qwen3-VL)
@pytest.mark.parametrize("strided", [False, True])
def test_rope_mrope(sec, strided):
    from gllm_b200.ops import sm100
    torch.manual_seed(5)
    t, hq, hkv, d = 40, 4, 2, 128
    q = torch.randn(t, hq, d, device=_dev()).bfloat16()
    k = torch.randn(t, hkv, d, device=_dev()).bfloat16()
    q_r, k_r = q.clone(), k.clone()
    pos = torch.randint(0, 300, (3, t + 24), device=_dev(), dtype=torch.int32)
    pos = pos[:, :t] if strided else pos[:, :t].contiguous()   # the runner passes a view of a [3, max_tokens] buffer
    cs = ref.build_cos_sin_cache(d, 512, 1e6).to(_dev())
    sm100.rope_kv_write(q, k, None, pos, cs, d, True, None, None, 1e-6, None, None, None, mrope_section=sec)
    ref.rope_kv_write(q_r, k_r, None, pos, cs, d, True, None, None, 1e-6, None, None, None, mrope_section=sec)
    assert _rel_err(q, q_r) < 8e-3 and _rel_err(k, k_r) < 8e-3


def _make_paged(seq_lens, q_lens, hq, hkv, d, page, device, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    b = len(seq_lens)
    max_blocks = max((s + page - 1) // page for s in seq_lens) + 1
    n_pages = sum((s + page - 1) // page for s in seq_lens) + 3
    perm = torch.randperm(n_pages, generator=g).tolist()
    bt = torch.zeros(b, max_blocks, dtype=torch.int32)
    c = 0
    for i, s in enumerate(seq_lens):
        n = (s + page - 1) // page
        bt[i, :n] = torch.tensor(perm[c:c + n], dtype=torch.int32)
        c += n
    shape = ref.kv_cache_shape(n_pages, hkv, d, page)
    kc = (torch.randn(shape, generator=g) * 0.5).bfloat16().to(device)
    vc = (torch.randn(shape, generator=g) * 0.5).bfloat16().to(device)
    t = sum(q_lens)
    q = (torch.randn(t, hq * d, generator=g) * 0.5).bfloat16().to(device)
    qsl = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32, device=device)
    sl = torch.tensor(seq_lens, dtype=torch.int32, device=device)
    return q, kc, vc, bt.to(device), sl, qsl


@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (8, 8, 128), (28, 4, 128), (16, 2, 64), (8, 1, 128)])
@pytest.mark.parametrize("splits", [None, 1, 4])
def test_attn_decode(hq, hkv, d, splits):
    from gllm_b200.ops import sm100
    seq_lens = [1, 5, 16, 17, 63, 64, 65, 200, 1000, 333]
    q_lens = [1] * len(seq_lens)
    q, kc, vc, bt, sl, qsl = _make_paged(seq_lens, q_lens, hq, hkv, d, 16, _dev())
    scale = 1.0 / math.sqrt(d)
    o = sm100.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d, len(seq_lens), len(seq_lens), 1,
                              max(seq_lens), splits=splits)
    torch.cuda.synchronize()
    o_ref = ref.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d)
    assert torch.isfinite(o.float()).all()
    assert _rel_err(o, o_ref) < 1e-2, _rel_err(o, o_ref)


@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (8, 8, 128), (28, 4, 128), (16, 2, 64)])
def test_attn_prefill_and_mixed(hq, hkv, d, monkeypatch):
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "ATTN_TC", False)     # the mma.sync kernel (fallback for shapes outside the tcgen05 one)
    # decode seqs first, then prefill chunks (some with prefix/chunk context)
    seq_lens = [7, 130, 40, 300, 129, 64, 1024]
    q_lens = [1, 1, 40, 100, 129, 3, 513]
    nd = 2
    q, kc, vc, bt, sl, qsl = _make_paged(seq_lens, q_lens, hq, hkv, d, 16, _dev(), seed=1)
    scale = 1.0 / math.sqrt(d)
    o = sm100.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d, nd, len(seq_lens), max(q_lens), max(seq_lens))
    torch.cuda.synchronize()
    o_ref = ref.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d)
    assert torch.isfinite(o.float()).all()
    assert _rel_err(o, o_ref) < 1e-2, _rel_err(o, o_ref)


@pytest.mark.parametrize("kv_tile", [128, 64])
@pytest.mark.parametrize("hq,hkv,d", [(32, 8, 128), (8, 8, 128), (28, 4, 128), (16, 2, 64)])
def test_prefill_attention_tc(hq, hkv, d, kv_tile, monkeypatch):
    """tcgen05 / TMEM prefill kernel vs the fp32 oracle: ragged chunks, prefix context, page-boundary cases."""
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "ATTN_TC", True)
    monkeypatch.setattr(sm100, "ATTN_TC_KV", kv_tile)
    seq_lens = [7, 130, 40, 300, 129, 64, 1024, 257]
    q_lens = [1, 1, 40, 100, 129, 3, 513, 257]
    nd = 2
    q, kc, vc, bt, sl, qsl = _make_paged(seq_lens, q_lens, hq, hkv, d, 16, _dev(), seed=1)
    scale = 1.0 / math.sqrt(d)
    o = sm100.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d, nd, len(seq_lens), max(q_lens), max(seq_lens))
    torch.cuda.synchronize()
    o_ref = ref.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d)
    assert torch.isfinite(o.float()).all()
    assert _rel_err(o, o_ref) < 1e-2, _rel_err(o, o_ref)


@pytest.mark.parametrize("page", [32, 64, 128])
@pytest.mark.parametrize("hq,hkv,d", [(8, 2, 128), (4, 4, 64)])
def test_prefill_attention_tc_page_sizes(hq, hkv, d, page, monkeypatch):
    """Pages below, at and above half of the 128 keys that the kernel walks at a time: two boxes of 64 rows for a page of 128,
    which ATTN_TC_KV = 128 admits."""
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "ATTN_TC", True)
    monkeypatch.setattr(sm100, "ATTN_TC_KV", max(64, page))
    q_lens, ctx = [1, 40, 127, 128, 300, 64], [127, 0, 129, 128, 1, 700]
    seq_lens = [a + b for a, b in zip(q_lens, ctx)]
    q, kc, vc, bt, sl, qsl = _make_paged(seq_lens, q_lens, hq, hkv, d, page, _dev(), seed=5)
    o = sm100.paged_attention(q, kc, vc, bt, sl, qsl, d ** -0.5, hq, d, 0, len(q_lens), max(q_lens), max(seq_lens))
    assert _rel_err(o, ref.paged_attention(q, kc, vc, bt, sl, qsl, d ** -0.5, hq, d)) < 1e-2


@pytest.mark.parametrize("hq,hkv,d", [(8, 1, 128), (4, 4, 128), (6, 2, 64)])
@pytest.mark.parametrize("page", [8, 16, 64])
@pytest.mark.parametrize("many", [False, True])       # few CTAs: one query tile each; many: two
def test_prefill_attention_tc_edges(hq, hkv, d, page, many, monkeypatch):
    """Chunks and contexts at the edges of the 128-row query tiles (16, 128 and 42 tokens), of their pairs and of the 128-key
    tiles; scores that grow along the keys so that the running reference of the exponentials moves; the same bits again."""
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "ATTN_TC", True)
    q_lens = [1, 15, 16, 17, 32, 33, 127, 128, 129, 255, 256, 257, 5, 300]
    ctx = [0, 1, 127, 128, 129, 0, 1, 500, 0, 1, 0, 255, 1000, 84]
    if many:
        q_lens, ctx = q_lens * 3, ctx * 3
    seq_lens = [a + b for a, b in zip(q_lens, ctx)]
    q, kc, vc, bt, sl, qsl = _make_paged(seq_lens, q_lens, hq, hkv, d, page, _dev(), seed=3)
    for i, n in enumerate(seq_lens):                  # scores rise by some 40 over a sequence
        for b in range((n + page - 1) // page):
            kc[bt[i, b].long()] *= 1 + 6.0 * b * page / 1024
    scale = 1.0 / math.sqrt(d)
    args = (q, kc, vc, bt, sl, qsl, scale, hq, d, 0, len(seq_lens), max(q_lens), max(seq_lens))
    o = sm100.paged_attention(*args)
    again = sm100.paged_attention(*args)
    o_ref = ref.paged_attention(q, kc, vc, bt, sl, qsl, scale, hq, d)
    assert torch.isfinite(o.float()).all() and torch.equal(o, again)
    assert _rel_err(o, o_ref) < 1e-2, _rel_err(o, o_ref)
    assert sm100.waits_given_up() == 0


def test_prefill_attention_of_more_sequences_than_a_grid_dimension():
    """65,600 sequences of one or two tokens: the blocks are counted in one dimension then."""
    from gllm_b200.ops import sm100
    torch.manual_seed(4)
    n, d = 65600, 64
    two = torch.arange(n) % 3 == 0
    lens = 1 + two.int()
    qsl = torch.cat([torch.zeros(1, dtype=torch.int32), lens.cumsum(0).int()]).to(_dev())
    q = torch.randn(int(lens.sum()), d, device=_dev()).bfloat16()
    kc, vc = (torch.randn(n, 1, 1, 8, d, device=_dev()).bfloat16() for _ in range(2))
    bt = torch.randperm(n, device=_dev()).int().view(n, 1)
    o = sm100.paged_attention(q, kc, vc, bt, lens.to(_dev()).int(), qsl, d ** -0.5, 1, d, 0, n, 2, 2).float()
    k, v = (x[bt[:, 0].long(), 0, 0].float() for x in (kc, vc))
    first, at = qsl[:-1].long(), two.to(_dev())
    assert _rel_err(o[first], v[:, 0]) < 1e-2
    s = torch.einsum("nd,nkd->nk", q[first[at] + 1].float(), k[at, :2]) * d ** -0.5
    assert _rel_err(o[first[at] + 1], torch.einsum("nk,nkd->nd", s.softmax(-1), v[at, :2])) < 1e-2


@pytest.mark.parametrize("window,bad,clean", [(None, 180, (40, 168)), (100, 60, (168, 340))])
@pytest.mark.parametrize("seqs", [1, 12])                   # one query tile per CTA, or two
def test_prefill_value_that_is_no_number(window, bad, clean, seqs):
    """A NaN in one cached value row reaches only query tiles of 128 rows that see a key of its 16-key step: not the tile whose
    last token (168 - 1) lies before that step, nor one whose window (from 168 - 99 on) starts behind it."""
    from gllm_b200.ops import sm100_seq as S
    h, d, page, ctx, n = 4, 128, 16, 40, 300
    q, kc, vc, bt, sl, qsl = _make_paged([ctx + n] * seqs, [n] * seqs, h, h, d, page, _dev(), seed=2)
    pos = torch.arange(ctx, ctx + n, dtype=torch.int32, device=_dev()).repeat(seqs)
    want = ref.window_attention(q, kc, vc, bt, sl, qsl, d ** -0.5, h, d, window, None)
    for i in range(seqs):
        vc[bt[i, bad // page].long(), :, :, bad % page] = float("nan")
    got = S.window_attention(q, kc, vc, bt, sl, qsl, pos, d ** -0.5, h, d, window, None, 0, n)
    ok = (pos >= clean[0]) & (pos < clean[1])
    assert _rel_err(got[ok], want[ok]) < 1e-2
    sees = (pos >= bad) & (pos < (bad + window if window else ctx + n))
    assert bool(torch.isnan(got[sees]).all())


@pytest.mark.parametrize("family", ["fp8", "attn", "mla", "gemm", "clusters", "gated clusters"])
def test_wait_that_gives_up_reaches_the_caller(family):
    """A wait limit of zero: whatever is not there at the first look is given up. The kernel returns, the engine's check raises,
    and the next call is right again."""
    from gllm_b200.model_runner import StepResult
    from gllm_b200.ops import lib, sm100
    torch.manual_seed(1)
    if family == "fp8":
        x, w = torch.randn(300, 1024, device=_dev()).bfloat16(), torch.randn(512, 1024, device=_dev()).to(torch.float8_e4m3fn)
        ws = torch.ones(4, 8, device=_dev())
        call = lambda: sm100.linear_fp8_block(x, w, ws)
        want = x.float() @ w.float().t()
    elif family == "gemm":
        x, w = torch.randn(600, 1024, device=_dev()).bfloat16(), torch.randn(6144, 1024, device=_dev()).bfloat16()
        call = lambda: sm100.linear(x, w)
        want = x.float() @ w.float().t()
    elif "clusters" in family:                                # 192 K blocks: every part of a cluster fills its ring more than once
        x, w = torch.randn(64, 12288, device=_dev()).bfloat16(), torch.randn(4096, 12288, device=_dev()).bfloat16() * 12288 ** -0.5
        call = lambda: sm100.linear(x, w)
        want = x.float() @ w.float().t()
        if family != "clusters":
            wi = ref.interleave_gate_up(w, 128)
            call = lambda: sm100.linear_silu_mul(x, wi)
            want = torch.nn.functional.silu(want[:, :2048]) * want[:, 2048:]
    elif family == "attn":
        lens = [300, 129]
        a = _make_paged(lens, lens, 8, 2, 128, 16, _dev(), seed=1)
        call = lambda: sm100.paged_attention(*a, 128 ** -0.5, 8, 128, 0, 2, 300, 300)
        want = ref.paged_attention(*a, 128 ** -0.5, 8, 128)
    else:
        cache = (torch.randn(500, 1, 9, 16, 64, device=_dev()) * 0.5).bfloat16()
        bt = torch.arange(500, dtype=torch.int32, device=_dev()).view(4, 125)
        q = (torch.randn(64, 16, 576, device=_dev()) * 0.3).bfloat16()       # shares of 14 tiles: copies are waited for
        pos, seq = torch.full((64,), 1999, dtype=torch.int32, device=_dev()), torch.arange(64, device=_dev()).int() % 4
        call = lambda: sm100.mla_attention(q, cache, bt, seq, pos, 192 ** -0.5)
        want = _mla_ref(q, cache, bt, seq, pos, 192 ** -0.5)
    assert _rel_err(call(), want) < 5e-2 and sm100.waits_given_up() == 0
    done = StepResult(tokens=torch.zeros(1, dtype=torch.int32), num_emit=1)
    try:
        lib.watch_waits(limit_ns=0)
        t0 = time.monotonic()
        call()
        torch.cuda.synchronize()
        assert time.monotonic() - t0 < 0.5                   # nothing waits for what was never issued (two seconds)
        with pytest.raises(RuntimeError, match="bounded wait"):
            done.tokens_list()
    finally:
        lib.watch_waits()
        lib.waits_gave_up(clear=True)
    assert _rel_err(call(), want) < 5e-2 and sm100.waits_given_up() == 0
    assert done.tokens_list() == [0]


@pytest.mark.parametrize("m,n,k", [(600, 6144, 64), (600, 6144, 1024), (4200, 4104, 4096)])
def test_gemm_on_pairs_that_gives_up_ends_soon(m, n, k):
    """Limits of nothing, 1 ns and 2 us: the two CTAs of a pair give up at different stages, and still no copy is waited for that was
    never issued (two seconds each). The sums of 64 K blocks are waited for longer than that."""
    from gllm_b200.ops import lib, sm100
    torch.manual_seed(k)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), torch.randn(n, k, device=_dev()).bfloat16()
    want = sm100.linear(x, w)
    torch.cuda.synchronize()
    try:
        for limit in (0, 1, 2000):
            lib.watch_waits(limit_ns=limit)
            for _ in range(5):
                t0 = time.monotonic()
                sm100.linear(x, w)
                torch.cuda.synchronize()
                assert time.monotonic() - t0 < 0.5, limit
            assert lib.waits_gave_up(clear=True) or (limit == 2000 and k < 4096), limit
    finally:
        lib.watch_waits()
        lib.waits_gave_up(clear=True)
    assert torch.equal(sm100.linear(x, w), want)


def test_wait_limit_does_not_count_the_kernel_before():
    """A GEMM on pairs of SMs starts while ten CTAs of the kernel before it still have a long product to sum up: what it waits for
    there is not a wait of its own. A wait ends within a suspension (as long as the limit here) of its limit, so the kernel before has to
    take longer than twice the limit."""
    from gllm_b200.ops import lib, sm100
    torch.manual_seed(1)
    x0, w0 = torch.randn(600, 1 << 17, device=_dev()).bfloat16(), torch.randn(256, 1 << 17, device=_dev()).bfloat16()
    x, w = torch.randn(600, 1024, device=_dev()).bfloat16(), torch.randn(6144, 1024, device=_dev()).bfloat16()
    want = x.float() @ w.float().t()
    sm100.linear(x0, w0), sm100.linear(x, w)
    assert sm100.waits_given_up() == 0
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    start.record(), sm100.linear(x0, w0), end.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(end) > 0.3
    try:
        lib.watch_waits(limit_ns=100_000)
        for _ in range(3):
            sm100.linear(x0, w0)
            got = sm100.linear(x, w)
        torch.cuda.synchronize()
        assert not lib.waits_gave_up()
    finally:
        lib.watch_waits()
        lib.waits_gave_up(clear=True)
    assert _rel_err(got, want) < 5e-2


def test_sampler_greedy_and_filter():
    from gllm_b200.ops import sm100
    torch.manual_seed(6)
    b, v = 33, 151936
    logits = (torch.randn(b, v, device=_dev()) * 3).bfloat16()
    tok = sm100.sample(logits)
    assert torch.equal(tok.long(), logits.float().argmax(-1))
    # temperature/top-k/top-p: every drawn token must lie in the oracle's support. fp32 logits so
    # that ties (which the kernel keeps, the sort-based oracle breaks arbitrarily) are improbable;
    # the oracle gets a hair more top-p mass to absorb x*(1/T) vs x/T rounding at the boundary.
    logits = torch.randn(b, v, device=_dev()) * 3
    temp = torch.full((b,), 0.8, device=_dev())
    tk = torch.full((b,), 50, device=_dev(), dtype=torch.int32)
    tp = torch.full((b,), 0.9, device=_dev())
    probs = ref.sample_filter(logits, temp, tk + 1, tp + 1e-3)
    for s in range(3):
        tok = sm100.sample(logits, temp, tk, tp, seed=123 + s)
        p_tok = probs.gather(1, tok.long().view(-1, 1))
        assert (p_tok > 0).all()
    # top-p only (no top-k) and top-k only
    tok = sm100.sample(logits, temp, torch.full((b,), -1, device=_dev(), dtype=torch.int32), tp, seed=5)
    probs = ref.sample_filter(logits, temp, None, tp + 1e-3)
    assert (probs.gather(1, tok.long().view(-1, 1)) > 0).all()
    tok = sm100.sample(logits, temp, tk, None, seed=6)
    probs = ref.sample_filter(logits, temp, tk + 1, None)
    assert (probs.gather(1, tok.long().view(-1, 1)) > 0).all()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("v", [1, 7, 8, 9, 8 * 1024 * 4 + 5, 50001])
def test_sampler_greedy_edges(v, dt):
    """The first largest element whatever the row's length and alignment: whole 16-byte chunks, remainders, unaligned rows, ties
    inside a chunk and across threads, a penalty on the winner."""
    from gllm_b200.ops import sm100
    torch.manual_seed(v)
    base = torch.randn(3, v + 3, device=_dev()).to(dt)
    for off in (0, 1, 3):
        z = base[:, off:off + v]
        z[1, :] = z[1].clamp(max=z[1].float().median().item())         # many ties at the top
        assert sm100.sample(z).tolist() == [int((r == r.max()).nonzero()[0, 0]) for r in z]
    seen = torch.full((3, (v + 31) // 32), -1, dtype=torch.int32, device=_dev())
    pen = torch.full((3,), 1.5, device=_dev())
    want = torch.where(z.float() > 0, z.float() / 1.5, z.float() * 1.5)
    assert sm100.sample(z, rep_penalty=pen, seen_bits=seen).tolist() == [int((r == r.max()).nonzero()[0, 0]) for r in want]


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("b,v", [(1, 24575), (1, 24576), (3, 49159), (13, 50001), (14, 50000), (32, 49152), (33, 49156), (69, 49152), (70, 49151), (2, 131072),
                                 (2, 131073)])
def test_sampler_rows_shared_by_a_cluster(b, v, dt):
    """Rows whose argmax pass eight, four, two CTAs or one share: ties within and across their parts, an unaligned row, rows that draw
    beside greedy ones (up to 256 KB by one CTA), whose tokens do not depend on how many CTAs share the row."""
    from gllm_b200.ops import sm100
    torch.manual_seed(b + v)
    base = torch.randn(b, v + 3, device=_dev()).to(dt)
    for off in (0, 3):
        z = base[:, off:off + v]
        z[0] = z[0].clamp(max=z[0].float().quantile(0.999).item())             # some ties, in all parts
        z[b - 1, v - 1] = 9.0                                                  # the row's end
        top = torch.empty(b, device=_dev())
        want = [int((r == r.max()).nonzero()[0, 0]) for r in z]
        assert sm100.sample(z, out_max=top).tolist() == want
        assert torch.equal(top, z.float().amax(-1))
    k = torch.tensor([1 if i % 2 else 40 for i in range(b)], dtype=torch.int32, device=_dev())
    temp, p = torch.full((b,), 0.7, device=_dev()), torch.full((b,), 0.9, device=_dev())
    got = sm100.sample(z, temp, k, p, seed=11).tolist()
    many = torch.cat([z, z.new_zeros(150, v)])                                 # one CTA to a row
    pad = lambda t, fill: torch.cat([t, torch.full((150,), fill, dtype=t.dtype, device=_dev())])
    assert sm100.sample(many, pad(temp, 1.0), pad(k, 1), pad(p, 1.0), seed=11).tolist()[:b] == got
    assert all(got[i] == want[i] for i in range(1, b, 2))


def test_sampler_distribution():
    from gllm_b200.ops import sm100
    torch.manual_seed(7)
    v = 64
    row = torch.randn(v, device=_dev()) * 2
    n = 20000
    logits = row.unsqueeze(0).repeat(n, 1).contiguous()
    temp = torch.full((n,), 1.3, device=_dev())
    tk = torch.full((n,), 20, device=_dev(), dtype=torch.int32)
    tp = torch.full((n,), 0.85, device=_dev())
    probs = ref.sample_filter(logits[:1], temp[:1], tk[:1], tp[:1])[0]
    tok = sm100.sample(logits, temp, tk, tp, seed=99)
    emp = torch.bincount(tok.long(), minlength=v).float() / n
    assert (emp[probs == 0] == 0).all()
    assert (emp - probs).abs().max().item() < 0.02


@pytest.mark.parametrize("t", [1, 64, 300])
@pytest.mark.parametrize("b,n,k", [(16, 512, 128), (16, 128, 512), (3, 256, 192)])
def test_gemm_batched_strided_views(t, b, n, k):
    """Batched mode of the tcgen05 GEMM (MLA weight absorption, K13): strided [T, B, K] operand through a 3-D TMA
    map, result written into a strided [T, B, N] view, vs an fp32 einsum."""
    from gllm_b200.ops import sm100
    torch.manual_seed(t + n)
    dev = _dev()
    a_full = (torch.randn(t, b, k + 64, device=dev) * 0.5).bfloat16()     # the operand is a column slice
    w = (torch.randn(b, n, k, device=dev) * 0.1).bfloat16()
    out_full = torch.full((t, b, n + 64), 7.0, device=dev, dtype=torch.bfloat16)
    a, out = a_full[:, :, :k], out_full[:, :, :n]
    sm100.gemm_batched(a, w, out)
    torch.cuda.synchronize()
    ref_o = torch.einsum("tbk,bnk->tbn", a.float(), w.float())
    assert _rel_err(out, ref_o) < 1e-2, _rel_err(out, ref_o)
    assert bool((out_full[:, :, n:] == 7.0).all())                         # nothing written outside the view


@pytest.mark.parametrize("tp", [2, 8])
def test_vocab_parallel_sampling_equals_the_full_vocab_kernel(tp):
    """vp_candidates_kernel on each vocab shard + vp_final_kernel on the gathered records draw the
    SAME token as sample_kernel on the full [B, V] row (the race's random numbers are keyed by token id) for greedy,
    top-k, top-k + top-p, nucleus-only, penalised and unfiltered rows — without ever holding the full logits."""
    from gllm_b200.ops import sm100
    torch.manual_seed(11)
    dev = _dev()
    v_full = 151936
    per = (v_full + tp - 1) // tp
    per = (per + 127) // 128 * 128                     # shards are padded: the last one ends with dead columns
    b = 24
    logits = torch.randn(b, tp * per, device=dev) * 3
    logits[:, v_full:] = 50.0                          # padding columns must never win
    base = torch.tensor([1, 20, 50, 200, 0, 0], dtype=torch.int32)
    top_k = base.repeat(b // 6).to(dev)
    top_k = torch.where(top_k <= 0, torch.full_like(top_k, v_full), top_k)
    top_p = torch.tensor([1.0, 0.9, 1.0, 0.8, 0.3, 1.0]).repeat(b // 6).to(dev)
    temp = torch.tensor([0.0, 0.7, 1.0, 1.2, 0.6, 1.0]).repeat(b // 6).to(dev)
    pen = torch.tensor([1.0, 1.3, 1.0, 1.1, 1.0, 1.2]).repeat(b // 6).to(dev)
    seen = torch.randint(-2 ** 31, 2 ** 31 - 1, (b, (tp * per + 31) // 32), dtype=torch.int64, device=dev).to(torch.int32)
    slots = torch.arange(b, dtype=torch.int32, device=dev)
    step = torch.tensor([5], dtype=torch.int64, device=dev)
    full = sm100.sample(logits[:, :v_full].contiguous(), temp, top_k, top_p, pen, seen, slots, seed=77, step=step)
    c = 256
    recs = []
    for r in range(tp):
        lo = r * per
        valid = max(0, min(per, v_full - lo))
        recs.append(sm100.vp_candidates(logits[:, lo:lo + per], valid, v_full, c, temp, top_k, top_p, pen, seen, slots,
                                        seed=77, step=step, vocab_offset=lo))
    toks = sm100.vp_final(torch.stack(recs).contiguous(), c, v_full, top_k, top_p, seed=77, step=step)
    torch.cuda.synchronize()
    assert int(toks.max()) < v_full
    assert torch.equal(toks, full), (toks.tolist(), full.tolist())
    # record hygiene: every shard returns its true top candidates and softmax statistics
    x = ref.apply_penalty_temperature(logits[:, :per], temp, None, None)
    rec0 = recs[0]
    row = 2                                            # top_k 50, no penalty on this row
    got = torch.sort(rec0[row, :50], descending=True).values
    want = torch.topk(logits[row, :per] / temp[row].clamp_min(1e-5), 50).values
    assert torch.allclose(got, want, rtol=1e-5, atol=1e-5)


def test_sampler_rep_penalty():
    from gllm_b200.ops import sm100
    torch.manual_seed(8)
    b, v = 4, 1000
    logits = torch.randn(b, v, device=_dev())
    seen = torch.zeros(b, (v + 31) // 32, dtype=torch.int32, device=_dev())
    top = logits.argmax(-1).to(torch.int32)
    rows = torch.arange(b, device=_dev(), dtype=torch.int32)
    sm100.mark_seen(seen, rows, top)
    pen = torch.full((b,), 50.0, device=_dev())
    tok = sm100.sample(logits, rep_penalty=pen, seen_bits=seen)
    mask = torch.zeros(b, v, dtype=torch.bool, device=_dev())
    mask[rows.long(), top.long()] = True
    exp = ref.sample(logits, rep_penalty=pen, seen_mask=mask)
    assert torch.equal(tok, exp)


@pytest.mark.parametrize("m", [1, 16, 17, 64, 100, 255, 256])
@pytest.mark.parametrize("n,k", [(4096, 4096), (6144, 4096), (4096, 12288), (1000, 512), (152064, 1024)])
@pytest.mark.parametrize("split", [0, 1, 3])
def test_gemm_smallm(m, n, k, split, monkeypatch):
    """swap-AB split-K decode GEMM (bias, forced splits, ragged N)."""
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "_FORCE_SPLIT", split)
    monkeypatch.setattr(sm100, "_SMALLM_MAX", 256)
    torch.manual_seed(m + n)
    x = (torch.randn(m, k, device=_dev()) * 0.5).bfloat16()
    w = (torch.randn(n, k, device=_dev()) * 0.05).bfloat16()
    b = torch.randn(n, device=_dev()).bfloat16()
    for bias in (None, b):
        y = sm100.linear(x, w, bias)
        yr = x.float() @ w.float().t() + (bias.float() if bias is not None else 0)
        assert _rel_err(y, yr) < 6e-3, _rel_err(y, yr)
    # back-to-back launches reuse the workspace/counters
    y2 = sm100.linear(x, w, None)
    assert torch.equal(y2, sm100.linear(x, w, None))


@pytest.mark.parametrize("m", [3, 64, 200])
@pytest.mark.parametrize("split", [0, 1, 2])
def test_gemm_smallm_silu(m, split, monkeypatch):
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "_FORCE_SPLIT", split)
    monkeypatch.setattr(sm100, "_SMALLM_MAX", 256)
    torch.manual_seed(m)
    i, k = 1536, 1024
    x = (torch.randn(m, k, device=_dev()) * 0.5).bfloat16()
    w = (torch.randn(2 * i, k, device=_dev()) * 0.05).bfloat16()
    y = sm100.linear_silu_mul(x, ref.interleave_gate_up(w, 128))
    h = x.float() @ w.float().t()
    yr = torch.nn.functional.silu(h[:, :i]) * h[:, i:]
    assert _rel_err(y, yr) < 1e-2


@pytest.mark.parametrize("e,k,renorm", [(8, 2, True), (60, 4, False), (128, 8, True), (256, 8, True)])
def test_moe_topk_softmax(e, k, renorm):
    from gllm_b200.ops import sm100_moe
    torch.manual_seed(e)
    logits = torch.randn(77, e, device=_dev()).bfloat16()
    w, ids = sm100_moe.topk_softmax(logits, k, renorm)
    w_r, ids_r = ref.topk_softmax(logits, k, renorm)
    # compare as sets per row (tie order may differ), weights by id
    dense = torch.zeros(77, e, device=_dev()).scatter(1, ids.long(), w)
    dense_r = torch.zeros(77, e, device=_dev()).scatter(1, ids_r.long(), w_r)
    assert torch.allclose(dense, dense_r, atol=2e-3, rtol=1e-2)


@pytest.mark.parametrize("scoring,bias", [("sigmoid", True), ("softmax", False)])
def test_moe_grouped_topk(scoring, bias):
    from gllm_b200.ops import sm100_moe
    torch.manual_seed(11)
    t, e, k, g, tg = 93, 256, 8, 8, 4
    logits = torch.randn(t, e, device=_dev()).bfloat16()
    b = (torch.randn(e, device=_dev()) * 0.1).float() if bias else None
    w, ids = sm100_moe.grouped_topk(logits, k, True, g, tg, scoring, b, 2.5)
    w_r, ids_r = ref.grouped_topk(logits, k, True, g, tg, scoring, b, 2.5)
    dense = torch.zeros(t, e, device=_dev()).scatter(1, ids.long(), w)
    dense_r = torch.zeros(t, e, device=_dev()).scatter(1, ids_r.long(), w_r)
    assert torch.allclose(dense, dense_r, atol=5e-3, rtol=2e-2)


@pytest.mark.parametrize("t,e,k,h,i,ep", [(5, 8, 2, 256, 512, False), (300, 8, 2, 512, 1024, False),
                                          (200, 16, 4, 256, 256, True), (1000, 64, 6, 256, 128, False)])
def test_moe_fused_experts(t, e, k, h, i, ep):
    from gllm_b200.ops import sm100_moe
    torch.manual_seed(t + e)
    x = (torch.randn(t, h, device=_dev()) * 0.5).bfloat16()
    e_local = e // 2 if ep else e
    w13 = (torch.randn(e_local, 2 * i, h, device=_dev()) * 0.05).bfloat16()
    w2 = (torch.randn(e_local, h, i, device=_dev()) * 0.05).bfloat16()
    logits = torch.randn(t, e, device=_dev()).bfloat16()
    w, ids = ref.topk_softmax(logits, k, True)
    emap = None
    if ep:
        emap = torch.full((e,), -1, dtype=torch.int32, device=_dev())
        emap[e // 2:] = torch.arange(e_local, dtype=torch.int32, device=_dev())
    w13_il = torch.stack([ref.interleave_gate_up(w13[j], 64) for j in range(e_local)])
    y = sm100_moe.fused_experts(x, w13_il, w2, w, ids, emap)
    y_ref = ref.fused_experts(x, w13, w2, w, ids, emap)
    assert torch.isfinite(y.float()).all()
    assert _rel_err(y, y_ref) < 2e-2, _rel_err(y, y_ref)


@pytest.mark.parametrize("counts", [(1, 15, 16, 17), (63, 0, 64, 65), (127, 128, 129, 300)])
def test_moe_expert_tiles_partly_filled(counts):
    """Only the rows that an expert has are loaded and stored: counts at the edges of the 16-row boxes and of the 128-row tiles,
    with a workspace full of NaN around them. Two bf16 roundings (the gated product, the result) of products of bf16 factors."""
    from gllm_b200.ops import sm100_moe
    torch.manual_seed(sum(counts))
    e, h, i, t = len(counts), 192, 256, sum(counts)
    x = torch.randn(t, h, device=_dev()).bfloat16()
    w13 = (torch.randn(e, 2 * i, h, device=_dev()) * h ** -0.5).bfloat16()
    w2 = (torch.randn(e, h, i, device=_dev()) * i ** -0.5).bfloat16()
    ids = torch.repeat_interleave(torch.arange(e), torch.tensor(counts))[torch.randperm(t)].to(torch.int32).to(_dev())[:, None]
    w13_il = torch.stack([ref.interleave_gate_up(w13[j], 64) for j in range(e)])
    one = torch.ones(t, 1, device=_dev())
    sm100_moe.fused_experts(x, w13_il, w2, one, ids)
    for b in sm100_moe._ws.values():
        if b.dtype == torch.bfloat16:
            b.fill_(float("nan"))
    y = sm100_moe.fused_experts(x, w13_il, w2, one, ids)
    g, u = torch.einsum("th,tnh->tn", x.float(), w13.float()[ids[:, 0].long()]).chunk(2, -1)
    want = torch.einsum("ti,thi->th", torch.nn.functional.silu(g) * u, w2.float()[ids[:, 0].long()])
    assert _rel_err(y, want) < 6e-3, _rel_err(y, want)


@pytest.mark.parametrize("m,k", [(7, 1152), (8 * 65535 + 9, 128)])       # the second: more row groups than a grid's y axis has
def test_fp8_quantiser_rows(m, k):
    """Scales amax / 448 (an approximate division, 2 ulp) and e4m3 values of rows before and past 524,280."""
    from gllm_b200.ops import sm100
    torch.manual_seed(k)
    x = torch.randn(m, k, device=_dev()).bfloat16()
    q, s = sm100.fp8_quant_group(x)
    amax = x.float().view(m, k // 128, 128).abs().amax(-1)
    assert torch.allclose(s.t(), amax / 448, rtol=2.0 ** -21, atol=0)
    back = q.float().view(m, k // 128, 128) * s.t()[..., None]
    # e4m3 keeps 3 bits behind the leading one (2^-4), and steps of 2^-9 below 2^-6
    err = (back - x.float().view(m, k // 128, 128)).abs()
    assert bool((err <= x.float().view(m, k // 128, 128).abs() * 2.0 ** -4 * 1.001 + s.t()[..., None] * 2.0 ** -10 * 1.001).all())


@pytest.mark.parametrize("m,n,k", [(1, 256, 128), (77, 1536, 512), (300, 4096, 7168), (1024, 2048, 2048),
                                   (64, 576, 7168),       # 576 = kv_a_proj_with_mqa (MLA): N not a multiple of 128
                                   (129, 8200, 640), (3000, 1032, 384), (2500, 4352, 1152)])   # tiles of 64, 128, 256
def test_gemm_fp8_block(m, n, k):
    from gllm_b200.ops import sm100
    torch.manual_seed(m)
    x = (torch.randn(m, k, device=_dev()) * 0.7).bfloat16()
    w = torch.randn(n, k, device=_dev()) * 0.05
    # block-quantise the weight like an HF fp8 checkpoint: per 128x128 block scale_inv = amax / 448
    nb, kb = (n + 127) // 128, k // 128
    wp = torch.zeros(nb * 128, k, device=_dev())
    wp[:n] = w
    blocks = wp.view(nb, 128, kb, 128)
    s_inv = (blocks.abs().amax(dim=(1, 3)) / 448.0).clamp_min(1e-8)
    w8 = (blocks / s_inv.view(nb, 1, kb, 1)).view(nb * 128, k)[:n].to(torch.float8_e4m3fn).contiguous()
    b = torch.randn(n, device=_dev()).bfloat16()
    y = sm100.linear_fp8_block(x, w8, s_inv.contiguous(), b)
    y_ref = ref.linear_fp8_block(x, w8, s_inv, b)
    assert _rel_err(y, y_ref) < 1e-2, _rel_err(y, y_ref)
    assert sm100.waits_given_up() == 0
    if n % 256 == 0:      # [gate ; up] weight with the gated epilogue: the activation leaves the fp32 sums, no bf16 between
        y = sm100.linear_fp8_block(x, w8, s_inv.contiguous(), silu=True)
        xq, xs = ref.fp8_quant_group(x)
        wide = w8.float() * s_inv.repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)
        g, u = ((xq.float() * xs.repeat_interleave(128, 1)) @ wide.t()).chunk(2, -1)
        assert _rel_err(y, torch.nn.functional.silu(g) * u) < 1e-2
    # and the quantiser alone
    q, s = sm100.fp8_quant_group(x)
    q_r, s_r = ref.fp8_quant_group(x)
    assert torch.allclose(s.t(), s_r, rtol=1e-5)
    assert _rel_err(q.float(), q_r.float()) < 3e-2


@contextlib.contextmanager
def _forced_split(parts):
    """A forced K split of the tiles on single SMs, which products of these sizes would otherwise leave to clusters (0: nothing forced)."""
    from gllm_b200.ops import lib
    lib.load().gllm_gemm_tune(parts, 512)
    try:
        yield
    finally:
        lib.load().gllm_gemm_tune(0, 512)


@pytest.mark.parametrize("split", [0, 2, 4])
@pytest.mark.parametrize("m", [64, 128, 200, 256, 384, 512])
@pytest.mark.parametrize("n,k", [(4096, 4096), (4096, 12288), (6144, 4096), (1000, 1536)])
def test_gemm_splitk_decode_shapes(m, n, k, split):
    """Decode-sized M as the dispatch has it (mostly clusters), and on the wide-tile split-K path (fp32 partials, last-arriver sum): exact
    shape sweep, bias, and back-to-back launches (tile counters re-arm themselves)."""
    from gllm_b200.ops import sm100
    torch.manual_seed(m + n + k)
    x = (torch.randn(m, k, device=_dev()) * 0.5).bfloat16()
    w = (torch.randn(n, k, device=_dev()) * 0.05).bfloat16()
    b = torch.randn(n, device=_dev()).bfloat16()
    with _forced_split(split):
        for bias in (None, b):
            y = sm100.linear(x, w, bias)
            yr = x.float() @ w.float().t() + (bias.float() if bias is not None else 0)
            assert _rel_err(y, yr) < 6e-3, _rel_err(y, yr)
        y2 = sm100.linear(x, w, None)
        for _ in range(3):
            assert torch.equal(y2, sm100.linear(x, w, None))   # deterministic slice-ordered reduction


@pytest.mark.parametrize("m", [64, 256, 384])
def test_gemm_splitk_silu(m):
    from gllm_b200.ops import sm100
    torch.manual_seed(m)
    i, k = 12288, 4096
    x = (torch.randn(m, k, device=_dev()) * 0.5).bfloat16()
    w = (torch.randn(2 * i, k, device=_dev()) * 0.02).bfloat16()
    y = sm100.linear_silu_mul(x, ref.interleave_gate_up(w, 128))
    h = x.float() @ w.float().t()
    yr = torch.nn.functional.silu(h[:, :i]) * h[:, i:]
    assert _rel_err(y, yr) < 1e-2


def _mla_ref(q_full, cache, bt, tok_seq, positions, scale):
    t, h, _ = q_full.shape
    out = torch.zeros(t, h, 512, dtype=torch.float32, device=q_full.device)
    for i in range(t):
        s = int(tok_seq[i]) if tok_seq is not None else i
        n = int(positions[i]) + 1
        lat = ref.gather_kv(cache, bt[s], n)[:, 0].float()          # [n, 576]
        att = torch.softmax((q_full[i].float() @ lat.t()) * scale, dim=-1)
        out[i] = att @ lat[:, :512]
    return out


@pytest.mark.parametrize("heads", [16, 8, 40])
@pytest.mark.parametrize("splits", [1, 3, None])
def test_mla_attention_decode(heads, splits):
    from gllm_b200.ops import sm100
    torch.manual_seed(7)
    page, b = 16, 5
    lens = [1, 63, 64, 300, 777]
    max_blocks = max((n + page - 1) // page for n in lens) + 1
    n_pages = sum((n + page - 1) // page for n in lens) + 2
    cache = (torch.randn(n_pages, 1, 9, page, 64, device=_dev()) * 0.5).bfloat16()
    perm = torch.randperm(n_pages)[: n_pages - 1].tolist()
    bt = torch.zeros(b, max_blocks, dtype=torch.int32)
    c = 0
    for i, n in enumerate(lens):
        k = (n + page - 1) // page
        bt[i, :k] = torch.tensor(perm[c:c + k], dtype=torch.int32)
        c += k
    bt = bt.to(_dev())
    q = (torch.randn(b, heads, 576, device=_dev()) * 0.3).bfloat16()
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=_dev())
    scale = 192 ** -0.5
    out = sm100.mla_attention(q, cache, bt, None, pos, scale, splits=splits)
    want = _mla_ref(q, cache, bt, None, pos, scale)
    assert _rel_err(out, want) < 1.5e-2, _rel_err(out, want)


@pytest.mark.parametrize("heads", [16, 40])
@pytest.mark.parametrize("tokens,longest", [(1, 5000), (3, 700), (149, 130), (300, 64)])
@pytest.mark.parametrize("page", [8, 64])
def test_mla_attention_shares(heads, tokens, longest, page):
    """Key tiles cut into one share per SM: shares with many tokens, tokens over many shares, more tokens than threads, lengths at
    the edges of a 64-key tile; a window and a sink in the first part. Probabilities are rounded once to bf16."""
    from gllm_b200.ops import sm100
    torch.manual_seed(tokens + page)
    lens = [longest] + [(1, 63, 64, 65, 128)[i % 5] for i in range(tokens - 1)]
    need = [-(-n // page) for n in lens]
    perm = torch.randperm(sum(need), device=_dev()).to(torch.int32)
    bt, at = torch.zeros(tokens, max(need), dtype=torch.int32, device=_dev()), 0
    for i, k in enumerate(need):
        bt[i, :k] = perm[at:at + k]
        at += k
    cache = (torch.randn(sum(need), 1, 9, page, 64, device=_dev()) * 0.5).bfloat16()
    q = (torch.randn(tokens, heads, 576, device=_dev()) * 0.3).bfloat16()
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=_dev())
    sink = torch.randn(heads, device=_dev())
    out = sm100.mla_attention(q, cache, bt, None, pos, 192 ** -0.5)
    win = sm100.mla_attention(q, cache, bt, None, pos, 192 ** -0.5, window=100, sink=sink)
    assert sm100.waits_given_up() == 0
    assert _rel_err(out, _mla_ref(q, cache, bt, None, pos, 192 ** -0.5)) < 1.5e-2
    for i, n in enumerate(lens):
        lat = ref.gather_kv(cache, bt[i], n)[-100:, 0].float()
        att = torch.softmax(torch.cat([q[i].float() @ lat.t() * 192 ** -0.5, sink[:, None]], -1), -1)[:, :-1]
        assert _rel_err(win[i], att @ lat[:, :512]) < 1.5e-2, i


def test_mla_attention_prefill_tokens_and_rope_cache():
    """Mixed batch: every token attends to its own causal prefix (tok_seq / positions); plus the fused
    rope + latent-cache write against the PyTorch oracle ops."""
    from gllm_b200.ops import sm100
    torch.manual_seed(8)
    page, heads = 16, 16
    q_lens, ctx = [40, 1, 70], [0, 130, 25]          # new tokens / already cached tokens per sequence
    b = len(q_lens)
    tot = [q + c for q, c in zip(q_lens, ctx)]
    max_blocks = max((n + page - 1) // page for n in tot) + 1
    n_pages = sum((n + page - 1) // page for n in tot) + 1
    cache = (torch.randn(n_pages, 1, 9, page, 64, device=_dev()) * 0.5).bfloat16()
    bt = torch.zeros(b, max_blocks, dtype=torch.int32)
    c = 0
    for i, n in enumerate(tot):
        k = (n + page - 1) // page
        bt[i, :k] = torch.arange(c, c + k, dtype=torch.int32)
        c += k
    tok_seq = torch.tensor(sum(([i] * q for i, q in enumerate(q_lens)), []), dtype=torch.int32)
    pos = torch.tensor(sum((list(range(cx, cx + q)) for q, cx in zip(q_lens, ctx)), []), dtype=torch.int32)
    t = int(tok_seq.numel())
    slots = torch.tensor([int(bt[s, p // page]) * page + p % page for s, p in zip(tok_seq.tolist(), pos.tolist())],
                         dtype=torch.int32)
    bt, tok_seq, pos, slots = bt.to(_dev()), tok_seq.to(_dev()), pos.to(_dev()), slots.to(_dev())
    # ---- rope + cache write ----
    qk_dim, nope = 192, 128
    qp = (torch.randn(t, heads, qk_dim, device=_dev()) * 0.5).bfloat16()
    kv_a = (torch.randn(t, 576, device=_dev()) * 0.5).bfloat16()
    kv_c = kv_a[:, :512].contiguous()
    cs = ref.build_cos_sin_cache(64, 512, 10000.0).to(_dev())
    q_full = torch.zeros(t, heads, 576, dtype=torch.bfloat16, device=_dev())
    cache2 = cache.clone()
    sm100.mla_rope_cache(qp[:, :, nope:], q_full, kv_a[:, 512:], kv_c, cs, pos, slots, cache2)
    q_pe = qp[:, :, nope:].contiguous()
    k_pe = kv_a[:, 512:].contiguous().view(t, 1, 64)
    ref.rope_kv_write(q_pe, k_pe, None, pos, cs, 64, False, None, None, 1e-6, None, None, None)
    cache_ref = cache.clone()
    ref.write_kv_cache(torch.cat([kv_c, k_pe.view(t, 64)], -1).view(t, 1, 576), None, cache_ref, None, slots)
    assert _rel_err(q_full[:, :, 512:], q_pe) < 8e-3
    assert _rel_err(cache2, cache_ref) < 8e-3
    # ---- attention over the freshly written cache ----
    q_full[:, :, :512] = (torch.randn(t, heads, 512, device=_dev()) * 0.3).bfloat16()
    scale = 192 ** -0.5
    out = sm100.mla_attention(q_full, cache2, bt, tok_seq, pos, scale)
    want = _mla_ref(q_full, cache2, bt, tok_seq, pos, scale)
    assert _rel_err(out, want) < 1.5e-2, _rel_err(out, want)


@pytest.mark.parametrize("t,e,k", [(77, 4, 2), (300, 8, 2), (5, 8, 4)])
def test_moe_fused_experts_fp8(t, e, k):
    """Grouped block-scaled fp8 expert GEMMs (SiLU-gate epilogue on interleaved tiles with per-64-row scales)
    against the de-quantised bf16 oracle."""
    from gllm_b200.layers.moe import _block_quant_rows64
    from gllm_b200.ops import sm100_moe
    torch.manual_seed(t + e)
    h, inter = 512, 256
    x = (torch.randn(t, h, device=_dev()) * 0.5).bfloat16()
    w13 = (torch.randn(e, 2 * inter, h, device=_dev()) * 0.05).bfloat16()
    w2 = (torch.randn(e, h, inter, device=_dev()) * 0.05).bfloat16()
    logits = torch.randn(t, e, device=_dev()).bfloat16()
    tw, ids = sm100_moe.topk_softmax(logits, k, True)
    q13, s13, q2, s2, d13, d2 = [], [], [], [], [], []
    for i in range(e):
        a, sa = _block_quant_rows64(w13[i])
        b, sb = _block_quant_rows64(w2[i])
        d13.append((a.float() * sa.repeat_interleave(64, 0).repeat_interleave(128, 1)).bfloat16())
        d2.append((b.float() * sb.repeat_interleave(64, 0).repeat_interleave(128, 1)).bfloat16())
        q13.append(ref.interleave_gate_up(a.view(torch.uint8), 64).view(torch.float8_e4m3fn))
        s13.append(ref.interleave_gate_up(sa, 1))
        q2.append(b)
        s2.append(sb)
    out = sm100_moe.fused_experts_fp8(x, torch.stack(q13), torch.stack(s13).contiguous(), torch.stack(q2),
                                      torch.stack(s2).contiguous(), tw, ids)
    def qdq(a):   # dynamic per-token-group(128) activation quantisation, as the kernel path does
        q, sc = ref.fp8_quant_group(a, 128)
        return (q.float().reshape(a.shape[0], -1, 128) * sc.unsqueeze(-1)).reshape(a.shape).to(a.dtype)

    want = torch.zeros(t, h, dtype=torch.float32, device=_dev())
    for i in range(e):
        tok, slot = torch.where(ids.long() == i)
        if tok.numel() == 0:
            continue
        hd = ref.silu_and_mul(torch.nn.functional.linear(qdq(x[tok]), d13[i]))
        ye = torch.nn.functional.linear(qdq(hd), d2[i]).float()
        want.index_add_(0, tok, ye * tw[tok, slot].float().unsqueeze(-1))
    # (bf16 rounding of the intermediate moves some values across e4m3 rounding boundaries: ~1.8 % measured)
    assert _rel_err(out, want) < 2.5e-2, _rel_err(out, want)
    # and within quantisation noise of the un-quantised-activation oracle
    assert _rel_err(out, ref.fused_experts(x, torch.stack(d13), torch.stack(d2), tw, ids)) < 8e-2


@pytest.mark.parametrize("heads,page", [(3, 16), (16, 64), (8, 8)])
@pytest.mark.parametrize("n_dec", [0, 2])
def test_mla_expanded_attention(heads, page, n_dec):
    """Expanded heads (128 key columns of their own + 64 shared, values 128 wide) over gathered latents: chunks and contexts at
    the edges of the 64-row gather tiles, 64-key and 128-query tiles; decoding sequences in front are left alone. Against fp32
    over the same bf16 latents and weights; keys and values are rounded once to bf16 (2^-9), like P."""
    from gllm_b200.ops import sm100
    torch.manual_seed(9)
    q_lens, ctx = [1] * n_dec + [1, 63, 64, 65, 128, 129, 40, 300], [7, 90][:n_dec] + [0, 1, 64, 0, 127, 0, 500, 3]
    lens = [a + b for a, b in zip(q_lens, ctx)]
    need = [-(-n // page) for n in lens]
    perm = torch.randperm(sum(need), device=_dev()).to(torch.int32)
    bt, at = torch.zeros(len(lens), max(need), dtype=torch.int32, device=_dev()), 0
    for i, k in enumerate(need):
        bt[i, :k] = perm[at:at + k]
        at += k
    cache = torch.randn(sum(need), 1, 9, page, 64, device=_dev()).bfloat16()
    w = (torch.randn(heads * 256, 512, device=_dev()) * 512 ** -0.5).bfloat16()
    t = sum(q_lens)
    q = torch.randn(t, heads, 192, device=_dev()).bfloat16()
    qsl = torch.tensor([0] + q_lens, device=_dev()).cumsum(0).to(torch.int32)
    sl = torch.tensor(lens, dtype=torch.int32, device=_dev())
    rows = sum(-(-n // 64) * 64 for n in lens[n_dec:])
    out = torch.full((t, heads, 128), 7.0, device=_dev()).bfloat16()
    scale = 192 ** -0.5
    sm100.mla_expanded_attention(q, cache, bt, sl, qsl, w, rows, n_dec, max(q_lens), scale, out)
    assert bool((out[:n_dec] == 7.0).all()) and sm100.waits_given_up() == 0
    want = torch.empty(t, heads, 128, device=_dev())
    for i, n in enumerate(lens):
        a, b = int(qsl[i]), int(qsl[i + 1])
        row = ref.gather_kv(cache, bt[i], n)[:, 0].float()
        kv = (row[:, :512] @ w.float().t()).view(n, heads, 256)
        k = torch.cat([kv[..., :128], row[:, None, 512:].expand(n, heads, 64)], -1)
        s = torch.einsum("qhd,khd->hqk", q[a:b].float(), k) * scale
        s.masked_fill_(torch.arange(n, device=_dev())[None] > torch.arange(n - (b - a), n, device=_dev())[:, None], float("-inf"))
        want[a:b] = torch.einsum("hqk,khd->qhd", s.softmax(-1), kv[..., 128:])
    assert _rel_err(out[n_dec:], want[n_dec:]) < 1.2e-2, _rel_err(out[n_dec:], want[n_dec:])


@pytest.mark.parametrize("decodes,q_lens,ctx", [(2, [40, 5, 70, 31], [0, 90, 200, 3]), (0, [31, 33], [65, 1]), (3, [100, 64], [64, 0])])
@pytest.mark.parametrize("kv_rows,latent_rows", [(1 << 20, 1 << 20), (320 * 3, 1 << 20), (1, 256)])    # heads: all, some, one
def test_latent_attention_block_mixed_batches(decodes, q_lens, ctx, kv_rows, latent_rows, monkeypatch):
    """The block on batches of decoding sequences, short and long portions, with limits that make it take rounds of heads and of
    sequences, against the same block that attends everything in the absorbed form; the cache after it bit for bit. Both round
    to bf16 at other places; 5 heads, so that a round is cut short."""
    from types import SimpleNamespace
    from gllm_b200.layers.rotary import build_rope
    from gllm_b200.models.decoder import ModelSpec
    from gllm_b200.models.deepseek_v2 import MLAAttention
    torch.manual_seed(4)
    dev, page, heads, width = _dev(), 16, 5, 256
    spec = ModelSpec(arch="DeepseekV3ForCausalLM", hidden_size=width, num_layers=1, num_heads=heads, num_kv_heads=heads, head_dim=192,
                     intermediate_size=64, vocab_size=64, rms_eps=1e-6, dtype=torch.bfloat16, use_mla=True,
                     extra={"qk_nope_head_dim": 128, "qk_rope_head_dim": 64, "v_head_dim": 128, "kv_lora_rank": 512,
                            "q_lora_rank": 0})
    att = MLAAttention(spec, 0, build_rope(64, 1024, 1e4, None, 64, False, device=dev), dev)
    for p in att.parameters():
        if p.dim() == 2:
            p.data.copy_(torch.randn(p.shape, device=dev) * p.shape[1] ** -0.5)
    att.process_weights()
    q, c = [1] * decodes + q_lens, [50, 1, 129][:decodes] + ctx
    lens = [a + b for a, b in zip(q, c)]
    need = [-(-n // page) for n in lens]
    perm, at = torch.randperm(sum(need)).tolist(), 0
    bt = torch.zeros(len(lens), max(need), dtype=torch.int32)
    for i, k in enumerate(need):
        bt[i, :k] = torch.tensor(perm[at:at + k])
        at += k
    qsl = np.concatenate([[0], np.cumsum(q)]).astype(np.int32)
    pos = torch.cat([torch.arange(a, a + b) for a, b in zip(c, q)]).int()
    seq = torch.repeat_interleave(torch.arange(len(q)), torch.tensor(q)).int()
    slots = torch.stack([bt[s, p // page] * page + p % page for s, p in zip(seq.tolist(), pos.tolist())]).int()
    g = lambda x: torch.as_tensor(x, dtype=torch.int32).to(dev)   # noqa: E731
    inp = SimpleNamespace(num_decode_seqs=decodes, num_seqs=len(q), padded_tokens=0, max_q_len=max(q),
                          batch=SimpleNamespace(query_start_loc=qsl, seq_lens=np.array(lens, np.int32)), positions=g(pos),
                          slot_mapping=g(slots), block_table=g(bt), tok_seq=g(seq), seq_lens=g(lens), query_start_loc=g(qsl))
    tpc = SimpleNamespace(materialize=lambda h: h)
    cache0 = torch.randn(sum(need), 1, 9, page, 64, device=dev).bfloat16()
    h = torch.randn(sum(q), width, device=dev).bfloat16()
    got = []
    for least, pairs in ((32, 0), (32, heads * 2400), (10 ** 6, 0)):
        monkeypatch.setattr(MLAAttention, "_EXPAND_MIN_TOKENS", least)
        monkeypatch.setattr(MLAAttention, "_EXPAND_MIN_PAIRS", pairs)
        monkeypatch.setattr(MLAAttention, "_EXPAND_KV_BYTES", kv_rows * 512)
        monkeypatch.setattr(MLAAttention, "_EXPAND_LATENT_BYTES", latent_rows * 1152)
        cache = cache0.clone()
        got.append((att(inp, h, SimpleNamespace(k_cache=[cache]), tpc), cache))
    for x in got[:2]:
        assert torch.equal(x[1], got[2][1])
        for a, b in zip(q, qsl):
            assert _rel_err(x[0][b:b + a], got[2][0][b:b + a]) < 1.2e-2


@pytest.mark.parametrize("m,n,k,act", [(3, 128, 64, None), (17, 200, 520, None), (33, 256, 8, "silu"), (64, 1000, 776, None),
                                       (100, 512, 4096, "gelu"), (129, 2112, 1024, None), (256, 384, 4104, None), (300, 136, 1536, None)])
@pytest.mark.parametrize("parts", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("smem", [108, 220])
def test_gemm_on_clusters(m, n, k, act, parts, smem):
    """K over the CTAs of a cluster: parts without a row of their own, with one K block or a ragged one, tiles past the last column
    and row, one and several tiles of rows, strided input and output, bias and both gates. fp32 sums of bf16 products, one rounding
    to bf16; gated ones also __expf and a division (2^-8 relative in all)."""
    from gllm_b200.ops import lib
    if parts > -(-k // 64):
        pytest.skip("no empty parts")
    torch.manual_seed(m + n)
    gated, n_out = act is not None, n // 2 if act else n
    x = torch.randn(m, k + 16, device=_dev()).bfloat16()[:, 8:8 + k]
    wide = torch.randn(n, k, device=_dev()).bfloat16() * k ** -0.5
    w = torch.zeros(n, k + 8, device=_dev(), dtype=torch.bfloat16)[:, :k]
    w.copy_(ref.interleave_gate_up(wide) if gated else wide)
    b = None if gated else torch.randn(n, device=_dev()).bfloat16()
    out = torch.full((m + 1, n_out + 8), 7.0, device=_dev()).bfloat16()
    y = x.double() @ wide.double().t()
    if gated:
        g, u = y.chunk(2, -1)
        want = (torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u
        tol = want.abs() * 2.0 ** -7 + 1e-3
    else:
        want = y + b.double()
        tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ wide.double().abs().t() + b.double().abs()) * k * 2.0 ** -24
    rows = min(256, -(-m // 16) * 16)
    for bt in {rows, max(16, -(-rows // 32) * 16)}:
        out.fill_(7.0)
        assert lib.load().gllm_gemm_bf16_cluster(x.data_ptr(), x.stride(0), w.data_ptr(), w.stride(0), out.data_ptr(), out.stride(0), m, n, k,
                                                 None if b is None else b.data_ptr(), int(gated), int(act == "gelu"), bt, parts,
                                                 smem * 1024, lib.stream_ptr()) == 0
        assert bool((out[m] == 7.0).all()) and bool((out[:, n_out:] == 7.0).all())
        assert bool(((out[:m, :n_out].double() - want).abs() <= tol).all())


@pytest.mark.parametrize("m,n,k", [(32, 16512, 72), (32, 19072, 72), (128, 12800, 264), (80, 12800, 264), (79, 12800, 264), (256, 10496, 1544),
                                   (128, 4608, 2368), (111, 4608, 2368), (384, 3072, 4416), (384, 3072, 4424), (128, 11008, 1536),
                                   (128, 11008, 1544), (128, 5760, 1032), (200, 3328, 2056)])
def test_linear_where_the_kernels_meet(m, n, k):
    """Sizes on both sides of the rules that choose between clusters and the other tiles, and tiles that fill the clusters of three and five
    that run at once to the last. fp32 sums of bf16 products in any order, one rounding."""
    from gllm_b200.ops import sm100
    torch.manual_seed(n + k)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), torch.randn(n, k, device=_dev()).bfloat16()
    want = x.double() @ w.double().t()
    tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    assert bool(((sm100.linear(x, w).double() - want).abs() <= tol).all())


@pytest.mark.parametrize("t,k,experts,held,valid", [(1, 1, 1, 1, None), (3, 8, 16, 16, None), (512, 8, 128, 128, None),
                                                    (513, 8, 256, 32, None), (2048, 2, 1024, 1024, None), (2049, 2, 1024, 700, None),
                                                    (600, 1, 8, 8, 37), (5000, 1, 8, 8, 4097), (40, 4, 300, 0, None),
                                                    (5000, 1, 8, 0, None), (16384, 1, 5, 5, None), (16385, 1, 5, 5, None),
                                                    (5000, 8, 256, 31, None), (17000, 8, 1024, 1024, None), (20000, 1, 8, 8, 37),
                                                    (40000, 1, 8, 8, 17001), (20000, 1, 8, 8, 0)])
@pytest.mark.parametrize("quant", [False, True])
def test_moe_routing_and_gather(t, k, experts, held, valid, quant):
    """Counts, padded offsets, tiles, places and rows of the forms of the routing (up to 4096 slots in one launch, up to 16,384 by one
    block, beyond by the CTAs of a cluster, the last of them in several steps), a rank that holds no expert among them, and quantised on the way the same bytes and scales as by the quantiser."""
    from gllm_b200.ops import lib
    torch.manual_seed(t + experts)
    dev, h, E = _dev(), 384, held
    ids = torch.randint(0, experts, (t, k), device=dev, dtype=torch.int32)
    ids[: t // 3] = ids[0, 0]                              # a liked expert: several tiles
    emap = None
    if held < experts:
        emap = torch.full((experts,), -1, dtype=torch.int32, device=dev)
        emap[torch.randperm(experts, device=dev)[:held]] = torch.arange(held, dtype=torch.int32, device=dev)
    x = torch.randn(t, h + 8, device=dev).bfloat16()[:, :h]
    if valid is not None:
        ids[valid:] = 10 ** 6                              # never looked at
    tiles = (t * k + 127) // 128 + E
    new = lambda *s, dtype=torch.int32: torch.full(s, -77, dtype=dtype, device=dev)   # noqa: E731
    meta, tile_expert, pos = new(2 + 3 * E + 1), new(tiles), new(t * k)
    nv = None if valid is None else torch.tensor([valid], dtype=torch.int32, device=dev)
    p = lambda v: None if v is None else v.data_ptr()      # noqa: E731
    L = lib.load()
    if quant:
        if nv is not None:
            pytest.skip("the quantised form takes every row")
        rows, scales = torch.zeros(tiles * 128, h, dtype=torch.uint8, device=dev), torch.zeros(h // 128, tiles * 128, device=dev)
        rc = L.gllm_moe_align_gather_fp8(p(ids), p(emap), t, k, E, p(meta), p(tile_expert), tiles, p(pos), p(x), x.stride(0), p(rows),
                                         p(scales), h, lib.stream_ptr())
    else:
        rows = torch.zeros(tiles * 128, h, dtype=torch.bfloat16, device=dev)
        rc = L.gllm_moe_align_gather(p(ids), p(emap), t, k, E, p(meta), p(tile_expert), tiles, p(pos), p(x), x.stride(0), p(rows), h,
                                     p(nv), lib.stream_ptr())
    assert rc == 0
    e = ids.flatten().long() if valid is None else ids.flatten().clamp(max=experts - 1).long()
    e = e if emap is None else emap[e].long()
    if valid is not None:
        e[valid:] = -1
    live = e >= 0
    cnt = torch.bincount(e[live], minlength=E)
    off = torch.cat([torch.zeros(1, dtype=torch.long, device=dev), ((cnt + 127) // 128 * 128).cumsum(0)])
    assert torch.equal(meta[2:2 + E].long(), cnt) and torch.equal(meta[2 + 2 * E:].long(), off)
    assert meta[0] == off[-1] // 128 and meta[1] == off[-1]
    want = torch.full((tiles,), -1, dtype=torch.int32, device=dev)
    want[: int(off[-1]) // 128] = torch.repeat_interleave(torch.arange(E, device=dev), (cnt + 127) // 128).int()
    assert torch.equal(tile_expert, want)
    assert bool((pos[~live] == -1).all())
    place, which = pos[live].long(), e[live]
    assert torch.equal(place.sort().values, torch.cat([torch.arange(int(o), int(o + c), device=dev) for o, c in zip(off, cnt)] or [place[:0]]))
    assert bool((place >= off[which]).all()) and bool((place < off[which] + cnt[which]).all())
    src = x.repeat_interleave(k, 0)[live]
    if not quant:
        assert torch.equal(rows[place], src)
    elif len(place):
        src = src.contiguous()
        q, s = torch.empty(len(place), h, dtype=torch.uint8, device=dev), torch.empty(h // 128, len(place), device=dev)
        assert L.gllm_fp8_quant_group(p(src), h, p(q), p(s), len(place), h, None, lib.stream_ptr()) == 0
        assert torch.equal(rows[place], q) and torch.equal(scales[:, place], s)


@pytest.mark.parametrize("heads,width", [(1, 256), (5, 512), (16, 8192)])
@pytest.mark.parametrize("q_lens,decodes", [([1], 1), ([1] * 33, 33), ([1] * 65 + [3, 7], 65), ([1] * 129, 129), ([20], 0)])
def test_latent_attention_block_in_one_call(heads, width, q_lens, decodes, monkeypatch):
    """The block launched by one native call is the block launched kernel by kernel, bit for bit: rows that take each of the GEMMs,
    one head, strided hidden states, decoding sequences and short portions."""
    from types import SimpleNamespace
    from gllm_b200.layers.rotary import build_rope
    from gllm_b200.models.decoder import ModelSpec
    from gllm_b200.models.deepseek_v2 import MLAAttention
    from gllm_b200.ops import sm100
    torch.manual_seed(6)
    dev, page = _dev(), 16
    spec = ModelSpec(arch="DeepseekV3ForCausalLM", hidden_size=width, num_layers=1, num_heads=heads, num_kv_heads=heads, head_dim=192,
                     intermediate_size=64, vocab_size=64, rms_eps=1e-6, dtype=torch.bfloat16, use_mla=True,
                     extra={"qk_nope_head_dim": 128, "qk_rope_head_dim": 64, "v_head_dim": 128, "kv_lora_rank": 512,
                            "q_lora_rank": 256})
    att = MLAAttention(spec, 0, build_rope(64, 1024, 1e4, None, 64, False, device=dev), dev)
    for p in att.parameters():
        p.data.copy_(torch.randn(p.shape, device=dev) * p.shape[-1] ** -0.5 if p.dim() == 2 else 1 + 0.1 * torch.randn(p.shape, device=dev))
    att.process_weights()
    ctx = [(37 * i) % 150 for i in range(len(q_lens))]
    lens = [a + b for a, b in zip(q_lens, ctx)]
    need = [-(-n // page) for n in lens]
    ids = torch.randperm(sum(need)).split(need)
    bt = torch.zeros(len(lens), max(need), dtype=torch.int32)
    for i, x in enumerate(ids):
        bt[i, :len(x)] = x
    qsl = np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)
    pos = torch.cat([torch.arange(a, a + b) for a, b in zip(ctx, q_lens)]).int()
    seq = torch.repeat_interleave(torch.arange(len(q_lens)), torch.tensor(q_lens)).int()
    slots = bt[seq.long(), pos.long() // page] * page + pos % page
    inp = SimpleNamespace(num_decode_seqs=decodes, num_seqs=len(q_lens), padded_tokens=0, max_q_len=max(q_lens),
                          batch=SimpleNamespace(query_start_loc=qsl, seq_lens=np.array(lens, np.int32)), positions=pos.to(dev),
                          slot_mapping=slots.int().to(dev), block_table=bt.to(dev), seq_lens=torch.tensor(lens).int().to(dev),
                          tok_seq=None if decodes == len(q_lens) else seq.to(dev), query_start_loc=torch.as_tensor(qsl).to(dev))
    tpc = SimpleNamespace(materialize=lambda h: h)
    cache0 = torch.randn(sum(need), 1, 9, page, 64, device=dev).bfloat16()
    h = torch.randn(sum(q_lens), width + 64, device=dev).bfloat16()[:, 32:32 + width]
    calls, got = [], []
    one = sm100.mla_block
    monkeypatch.setattr(sm100, "mla_block", lambda *a: calls.append(1) or one(*a))
    for forced in (0, 1):
        monkeypatch.setattr(sm100, "gemm_forced", lambda: bool(forced))
        cache = cache0.clone()
        got.append((att(inp, h, SimpleNamespace(k_cache=[cache]), tpc), cache))
    assert len(calls) == 1
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k,act", [(8, 8, 0), (5, 264, 0), (4100, 1024, 0), (640, 6144, 0), (512, 1032, 1), (6144, 1024, 1), (64, 12280, 0)])
def test_norm_with_the_product_behind_it(m, n, k, act):
    """rmsnorm(y + residual) formed by the one-or-two-row product: the sum bit for bit that of the norm kernel, the product within the
    roundings of fp32 sums of bf16 products and of normed values that may round to the other neighbour (2^-8 each, not all one way)."""
    from gllm_b200.ops import sm100
    torch.manual_seed(n + k)
    y = torch.randn(m, k + 16, device=_dev()).bfloat16()[:, 8:8 + k]
    res, w = torch.randn(m, k, device=_dev()).bfloat16(), (1 + 0.2 * torch.randn(k, device=_dev())).bfloat16()
    wt = torch.randn(n, k + 8, device=_dev()).bfloat16()[:, :k] * k ** -0.5
    b = None if act else torch.randn(n, device=_dev()).bfloat16()
    out = torch.full_like(res, 7.0)
    got = sm100.norm_linear(y, res, out, w, 1e-6, wt, b, act)
    want_res = res.clone()
    normed, _ = sm100.rmsnorm(y, w, 1e-6, want_res)
    assert got is not None and torch.equal(out, want_res)
    want = sm100.linear_silu_mul(normed, wt) if act else sm100.linear(normed, wt, b)
    assert got.shape == want.shape and _rel_err(got, want) < 6e-3


@pytest.mark.parametrize("m,k", [(1, 24584), (1, 24576), (2, 12288), (2, 12296)])
def test_norm_that_no_product_takes(m, k):
    """A deferred norm whose product is too large for the kernel is formed by the norm's own: rows beyond its shared memory, or rows
    that fill it to the last byte and leave nothing for the sums of squares."""
    from gllm_b200.layers import functional as Fn
    torch.manual_seed(3)
    y, res = torch.randn(m, k, device=_dev()).bfloat16(), torch.randn(m, k, device=_dev()).bfloat16()
    w, wt = torch.ones(k, device=_dev()).bfloat16(), torch.randn(64, k, device=_dev()).bfloat16() * k ** -0.5
    h = Fn.NormedSum(y, res, w, 1e-6)
    got = h.linear(wt)
    want_res = res.clone()
    normed, _ = Fn.rmsnorm(y, w, 1e-6, want_res)
    assert torch.equal(h.residual, want_res) and torch.equal(got, Fn.linear(normed, wt))
    assert torch.equal(Fn.NormedSum(y, res, w, 1e-6).tensor(), normed)


@pytest.mark.parametrize("m,k,deferred", [(1, 3072, True), (1, 3080, False), (2, 1024, True), (2, 1032, False), (3, 512, False)])
def test_rows_whose_norm_is_deferred(m, k, deferred):
    """Short rows leave their norm to the product behind it, longer ones do not; either way the product and the sum are those of the
    norm and the product by themselves (fp32 sums in another order: 2^-8 of some normed values)."""
    from gllm_b200.layers import functional as Fn
    from gllm_b200.parallel.tp import TPComm
    torch.manual_seed(k)
    a, w1, w2 = torch.randn(m, 256, device=_dev()).bfloat16(), torch.randn(k, 256, device=_dev()).bfloat16(), torch.randn(384, k, device=_dev()).bfloat16()
    res, nw, tpc = torch.randn(m, k, device=_dev()).bfloat16(), (1 + 0.2 * torch.randn(k, device=_dev())).bfloat16(), TPComm()
    normed, want = Fn.rmsnorm(Fn.linear(a, w1), nw, 1e-6, res.clone())
    h, got = tpc.row_linear_add_norm(a, w1, res, nw, 1e-6, defer=True)
    assert isinstance(h, Fn.NormedSum) == deferred
    assert _rel_err(tpc.col_linear(h, w2), Fn.linear(normed, w2)) < 6e-3 and torch.equal(got, want)


@pytest.mark.parametrize("where", ["layer", "layer behind", "attention", "all modules", None])
def test_hooks_see_tensors_between_layers(where, monkeypatch):
    """A hook between two layers sees the normed input and the residual stream as tensors that are there: the norm is not left to the
    next layer's first product then. Both forms round alike but for the order of the fp32 sums."""
    from types import SimpleNamespace
    from gllm_b200.layers import functional as Fn
    from gllm_b200.models.decoder import CausalLM, ModelSpec
    from gllm_b200.parallel.tp import TPComm
    torch.manual_seed(11)
    spec = ModelSpec(arch="Qwen3ForCausalLM", hidden_size=512, num_layers=3, num_heads=4, num_kv_heads=2, head_dim=128,
                     intermediate_size=1024, vocab_size=128, max_position=64)
    model = CausalLM(spec, _dev())
    for w in model.parameters():
        w.data.copy_(torch.randn_like(w) * (0.05 if w.dim() > 1 else 1.0))
    inp = SimpleNamespace(tokens=torch.tensor([5, 77], dtype=torch.int32, device=_dev()))
    deferred, made = [], Fn.NormedSum.__init__
    monkeypatch.setattr(Fn.NormedSum, "__init__", lambda self, *a: deferred.append(1) or made(self, *a))

    def run():
        seen = []

        def keep(module, args, out=None):
            values = args if out is None or module is model.layers[1].attn else out if isinstance(out, tuple) else (out,)
            seen.extend(x.clone() for x in values if isinstance(x, (torch.Tensor, Fn.NormedSum)))
        hook = {"layer": lambda: model.layers[0].register_forward_hook(keep),
                "layer behind": lambda: model.layers[1].register_forward_pre_hook(keep),
                "attention": lambda: model.layers[1].attn.register_forward_hook(keep),
                "all modules": lambda: torch.nn.modules.module.register_module_forward_hook(keep), None: lambda: None}[where]()
        try:
            return [*model(inp, None, TPComm()), *seen]
        finally:
            if hook is not None:
                hook.remove()

    got = run()
    between = {"layer behind": 2, "all modules": 2, None: 0}.get(where, 1)    # the middle layer's hook speaks for both its sides
    assert len(deferred) == 5 - between                     # three norms inside layers, two between them
    monkeypatch.setattr(Fn.NormedSum, "takes", staticmethod(lambda *a: False))
    want = run()
    assert len(got) == len(want) and (len(got) == 2) == (where is None)
    assert all(_rel_err(a, b) < 2e-2 for a, b in zip(got, want))


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("n,k", [(1, 8), (5, 264), (130, 1024), (4097, 1024), (4100, 2056), (257, 6144), (640, 8192)])
def test_linear_few_rows(m, n, k):
    """One and two rows: a warp per weight row with the whole of K. Rows and columns beyond the last block, K below one 16-byte
    load per lane, K over several chunks, strided input and output, a bias. fp32 sums of bf16 products, one rounding to bf16."""
    from gllm_b200.ops import sm100
    torch.manual_seed(n + k)
    x = torch.randn(m, k + 16, device=_dev()).bfloat16()[:, 8:8 + k]
    w = torch.randn(n, k + 8, device=_dev()).bfloat16()[:, :k]
    b = torch.randn(n, device=_dev()).bfloat16()
    out = torch.full((m + 1, n + 8), 7.0, device=_dev()).bfloat16()
    sm100.linear(x, w, b, out=out[:m, :n])
    want = x.double() @ w.double().t() + b.double()
    assert bool((out[m] == 7.0).all()) and bool((out[:, n:] == 7.0).all())
    tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    assert bool(((out[:m, :n].double() - want).abs() <= tol).all())
    if k >= 1024:
        gu = torch.randn(512, k, device=_dev()).bfloat16() * k ** -0.5
        inter = ref.interleave_gate_up(gu)
        for act, f in (("silu", torch.nn.functional.silu), ("gelu", lambda z: torch.nn.functional.gelu(z, approximate="tanh"))):
            g, u = (x.float() @ gu.float().t()).chunk(2, -1)
            assert _rel_err(sm100.linear_silu_mul(x, inter, act=act), f(g) * u) < 6e-3      # one bf16 rounding and fast exp


@pytest.mark.parametrize("m,n", [(1, 9472), (1, 9473), (2, 2368), (2, 2369)])       # 148 SMs x 16 warps: four full rounds, one
@pytest.mark.parametrize("gated", [False, True])
def test_linear_few_rows_at_the_rules_border(m, n, gated):
    """The last matrix that the plain-core kernel takes and the first that goes to the tensor-core one, K = 4096 (131 KB a round
    and SM; gated, two rows per warp: half as many rounds)."""
    from gllm_b200.ops import sm100
    torch.manual_seed(n)
    x = torch.randn(m, 4096, device=_dev()).bfloat16()
    if not gated:
        w = torch.randn(n, 4096, device=_dev()).bfloat16()
        want = x.double() @ w.double().t()
        tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * 4096 * 2.0 ** -24
        assert bool(((sm100.linear(x, w).double() - want).abs() <= tol).all())
        return
    w = torch.randn(n // 256 * 256 + 256 * (n & 1), 4096, device=_dev()).bfloat16() * 4096 ** -0.5
    g, u = (x.float() @ w.float().t()).chunk(2, -1)
    assert _rel_err(sm100.linear_silu_mul(x, ref.interleave_gate_up(w)), torch.nn.functional.silu(g) * u) < 6e-3


@pytest.mark.parametrize("bn", [32, 192])
def test_gemm_gated_refuses_tile_widths_without_a_gated_form(bn, monkeypatch):
    """The plain epilogue would store twice the output's columns."""
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "_FORCE_BN", bn)
    x, w = torch.randn(64, 128, device=_dev()).bfloat16(), torch.randn(256, 128, device=_dev()).bfloat16()
    with pytest.raises(RuntimeError):
        sm100.linear(x, w, epi=1)


@pytest.mark.parametrize("m", [3, 17, 32])
@pytest.mark.parametrize("ldc,shift", [(13, 0), (514, 1), (516, 2), (516, 4)])     # the last one: 8-byte boundaries
def test_gemm_smallm_any_output(m, ldc, shift):
    """Outputs whose rows lie off the 8-byte boundaries that the split-K sums are stored on: element-wise stores instead."""
    from gllm_b200.ops import sm100
    torch.manual_seed(ldc + m)
    n, k = (5, 4096) if ldc == 13 else (512, 4096)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), torch.randn(n, k, device=_dev()).bfloat16()
    buf = torch.full((m * ldc + 8,), 7.0, device=_dev()).bfloat16()
    want = x.double() @ w.double().t()
    tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    out = torch.as_strided(buf, (m, n), (ldc, 1), shift)
    sm100.linear(x, w, out=out)
    assert bool(((out.double() - want).abs() <= tol).all())
    if ldc != 13:
        gated = torch.as_strided(buf, (m, n // 2), (ldc, 1), shift)
        wk = w * k ** -0.5
        g, u = (x.float() @ wk.float().t()).chunk(2, -1)
        sm100.linear_silu_mul(x, ref.interleave_gate_up(wk), out=gated)
        assert _rel_err(gated, torch.nn.functional.silu(g) * u) < 6e-3      # one bf16 rounding and fast exp
    written = torch.zeros_like(buf, dtype=torch.bool)
    torch.as_strided(written, (m, n), (ldc, 1), shift).fill_(True)
    assert bool((buf[~written] == 7.0).all())


@pytest.mark.parametrize("act", ["silu", "gelu", "glu"])
@pytest.mark.parametrize("m,f,k", [(64, 1536, 4096), (100, 2048, 7168), (128, 1792, 4096)])
def test_gemm_gated_split_in_eight(m, f, k, act):
    """K in eight parts, each of whose CTAs gates 16 columns of a tile: what the rule of that kernel chooses here, though clusters take the
    silu and gelu forms if nothing is forced. fp32 sums in the order of the parts, one rounding."""
    from gllm_b200.ops import lib, ref, sm100, sm100_latent
    torch.manual_seed(f)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), (torch.randn(2 * f, k, device=_dev()) * k ** -0.5).bfloat16()
    units = lib.load().gllm_gemm_bf16_tiles_covering(m, 2 * f, k, 1, 256, 0, m, sm100._SMALLM_WS_FLOATS * 4, sm100._SPLITK_MAX_TILES)
    assert units == f // 128 * 8
    wi = ref.interleave_gate_up(w, 128)
    g, u = (x.double() @ w.double().t()).chunk(2, -1)
    if act == "glu":
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        want, call = g * torch.sigmoid(1.7 * g) * (u + 1), lambda: sm100_latent.linear_glu_clamp(x, wi, 1.5, 1.7)
    else:
        want = (torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u
        call = lambda: sm100.linear_silu_mul(x, wi, act=act)  # noqa: E731
    for split in (8, 8, 8, 0):                               # the counters of a tile are set back behind each product; as dispatched
        with _forced_split(split):
            got = call()
        assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -16 * (1 + want.abs())).all())


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("m", [64, 600, 2305])
def test_gemm_gated_at_a_forced_tile_width(bn, m, monkeypatch):
    """A forced width of a gated product says how gate and up rows alternate (blocks of half of it): no other tiles may be taken.
    One rounding of the output; the gate is fp32 on fp32 sums."""
    from gllm_b200.ops import ref, sm100
    torch.manual_seed(bn)
    monkeypatch.setattr(sm100, "_FORCE_BN", bn)
    f, k = 4992, 136
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), (torch.randn(2 * f, k, device=_dev()) * k ** -0.5).bfloat16()
    g, u = (x.double() @ w.double().t()).chunk(2, -1)
    want = torch.nn.functional.silu(g) * u
    got = sm100.linear(x, ref.interleave_gate_up(w, bn // 2), epi=1)
    assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -16 * (1 + want.abs())).all())


def test_gemm_refuses_unaligned_output():
    """The tiled GEMMs store 16 bytes at a time: an output or bias off that boundary is an error, never a launch."""
    from gllm_b200.ops import sm100
    x, w = torch.randn(64, 256, device=_dev()).bfloat16(), torch.randn(256, 256, device=_dev()).bfloat16()
    buf = torch.zeros(64 * 264 + 8, device=_dev()).bfloat16()
    off = torch.as_strided(buf, (64, 256), (264, 1), 4)
    w8, ws = w.to(torch.float8_e4m3fn), torch.ones(2, 2, device=_dev())
    for call in (lambda: sm100.linear(x, w, out=off), lambda: sm100.linear(x, w, buf[4:260]),
                 lambda: sm100.linear_fp8_block(x, w8, ws, out=off), lambda: sm100.linear_fp8_block(x, w8, ws, buf[4:260]),
                 lambda: sm100.linear_fp8_block(x, w8, ws, out=torch.as_strided(buf, (64, 256), (260, 1)))):
        with pytest.raises(RuntimeError):
            call()
    assert bool((buf == 0).all())


@pytest.mark.parametrize("m,n,k", [(1, 8, 64), (128, 192, 128), (129, 184, 72), (300, 200, 1000), (2100, 576, 328)])
def test_gemm_tiles_of_192(m, n, k, monkeypatch):
    """Tiles 192 wide: columns and rows beyond the last tile, K not a multiple of a 64-deep block, a bias; fp32 sums, one rounding."""
    from gllm_b200.ops import sm100
    monkeypatch.setattr(sm100, "_FORCE_BN", 192)
    torch.manual_seed(n + k)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), torch.randn(n, k, device=_dev()).bfloat16()
    b = torch.randn(n, device=_dev()).bfloat16()
    want = x.double() @ w.double().t() + b.double()
    tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    assert bool(((sm100.linear(x, w, b).double() - want).abs() <= tol).all())


@pytest.mark.parametrize("m,n,k", [(513, 5000, 8), (600, 6136, 264), (769, 5128, 1000), (4200, 4104, 136), (2305, 19208, 64)])
def test_gemm_on_pairs_of_sms(m, n, k):
    """Sizes that run on pairs: rows and columns beyond the last tile of 256 (one row, one CTA's half, eight columns), one to four
    rounds, K not a multiple of a 64-deep block; rows of the output on a wider stride, the row behind the last untouched. fp32
    sums, one rounding."""
    from gllm_b200.ops import sm100
    torch.manual_seed(n + k)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), torch.randn(n, k, device=_dev()).bfloat16()
    b = torch.randn(n, device=_dev()).bfloat16()
    buf = torch.full((m + 1, n + 8), 7.0, device=_dev(), dtype=torch.bfloat16)
    sm100.linear(x, w, b, out=buf[:m, :n])
    want = x.double() @ w.double().t() + b.double()
    tol = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * k * 2.0 ** -24
    assert bool(((buf[:m, :n].double() - want).abs() <= tol).all())
    assert bool((buf[m] == 7).all()) and bool((buf[:, n:] == 7).all())


@pytest.mark.parametrize("act", ["silu", "gelu", "glu"])
@pytest.mark.parametrize("m,f,k", [(600, 2944, 264), (2305, 4992, 72), (33, 128, 72), (64, 12288, 136), (128, 4736, 200)])
def test_gemm_gated_tiles(m, f, k, act):
    """On pairs of SMs, where both halves of a gated tile lie in each CTA; up to 128 rows in tiles of 96 features, whose rows
    straddle the blocks that gate and up rows alternate in. One rounding of the output; the gate functions are fp32 on fp32 sums."""
    from gllm_b200.ops import ref, sm100, sm100_latent
    torch.manual_seed(f)
    x, w = torch.randn(m, k, device=_dev()).bfloat16(), (torch.randn(2 * f, k, device=_dev()) * k ** -0.5).bfloat16()
    wi = ref.interleave_gate_up(w, 128)
    g, u = (x.double() @ w.double().t()).chunk(2, -1)
    if act == "glu":
        got = sm100_latent.linear_glu_clamp(x, wi, 1.5, 1.7)
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        want = g * torch.sigmoid(1.7 * g) * (u + 1)
    else:
        got = sm100.linear_silu_mul(x, wi, act=act)
        want = (torch.nn.functional.silu(g) if act == "silu" else torch.nn.functional.gelu(g, approximate="tanh")) * u
    assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -16 * (1 + want.abs())).all())


@pytest.mark.parametrize("t,widths", [(1, (1536, 512)), (5, (8, 8192)), (130, (72, 1000))])
def test_rmsnorm_two(t, widths):
    """Two norms over column ranges of the same rows: each as the single one has it (fp32 sums in another order, one rounding)."""
    from gllm_b200.ops import sm100
    torch.manual_seed(t)
    x = torch.randn(t, sum(widths) + 64, device=_dev()).bfloat16()
    x1, x2 = x[:, :widths[0]], x[:, widths[0]:sum(widths)]
    w1, w2 = (torch.randn(n, device=_dev()).bfloat16() for n in widths)
    for got, v, w in zip(sm100.rmsnorm_two(x1, w1, x2, w2, 1e-6), (x1, x2), (w1, w2)):
        want = v.double() * torch.rsqrt(v.double().square().mean(-1, keepdim=True) + 1e-6) * w.double()
        assert got.is_contiguous() and bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-6).all())


@pytest.mark.parametrize("seqs,blocks,tokens", [(1, 1, 1), (3, 7, 3), (64, 60, 64), (64, 70, 4100), (200, 100, 5000)])
def test_batch_arrays_reach_their_buffers(seqs, blocks, tokens):
    """A step's arrays on the device are the host's, whether they go in the staging block or are copied by themselves (more than
    4096 words each, or beyond the block's 16,384), over several steps that alternate the staging buffers; rows beyond them stay."""
    import numpy as np
    from gllm_b200.input_data import BatchArrays, InputData
    inp, rng = InputData(6000, 256, 128, "cuda:0"), np.random.RandomState(seqs)
    i32, f32 = np.int32, np.float32
    for step in range(3):
        ints = lambda n: rng.randint(0, 1 << 30, n).astype(i32)
        b = BatchArrays(tokens=ints(tokens), positions=ints(tokens), slot_mapping=ints(tokens),
                        block_table=rng.randint(0, 1 << 30, (seqs, blocks)).astype(i32), seq_lens=ints(seqs),
                        query_start_loc=ints(seqs + 1), logits_idx=ints(seqs), emit_seq=np.arange(seqs, dtype=i32),
                        temperature=rng.rand(seqs).astype(f32), top_k=ints(seqs), top_p=rng.rand(seqs).astype(f32),
                        rep_penalty=rng.rand(seqs).astype(f32), state_slot=ints(seqs), num_decode_seqs=0, num_seqs=seqs,
                        num_tokens=tokens, max_q_len=2, max_seq_len=9, rec_slots=ints(seqs), all_greedy=False)
        inp.load(b)
        for pair, want in ((inp._tokens, b.tokens), (inp._positions, b.positions), (inp._slots, b.slot_mapping),
                           (inp._seq_lens, b.seq_lens), (inp._qsl, b.query_start_loc), (inp._logits_idx, b.logits_idx),
                           (inp._temperature, b.temperature), (inp._top_k, b.top_k), (inp._top_p, b.top_p),
                           (inp._rep_penalty, b.rep_penalty), (inp._state_slot, b.state_slot), (inp._rec_slots, b.rec_slots)):
            got = pair[1].cpu().numpy()
            assert np.array_equal(got[:len(want)], want) and not got[len(want):].any()
        table = inp._block_table[1].cpu().numpy()
        assert np.array_equal(table[:seqs, :blocks], b.block_table) and not table[seqs:].any() and not table[:, blocks:].any()
