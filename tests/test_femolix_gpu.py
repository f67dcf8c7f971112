"""Femolix on the sm_100a kernels: every new kernel of csrc/seq against its unfused PyTorch form, and the engine
scenarios of test_femolix_cpu.py (chunking, mixed batches, page / slot re-use, generation, CUDA-graph decode) against
the plain oracle, in fp32 (tight) and bf16 (rounding-sized tolerance)."""
import numpy as np
import pytest
import torch

import femolix_oracle as oracle
import femolix_util as U
from test_femolix_cpu import CONFIGS, _chunk_probe, toks

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL32 = 2e-4


def row_errs(got, want):
    d = got - want
    d = d - d.mean(-1, keepdims=True)
    w = want - want.mean(-1, keepdims=True)
    return np.sqrt((d ** 2).mean(-1)) / (np.sqrt((w ** 2).mean(-1)) + 1e-9)


class Expect:
    """What a run is held to. fp32: the oracle, tightly. bf16: the error that rounding alone causes is measured by
    running the unfused PyTorch forms on the CPU with the same rounding points (bf16 weights, activations and cache,
    fp32 accumulation); the kernels may be at most twice as far from the oracle, on the median row and, for models
    without discrete choices, on the worst row. In models with a router, one bf16 rounding can flip a close call
    in these tiny sizes and move every later row by tens of percent on either device: there only the median is held,
    loosely; their exactness is what the fp32 runs and the kernel tests establish."""

    def __init__(self, cfg, w, path, tokens, dtype):
        self.want = U.expected_logits(cfg, w, tokens)
        self.dtype = dtype
        self.routed = any(L["mlp"] and L["mlp"]["kind"] == "moe" and
                          L["mlp"]["router"]["top"] < L["mlp"]["router"]["experts"] for L in cfg["layers"])
        if dtype == "bfloat16":
            s = U.session(path, "bfloat16", "cpu", max_tokens=max(256, len(tokens) + 64), page_size=16)
            got = s.step([{"id": "r", "tokens": tokens, "want": list(range(len(tokens)))}], ["r"])
            self.noise = row_errs(got, self.want)

    def check(self, got):
        e = row_errs(got, self.want)
        if self.dtype == "float32":
            assert e.max() < TOL32
        elif self.routed:
            assert np.median(e) < max(2 * np.median(self.noise), 0.25)
        else:
            assert np.median(e) <= 2 * np.median(self.noise) + 1e-2
            assert e.max() <= 2 * self.noise.max() + 2e-2


def close(a, b, tol):
    return (a.float() - b.float()).abs().max().item() <= tol * (b.float().abs().max().item() + 1e-9)


def _batch(qlens, ctx, ps, pages):
    qsl = torch.tensor([0] + np.cumsum(qlens).tolist(), dtype=torch.int32, device=DEV)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    per = max((c + q + ps - 1) // ps for c, q in zip(ctx, qlens))
    bt = torch.randperm(pages - 1)[: len(qlens) * per].reshape(len(qlens), per).to(torch.int32).to(DEV)
    pos = torch.cat([torch.arange(c, c + q) for c, q in zip(ctx, qlens)]).to(torch.int32).to(DEV)
    seqi = torch.cat([torch.full((q,), i) for i, q in enumerate(qlens)]).to(DEV)
    slots = (bt[seqi, (pos // ps).long()] * ps + pos % ps).to(torch.int32)
    return qsl, sl, bt, pos, slots


@pytest.mark.parametrize("dt,tol", [(torch.float32, 3e-5), (torch.bfloat16, 2e-2)])
def test_kernels_against_unfused_ops(dt, tol):
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(0)
    T, W = 37, 200
    x = torch.randn(T, W, device=DEV)
    y, w = torch.randn(T, W, device=DEV).to(dt), (torch.rand(W, device=DEV) + 0.5).to(dt)
    x1, x2 = x.clone(), x.clone()
    h1, h2 = S.postnorm(x1, y, 1.75, w, 1e-5, dt), ref.postnorm(x2, y, 1.75, w, 1e-5, dt)
    assert close(h1, h2, tol) and close(x1, x2, 1e-5)
    gu = torch.randn(T, 2 * 50, device=DEV).to(dt)
    assert close(S.silu_mul(gu), ref.silu_mul(gu), tol)
    z = (torch.randn(T, 77, device=DEV) * 20).to(dt)
    assert close(S.softcap(z.clone(), 12.0), ref.softcap(z, 12.0), tol)
    # router: ids exact (random logits have no near ties), weights close
    hh, wr = torch.randn(T, W, device=DEV).to(dt), torch.randn(11, W, device=DEV).to(dt)
    for k in (1, 2, 11):
        w2, i2 = ref.router_topk(hh, wr, k)
        for path in ("token", "gemm"):
            w1, i1 = S.router_topk(hh, wr, k, force=path)
            assert torch.equal(i1, i2) and close(w1, w2, 1e-4), (k, path)
    if dt == torch.bfloat16:          # tensor-core logits: ragged token and expert counts, two expert tiles
        for tt, ee, ww in ((37, 11, 208), (300, 70, 64), (64, 8, 16), (1000, 64, 512)):
            hb = torch.randn(tt, ww + 16, device=DEV).to(dt)[:, :ww]
            wb = torch.randn(ee, ww, device=DEV).to(dt)
            w2, i2 = ref.router_topk(hb, wb, 2)
            w1, i1 = S.router_topk(hb, wb, 2, force="mma")
            assert torch.equal(i1, i2) and close(w1, w2, 1e-4), (tt, ee, ww)
    # plain experts
    E, F = 5, 24
    w13, w2_ = (torch.randn(E, 2 * F, W, device=DEV) * W ** -0.5).to(dt), (torch.randn(E, W, F, device=DEV) * F ** -0.5).to(dt)
    wt, ids = ref.router_topk(hh, wr[:E], 2)
    assert close(S.routed_experts(hh, w13, w2_, wt, ids), ref.fused_experts(hh, w13, w2_, wt, ids, None), tol)
    # q/k norm + rotation + cache write, then chunk / window attention on the plain kernel, odd head sizes
    for D, Dv, rot in ((40, 72, 24), (8, 4, 6), (64, 64, 32), (20, 36, 0)):
        H, G, ps = 6, 2, 16
        qlens, ctx = [5, 1, 30], [17, 40, 0]
        qsl, sl, bt, pos, slots = _batch(qlens, ctx, ps, 32)
        Tt = sum(qlens)
        kc = torch.randn(ref.kv_cache_shape(32, G, D, ps), device=DEV).to(dt)
        vc = torch.randn(ref.kv_cache_shape(32, G, Dv, ps), device=DEV).to(dt)
        qkv = torch.randn(Tt, H * D + G * D + G * Dv + 8, device=DEV).to(dt)
        qn, kn = torch.randn(D, device=DEV).to(dt), torch.randn(D, device=DEV).to(dt)
        kc2, vc2 = kc.clone(), vc.clone()
        big = pos + 5000                                   # far positions: angles need more than fp32 products
        q1 = S.qk_norm_rope_kv_write(qkv, H, G, D, Dv, qn, kn, 1e-5, big, rot, 5000.0, kc, vc, slots)
        q2 = ref.qk_norm_rope_kv_write(qkv, H, G, D, Dv, qn, kn, 1e-5, big, rot, 5000.0, kc2, vc2, slots)
        assert close(q1, q2, tol) and close(kc, kc2, tol) and torch.equal(vc, vc2)
        sink = torch.randn(H, device=DEV)
        for wn, ch, sk in ((None, 7, None), (None, 16, None), (5, 12, sink), (None, 1, None), (None, None, None)):
            joint = torch.zeros(Tt, H * Dv + 8, device=DEV).to(dt)
            a1 = S.window_attention(q2, kc2, vc2, bt, sl, qsl, pos, 0.2, H, D, wn, sk, chunk=ch, v_dim=Dv,
                                    out_scale=1.2, out=joint[:, 8:])
            a2 = ref.window_attention(q2, kc2, vc2, bt, sl, qsl, 0.2, H, D, wn, sk, chunk=ch, v_dim=Dv, out_scale=1.2)
            assert close(a1, a2, tol), (D, wn, ch)
            assert joint[:, :8].abs().max().item() == 0
    # matrix-state recurrences with carried state, grouped heads, padded value columns
    for Hh, Gq, D, V, delta in ((4, 2, 32, 24, True), (2, 2, 64, 48, False), (3, 1, 5, 3, True), (2, 2, 48, 40, False),
                                (1, 1, 128, 16, True), (2, 1, 128, 40, True), (2, 2, 192, 8, False)):
        # head sizes above 64 take the 8-lanes-per-column form when the chunks are long
        qlens, ctx = ([40, 1, 70], [17, 40, 0]) if (D > 64 and V != 16) else ([5, 1, 30], [17, 40, 0])
        qsl, sl, _, _, _ = _batch(qlens, ctx, 16, 32)
        Tt = sum(qlens)
        rs = torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV)
        q, k = torch.randn(Tt, Gq * D + 3, device=DEV).to(dt), torch.randn(Tt, Gq * D, device=DEV).to(dt)
        v = torch.randn(Tt, Hh * V, device=DEV).to(dt)
        beta, a = torch.randn(Tt, Hh, device=DEV).to(dt), torch.randn(Tt, Hh, device=DEV).to(dt)
        neg_a, dtb = -torch.rand(Hh, device=DEV) * 2, torch.randn(Hh, device=DEV)
        decay = torch.tensor([0.9, 1.0, 0.5, 0.99][:Hh], device=DEV)
        st1 = torch.randn(5, Hh, D, V, device=DEV) * 0.3
        st2 = st1.clone()
        args = (beta, a, neg_a, dtb, None) if delta else (None, None, None, None, decay)
        o1 = S.linear_state_scan(q[:, :Gq * D], k, v, *args, st1, rs, sl, qsl, Hh, Gq, D, V, not delta, delta,
                                 D ** -0.5 if delta else 1.0, delta)
        o2 = ref.linear_state_scan(q[:, :Gq * D], k, v, *args, st2, rs, sl, qsl, Hh, Gq, D, V, not delta, delta,
                                   D ** -0.5 if delta else 1.0, delta)
        assert close(o1, o2, 2e-4), (Hh, D, V, delta)
        assert close(st1, st2, 2e-4)
        assert torch.equal(st1[1], st2[1]) and torch.equal(st1[4], st2[4])      # untouched slots
        gate, nw = torch.randn(Tt, Hh * V + 5, device=DEV).to(dt), torch.randn(V, device=DEV).to(dt)
        for group, wv, act in ((V, nw, "silu"), (Hh * V, torch.randn(Hh * V, device=DEV).to(dt), "sigmoid")):
            joint = torch.zeros(Tt, Hh * V + 2, device=DEV).to(dt)
            g1 = S.gated_group_norm(o2, gate[:, :Hh * V], wv, group, 1e-5, act, 0.5, joint[:, 2:])
            g2 = ref.gated_group_norm(o2, gate[:, :Hh * V], wv, group, 1e-5, act, 0.5, None, dt)
            assert close(g1, g2, tol)


@pytest.mark.parametrize("group,ngroups,ntok,pad", [(128, 1, 1, 0), (128, 3, 7, 4), (256, 1, 5, 8), (256, 3, 33, 4), (128, 5, 3, 1),
                                                    (384, 2, 9, 4)])
@pytest.mark.parametrize("act", ["silu", "sigmoid"])
def test_gated_group_norm_wide_rows(group, ngroups, ntok, pad, act):
    """bf16 groups of 128 and 256: several groups per warp, the last ones missing, rows whose stride (pad 1) or group keeps them
    on the element-wise kernel. One bf16 rounding."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(group + ntok)
    n = group * ngroups
    o = torch.randn(ntok, n, device=DEV)
    gate = torch.randn(ntok, n + pad, device=DEV).bfloat16()[:, :n]
    out = torch.zeros(ntok, n + pad, device=DEV).bfloat16()
    for w in (torch.randn(group, device=DEV).bfloat16(), torch.randn(n, device=DEV).bfloat16()):
        got = S.gated_group_norm(o, gate, w, group, 1e-5, act, 0.5, out[:, :n])
        want = ref.gated_group_norm(o, gate.float(), w.float(), group, 1e-5, act, 0.5, None, torch.float32)
        assert bool(((got.float() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-6).all())
        assert out[:, n:].abs().sum().item() == 0


@pytest.mark.parametrize("group,ngroups,ntok", [(128, 3, 7001), (256, 3, 5001), (128, 8, 3000)])
def test_gated_group_norm_groups_of_a_warp(group, ngroups, ntok):
    """As many groups as a warp takes four (two of 256) at a time, the last warp with fewer, groups of very different size so that one's
    root cannot stand for another's; weights of a group, of a row, and of a length that neither is. One bf16 rounding."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(ntok)
    n = group * ngroups
    o = (torch.randn(ntok, ngroups, group, device=DEV) * torch.exp(torch.randn(ntok, ngroups, 1, device=DEV) * 3)).view(ntok, n)
    gate = torch.randn(ntok, n, device=DEV).bfloat16()
    out = torch.empty(ntok, n, device=DEV).bfloat16()
    for w in (torch.randn(group, device=DEV).bfloat16(), torch.randn(n, device=DEV).bfloat16(), torch.randn(64, device=DEV).bfloat16()):
        got = S.gated_group_norm(o, gate, w, group, 1e-5, "silu", 1.0, out)
        full = w.float().repeat(n // w.shape[0])
        want = ref.gated_group_norm(o, gate.float(), full, group, 1e-5, "silu", 1.0, None, torch.float32)
        assert bool(((got.float() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-6).all())


@pytest.mark.parametrize("act", ["silu", "sigmoid"])
def test_gated_group_norm_gates_one_by_one(act):
    """Unit rows (norm exactly 1) and gates from -100 to 100: the product before the bf16 rounding is within 2^-20 of float64 at any
    gate, so a result is at most half a bf16 step and that away."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(3)
    n, T = 4096, 64
    o = torch.ones(T, n, device=DEV)
    gate = (torch.rand(T, n, device=DEV) * 200 - 100).bfloat16()
    gate[0, :3] = torch.tensor([float("inf"), float("nan"), -float("inf")], device=DEV)
    w = (1 + torch.rand(n, device=DEV)).bfloat16()
    scale = 1 + torch.rand(1).item()
    got = S.gated_group_norm(o, gate, w, 128, 0.0, act, scale).double()
    sg = torch.sigmoid(gate.double())
    want = w.double() * float(torch.tensor(scale, dtype=torch.float32)) * (sg if act == "sigmoid" else gate.double() * sg)
    step = torch.exp2(torch.floor(torch.log2(want.abs().clamp(min=2.0 ** -126))) - 7)
    ok = (got - want).abs() <= step / 2 + want.abs() * 2.0 ** -20
    assert bool(ok[1:].all()) and bool(ok[0, 3:].all())
    assert bool(torch.isnan(got[0, 1])) and float(got[0, 0]) == float(want[0, 0].float().bfloat16())
    assert bool(torch.isnan(got[0, 2])) if act == "silu" else float(got[0, 2]) == 0.0


@pytest.mark.parametrize("taps", [1, 2, 4])
@pytest.mark.parametrize("qlens", [[600], [1, 1, 2050, 3, 1, 4, 5], [17, 1, 15, 700]])
def test_conv_rows_fetched_ahead(qlens, taps):
    """Blocks of 8 rows, one fetched ahead, and of 16, all fetched ahead in groups of four: sequence borders at every place of a group,
    a last block cut short."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(taps)
    ns, C = len(qlens), 36
    ctx = [5 * (i % 2) for i in range(ns)]
    qsl = torch.tensor([0] + qlens, device=DEV).cumsum(0).to(torch.int32)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    rs = torch.randperm(ns + 1, device=DEV)[:ns].to(torch.int32)
    xz = torch.randn(sum(qlens), 2 * C, device=DEV).bfloat16()
    w, b = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV)
    st = torch.randn(ns + 1, max(taps - 1, 1), C, device=DEV).bfloat16()[:, :max(taps - 1, 1)]
    st1, st2 = st.clone(), st.clone()
    c1, c2 = S.causal_conv_silu(xz, C, w, b, st1, rs, sl, qsl), ref.causal_conv_silu(xz, C, w, b, st2, rs, sl, qsl)
    assert close(c1, c2, 1e-2) and torch.equal(st1, st2)


@pytest.mark.parametrize("act", ["silu", "none"])
@pytest.mark.parametrize("taps", [1, 3, 4])
def test_conv_groups_without_a_border(taps, act):
    """Groups of four rows that lie inside one sequence go side by side, the others row by row: sequences that end at each place of a
    group, single tokens between them, the block's last group cut short, an input bias. The sum of at most 5 terms and the sigmoid
    are fp32: their errors are far below the rounding to bf16 of the result, 2^-8 of it or of its terms where they cancel."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(taps)
    qlens = [1, 4, 5, 6, 7, 8, 1, 9, 2100, 2, 3, 1, 17]
    ns, t, C = len(qlens), sum(qlens), 1028
    ctx = [3 * (i % 2) for i in range(ns)]
    qsl = torch.tensor([0] + qlens, device=DEV).cumsum(0).to(torch.int32)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    rs = torch.randperm(ns + 1, device=DEV)[:ns].to(torch.int32)
    xz = torch.randn(t, C + 4, device=DEV).bfloat16()
    w, b, ib = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV), torch.randn(C, device=DEV)
    st1 = torch.randn(ns + 1, max(taps - 1, 1), C, device=DEV).bfloat16()
    st2 = st1.clone()
    got = S.causal_conv_silu(xz, C, w, b, st1, rs, sl, qsl, act=act, in_bias=ib)
    want = ref.causal_conv_silu(xz.float(), C, w, b, st2.float(), rs, sl, qsl, act=act, in_bias=ib)
    ref.causal_conv_silu(xz, C, w, b, st2, rs, sl, qsl, act=act, in_bias=ib)
    assert torch.equal(st1, st2)
    assert bool(((got.float() - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -16).all())


@pytest.mark.parametrize("C", [5120, 10240])
@pytest.mark.parametrize("qlens", [[4100], [1, 1, 700, 13, 1500, 18, 1, 1866]])
def test_conv_rows_beyond_the_ring(C, qlens):
    """Blocks of 32 (5120 channels) and 64 rows, which fill each of the 16 places of the ring twice and four times: borders inside a
    block, a last block cut short. Element by element: the sum and the sigmoid are fp32 (2^-18 at any input here), one rounding."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(C)
    ns, t, taps = len(qlens), sum(qlens), 4
    ctx = [5 * (i % 2) for i in range(ns)]
    qsl = torch.tensor([0] + qlens, device=DEV).cumsum(0).to(torch.int32)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    rs = torch.randperm(ns + 1, device=DEV)[:ns].to(torch.int32)
    xz = (torch.randn(t, C, device=DEV) * 4).bfloat16()
    w, b = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV)
    st1 = torch.randn(ns + 1, taps - 1, C, device=DEV).bfloat16()
    st2, st0 = st1.clone(), st1.clone()
    got = S.causal_conv_silu(xz, C, w, b, st1, rs, sl, qsl)
    assert close(got, ref.causal_conv_silu(xz, C, w, b, st2, rs, sl, qsl), 1e-2) and torch.equal(st1, st2)
    for s in range(ns):
        a, e = int(qsl[s]), int(qsl[s + 1])
        before = st0[rs[s]].double() if ctx[s] else torch.zeros(taps - 1, C, dtype=torch.float64, device=DEV)
        x = torch.cat([before, xz[a:e].double()])
        terms = [w[:, j].double() * x[j:j + e - a] for j in range(taps)]
        acc, size = sum(terms) + b.double(), sum(v.abs() for v in terms) + b.double().abs()
        want = acc * torch.sigmoid(acc)
        tol = want.abs() * (2.0 ** -8 + 2.0 ** -17) + size * 2.0 ** -22 * (1 + acc.abs()) * torch.sigmoid(acc)   # sum of 5, times silu'
        assert bool(((got[a:e].double() - want).abs() <= tol).all())


def test_tensor_core_attention_with_chunk_mask_and_strided_output():
    """bf16, head size 64 / 128 with equal value size: the chunk mask runs on the tensor-core kernels (decode and
    prefill) and must agree with the plain kernel and the PyTorch form, also when it writes a scaled column slice."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(1)
    dt = torch.bfloat16
    for D, ps, ch in ((64, 16, 24), (128, 16, 100), (64, 64, 7), (128, 8, 64)):
        H, G = 8, 2
        for qlens, ctx in (([1, 1, 1], [130, 63, 0]), ([70, 3, 150], [17, 140, 0]), ([1, 1, 90], [99, 5, 31])):
            qsl, sl, bt, pos, _ = _batch(qlens, ctx, ps, 64)
            Tt = sum(qlens)
            nd = sum(1 for q in qlens if q == 1) if qlens[0] == 1 else 0
            nd = nd if all(q == 1 for q in qlens[:nd]) else 0
            kc = torch.randn(ref.kv_cache_shape(64, G, D, ps), device=DEV).to(dt)
            vc = torch.randn(ref.kv_cache_shape(64, G, D, ps), device=DEV).to(dt)
            q = torch.randn(Tt, H * D, device=DEV).to(dt)
            joint = torch.zeros(Tt, H * D + 64, device=DEV).to(dt)
            a1 = S.window_attention(q, kc, vc, bt, sl, qsl, pos, D ** -0.5, H, D, None, None, num_decode_seqs=nd,
                                    max_q_len=max(qlens), chunk=ch, v_dim=D, out_scale=1.2, out=joint[:, 64:])
            a0 = S.window_attention(q, kc, vc, bt, sl, qsl, pos, D ** -0.5, H, D, None, None, simt=True, chunk=ch,
                                    v_dim=D, out_scale=1.2)
            a2 = ref.window_attention(q, kc, vc, bt, sl, qsl, D ** -0.5, H, D, None, None, chunk=ch, v_dim=D,
                                      out_scale=1.2)
            assert close(a0, a2, 2e-2) and close(a1, a2, 2e-2), (D, ps, ch, qlens)
            assert joint[:, :64].abs().max().item() == 0


def test_grouped_gemm_experts_match_plain_experts():
    from gllm_b200.layers.moe import SelectedSoftmaxMoE
    torch.manual_seed(2)
    W, F, E = 384, 128, 8
    m = SelectedSoftmaxMoE(E, 2, W, F, torch.bfloat16, DEV)
    assert m.interleaved
    m.router_w.data.copy_(torch.randn(E, W) * 0.3)
    gates = [torch.randn(F, W) * W ** -0.5 for _ in range(E)]
    ups = [torch.randn(F, W) * W ** -0.5 for _ in range(E)]
    downs = [torch.randn(W, F) * F ** -0.5 for _ in range(E)]
    for e in range(E):
        m.load_expert(e, gates[e].bfloat16().to(DEV), ups[e].bfloat16().to(DEV), downs[e].bfloat16().to(DEV))
    h = torch.randn(150, W, device=DEV).bfloat16()
    got = m(h).float().cpu()
    hd = h.double().cpu()
    z = hd @ m.router_w.double().cpu().T
    val, idx = torch.topk(z, 2, -1)
    wt = torch.softmax(val, -1)
    want = torch.zeros(150, W, dtype=torch.float64)
    for t in range(150):
        for j in range(2):
            e = int(idx[t, j])
            g, u, d = gates[e].bfloat16().double(), ups[e].bfloat16().double(), downs[e].bfloat16().double()
            want[t] += wt[t, j] * (d @ (torch.nn.functional.silu(g @ hd[t]) * (u @ hd[t])))
    assert close(got, want.float(), 3e-2)


@pytest.fixture(scope="module")
def models():
    out = {}
    for i, (name, cfg) in enumerate(CONFIGS.items()):
        w = U.random_weights(cfg, seed=40 + i)
        out[name] = (cfg, w, U.save_model(cfg, w))
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(CONFIGS))
def test_whole_prompt_and_decoding(models, name, dtype):
    cfg, w, path = models[name]
    t = toks(45, cfg["vocab"], 1)
    ex = Expect(cfg, w, path, t, dtype)
    s = U.session(path, dtype, DEV)
    ex.check(U.run_chunks(s, "a", t, [len(t)]))
    ex.check(U.run_chunks(s, "b", t, [20]))
    ex.check(U.run_chunks(s, "c", t, [2, 2, 7, 1, 1, 13, 2]))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_mixed_batches_reuse_pages_and_slots(models, dtype):
    cfg, w, path = models["mixed"]
    v = cfg["vocab"]
    reqs = {k: toks(n, v, 20 + i) for i, (k, n) in enumerate([("a", 30), ("b", 9), ("c", 17), ("d", 2), ("e", 26),
                                                              ("f", 12)])}
    ex = {k: Expect(cfg, w, path, t, dtype) for k, t in reqs.items()}
    s = U.session(path, dtype, DEV, max_tokens=64, page_size=4, state_slots=3)
    plan = [[("a", 11), ("b", 9)], [("a", 1), ("c", 5)], [("a", 2), ("c", 1)], [("c", 11), ("a", 16), ("d", 2)],
            [("e", 3)], [("e", 1), ("f", 12)], [("e", 22)]]
    got = U.run_plan(s, reqs, plan)
    for k in reqs:
        ex[k].check(got[k])
    mm = s.scheduler.mm
    assert mm.get_num_free_state_slots() == 3 and mm.get_num_free_pages() == mm.usable_pages


@pytest.mark.parametrize("chunk,page_size", [(8, 4), (5, 4), (16, 16), (6, 8)])
def test_chunk_edges_on_the_kernels(chunk, page_size):
    for back in range(0, chunk + 2):
        want, outs, offset = _chunk_probe(chunk, page_size, back, DEV, torch.float32)
        for o in outs:
            assert torch.allclose(o, want, atol=1e-4, rtol=1e-4), (chunk, back)
        assert (outs[0][-1, 0].item() > 2.5) == (back <= offset)


def test_tensor_core_sized_model_in_bf16():
    """Head size 64 = value size, ff % 64 == 0, width % 128 == 0: tcgen05 GEMMs, tensor-core chunk attention and
    the grouped expert GEMMs carry the model; logits must stay within rounding of the oracle."""
    cfg = U.make_config([U.parallel(heads=4, kv_heads=2, dim=64, vdim=64, chunk=24, rot=32, rheads=2, rdim=32,
                                    rvdim=32, decay=(0.9, 0.99), mlp=U.moe(experts=8, top=2, ff=64)),
                         U.delta(heads=4, kv_heads=2, dim=32, vdim=32, mlp=U.dense(128))], width=128, vocab=96)
    w = U.random_weights(cfg, 5)
    path = U.save_model(cfg, w)
    t = toks(150, cfg["vocab"], 4)
    s = U.session(path, "bfloat16", DEV, max_tokens=512, page_size=16)
    ex = Expect(cfg, w, path, t, "bfloat16")
    ex.check(U.run_chunks(s, "a", t, [150]))
    ex.check(U.run_chunks(s, "b", t, [100, 30, 2]))
    # the same sizes without a router: every row within twice the rounding noise
    cfg2 = U.make_config([U.parallel(heads=4, kv_heads=2, dim=64, vdim=64, chunk=24, rot=32, rheads=2, rdim=32,
                                     rvdim=32, decay=(0.9, 0.99), mlp=U.dense(128)),
                          U.delta(heads=4, kv_heads=2, dim=32, vdim=32, mlp=U.dense(256))], width=128, vocab=96)
    w2 = U.random_weights(cfg2, 6)
    path2 = U.save_model(cfg2, w2)
    s2 = U.session(path2, "bfloat16", DEV, max_tokens=512, page_size=16)
    ex2 = Expect(cfg2, w2, path2, t, "bfloat16")
    ex2.check(U.run_chunks(s2, "a", t, [150]))
    ex2.check(U.run_chunks(s2, "b", t, [100, 30, 2]))


def test_greedy_generation_with_cuda_graphs(models):
    from gllm_b200.engine.llm_engine import LLM
    cfg, w, path = models["mixed"]
    llm = LLM(path, dtype="float32", page_size=4, maxp=16, maxd=8, num_gpu_pages=64, model_max_length=96,
              log_stats=False, num_state_slots=4, max_cuda_graph_bs=4)
    prompts = [toks(21, cfg["vocab"], 31), toks(3, cfg["vocab"], 32), toks(9, cfg["vocab"], 33)]
    lens = [7, 12, 5]
    seqs = llm.generate(tokens=prompts, output_lens=lens, temperature=0.0, top_k=1)
    assert llm.worker.runner.stats["graph_steps"] > 0
    for p, n, s in zip(prompts, lens, seqs):
        cur = list(p)
        for _ in range(n):
            cur.append(int(oracle.forward(cfg, w, cur, torch.float64)[-1].argmax()))
        assert s.token_ids == cur


def _delta_exact(q, k, v, beta, a, neg_a, dt_bias, st, qsl, sl, H, G, D, V):
    """The delta rule token by token in float64."""
    f = lambda x: x.double().cpu()   # noqa: E731
    q, k, v, beta, a, neg_a, dt_bias, st = (f(x) for x in (q, k, v, beta, a, neg_a, dt_bias, st))
    out, ends = torch.empty(q.shape[0], H * V, dtype=torch.float64), st.clone()
    for s in range(len(sl)):
        q0, q1 = int(qsl[s]), int(qsl[s + 1])
        S = st[s].clone() if int(sl[s]) > q1 - q0 else torch.zeros(H, D, V, dtype=torch.float64)
        for t in range(q0, q1):
            qq, kk = (x[t].view(G, D) / torch.sqrt((x[t].view(G, D) ** 2).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
            qq, kk = (qq * D ** -0.5).repeat_interleave(H // G, 0), kk.repeat_interleave(H // G, 0)
            S = S * torch.exp(neg_a * torch.nn.functional.softplus(a[t] + dt_bias)).view(H, 1, 1)
            u = torch.sigmoid(beta[t]).view(H, 1) * (v[t].view(H, V) - torch.einsum("hdv,hd->hv", S, kk))
            S = S + kk.unsqueeze(-1) * u.unsqueeze(1)
            out[t] = torch.einsum("hdv,hd->hv", S, qq).reshape(-1)
        if q1 > q0:
            ends[s] = S
    return out, ends


@pytest.mark.parametrize("H,G,D,V", [(4, 2, 128, 128), (3, 3, 64, 72), (2, 1, 40, 8), (2, 2, 120, 136)])
@pytest.mark.parametrize("lens,ctx", [([1, 32, 31, 64, 65, 200], [5, 0, 9, 0, 70, 0]), ([130], [0]), ([33, 3], [1, 0]),
                                      ([16, 15, 24, 17], [0, 3, 7, 0]), ([16], [0])])
@pytest.mark.parametrize("decay", ["slow", "fast"])
def test_chunked_delta_rule(H, G, D, V, lens, ctx, decay):
    """Chunked against token-serial, both against float64 from the same bf16 inputs: tile edges, ragged and short portions
    (below 16 tokens the serial kernel takes them), carried state, decays that wipe the state. The chunked form keeps the
    serial one's accuracy (a fixed 2e-6 covers the few-token cases, where either is a handful of fp32 roundings)."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(D + len(lens))
    dev, t, n = "cuda", sum(lens), len(lens)
    qkv = torch.randn(t, 2 * G * D + H * V, device=dev).bfloat16()
    q, k, v = qkv[:, :G * D], qkv[:, G * D:2 * G * D], qkv[:, 2 * G * D:]
    ba = torch.randn(t, 2 * H, device=dev).bfloat16()
    beta, a = ba[:, :H], ba[:, H:]
    if decay == "fast":
        a[t // 2] = 300.0                       # one token whose decay is an exact zero
    neg_a = -torch.rand(H, device=dev) * (1.0 if decay == "slow" else 16.0)
    dt_bias = torch.full((H,), -4.0 if decay == "slow" else 0.5, device=dev)
    st0 = torch.randn(n, H, D, V, device=dev)
    qsl = torch.tensor([0] + lens, device=dev).cumsum(0).to(torch.int32)
    sl = torch.tensor([x + c for x, c in zip(lens, ctx)], device=dev, dtype=torch.int32)
    rs = torch.arange(n, device=dev, dtype=torch.int32)
    exact = _delta_exact(q, k, v, beta, a, neg_a, dt_bias, st0, qsl, sl, H, G, D, V)
    err = {}
    for name, mx in (("chunk", max(lens)), ("serial", None)):
        st = st0.clone()
        o = S.linear_state_scan(q, k, v, beta, a, neg_a, dt_bias, None, st, rs, sl, qsl, H, G, D, V, False, True, D ** -0.5,
                                True, max_q_len=mx)
        err[name] = [float((x.double().cpu() - e).norm() / e.norm()) for x, e in ((o, exact[0]), (st, exact[1]))]
    for c, s in zip(err["chunk"], err["serial"]):
        assert c <= max(1.2 * s, 2e-6), err


@pytest.mark.parametrize("lens", [[5], [20], [40], [5, 40]])
def test_delta_rule_with_a_bound_on_the_lengths(lens):
    """`max_q_len` may be larger than every portion: each portion is computed, by the kernel that its own length asks for."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(lens[0])
    dev, t, n, H, D, V = "cuda", sum(lens), len(lens), 2, 128, 64
    q, k, v = (torch.randn(t, H * w, device=dev).bfloat16() for w in (D, D, V))
    beta, a = (torch.randn(t, H, device=dev).bfloat16() for _ in range(2))
    neg_a, dt_bias = -torch.rand(H, device=dev), torch.zeros(H, device=dev)
    qsl = torch.tensor([0] + lens, device=dev).cumsum(0).to(torch.int32)
    sl, rs = torch.tensor(lens, device=dev, dtype=torch.int32), torch.arange(n, device=dev, dtype=torch.int32)
    got = []
    for bound in (max(lens), 1000):
        st = torch.zeros(n, H, D, V, device=dev)
        torch.full((t, H * V), 3.0, device=dev)              # what an unwritten output is likely to hold
        got.append((S.linear_state_scan(q, k, v, beta, a, neg_a, dt_bias, None, st, rs, sl, qsl, H, H, D, V, False, True, 1.0,
                                        True, max_q_len=bound), st))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and bool(got[0][1].abs().sum() > 0)


@pytest.mark.parametrize("what", ["v", "k", "q", "beta", "a"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("at", [0, 13, 30, 47, 70, 127])
def test_chunked_delta_rule_keeps_earlier_tokens_clean(what, value, at):
    """One element that is no number: the chunked form is finite exactly where the token-serial one is (the tokens before it, and
    for a value the other columns), with the same results there, and the state alike."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(at)
    dev, H, D, V, lens = "cuda", 2, 128, 72, [40, 150, 35]
    t, n = sum(lens), len(lens)
    x = {"q": torch.randn(t, H * D), "k": torch.randn(t, H * D), "v": torch.randn(t, H * V), "beta": torch.randn(t, H),
         "a": torch.randn(t, H)}
    row = lens[0] + at                                       # in the middle sequence
    x[what][row, H - 1 if what in ("beta", "a") else 5] = value
    x = {name: y.to(dev).bfloat16() for name, y in x.items()}
    neg_a, dt_bias = -torch.rand(H, device=dev) * 0.2, torch.zeros(H, device=dev)
    qsl = torch.tensor([0] + lens, device=dev).cumsum(0).to(torch.int32)
    sl, rs = torch.tensor([45, 150, 35], device=dev, dtype=torch.int32), torch.arange(n, device=dev, dtype=torch.int32)
    st0, got = torch.randn(n, H, D, V, device=dev), []
    for mx in (max(lens), None):
        st = st0.clone()
        got.append((S.linear_state_scan(x["q"], x["k"], x["v"], x["beta"], x["a"], neg_a, dt_bias, None, st, rs, sl, qsl, H, H,
                                        D, V, False, True, D ** -0.5, True, max_q_len=mx), st))
    for c, s in zip(*got):
        fin = torch.isfinite(s)
        assert torch.equal(torch.isfinite(c), fin)
        zero = torch.zeros_like(s)
        a, b = torch.where(fin, c, zero), torch.where(fin, s, zero)
        assert float((a - b).norm()) <= 2e-5 * float(b.norm())      # sums of some 150 tokens in fp32, in another order
    assert bool(torch.isfinite(got[0][0][:row]).all())


@pytest.mark.parametrize("state", [True, False])
@pytest.mark.parametrize("unit", [True, False])
def test_chunked_delta_rule_in_rounds_of_heads(state, unit, monkeypatch):
    """A workspace for two of three heads: rounds of two and one, each with its own strides, the same bits as all at once. Without
    a carried state, and without unit lengths; against the token-serial kernel (fp32 sums over some 100 tokens in another order)."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(3)
    dev, H, D, V, lens, ctx = "cuda", 3, 64, 40, [70, 5, 33, 128], [4, 0, 9, 0]
    t, n = sum(lens), len(lens)
    q, k, v = (torch.randn(t, H * w, device=dev) for w in (D, D, V))
    q, k, v = q.bfloat16(), (k if unit else k * D ** -0.5).bfloat16(), v.bfloat16()
    beta, a = (torch.randn(t, H, device=dev).bfloat16() for _ in range(2))
    neg_a, dt_bias = -torch.rand(H, device=dev), torch.zeros(H, device=dev)
    qsl = torch.tensor([0] + lens, device=dev).cumsum(0).to(torch.int32)
    sl = torch.tensor([x + c for x, c in zip(lens, ctx)], device=dev, dtype=torch.int32)
    rs = torch.randperm(n, device=dev).to(torch.int32)
    st0, got = torch.randn(n, H, D, V, device=dev), []
    slots, unit_bytes = t // 64 + n, S._L().gllm_delta_unit_bytes()
    for work, mx in ((1 << 28, max(lens)), (2 * slots * unit_bytes, max(lens)), (1 << 28, None)):
        monkeypatch.setattr(S, "_DELTA_WORK_BYTES", work)
        st = st0.clone()
        o = S.linear_state_scan(q, k, v, beta, a, neg_a, dt_bias, None, st if state else None, rs if state else None, sl, qsl, H, H,
                                D, V, False, unit, 0.3, True, max_q_len=mx)
        got.append((o, st))
    for whole, rounds, serial in zip(*got):
        assert torch.equal(whole, rounds)
        assert float((whole - serial).norm()) <= 1e-5 * float(serial.norm())
