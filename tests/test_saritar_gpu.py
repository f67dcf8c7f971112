"""Saritar on the sm_100a kernels: every kernel of csrc/seq against its unfused PyTorch form, and the engine
scenarios of test_saritar_cpu.py (chunking, mixed batches, page / slot re-use, generation, CUDA-graph decode) against
the plain oracle, in fp32 (tight) and bf16 (rounding-sized tolerance)."""
import numpy as np
import pytest
import torch

import saritar_oracle as oracle
import saritar_util as U
from test_saritar_cpu import CONFIGS, toks

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOLS = {"float32": 2e-4, "bfloat16": 6e-2}


def close(a, b, tol):
    return (a.float() - b.float()).abs().max().item() <= tol * (b.float().abs().max().item() + 1e-9)


@pytest.mark.parametrize("dt,tol", [(torch.float32, 2e-5), (torch.bfloat16, 2e-2)])
def test_kernels_against_unfused_ops(dt, tol):
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(0)
    T, W = 37, 200
    x = torch.randn(T, W, device=DEV)
    y, wp, wq = (torch.randn(*s, device=DEV).to(dt) for s in ((T, W), (W,), (W,)))
    add = torch.randn(T, W, device=DEV)
    x1, x2 = x.clone(), x.clone()
    assert close(S.resid_norm(x1, y, wp, add, wq, 1e-5, dt), ref.resid_norm(x2, y, wp, add, wq, 1e-5, dt), tol)
    assert close(x1, x2, 1e-5)
    x3 = x.clone()
    assert S.resid_norm(x3, y, wp, None, None, 1e-5, dt) is None and not torch.equal(x3, x)
    for m, k, n in ((45, 72, 50), (1, 10, 3), (130, 192, 768), (3, 384, 64), (70, 64, 192)):
        a, w = torch.randn(m, k, device=DEV).to(dt), torch.randn(n, k, device=DEV).to(dt)
        assert close(S.linear_any(a, w), (a.float() @ w.float().T).to(dt), tol), (m, k, n)
    for D, N, taps in ((48, 24, 4), (64, 16, 2), (8, 1, 1), (128, 40, 3)):
        H, G, ps, win = 6, 2, 16, 20
        qlens, ctx = [5, 1, 30], [17, 40, 0]
        Tt = sum(qlens)
        qsl = torch.tensor([0, 5, 6, 36], dtype=torch.int32, device=DEV)
        sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
        kshape = ref.kv_cache_shape(32, G, D, ps)
        kc, vc = torch.randn(kshape, device=DEV).to(dt), torch.randn(kshape, device=DEV).to(dt)
        bt = torch.randperm(31)[:12].reshape(3, 4).to(torch.int32).to(DEV)
        pos = torch.cat([torch.arange(c, c + q) for c, q in zip(ctx, qlens)]).to(torch.int32).to(DEV)
        seqi = torch.cat([torch.full((q,), i) for i, q in enumerate(qlens)]).to(DEV)
        slots = (bt[seqi, (pos // ps).long()] * ps + pos % ps).to(torch.int32)
        qk = torch.randn(Tt, (H + G) * D, device=DEV).to(dt)
        qn, kn = torch.randn(D, device=DEV).to(dt), torch.randn(D, device=DEV).to(dt)
        kc2, vc2 = kc.clone(), vc.clone()
        q1 = S.qk_norm_kv_write(qk, H, G, D, qn, kn, 1e-5, kc, vc, slots)
        q2 = ref.qk_norm_kv_write(qk, H, G, D, qn, kn, 1e-5, kc2, vc2, slots)
        assert close(q1, q2, tol) and close(kc, kc2, tol) and torch.equal(vc, vc2)
        sink = torch.randn(H, device=DEV)
        for wn, sk in ((win, sink), (None, None), (3, sink), (1, None)):
            a1 = S.window_attention(q2, kc2, vc2, bt, sl, qsl, pos, 0.2, H, D, wn, sk)
            a2 = ref.window_attention(q2, kc2, vc2, bt, sl, qsl, 0.2, H, D, wn, sk)
            assert close(a1, a2, tol), (D, wn)
        C, R = 100, 10
        xz = torch.randn(Tt, 2 * C, device=DEV).to(dt)
        cw, cb = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV)
        cs = torch.randn(5, max(taps - 1, 1), C, device=DEV).to(dt)
        cs2 = cs.clone()
        rs = torch.tensor([3, 0, 2], dtype=torch.int32, device=DEV)
        c1 = S.causal_conv_silu(xz, C, cw, cb, cs, rs, sl, qsl)
        c2 = ref.causal_conv_silu(xz, C, cw, cb, cs2, rs, sl, qsl)
        assert close(c1, c2, tol) and (taps == 1 or torch.equal(cs, cs2))
        proj, dtr = torch.randn(Tt, R + 2 * N, device=DEV).to(dt), torch.randn(Tt, C, device=DEV).to(dt)
        A, Dk, db = -torch.rand(C, N, device=DEV) * 2, torch.randn(C, device=DEV), torch.randn(C, device=DEV)
        ss = torch.randn(5, N, C, device=DEV)
        ss2 = ss.clone()
        y1 = S.selective_scan(c2, dtr, proj, xz, A, Dk, db, ss, rs, sl, qsl, C, N, R)
        y2 = ref.selective_scan(c2, dtr, proj, xz, A, Dk, db, ss2, rs, sl, qsl, C, N, R)
        assert close(y1, y2, tol) and close(ss, ss2, 1e-5)
        assert torch.equal(S.relu2(xz), ref.relu2(xz))


@pytest.mark.parametrize("dt,tol", [(torch.float32, 2e-5), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("N,C", [(16, 96), (24, 100), (8, 64), (40, 32)])
def test_scan_and_conv_on_long_chunks(dt, tol, N, C):
    """few long sequences take the 4-threads-per-channel scan"""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(2)
    qlens, ctx, R, taps = [70, 33], [0, 9], 6, 4
    Tt = sum(qlens)
    qsl = torch.tensor([0, 70, 103], dtype=torch.int32, device=DEV)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    rs = torch.tensor([1, 0], dtype=torch.int32, device=DEV)
    xz = torch.randn(Tt, 2 * C, device=DEV).to(dt)
    cw, cb = torch.randn(C, taps, device=DEV), torch.randn(C, device=DEV)
    cs = torch.randn(3, taps - 1, C, device=DEV).to(dt)
    cs2 = cs.clone()
    c1 = S.causal_conv_silu(xz, C, cw, cb, cs, rs, sl, qsl)
    c2 = ref.causal_conv_silu(xz, C, cw, cb, cs2, rs, sl, qsl)
    assert close(c1, c2, tol) and torch.equal(cs, cs2)
    proj, dtr = torch.randn(Tt, R + 2 * N, device=DEV).to(dt), torch.randn(Tt, C, device=DEV).to(dt)
    A, Dk, db = -torch.rand(C, N, device=DEV) * 2, torch.randn(C, device=DEV), torch.randn(C, device=DEV)
    ss = torch.randn(3, N, C, device=DEV)
    ss2 = ss.clone()
    y1 = S.selective_scan(c2, dtr, proj, xz, A, Dk, db, ss, rs, sl, qsl, C, N, R)
    y2 = ref.selective_scan(c2, dtr, proj, xz, A, Dk, db, ss2, rs, sl, qsl, C, N, R)
    assert close(y1, y2, tol) and close(ss, ss2, 1e-5)


@pytest.mark.parametrize("D", [64, 128])
def test_window_and_sink_on_the_tensor_core_attention(D):
    """decode rows first, then prompt portions; contexts over several 64-key tiles; windows that end inside, at
    and beyond tile and page borders."""
    from gllm_b200.ops import ref, sm100_seq as S
    torch.manual_seed(1)
    bf, H, G, ps = torch.bfloat16, 8, 2, 16
    qlens, ctx = [1, 1, 1, 70, 5, 200], [0, 63, 300, 130, 64, 0]
    B, Tt = len(qlens), sum(qlens)
    qsl = torch.tensor([0] + torch.tensor(qlens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    npp = 20
    bt = torch.randperm(B * npp)[: B * npp].reshape(B, npp).to(torch.int32).to(DEV)
    kshape = ref.kv_cache_shape(B * npp + 1, G, D, ps)
    kc, vc = torch.randn(kshape, device=DEV).to(bf), torch.randn(kshape, device=DEV).to(bf)
    pos = torch.cat([torch.arange(c, c + q) for c, q in zip(ctx, qlens)]).to(torch.int32).to(DEV)
    q = torch.randn(Tt, H * D, device=DEV).to(bf)
    sink = torch.randn(H, device=DEV) * 2
    for wn, sk in ((72, sink), (64, sink), (65, None), (1, sink), (16, None), (None, sink), (None, None), (250, sink)):
        want = ref.window_attention(q, kc, vc, bt, sl, qsl, D ** -0.5, H, D, wn, sk)
        got = S.window_attention(q, kc, vc, bt, sl, qsl, pos, D ** -0.5, H, D, wn, sk, num_decode_seqs=3,
                                 max_q_len=max(qlens))
        plain = S.window_attention(q, kc, vc, bt, sl, qsl, pos, D ** -0.5, H, D, wn, sk, simt=True)
        assert close(got, want, 2e-2), (D, wn, sk is not None)
        assert close(plain, want, 2e-2), (D, wn, sk is not None)


@pytest.fixture(scope="module")
def models():
    out = {}
    for i, (name, cfg) in enumerate(CONFIGS.items()):
        w = U.random_weights(cfg, seed=10 + i)
        out[name] = (cfg, w, U.save_model(cfg, w))
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(CONFIGS))
def test_chunked_and_decoded_match_oracle(models, name, dtype):
    cfg, w, path = models[name]
    t = toks(45, cfg["vocab"], 2)
    want = U.expected_logits(cfg, w, t)
    s = U.session(path, dtype=dtype, device=DEV)
    for k, cuts in enumerate(([len(t)], [], [2, 2, 3, 17, 2], [30])):
        assert U.rel_err(U.run_chunks(s, "r%d" % k, t, cuts), want) < TOLS[dtype], cuts


def test_engine_on_the_tensor_core_attention_path():
    cfg = U.make_config([U.with_mlp(U.attn(heads=4, kv_heads=2, dim=64, window=40, scale=0.125), ff=96),
                         U.mamba(inner=64, state=16, dt_rank=8, conv=4),
                         U.attn(heads=2, kv_heads=1, dim=128, window=70, scale=0.09)], width=64, loop=(0, 2, 2))
    w = U.random_weights(cfg, seed=77)
    path = U.save_model(cfg, w)
    t = toks(150, cfg["vocab"], 4)
    want = U.expected_logits(cfg, w, t)
    s = U.session(path, dtype="bfloat16", device=DEV, max_tokens=512, page_size=16)
    for k, cuts in enumerate(([len(t)], [100] + [1] * 50, [2, 62, 3, 64, 17, 2])):
        assert U.rel_err(U.run_chunks(s, "r%d" % k, t, cuts), want) < TOLS["bfloat16"], cuts


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_mixed_batches_reuse_pages_and_slots(models, dtype):
    cfg, w, path = models["mixed_loop"]
    v = cfg["vocab"]
    reqs = {k: toks(n, v, 20 + i) for i, (k, n) in enumerate([("a", 30), ("b", 9), ("c", 17), ("d", 2), ("e", 26), ("f", 12)])}
    want = {k: U.expected_logits(cfg, w, t) for k, t in reqs.items()}
    s = U.session(path, dtype=dtype, device=DEV, max_tokens=64, page_size=4, state_slots=3)
    at, got = {k: 0 for k in reqs}, {k: [] for k in reqs}
    plan = [[("a", 11), ("b", 9)], [("a", 1), ("c", 5)], [("a", 2), ("c", 1)], [("c", 11), ("a", 16), ("d", 2)],
            [("e", 3)], [("e", 1), ("f", 12)], [("e", 22)]]
    for step in plan:
        entries, end = [], []
        for k, n in step:
            entries.append({"id": k, "tokens": reqs[k][at[k]:at[k] + n], "want": list(range(n))})
            at[k] += n
            if at[k] == len(reqs[k]):
                end.append(k)
        out, o = s.step(entries, end), 0
        for k, n in step:
            got[k].append(out[o:o + n])
            o += n
    for k in reqs:
        assert U.rel_err(np.concatenate(got[k], 0), want[k]) < TOLS[dtype], k


@pytest.mark.parametrize("graphs", [False, True])
def test_greedy_generation_on_the_gpu(models, graphs):
    from gllm_b200.engine.llm_engine import LLM
    cfg, w, path = models["mixed_loop"]
    llm = LLM(path, dtype="float32", page_size=4, maxp=32, maxd=8, num_gpu_pages=64, model_max_length=96,
              log_stats=False, num_state_slots=3, disable_cuda_graph=not graphs, max_cuda_graph_bs=4)
    prompts = [toks(21, cfg["vocab"], 31), toks(3, cfg["vocab"], 32), toks(9, cfg["vocab"], 33)]
    lens = [7, 12, 5]
    seqs = llm.generate(tokens=prompts, output_lens=lens, temperature=0.0, top_k=1)
    if graphs:
        assert llm.worker.runner.stats["graph_steps"] > 0
    for p, n, s in zip(prompts, lens, seqs):
        cur = list(p)
        for _ in range(n):
            cur.append(int(oracle.forward(cfg, w, cur, torch.float64)[-1].argmax()))
        assert s.token_ids == cur


@pytest.mark.parametrize("N,C", [(16, 130), (5, 64), (12, 257)])
@pytest.mark.parametrize("qlens,ctx", [([1, 128, 127, 129, 300], [4, 0, 2, 66, 0]), ([193], [0])])
def test_scan_cut_in_time(N, C, qlens, ctx, monkeypatch):
    """Portions of 128 tokens and more in pieces of 64; both forms against float64 from the same fp32 inputs. The cut form adds
    one product of a summed decay per piece and no other rounding: as accurate as the serial form."""
    from gllm_b200.ops import sm100, sm100_seq as S
    monkeypatch.setattr(S, "scan_piece", lambda *a: 64)
    monkeypatch.setattr(S, "_SCAN_UNCUT", 127)
    torch.manual_seed(N + len(qlens))
    R, t, n = 6, sum(qlens), len(qlens)
    qsl = torch.tensor([0] + qlens, device=DEV).cumsum(0).to(torch.int32)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    rs = torch.randperm(n + 2, device=DEV)[:n].to(torch.int32)
    x, dtr, xz = (torch.randn(t, w, device=DEV) for w in (C, C, 2 * C))
    proj = torch.randn(t, R + 2 * N, device=DEV)
    A, Dk, db = -torch.rand(C, N, device=DEV) * 4, torch.randn(C, device=DEV), torch.full((C,), -3.0, device=DEV)
    st0 = torch.randn(n + 2, N, C, device=DEV)
    xd, dtd, zd, pd, Ad, Dd, dbd, sd = (v.double().cpu() for v in (x, dtr, xz[:, C:], proj, A, Dk, db, st0))
    want, ends = torch.empty(t, C, dtype=torch.float64), sd.clone()
    for s in range(n):
        a, b, slot = int(qsl[s]), int(qsl[s + 1]), int(rs[s])
        h = sd[slot].t().clone() if ctx[s] else torch.zeros(C, N, dtype=torch.float64)
        for i in range(a, b):
            step = torch.nn.functional.softplus(dtd[i] + dbd)
            h = torch.exp(step[:, None] * Ad) * h + (step * xd[i])[:, None] * pd[i, R:R + N]
            want[i] = (h @ pd[i, R + N:] + Dd * xd[i]) * torch.nn.functional.silu(zd[i])
        ends[slot] = h.t()
    err = []
    for mx, launches in ((max(qlens), 3), (None, 1)):
        st, before = st0.clone(), sm100.launches()
        y = S.selective_scan(x, dtr, proj, xz, A, Dk, db, st, rs, sl, qsl, C, N, R, max_q_len=mx)
        assert sm100.launches() - before == launches
        err.append([float((g.double().cpu() - e).norm() / e.norm()) for g, e in ((y, want), (st, ends))])
    for cut, serial in zip(*err):
        assert cut <= max(1.2 * serial, 1e-6), err


@pytest.mark.parametrize("lens,cut", [([5], False), ([100], False), ([100, 130], False), ([400, 400], True), ([300, 7, 128, 400], True)])
def test_scan_with_a_bound_on_the_lengths(lens, cut):
    """`max_q_len` may be larger than every portion: each portion is computed, also where the bound makes the batch one that is cut.
    Portions of up to 128 tokens are walked whole in both: the same state bit for bit; longer ones within fp32 roundings (2^-23 a
    token); outputs within one bf16 rounding."""
    from gllm_b200.ops import sm100, sm100_seq as S
    torch.manual_seed(lens[0])
    N, C, R, t, n = 8, 70, 4, sum(lens), len(lens)
    qsl = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    sl, rs = torch.tensor(lens, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
    x, dtr, xz = (torch.randn(t, w, device=DEV).bfloat16() for w in (C, C, 2 * C))
    proj = torch.randn(t, R + 2 * N, device=DEV).bfloat16()
    A, Dk, db = -torch.rand(C, N, device=DEV) * 4, torch.randn(C, device=DEV), torch.full((C,), -3.0, device=DEV)
    got = []
    for bound, launches in ((max(lens), 1), (1000, 3 if cut else 1)):
        st, before = torch.zeros(n, N, C, device=DEV), sm100.launches()
        torch.full((t, C), 3.0, device=DEV).bfloat16()       # what an unwritten output is likely to hold
        got.append((S.selective_scan(x, dtr, proj, xz, A, Dk, db, st, rs, sl, qsl, C, N, R, max_q_len=bound), st))
        assert sm100.launches() - before == launches
    (a, sa), (b, sb) = got
    for s, m in enumerate(lens):
        assert bool(sa[s].abs().sum() > 0)
        assert torch.equal(sa[s], sb[s]) if m <= 128 or not cut else float((sa[s] - sb[s]).norm() / sa[s].norm()) <= m * 2.0 ** -23
    # sums of eight terms in fp32, of either form's states, and a rounding of 2^-8 each
    assert bool(((a.float() - b.float()).abs() <= a.float().abs() * 2.0 ** -7 + 1e-5).all())


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("state", [True, False])
def test_scan_in_rounds_of_channels(dt, state, monkeypatch):
    """Portions cut in pieces of 64 with a workspace for 128 channels: rounds of 128, 128 and 1, the same bits as all at once; with and
    without a carried state, in fp32 and bf16. Against the token-serial kernel: fp32 sums in another order, and for bf16 outputs one
    rounding (2^-8)."""
    from gllm_b200.ops import sm100, sm100_seq as S
    monkeypatch.setattr(S, "scan_piece", lambda *a: 64)
    torch.manual_seed(5)
    N, C, R, qlens, ctx = 12, 257, 6, [150, 7, 129, 256], [4, 0, 0, 66]
    t, n = sum(qlens), len(qlens)
    qsl = torch.tensor([0] + qlens, device=DEV).cumsum(0).to(torch.int32)
    sl = torch.tensor([c + q for c, q in zip(ctx, qlens)], dtype=torch.int32, device=DEV)
    rs = torch.randperm(n, device=DEV).to(torch.int32)
    x, dtr, xz = (torch.randn(t, w, device=DEV).to(dt) for w in (C, C, 2 * C))
    proj = torch.randn(t, R + 2 * N, device=DEV).to(dt)
    A, Dk, db = -torch.rand(C, N, device=DEV) * 4, torch.randn(C, device=DEV), torch.full((C,), -3.0, device=DEV)
    st0, got = torch.randn(n, N, C, device=DEV), []
    for work, mx, launches in ((1 << 28, max(qlens), 3), (0, max(qlens), 9), (1 << 28, None, 1)):
        monkeypatch.setattr(S, "_SCAN_WORK_BYTES", work)
        st, before = st0.clone(), sm100.launches()
        o = S.selective_scan(x, dtr, proj, xz, A, Dk, db, st if state else None, rs if state else None, sl, qsl, C, N, R,
                             max_q_len=mx)
        assert sm100.launches() - before == launches
        got.append((o, st))
    for (whole, rounds, serial), tol in zip(zip(*got), (1e-5 if dt == torch.float32 else 2.0 ** -8, 1e-5)):
        assert torch.equal(whole, rounds)
        assert float((whole.float() - serial.float()).norm()) <= tol * float(serial.float().norm())


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,C", [(16, 128), (16, 2176), (9, 65), (8, 64), (3, 34), (1, 7)])
@pytest.mark.parametrize("piece", [None, 16, 40])
def test_scan_walk_against_float64(dt, N, C, piece, monkeypatch):
    """Portions around the 16 tokens between two barriers, whole and cut in pieces, with two and four lanes per channel (2176
    channels fill the machine), steps from 0 (inputs of -60) to 60. fp32: a state keeps at most max(len) rounded sums of relative
    error 2^-23 each; bf16 outputs are rounded once (2^-8), their inputs are exact in float64."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(N)
    lens, ctx, R = [1, 15, 16, 17, 0, 33, 100, 2] + [20] * (16 if C > 2000 else 0), [4, 0, 3, 0, 0, 66, 1, 0] + [0] * 16, 5
    lens, ctx = [n for n in lens if n], [c for n, c in zip(lens, ctx) if n]
    t, n = sum(lens), len(lens)
    qsl = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    sl = torch.tensor([a + b for a, b in zip(lens, ctx)], dtype=torch.int32, device=DEV)
    rs = torch.randperm(n, device=DEV).to(torch.int32)
    x, dtr, xz = (torch.randn(t, w, device=DEV).to(dt) for w in (C, C, 2 * C))
    dtr[0, 0], dtr[1, C - 1], dtr[-1, 0] = 60.0, -60.0, 20.5
    proj = torch.randn(t, R + 2 * N, device=DEV).to(dt)
    A, Dk, db = -torch.rand(C, N, device=DEV) * 4, torch.randn(C, device=DEV), torch.full((C,), -3.0, device=DEV)
    st0 = torch.randn(n, N, C, device=DEV)
    if piece:
        monkeypatch.setattr(S, "scan_piece", lambda *a: piece)
        monkeypatch.setattr(S, "_SCAN_UNCUT", 0)
    st = st0.clone()
    got = S.selective_scan(x, dtr, proj, xz, A, Dk, db, st, rs, sl, qsl, C, N, R, max_q_len=max(lens))
    want, ends, at = torch.empty(t, C, dtype=torch.float64, device=DEV), st0.double(), 0
    for i, q in enumerate(lens):
        h = st0[rs[i]].double() if ctx[i] else torch.zeros(N, C, dtype=torch.float64, device=DEV)
        for k in range(at, at + q):
            s = torch.nn.functional.softplus(dtr[k].double() + db.double(), threshold=50)
            h = torch.exp(s * A.double().t()) * h + (s * x[k].double()) * proj[k, R:R + N].double()[:, None]
            y = (h * proj[k, R + N:].double()[:, None]).sum(0) + Dk.double() * x[k].double()
            want[k] = y * torch.nn.functional.silu(xz[k, C:].double())
        ends[rs[i]] = h
        at += q
    bound = max(lens) * 2.0 ** -23
    assert float((st.double() - ends).norm() / ends.norm()) < bound
    assert float((got.double() - want).norm() / want.norm()) < bound + (2.0 ** -8 if dt == torch.bfloat16 else 0)


@pytest.mark.parametrize("lo,hi", [(-20, -10), (-7, -3), (-3, 3), (3, 25), (-100, -80)])
def test_scan_steps_and_gates_one_by_one(lo, hi):
    """Portions of one token from empty states with x = B = 1, C = 0, D = 1: the states are softplus(dt), the outputs silu(z). The 2^x
    unit is within 2^-22 (2 ulp; twice that where it squares a result to reach denormals, below -87), two to three further roundings of
    2^-24 each; in the denormals their spacing. Infinities and NaN as the token-serial kernel has them."""
    from gllm_b200.ops import sm100_seq as S
    n, C, N = 40, 1030, 3
    torch.manual_seed(hi)
    v = torch.rand(n, C, device=DEV) * (hi - lo) + lo
    v[3, :5] = torch.tensor([float("inf"), -float("inf"), float("nan"), 0.0, -0.0], device=DEV)
    proj = torch.cat([torch.ones(n, N, device=DEV), torch.zeros(n, N, device=DEV)], 1)
    qsl, ones = torch.arange(n + 1, device=DEV, dtype=torch.int32), torch.ones(n, C, device=DEV)
    got = []
    for mx in (2, None):
        st = torch.empty(n, N, C, device=DEV)
        y = S.selective_scan(ones, v, proj, torch.cat([ones, v], 1), -torch.rand(C, N, device=DEV), ones[0], torch.zeros(C, device=DEV), st,
                             qsl[:n], qsl[:n] * 0 + 1, qsl, C, N, 0, max_q_len=mx)
        got.append((st[:, N - 1], y))
    d = v.double()
    for one, serial, want in zip(*got, (torch.logaddexp(d, torch.zeros_like(d)), d * torch.sigmoid(d))):
        fine = torch.isfinite(d)
        assert bool(((one.double() - want).abs() <= want.abs() * 2.0 ** (-21.4 if lo > -80 else -20.4) + 2.0 ** -148 * (1 + d.abs()))[fine].all())
        assert torch.equal(torch.nan_to_num(one[3, :3], 7.0, 8.0, 9.0), torch.nan_to_num(serial[3, :3], 7.0, 8.0, 9.0))


@pytest.mark.parametrize("lens,C", [([2048] * 4, 1024), ([600, 130], 96)])
def test_scan_states_that_decay_slowly(lens, C):
    """Decays around 0.9999 to 0.99 over whole portions. Against float64: the 2^x unit's errors (at most 2^-23 in a token, of one
    sign) add up over 64 tokens and not over the portion."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(C)
    N, t, n = 16, sum(lens), len(lens)
    qsl = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    sl, rs = torch.tensor(lens, dtype=torch.int32, device=DEV) + 1, torch.arange(n, dtype=torch.int32, device=DEV)
    steps = 10.0 ** -torch.linspace(2, 4, C, device=DEV, dtype=torch.float64)
    raw = torch.log(torch.expm1(steps * (0.8 + 0.4 * torch.rand(t, C, device=DEV)))).float()
    x, xz = torch.randn(t, C, device=DEV), torch.randn(t, 2 * C, device=DEV)
    proj, st0 = torch.randn(t, 2 * N, device=DEV), torch.randn(n, N, C, device=DEV)
    A, st = -(0.5 + torch.rand(C, N, device=DEV)), st0.clone()
    S.selective_scan(x, raw, proj, xz, A, torch.zeros(C, device=DEV), torch.zeros(C, device=DEV), st, rs, sl, qsl, C, N, 0, max_q_len=max(lens))
    for s in range(n):
        h = st0[s].double()
        for k in range(int(qsl[s]), int(qsl[s + 1])):
            dt = torch.nn.functional.softplus(raw[k].double())
            h = torch.exp(dt * A.double().t()) * h + (dt * x[k].double()) * proj[k, :N].double()[:, None]
        err = (st[s].double() - h).norm(dim=0) / h.norm(dim=0)              # per channel
        assert float(err.max()) <= 64 * 2.0 ** -23, float(err.max())


@pytest.mark.parametrize("L", [1, 5, 64, 70])
def test_scan_with_infinite_rates(L):
    """A = -inf forgets everything at every step, also in portions that end inside a group of four tokens."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(L)
    N, C, i32 = 3, 40, torch.int32
    A = -torch.rand(C, N, device=DEV)
    A[::3] = -float("inf")
    x, raw, xz, proj = (torch.randn(L, w, device=DEV) for w in (C, C, 2 * C, 2 * N))
    z, st = torch.zeros(C, device=DEV), torch.randn(1, N, C, device=DEV)
    y = S.selective_scan(x, raw, proj, xz, A, z, z, st, torch.zeros(1, dtype=i32, device=DEV), torch.tensor([L + 1], dtype=i32, device=DEV),
                         torch.tensor([0, L], dtype=i32, device=DEV), C, N, 0, max_q_len=max(L, 2))
    dx = torch.nn.functional.softplus(raw.double()) * x.double()
    want = dx[:, None, ::3] * proj[:, :N, None].double()                    # [token, state, channel]
    assert bool(((st[0, :, ::3].double() - want[-1]).abs() <= want[-1].abs() * 2.0 ** -20).all())
    out = (want * proj[:, N:, None].double()).sum(1) * torch.nn.functional.silu(xz[:, C::3].double())
    assert bool(((y[:, ::3].double() - out).abs() <= 2.0 ** -20 * (want.abs() * proj[:, N:, None].abs()).sum(1) * 20).all())
    assert bool(torch.isfinite(y).all()) and bool(torch.isfinite(st).all())


@pytest.mark.parametrize("N,C", [(16, 96), (5, 2048)])
def test_scan_of_a_short_portion_beside_a_long_one(N, C):
    """Portions of up to 128 tokens alone, and beside one that is cut in pieces: the same states bit for bit, outputs of the same terms
    (at most 16, 2^-23 each for the order of the sum)."""
    from gllm_b200.ops import sm100_seq as S
    torch.manual_seed(C)
    lens, R = [100, 1500, 128, 1, 7], 3
    t, n = sum(lens), len(lens)
    assert S.scan_piece(t, 1500, C) < 128 and S.scan_piece(128, 128, C) == 128
    qsl = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    rs, sl = torch.arange(n, dtype=torch.int32, device=DEV), torch.tensor(lens, dtype=torch.int32, device=DEV) + 1
    x, raw, xz, proj = (torch.randn(t, w, device=DEV) for w in (C, C, 2 * C, R + 2 * N))
    A, z, st0 = -torch.rand(C, N, device=DEV), torch.zeros(C, device=DEV), torch.randn(n, N, C, device=DEV)
    st = st0.clone()
    y = S.selective_scan(x, raw, proj, xz, A, z, z, st, rs, sl, qsl, C, N, R, max_q_len=1500)
    for s in (0, 2, 3, 4):
        a, b, one = int(qsl[s]), int(qsl[s + 1]), st0[s:s + 1].clone()
        ys = S.selective_scan(x[a:b], raw[a:b], proj[a:b], xz[a:b], A, z, z, one, rs[:1], sl[s:s + 1], qsl[s:s + 2] - a, C, N, R, max_q_len=128)
        assert torch.equal(one[0], st[s])
        most = torch.nn.functional.silu(xz[a:b, C:]).abs() * (y[a:b].abs() + 16 * 30)         # |state| |C| below 30
        assert bool(((ys - y[a:b]).abs() <= 2.0 ** -20 * most).all())
