"""Numerics of every sm_100a kernel against the plain-PyTorch fp32 reference of the
same op (monarch_b200.ops.reference)."""
import pytest
import torch

from monarch_b200 import ops
from monarch_b200.ops import kernels as K
from monarch_b200.ops import reference as R

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    torch.cuda.synchronize()
    K.check_status()


@pytest.fixture(params=[1, 2], ids=["cta1", "cta_pair"])
def gemm_impl(request):
    """Run the test under both GEMM kernels (single-CTA tiles and cta_group::2 pairs)."""
    before = K.gemm_impl()
    K.set_gemm_impl(request.param)
    yield request.param
    K.set_gemm_impl(before)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K_", [(128, 256, 64), (256, 512, 256), (384, 768, 1024),
                                    (304, 520, 200), (8, 24, 72), (1024, 4096, 4096)])
def test_gemm_matches_fp32(gemm_impl, a_mn, b_mn, M, N, K_):
    torch.manual_seed(0)
    a = torch.randn((K_, M) if a_mn else (M, K_), device="cuda", dtype=bf16)
    b = torch.randn((K_, N) if b_mn else (N, K_), device="cuda", dtype=bf16)
    c = ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    ref = R.gemm(a, b, a_mn, b_mn)
    assert c.shape == (M, N)
    assert _rel(c, ref) < 5e-3, _rel(c, ref)


def test_gemm_residual_and_accumulate(gemm_impl):
    torch.manual_seed(1)
    M, N, K_ = 512, 1024, 512
    a = torch.randn(M, K_, device="cuda", dtype=bf16)
    b = torch.randn(N, K_, device="cuda", dtype=bf16)
    r = torch.randn(M, N, device="cuda", dtype=bf16)
    c = ops.gemm(a, b, residual=r)
    assert _rel(c, R.gemm(a, b, residual=r)) < 5e-3
    c0 = torch.randn(M, N, device="cuda", dtype=bf16)
    c1 = c0.clone()
    ops.gemm(a, b, out=c1, accumulate=True)
    assert _rel(c1, R.gemm(a, b, accumulate_into=c0)) < 5e-3


def test_gemm_strided_views(gemm_impl):
    torch.manual_seed(2)
    big = torch.randn(512, 1024, device="cuda", dtype=bf16)
    a = big[:, 256:768]           # [512, 512], ld 1024
    b = torch.randn(256, 512, device="cuda", dtype=bf16)
    out_big = torch.zeros(512, 512, device="cuda", dtype=bf16)
    out = out_big[:, 128:384]
    ops.gemm(a, b, out=out)
    assert _rel(out, R.gemm(a, b)) < 5e-3
    assert out_big[:, :128].abs().max() == 0 and out_big[:, 384:].abs().max() == 0


def test_gemm_many_tiles_persistent(gemm_impl):
    # more tiles than SMs: exercises the persistent loop and TMEM double buffering
    torch.manual_seed(3)
    M, N, K_ = 4096, 4096, 512
    a = torch.randn(M, K_, device="cuda", dtype=bf16)
    b = torch.randn(N, K_, device="cuda", dtype=bf16)
    c = ops.gemm(a, b)
    ref = (a.float() @ b.float().t())
    assert _rel(c, ref) < 5e-3


@pytest.mark.parametrize("rows,d", [(64, 256), (1000, 2048), (512, 4096), (33, 8192)])
def test_rmsnorm(rows, d):
    torch.manual_seed(0)
    x = torch.randn(rows, d, device="cuda", dtype=bf16)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(bf16)
    y, rstd = ops.rmsnorm_fwd(x, w, 1e-5)
    yr, rstdr = R.rmsnorm_fwd(x, w, 1e-5)
    assert _rel(y, yr) < 5e-3 and _rel(rstd, rstdr) < 1e-5
    dy = torch.randn(rows, d, device="cuda", dtype=bf16)
    dres = torch.randn(rows, d, device="cuda", dtype=bf16)
    dw = torch.zeros(d, device="cuda", dtype=bf16)
    dx = ops.rmsnorm_bwd(dy, x, w, rstd, dw, dres=dres)
    dxr, dwr = R.rmsnorm_bwd(dy, x, w, rstdr)
    assert _rel(dx, dxr + dres.float()) < 6e-3
    assert _rel(dw, dwr) < 6e-3
    # second call reuses the scratch buffer and accumulates
    ops.rmsnorm_bwd(dy, x, w, rstd, dw, accumulate=True)
    assert _rel(dw, 2 * dwr) < 1e-2


def test_rope_forward_inverse():
    torch.manual_seed(0)
    S, Hq, Hkv, hd, B = 64, 4, 2, 128, 2
    cos, sin = R.rope_tables(S, hd, 500000.0, device="cuda")
    qkv = torch.randn(B * S, (Hq + 2 * Hkv) * hd, device="cuda", dtype=bf16)
    orig = qkv.clone()
    ops.rope_(qkv, cos, sin, S, Hq + Hkv, hd)
    ref = R.rope(orig[:, : (Hq + Hkv) * hd].float().reshape(B * S, Hq + Hkv, hd), cos, sin, S)
    assert _rel(qkv[:, : (Hq + Hkv) * hd], ref.reshape(B * S, -1)) < 5e-3
    assert torch.equal(qkv[:, (Hq + Hkv) * hd:], orig[:, (Hq + Hkv) * hd:])
    ops.rope_(qkv, cos, sin, S, Hq + Hkv, hd, inverse=True)
    assert _rel(qkv, orig) < 1e-2


def test_swiglu():
    torch.manual_seed(0)
    gu = torch.randn(300, 2 * 1024, device="cuda", dtype=bf16)
    dh = torch.randn(300, 1024, device="cuda", dtype=bf16)
    assert _rel(ops.swiglu_fwd(gu), R.swiglu_fwd(gu)) < 5e-3
    assert _rel(ops.swiglu_bwd(gu, dh), R.swiglu_bwd(gu, dh)) < 5e-3


@pytest.mark.parametrize("rows,V", [(64, 512), (37, 32000), (16, 128256)])
def test_cross_entropy(rows, V):
    torch.manual_seed(0)
    logits = (3 * torch.randn(rows, V, device="cuda")).to(bf16)
    tg = torch.randint(0, V, (rows,), device="cuda")
    lr, gr = R.cross_entropy(logits, tg, 1.0 / rows)
    loss = ops.cross_entropy_(logits, tg, 1.0 / rows)
    assert torch.allclose(loss, lr, atol=2e-3, rtol=1e-3)
    assert _rel(logits, gr) < 1e-2


def test_adamw_matches_reference():
    torch.manual_seed(0)
    n = 100003
    p = torch.randn(n, device="cuda")
    m = torch.zeros(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    pb = torch.empty(n, device="cuda", dtype=bf16)
    pr, mr, vr = p.clone(), m.clone(), v.clone()
    for step in range(1, 4):
        g = torch.randn(n, device="cuda").to(bf16)
        ops.adamw_(p, m, v, g, pb, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, wd=0.1, step=step)
        pr, mr, vr = R.adamw(pr, mr, vr, g, 1e-2, 0.9, 0.95, 1e-8, 0.1, step)
    assert torch.allclose(p, pr, atol=1e-5) and torch.allclose(m, mr, atol=1e-6)
    assert torch.allclose(v, vr, atol=1e-6)
    assert torch.equal(pb, p.to(bf16))


def test_embedding():
    torch.manual_seed(0)
    table = torch.randn(1000, 256, device="cuda", dtype=bf16)
    ids = torch.randint(0, 1000, (777,), device="cuda")
    assert torch.equal(ops.embedding_fwd(table, ids), table[ids])
    dout = torch.randn(777, 256, device="cuda", dtype=bf16)
    dt = torch.zeros(1000, 256, device="cuda", dtype=bf16)
    ops.embedding_bwd_(dout, ids, dt)
    ref = torch.zeros(1000, 256, device="cuda").index_add_(0, ids, dout.float())
    assert _rel(dt, ref) < 1e-2


def test_sumsq():
    x = torch.randn(1 << 20, device="cuda", dtype=bf16)
    s = ops.sumsq(x)
    assert abs(s.item() - x.float().pow(2).sum().item()) / s.item() < 1e-3


def test_engine_gpu_matches_cpu_fp32():
    """The whole explicit step on the GPU kernels (bf16) against the same engine run with
    the fp32 CPU reference ops."""
    from monarch_b200.models import PRESETS, LlamaEngine, LocalParamStore, ParamLayout
    cfg = PRESETS["tiny"]
    layout = ParamLayout(cfg)
    g_st = LocalParamStore(layout, "cuda", seed=5, init_std=0.05)
    c_st = LocalParamStore(layout, "cpu", seed=5, init_std=0.05)
    c_st.master.copy_(g_st.master.cpu())
    c_st.params = g_st.params.cpu().float()
    c_st.grads = torch.zeros(layout.total)
    S = 128
    torch.manual_seed(0)
    tokens = torch.randint(0, cfg.vocab, (2, S))
    targets = torch.randint(0, cfg.vocab, (2, S))
    lg = LlamaEngine(cfg, g_st, S).forward_backward(tokens.cuda(), targets.cuda())
    lc = LlamaEngine(cfg, c_st, S).forward_backward(tokens, targets)
    assert abs(lg.item() - lc.item()) < 3e-2, (lg.item(), lc.item())
    assert _rel(g_st.grads.cpu(), c_st.grads) < 5e-2, _rel(g_st.grads.cpu(), c_st.grads)
    assert K.launch_count > 0


def test_optimizer_overlapped_with_backward_is_bit_identical():
    """With the hyper-parameters known before backward the resident store updates every unit
    on a side stream right after its backward; the parameters after two steps equal, bit for
    bit, those of a store that runs one AdamW launch at the end of the step."""
    from monarch_b200.models import PRESETS, LlamaEngine, LocalParamStore, ParamLayout
    for preset in ("tiny", "tiny-tied"):
        cfg = PRESETS[preset]
        layout = ParamLayout(cfg)
        S = 128
        g = torch.Generator().manual_seed(3)
        # no token twice within a batch: the embedding backward adds rows atomically, and
        # only then is the order of the additions irrelevant to the last bit
        toks = torch.stack([torch.randperm(cfg.vocab, generator=g)[: 2 * S].reshape(2, S)
                            for _ in range(3)]).cuda()
        a_st = LocalParamStore(layout, "cuda", seed=5, init_std=0.05)
        b_st = LocalParamStore(layout, "cuda", seed=5, init_std=0.05)
        ea, eb = LlamaEngine(cfg, a_st, S), LlamaEngine(cfg, b_st, S)
        for step in range(2):
            a_st.set_hyper(lr=1e-2)
            la = ea.forward_backward(toks[step], toks[step + 1])
            assert a_st._updated_units == len(layout.units)
            ea.optimizer_step(1e-2)
            lb = eb.forward_backward(toks[step], toks[step + 1])
            eb.optimizer_step(1e-2)
            torch.cuda.synchronize()
            assert float(la) == float(lb)
        assert torch.equal(a_st.params, b_st.params) and torch.equal(a_st.master, b_st.master)
        assert torch.equal(a_st.m, b_st.m) and torch.equal(a_st.v, b_st.v)
        assert a_st.step_count == b_st.step_count == 2


# (M, N, K): what each tile of the plain product covers -- 128x64 and its splits (few rows, long
# K; fewer rows and columns than a tile; remainders in M, N and K), 128x128 and its splits in 2, 4
# and 8 parts, 128x256, the CTA pair, one row, and a K beyond 20000
GEMM_SHAPES = [(200, 768, 256), (1, 264, 4096), (64, 512, 4104), (96, 4096, 4096), (8, 24, 1032),
               (333, 1496, 1096), (1000, 2048, 1544), (257, 6144, 1024), (2048, 2048, 2056),
               (8, 8200, 2056), (24, 1496, 8200), (100, 1032, 20008), (2040, 4104, 1096),
               (250, 12008, 264)]


def test_gemm_shapes_reach_every_tile_and_split():
    plans = {K.gemm_plan(M, N, K_, K_, K_, N + 8) for M, N, K_ in GEMM_SHAPES}
    assert plans == {(0, 1), (256, 1), (128, 1), (128, 2), (128, 4), (128, 8), (64, 1), (64, 2),
                     (64, 4), (64, 8)}


@pytest.mark.parametrize("M,N,K_", GEMM_SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_gemm_tile_choice(M, N, K_, a_mn, b_mn):
    """Every tile and split the product can choose, against 64 bits: the only rounding is that
    of the bf16 result (2^-9 at most, 1.7e-3 in the 2-norm) plus fp32 sums of K terms."""
    if a_mn and M % 8:
        M += 8 - M % 8
    torch.manual_seed(4)
    a = torch.randn((K_, M) if a_mn else (M, K_), device="cuda", dtype=bf16)
    b = torch.randn((K_, N) if b_mn else (N, K_), device="cuda", dtype=bf16)
    r = torch.randn(M, N, device="cuda", dtype=bf16)
    wide = torch.full((M, N + 8), 7.0, device="cuda", dtype=bf16)
    ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=wide[:, :N], residual=r)
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double() + r.double()
    err = ((wide[:, :N].double() - ref).norm() / ref.norm()).item()
    assert err < 2.5e-3, err
    assert (wide[:, N:] == 7).all()
    first = wide[:, :N].clone()
    ops.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=wide[:, :N], accumulate=True)
    assert _rel(wide[:, :N], ref - r.double() + first.double()) < 2.5e-3


# one row, rows that leave the last block short, more rows than a ring has stages and than there
# are blocks; d: one chunk, a remainder of a warp's chunk, both sides of every variant's limit
@pytest.mark.parametrize("rows,d", [(1, 8), (5, 264), (3000, 512), (77, 2048), (700, 2056),
                                    (1201, 4096), (19, 4104), (333, 5120), (2, 8192)])
def test_rmsnorm_row_lengths(rows, d):
    torch.manual_seed(1)
    x = torch.randn(rows, d, device="cuda", dtype=bf16)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(bf16)
    dy = torch.randn(rows, d, device="cuda", dtype=bf16)
    dres = torch.randn(rows, d, device="cuda", dtype=bf16)
    y, rstd = ops.rmsnorm_fwd(x, w, 1e-5)
    yr, rstdr = R.rmsnorm_fwd(x.double(), w.double(), 1e-5)
    # bf16 results are off by their rounding (1.7e-3 in the 2-norm), rstd by fp32 sums
    assert _rel(y, yr) < 3e-3 and _rel(rstd, rstdr) < 1e-6
    for res in (dres, None):
        dw = torch.zeros(d, device="cuda", dtype=bf16)
        dx = ops.rmsnorm_bwd(dy, x, w, rstd, dw, dres=res)
        dxr, dwr = R.rmsnorm_bwd(dy, x, w, rstdr.float())
        assert _rel(dx, dxr if res is None else dxr + res.float()) < 3e-3
        assert _rel(dw, dwr) < 3e-3


def test_rmsnorm_fwd_longer_than_registers():
    x = torch.randn(3, 8200, device="cuda", dtype=bf16)
    w = torch.ones(8200, device="cuda", dtype=bf16)
    y, _ = ops.rmsnorm_fwd(x, w, 1e-5)
    assert _rel(y, R.rmsnorm_fwd(x, w, 1e-5)[0]) < 3e-3


# head sizes with 1, 4, 8, 32 threads per head and two that take the general kernel; heads that
# leave the last batch of a thread short
@pytest.mark.parametrize("hd,heads", [(16, 3), (64, 40), (128, 1), (128, 41), (512, 2), (1024, 2), (48, 5)])
@pytest.mark.parametrize("rows,S", [(7, 4), (130, 64)])
def test_rope_head_sizes(hd, heads, rows, S):
    torch.manual_seed(2)
    cos, sin = R.rope_tables(S, hd, 10000.0, device="cuda")
    x = torch.randn(rows, heads * hd + 16, device="cuda", dtype=bf16)
    before = x.clone()
    for inverse in (False, True):
        y = before.clone()
        ops.rope_(y, cos, sin, S, heads, hd, inverse=inverse)
        ref = R.rope(before[:, : heads * hd].float().reshape(rows, heads, hd), cos, sin, S, inverse)
        assert _rel(y[:, : heads * hd], ref.reshape(rows, -1)) < 3e-3
        assert torch.equal(y[:, heads * hd:], before[:, heads * hd:])


@pytest.mark.parametrize("rows,F", [(1, 8), (3, 264), (5, 2048), (2, 2056)])
def test_swiglu_row_lengths(rows, F):
    gu = torch.randn(rows, 2 * F, device="cuda", dtype=bf16)
    dh = torch.randn(rows, F, device="cuda", dtype=bf16)
    assert _rel(ops.swiglu_fwd(gu), R.swiglu_fwd(gu)) < 3e-3
    assert _rel(ops.swiglu_bwd(gu, dh), R.swiglu_bwd(gu, dh)) < 3e-3


# both sides of the block sizes' limits, and lengths with a scalar remainder
@pytest.mark.parametrize("V", [8, 513, 4096, 4100, 65536, 65541, 100003])
def test_cross_entropy_vocabularies(V):
    torch.manual_seed(3)
    rows, ld = 5, (V + 15) // 8 * 8
    wide = (3 * torch.randn(rows, ld, device="cuda")).to(bf16)
    rest = wide[:, V:].clone()
    tg = torch.tensor([0, V - 1, V // 2, 1, 7], device="cuda")
    lr, gr = R.cross_entropy(wide[:, :V], tg, 0.25)
    loss = ops.cross_entropy_(wide[:, :V], tg, 0.25)
    assert torch.allclose(loss, lr, atol=2e-4, rtol=1e-4)
    assert _rel(wide[:, :V], gr) < 3e-3
    assert torch.equal(wide[:, V:], rest)


# 16-byte reductions (d % 8 == 0), pairs for the others; every token once, then many of one
@pytest.mark.parametrize("d", [8, 250, 2056])
def test_embedding_bwd_widths(d):
    torch.manual_seed(4)
    ids = torch.randperm(300, device="cuda")[:200]
    dout = torch.randn(200, d, device="cuda", dtype=bf16)
    base = torch.randn(300, d, device="cuda", dtype=bf16)
    dt = base.clone()
    ops.embedding_bwd_(dout, ids, dt)
    ref = base.clone()
    ref[ids] += dout
    assert torch.equal(dt, ref)
    one = torch.zeros(3, d, device="cuda", dtype=bf16)
    ops.embedding_bwd_(torch.ones(100, d, device="cuda", dtype=bf16),
                       torch.full((100,), 1, device="cuda"), one)
    assert (one[1] == 100).all() and one[0].abs().max() == 0 and one[2].abs().max() == 0


# the fused tiles and their remainders in rows, K and (backward) F; F that takes the separate
# kernels (200 % 64, 24 % 32), products split along K, more than one wave of small tiles and K too
# long for them, pair tiles on both sides of the limits in K, in rows and in tiles
@pytest.mark.parametrize("T,F,K_", [(1, 64, 64), (256, 512, 256), (200, 384, 136), (300, 96, 72),
                                    (130, 2048, 128), (77, 200, 64), (50, 24, 64), (64, 512, 4096),
                                    (2049, 4096, 1024), (1100, 8192, 3080), (1030, 1024, 1088),
                                    (4097, 512, 256), (4100, 2048, 2568), (4100, 2048, 4104),
                                    (8200, 8192, 256)])
def test_gemm_swiglu_equals_the_separate_kernels(gemm_impl, T, F, K_):
    """The fused epilogues round where the separate kernels store, and the products add along K in
    the same order: the same bits."""
    torch.manual_seed(5)
    a = torch.randn(T, K_, device="cuda", dtype=bf16)
    w = (0.1 * torch.randn(2 * F, K_, device="cuda")).to(bf16)
    gu_ref = ops.gemm(a, w)
    h_ref = ops.swiglu_fwd(gu_ref)
    h, gu = ops.gemm_swiglu(a, w)
    assert torch.equal(gu, gu_ref) and torch.equal(h, h_ref)
    h2, none = ops.gemm_swiglu(a, w, keep_gu=False)
    assert none is None and torch.equal(h2, h)
    dy = torch.randn(T, K_, device="cuda", dtype=bf16)
    wd = (0.1 * torch.randn(K_, F, device="cuda")).to(bf16)
    ref = ops.swiglu_bwd(gu, ops.gemm(dy, wd, b_mn=True))
    assert torch.equal(ops.gemm_swiglu_bwd(dy, wd, gu), ref)


def test_rmsnorm_bwd_on_two_streams_shares_no_scratch(monkeypatch):
    """The partial weight-gradient sums of a call are read by its second kernel, while a call on
    another stream may already write its own."""
    lib, used = K.lib(), []

    class Recorder:
        def __getattr__(self, name):
            return getattr(lib, name)

        def mb200_rmsnorm_bwd(self, *args):
            used.append(args[6])
            return lib.mb200_rmsnorm_bwd(*args)

    monkeypatch.setattr(K, "lib", lambda: Recorder())
    x = torch.randn(64, 512, device="cuda", dtype=bf16)
    w = torch.ones(512, device="cuda", dtype=bf16)
    _, rstd = ops.rmsnorm_fwd(x, w, 1e-5)
    dw = torch.empty(2, 512, device="cuda", dtype=bf16)
    torch.cuda.synchronize()
    for i, st in enumerate((torch.cuda.Stream(), torch.cuda.Stream())):
        with torch.cuda.stream(st):
            ops.rmsnorm_bwd(x, x, w, rstd, dw[i])
    torch.cuda.synchronize()
    assert len(set(used)) == 2 and torch.equal(dw[0], dw[1])


def test_checkpointing_keeps_the_residual_stream_only_when_asked(monkeypatch):
    """What the forward has left when the loss is computed differs by exactly the switch's cost,
    and the gradients have the same bits: the recomputed projection is the same product."""
    from monarch_b200.models import LlamaConfig, LlamaEngine, LocalParamStore, ParamLayout
    cfg = LlamaConfig(vocab=512, d=256, n_layers=6, n_heads=2, n_kv_heads=1, ffn=512)
    T = 2048
    tok = torch.randint(0, cfg.vocab, (1, T), device="cuda")
    held, grads, loss = {}, {}, ops.cross_entropy_

    def requested():   # what was asked for, not the blocks that the allocator found for it
        return torch.cuda.memory_stats()["requested_bytes.all.current"]

    def counted(*args):
        held[keep] = requested() - base
        return loss(*args)

    monkeypatch.setattr(ops, "cross_entropy_", counted)
    cost = cfg.n_layers * T * cfg.d * 2
    for keep, limit in ((False, None), (True, 0), (None, cost - 1), (None, cost)):
        if limit is not None:
            monkeypatch.setattr(LlamaEngine, "KEEP_RESIDUAL_BYTES", limit)
        st = LocalParamStore(ParamLayout(cfg), "cuda", seed=1)
        eng = LlamaEngine(cfg, st, T, keep_residual=keep)
        keep = (keep, limit)
        base = requested()
        eng.forward_backward(tok, tok)
        grads[keep] = [g.clone() for u in range(cfg.n_layers + 2) for g in st.unit_grads(u).values()]
    no, yes = (False, None), (True, 0)
    assert held[yes] - held[no] == cost, held
    assert held[None, cost - 1] == held[no] and held[None, cost] == held[yes], held
    assert all(torch.equal(a, b) for a, b in zip(grads[no][1:], grads[yes][1:]))


# both sides of every limit in rows and width that the choice of warps per row has, with a last
# block that is not full
@pytest.mark.parametrize("rows,d", [(2048, 264), (2049, 512), (2047, 1024), (2049, 1024), (2049, 1040), (3, 2048),
                                    (767, 4096), (769, 3080), (2049, 5120), (2047, 6144),
                                    (2049, 6152), (9, 8192)])
def test_rmsnorm_forward_row_counts(rows, d):
    x = torch.randn(rows, d, device="cuda", dtype=bf16)
    w = (1 + 0.1 * torch.randn(d, device="cuda")).to(bf16)
    y, rstd = ops.rmsnorm_fwd(x, w, 1e-5)
    yr, rstdr = R.rmsnorm_fwd(x.double(), w.double(), 1e-5)
    assert _rel(y, yr) < 3e-3 and _rel(rstd, rstdr) < 1e-6   # as in test_rmsnorm_row_lengths


# rows and heads on both sides of where a row gets more threads; a row's heads in several batches
@pytest.mark.parametrize("rows,heads", [(1, 3), (64, 80), (600, 41), (2050, 20), (4099, 9), (9000, 1),
                                        (9000, 17)])
@pytest.mark.parametrize("hd", [16, 64, 128, 512])
def test_rope_row_and_head_counts(rows, heads, hd):
    cos, sin = R.rope_tables(500, hd, 10000.0, device="cuda")
    x = torch.randn(rows, heads * hd + 8, device="cuda", dtype=bf16)
    y = x.clone()
    ops.rope_(y, cos, sin, 500, heads, hd)
    ref = R.rope(x[:, : heads * hd].float().reshape(rows, heads, hd), cos, sin, 500, False)
    assert _rel(y[:, : heads * hd], ref.reshape(rows, -1)) < 3e-3
    assert torch.equal(y[:, heads * hd:], x[:, heads * hd:])


# several rows per block, with rows left over; a block's chunks that are no whole number of warps
@pytest.mark.parametrize("rows,F", [(300, 24), (1001, 120), (77, 2040), (513, 1000)])
def test_swiglu_short_rows(rows, F):
    gu = torch.randn(rows, 2 * F, device="cuda", dtype=bf16)
    dh = torch.randn(rows, F, device="cuda", dtype=bf16)
    assert _rel(ops.swiglu_fwd(gu), R.swiglu_fwd(gu)) < 3e-3
    assert _rel(ops.swiglu_bwd(gu, dh), R.swiglu_bwd(gu, dh)) < 3e-3


@pytest.mark.parametrize("rows,d", [(301, 64), (77, 2040)])
def test_embedding_bwd_short_rows(rows, d):
    ids = torch.randperm(400, device="cuda")[:rows]
    dout = torch.randn(rows, d, device="cuda", dtype=bf16)
    dt = torch.zeros(400, d, device="cuda", dtype=bf16)
    ops.embedding_bwd_(dout, ids, dt)
    ref = torch.zeros_like(dt)
    ref[ids] = dout
    assert torch.equal(dt, ref)


@pytest.mark.parametrize("rows,V", [(512, 6144), (513, 6152), (511, 6144), (600, 16384), (600, 16396),
                                    (5, 65535), (5, 65536)])
def test_cross_entropy_block_sizes(rows, V):
    ld = (V + 15) // 8 * 8
    wide = (3 * torch.randn(rows, ld, device="cuda")).to(bf16)
    tg = torch.randint(0, V, (rows,), device="cuda")
    tg[:2] = torch.tensor([0, V - 1])
    lr, gr = R.cross_entropy(wide[:, :V], tg, 0.25)
    loss = ops.cross_entropy_(wide[:, :V], tg, 0.25)
    assert torch.allclose(loss, lr, atol=2e-4, rtol=1e-4)   # as in test_cross_entropy_vocabularies
    assert _rel(wide[:, :V], gr) < 3e-3
