"""Numerics of every sm_100a kernel against the fp32 PyTorch reference of the same op
(the CPU path of the same ``ops`` function)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def rel(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return ((a - b).norm() / b.norm().clamp_min(1e-12)).item()


def bf(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


@pytest.fixture(autouse=True)
def _seed_and_status():
    from dhellam_b200 import kernels as K
    torch.manual_seed(1234)
    yield
    torch.cuda.synchronize()
    st = K.read_status()
    assert st.code == 0, f"device status {st.code} at {st.where}"


@pytest.fixture(params=[False, True], ids=["atomic", "reproducible"])
def reduction_mode(request):
    """The kernels with cross-CTA reductions in both forms: order-dependent atomics (default) and the
    fixed-order forms of the reproducible mode."""
    from dhellam_b200 import kernels as K
    K.set_deterministic(request.param)
    yield request.param
    K.set_deterministic(False)


@pytest.fixture(params=[1, 2], ids=["single_cta", "cta_pair"])
def gemm_mode(request):
    from dhellam_b200.ops.gemm import set_gemm_mode
    set_gemm_mode(request.param)
    yield request.param
    set_gemm_mode(0)


@pytest.mark.parametrize("M,N,K_", [(128, 256, 64), (384, 1280, 1024), (200, 264, 136), (1024, 1024, 4096), (8, 4096, 256),
                                    (2048, 1536, 2048), (1100, 520, 328)])
def test_gemm_three_layouts(M, N, K_, gemm_mode):
    from dhellam_b200.ops.gemm import gemm_nn, gemm_nt, gemm_tn_acc
    x, w, dy = bf(M, K_), bf(N, K_), bf(M, N)
    assert rel(gemm_nt(x, w), x.float() @ w.float().t()) < 5e-3
    assert rel(gemm_nn(dy, w), dy.float() @ w.float()) < 5e-3
    g = torch.ones(N, K_, device=DEV)
    gemm_tn_acc(dy, x, g)
    assert rel(g, 1 + dy.float().t() @ x.float()) < 1e-4
    g2 = torch.full((N, K_), 7.0, device=DEV)
    gemm_tn_acc(dy, x, g2, accumulate=False)
    assert rel(g2, dy.float().t() @ x.float()) < 1e-4


@pytest.mark.parametrize("split", [2, 3, 4])
def test_gemm_weight_gradient_split_along_k_adds_atomically(split):
    """An accumulating GEMM may be cut into ``split`` work items per tile that each add their share
    into the fp32 output with the reducing bulk store; the result must not depend on the split."""
    from dhellam_b200.ops.gemm import gemm_tn_acc, set_gemm_mode, set_gemm_splitk
    set_gemm_mode(2)
    try:
        for M, N, K_ in ((4096, 520, 392), (1000, 256, 256), (8192, 1280, 512)):
            dy, x = bf(M, N), bf(M, K_)
            ref = 3.0 + dy.float().t() @ x.float()
            set_gemm_splitk(split)
            g = torch.full((N, K_), 3.0, device=DEV)
            gemm_tn_acc(dy, x, g)
            assert rel(g, ref) < 1e-4, (M, N, K_, rel(g, ref))
    finally:
        set_gemm_splitk(-1)
        set_gemm_mode(0)


@pytest.mark.parametrize("M,N,K_,kind", [(16384, 1280, 8192, "nt"), (16384, 8192, 1024, "nt"), (16384, 7168, 8192, "nn"),
                                         (16384, 16032, 2048, "nt"), (16384, 3584, 8192, "tn"), (16384, 1280, 8192, "tn")])
def test_gemm_headline_shapes_against_fp32(M, N, K_, kind):
    """The per-GPU shapes of the 8-way tensor-parallel headline run (16384 rows) against an fp32 product."""
    from dhellam_b200.ops.gemm import gemm_nn, gemm_nt, gemm_tn_acc
    if kind == "nt":
        x, w = bf(M, K_), bf(N, K_, scale=0.05)
        got, ref = gemm_nt(x, w), x.float() @ w.float().t()
        tol = 5e-3
    elif kind == "nn":
        dy, w = bf(M, N), bf(N, K_, scale=0.05)
        got, ref = gemm_nn(dy, w), dy.float() @ w.float()
        tol = 5e-3
    else:
        dy, x = bf(M, N, scale=0.1), bf(M, K_)
        got = torch.ones(N, K_, device=DEV)
        gemm_tn_acc(dy, x, got)
        ref = 1 + dy.float().t() @ x.float()
        tol = 1e-4
    assert rel(got, ref) < tol, rel(got, ref)


def test_gemm_sm_budget_and_strided_output(gemm_mode):
    from dhellam_b200.ops.gemm import gemm_nt
    x, w = bf(512, 512), bf(768, 512)
    big = torch.zeros(512, 1024, dtype=torch.bfloat16, device=DEV)
    out = gemm_nt(x, w, out=big[:, :768], sm_budget=16)
    assert rel(out, x.float() @ w.float().t()) < 5e-3
    assert float(big[:, 768:].abs().max()) == 0.0


@pytest.mark.parametrize("M,N,Kd", [(8, 512, 64), (1, 8, 520), (129, 136, 1000), (300, 1024, 576), (128, 128, 8192)])
@pytest.mark.parametrize("cluster", [1, 2, 4, 8])
def test_gemm_cluster_k(M, N, Kd, cluster):
    """The small-output kernel with K over 1 to 8 CTAs: edges of tiles in M and N, K that is no multiple of a k-block or has fewer
    k-blocks than CTAs, all operand majors, fp32 outputs stored and accumulated, a strided output.  Only the order of fp32
    sums differs from the reference's."""
    from dhellam_b200.ops.gemm import gemm_nn, gemm_nt, gemm_tn_acc, set_gemm_cluster_k
    x, w, dy = bf(M, Kd), bf(N, Kd), bf(M, N)
    big = torch.zeros(M, N + 64, dtype=torch.bfloat16, device=DEV)
    xt, dyt, g = bf(Kd, 8 * ((M + 7) // 8)), bf(Kd, N), torch.ones(N, 8 * ((M + 7) // 8), device=DEV)
    set_gemm_cluster_k(cluster)
    try:
        gemm_nt(x, w, out=big[:, :N])
        f = gemm_nt(x, w, out_dtype=torch.float32)
        dx = gemm_nn(dy, w)
        gemm_tn_acc(dyt, xt, g)
        again = gemm_nt(x, w, out_dtype=torch.float32)
    finally:
        set_gemm_cluster_k(-1)
    ref = x.double() @ w.double().t()
    assert rel(big[:, :N], ref) < 5e-3 and float(big[:, N:].abs().max()) == 0.0
    assert rel(f, ref) < 1e-5 and torch.equal(f, again)
    assert rel(dx, dy.double() @ w.double()) < 5e-3
    assert rel(g, 1 + dyt.double().t() @ xt.double()) < 1e-5


@pytest.mark.parametrize("M,N,Kd", [(128, 4224, 512), (64, 4352, 1024), (8, 4608, 512), (64, 8192, 12288), (129, 6144, 4096),
                                    (129, 6144, 4032), (16, 12288, 4096), (64, 12288, 4096), (300, 6528, 4096)])
def test_gemm_by_the_rule(M, N, Kd):
    """No kernel forced: problems on both sides of the lines between the kernels, bf16 and fp32 outputs, stored and accumulated.
    bf16 rounding, and fp32 sums of Kd products in another order."""
    from dhellam_b200.ops.gemm import gemm_nn, gemm_nt, gemm_tn_acc
    x, w = bf(M, Kd), bf(N, Kd, scale=0.05)
    ref = x.double() @ w.double().t()
    assert rel(gemm_nt(x, w), ref) < 5e-3 and rel(gemm_nt(x, w, out_dtype=torch.float32), ref) < 1e-5
    assert rel(gemm_nn(x, w.t().contiguous()), ref) < 5e-3
    rows = 8 * ((M + 7) // 8)                              # fp32 rows of the accumulated output: M of them are looked at
    dy = torch.zeros(Kd, rows, dtype=torch.bfloat16, device=DEV)
    dy[:, :M] = x.t()
    g = torch.ones(rows, N, device=DEV)
    gemm_tn_acc(dy, w.t().contiguous(), g)
    assert rel(g[:M] - 1, ref) < 1e-5 + 1e-7 * math.sqrt(M * N) / ref.norm().item()


@pytest.mark.parametrize("rows,h", [(64, 256), (300, 4096), (257, 8192), (33, 1024)])
def test_rmsnorm(rows, h, reduction_mode):
    from dhellam_b200.ops.norm import rmsnorm_bwd, rmsnorm_fwd
    x, w, dy, res = bf(rows, h), bf(h) * 0.1 + 1, bf(rows, h), bf(rows, h)
    y, rstd = rmsnorm_fwd(x, w, 1e-5)
    yr, rstdr = rmsnorm_fwd(x.cpu().float(), w.cpu().float(), 1e-5)
    assert rel(y, yr) < 5e-3 and rel(rstd, rstdr) < 1e-4
    mg = torch.zeros(h, device=DEV)
    dx, _ = rmsnorm_bwd(dy, x, w, rstd, weight_main_grad=mg, residual_grad=res)
    mgr = torch.zeros(h)
    dxr, _ = rmsnorm_bwd(dy.cpu().float(), x.cpu().float(), w.cpu().float(), rstdr, weight_main_grad=mgr, residual_grad=res.cpu().float())
    assert rel(dx, dxr) < 5e-3 and rel(mg, mgr) < 2e-3


@pytest.mark.parametrize("rows,h", [(64, 256), (129, 5120)])
def test_layernorm(rows, h, reduction_mode):
    from dhellam_b200.ops.norm import layernorm_bwd, layernorm_fwd
    x, w, b, dy = bf(rows, h) + 0.5, bf(h) * 0.1 + 1, bf(h) * 0.1, bf(rows, h)
    y, mu, rstd = layernorm_fwd(x, w, b, 1e-5)
    yr, mur, rstdr = layernorm_fwd(x.cpu().float(), w.cpu().float(), b.cpu().float(), 1e-5)
    assert rel(y, yr) < 5e-3 and rel(mu, mur) < 1e-3 and rel(rstd, rstdr) < 1e-3
    dx, dw, db = layernorm_bwd(dy, x, w, mu, rstd)
    dxr, dwr, dbr = layernorm_bwd(dy.cpu().float(), x.cpu().float(), w.cpu().float(), mur, rstdr)
    assert rel(dx, dxr) < 6e-3 and rel(dw, dwr) < 2e-3 and rel(db, dbr) < 2e-3


def test_swiglu_gelu():
    from dhellam_b200.ops.activation import gelu_bwd, gelu_fwd, swiglu_bwd, swiglu_fwd
    y, d = bf(300, 2 * 1032), bf(300, 1032)
    assert rel(swiglu_fwd(y), swiglu_fwd(y.cpu().float())) < 5e-3
    assert rel(swiglu_bwd(d, y), swiglu_bwd(d.cpu().float(), y.cpu().float())) < 5e-3
    x, dx = bf(77, 1024), bf(77, 1024)
    assert rel(gelu_fwd(x), gelu_fwd(x.cpu().float())) < 5e-3
    assert rel(gelu_bwd(dx, x), gelu_bwd(dx.cpu().float(), x.cpu().float())) < 5e-3


def test_bias_dropout_add_mask_matches_cpu_model():
    from dhellam_b200.ops.bda import bda_bwd, bda_fwd
    x, r, b = bf(130, 512), bf(130, 512), bf(512)
    for p in (0.0, 0.1):
        out = bda_fwd(x, r, b, p, seed=99)
        ref = bda_fwd(x.cpu().float(), r.cpu().float(), b.cpu().float(), p, seed=99)
        assert rel(out, ref) < 5e-3
    dx = bda_bwd(x, 0.1, seed=99)
    assert rel(dx, bda_bwd(x.cpu().float(), 0.1, seed=99)) < 5e-3


def test_rope_roundtrip_and_reference():
    from dhellam_b200.ops.rope import rope_apply_, rope_table
    T, nq, nkv, d = 96, 4, 2, 128
    qkv = bf(T, (nq + 2 * nkv) * d)
    pos = torch.randint(0, 64, (T,), dtype=torch.int32, device=DEV)
    cos, sin = rope_table(64, d, 500000.0, DEV)
    ref = rope_apply_(qkv.cpu().float().clone(), pos.cpu(), cos.cpu(), sin.cpu(), nq, nkv, d)
    orig = qkv.clone()
    out = rope_apply_(qkv, pos, cos, sin, nq, nkv, d)
    assert rel(out, ref) < 5e-3
    back = rope_apply_(out, pos, cos, sin, nq, nkv, d, inverse=True)
    assert rel(back, orig) < 1e-2


def test_embedding_and_cross_entropy(reduction_mode):
    from dhellam_b200.ops.embedding import embedding_bwd, embedding_fwd
    from dhellam_b200.ops.loss import ce_combine_stats, ce_local_stats, vocab_parallel_ce_bwd_
    T, h, Vl, v0 = 200, 256, 1000, 500
    tok = torch.randint(0, 2000, (T,), dtype=torch.int32, device=DEV)
    w = bf(Vl, h)
    assert rel(embedding_fwd(tok, w, v0), embedding_fwd(tok.cpu(), w.cpu().float(), v0)) < 1e-6
    d = bf(T, h)
    mg, mgr = torch.zeros(Vl, h, device=DEV), torch.zeros(Vl, h)
    embedding_bwd(d, tok, mg, v0)
    embedding_bwd(d.cpu().float(), tok.cpu(), mgr, v0)
    assert rel(mg, mgr) < 1e-5
    for dtype, Vc in ((torch.bfloat16, 1000), (torch.bfloat16, 1003), (torch.float32, 777)):
        buf = (torch.randn(T, 1008, device=DEV) * 3).to(dtype)
        logits = buf[:, :Vc]
        st = ce_local_stats(logits, tok, v0)
        str_ = ce_local_stats(logits.cpu().float(), tok.cpu(), v0)
        loss, lse = ce_combine_stats(st.unsqueeze(0))
        lossr, lser = ce_combine_stats(str_.unsqueeze(0))
        assert rel(lse, lser) < 1e-4 and rel(loss, lossr) < 1e-4
        gt = torch.rand(T, device=DEV)
        ref = vocab_parallel_ce_bwd_(logits.cpu().float().clone(), tok.cpu(), lser, gt.cpu(), v0)
        out = vocab_parallel_ce_bwd_(buf.clone()[:, :Vc], tok, lse, gt, v0)
        assert rel(out, ref) < 1e-2


def test_adam_and_sum_squares(reduction_mode):
    from dhellam_b200.optim.adam import adam_update, sum_squares
    n = 4096 * 3 + 4
    master = torch.randn(n, device=DEV)
    p = master.to(torch.bfloat16)
    m, v, g = torch.zeros(n, device=DEV), torch.zeros(n, device=DEV), torch.randn(n, device=DEV)
    ref = [t.cpu().clone() for t in (p.float(), master, m, v, g)]
    for step in (1, 2):
        adam_update(p, master, m, v, g, 1e-2, 0.9, 0.95, 1e-8, 0.1, step, 0.5)
        adam_update(ref[0], ref[1], ref[2], ref[3], ref[4], 1e-2, 0.9, 0.95, 1e-8, 0.1, step, 0.5)
    assert rel(master, ref[1]) < 1e-5 and rel(m, ref[2]) < 1e-5 and rel(v, ref[3]) < 1e-5 and rel(p, ref[1]) < 5e-3
    assert abs(float(sum_squares(g)) - float((g.double() ** 2).sum())) / float((g.double() ** 2).sum()) < 1e-4


def test_router_topk():
    from dhellam_b200.ops.moe import router_topk_fwd
    T, h, E, k = 333, 512, 8, 2
    x, w = bf(T, h), bf(E, h, scale=0.05)
    probs, topi, gates = router_topk_fwd(x, w, k)
    pr, ti, gr = router_topk_fwd(x.cpu().float(), w.cpu().float(), k)
    assert rel(probs, pr) < 1e-3
    same = (topi.cpu() == ti).all(dim=1)
    assert same.float().mean() > 0.99            # near-ties may order differently in bf16 vs fp32 accumulation
    assert rel(gates.cpu()[same], gr[same]) < 1e-3


@pytest.mark.parametrize("rows,h", [(1, 8), (3, 264), (700, 1000), (5, 8192), (4, 8200), (2, 16384)])
@pytest.mark.parametrize("kind", ["rms", "layer"])
@pytest.mark.parametrize("residual", [False, True], ids=["plain", "residual"])
def test_norm_backward_row_lengths(rows, h, kind, residual):
    """One vector per thread (up to 8192 elements, lanes to spare at 264 and 1000), several beyond; more rows than CTAs; with and
    without a residual, and a gradient buffer that is only 4-byte aligned.  bf16 results: 1e-2; fp32 sums: 1e-3."""
    from dhellam_b200.ops.norm import layernorm_bwd, layernorm_fwd, rmsnorm_bwd, rmsnorm_fwd
    x, w, b, dy, res = bf(rows, h), bf(h), bf(h), bf(rows, h), bf(rows, h) if residual else None
    grads = torch.zeros(2, h + 1, device=DEV)
    dw, db, dwr, dbr = grads[0, 1:], grads[1, 1:], torch.zeros(h), torch.zeros(h)
    cpu = lambda *t: [a if a is None else a.cpu().float() for a in t]
    xc, wc, bc, dyc, rc = cpu(x, w, b, dy, res)
    if kind == "rms":
        _, rstd = rmsnorm_fwd(x, w)
        dx, _ = rmsnorm_bwd(dy, x, w, rstd, weight_main_grad=dw, residual_grad=res)
        dxr, _ = rmsnorm_bwd(dyc, xc, wc, rstd.cpu(), weight_main_grad=dwr, residual_grad=rc)
    else:
        _, mu, rstd = layernorm_fwd(x, w, b)
        dx, _, _ = layernorm_bwd(dy, x, w, mu, rstd, weight_main_grad=dw, bias_main_grad=db, residual_grad=res)
        dxr, _, _ = layernorm_bwd(dyc, xc, wc, mu.cpu(), rstd.cpu(), weight_main_grad=dwr, bias_main_grad=dbr, residual_grad=rc)
        assert rel(db, dbr) < 1e-3
    assert rel(dx, dxr) < 1e-2 and rel(dw, dwr) < 1e-3


@pytest.mark.parametrize("Sq,Sk,B,Hq,Hk,causal", [(128, 128, 1, 1, 1, True), (256, 256, 2, 4, 2, True), (384, 384, 1, 2, 1, False),
                                                     (200, 200, 2, 2, 2, True), (128, 256, 1, 2, 1, False), (256, 128, 1, 2, 2, False)])
def test_attention_forward_backward(Sq, Sk, B, Hq, Hk, causal):
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd
    d = 128
    # strided views into packed buffers, as the engine uses them
    qkv = bf(Sq, B, Hq + 2 * Hk, d)
    q = qkv[:, :, :Hq]
    if Sk == Sq:
        k, v = qkv[:, :, Hq:Hq + Hk], qkv[:, :, Hq + Hk:]
    else:
        kv = bf(Sk, B, 2 * Hk, d)
        k, v = kv[:, :, :Hk], kv[:, :, Hk:]
    scale = 1.0 / math.sqrt(d)
    o, lse = attn_fwd(q, k, v, causal, scale)
    qc, kc, vc = q.cpu().float(), k.cpu().float(), v.cpu().float()
    oref, lref = attn_fwd(qc, kc, vc, causal, scale)
    assert rel(o, oref) < 1e-2, rel(o, oref)
    assert rel(lse, lref) < 1e-3
    do = bf(Sq, B, Hq, d)
    dq, dk, dv = attn_bwd(do, q, k, v, o, lse, causal, scale)
    dqr, dkr, dvr = attn_bwd(do.cpu().float(), qc, kc, vc, oref, lref, causal, scale)
    assert rel(dq, dqr) < 2e-2, ("dq", rel(dq, dqr))
    assert rel(dk, dkr) < 2e-2, ("dk", rel(dk, dkr))
    assert rel(dv, dvr) < 2e-2, ("dv", rel(dv, dvr))


@pytest.mark.parametrize("Sq,Sk,B,Hq,Hk", [(4096, 4096, 1, 8, 1), (1024, 2048, 2, 4, 2), (2048, 2048, 4, 16, 2)])
def test_attention_large_shapes_against_fp32(Sq, Sk, B, Hq, Hk):
    """Causal attention at the sizes the training step uses, against plain fp32 PyTorch (explicit softmax and
    autograd on the GPU): 4096 positions with eight query heads on one KV head (the dK/dV kernel then splits the
    heads of that KV head over several CTAs), more keys than queries (mask aligned to the last key, the
    context-parallel case), and a batch that fills the GPU without a head split."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd
    d = 128
    scale = 1.0 / math.sqrt(d)
    q, k, v, do = bf(Sq, B, Hq, d), bf(Sk, B, Hk, d), bf(Sk, B, Hk, d), bf(Sq, B, Hq, d)
    o, lse = attn_fwd(q, k, v, True, scale)
    dq, dk, dv = attn_bwd(do, q, k, v, o, lse, True, scale)
    qf, kf, vf = (t.float().requires_grad_() for t in (q, k, v))
    g = Hq // Hk
    sc = torch.einsum("sbhd,tbhd->bhst", qf, kf.repeat_interleave(g, dim=2)) * scale
    i = torch.arange(Sq, device=DEV).unsqueeze(1)
    j = torch.arange(Sk, device=DEV).unsqueeze(0)
    sc = sc.masked_fill(j > i + (Sk - Sq), float("-inf"))
    ref_lse = torch.logsumexp(sc, dim=-1)
    oref = torch.einsum("bhst,tbhd->sbhd", torch.softmax(sc, dim=-1), vf.repeat_interleave(g, dim=2))
    oref.backward(do.float())
    assert rel(o, oref.detach()) < 1e-2 and rel(lse, ref_lse.detach()) < 1e-3
    assert rel(dq, qf.grad) < 2e-2, ("dq", rel(dq, qf.grad))
    assert rel(dk, kf.grad) < 2e-2, ("dk", rel(dk, kf.grad))
    assert rel(dv, vf.grad) < 2e-2, ("dv", rel(dv, vf.grad))


def _peaked_scores(kind, Sq, Sk, Hq, Hk):
    """Inputs whose softmax has few dominant keys, as trained models have: scores with a standard deviation of 3 or 6, scores
    that rise with the key index (every key block has a new maximum), one key that outgrows the others by more than 2^8."""
    d = 128
    q, k, v = bf(Sq, 1, Hq, d), bf(Sk, 1, Hk, d), bf(Sk, 1, Hk, d)
    if kind in ("std3", "std6"):
        q *= float(kind[3:])
    elif kind == "rising":
        k[:, :, :, 0] = torch.linspace(-8, 8, Sk, device=DEV)[:, None, None].to(torch.bfloat16)
        q[:, :, :, 0] = 12.0
    else:
        k[Sk // 2] = 40.0 * q[Sq // 2, :, :Hk] / q[Sq // 2, :, :Hk].float().norm(dim=-1, keepdim=True)
    return q, k, v


def _running_maximum_reference(q, k, v, causal, scale):
    """``(out, lse, out as flash attention rounds it)`` in 64 bits: the third divides sums whose probabilities are rounded to
    bf16 relative to the running maximum of blocks of 128 keys, the only rounding of a forward pass besides that of its result."""
    Sq, Hq, Sk = q.shape[0], q.shape[2], k.shape[0]
    g = Hq // k.shape[2]
    qd, kd, vd = (t[:, 0].transpose(0, 1).double() for t in (q, k, v))
    kd, vd = kd.repeat_interleave(g, 0), vd.repeat_interleave(g, 0)
    s = qd @ kd.transpose(1, 2) * scale
    if causal:
        s.masked_fill_(torch.arange(Sk, device=DEV)[None] > torch.arange(Sq, device=DEV)[:, None] + (Sk - Sq), float("-inf"))
    lse = torch.logsumexp(s, -1)
    exact = torch.softmax(s, -1) @ vd
    pad = -Sk % 128
    s = torch.nn.functional.pad(s, (0, pad), value=float("-inf")).view(Hq, Sq, -1, 128)
    run = s.amax(-1).cummax(-1).values
    p = torch.exp(s - run[..., None])
    w = torch.exp(run - run[..., -1:])[..., None]
    num = (p.to(torch.bfloat16).double() * w).view(Hq, Sq, -1)[..., :Sk] @ vd
    rounded = (num / (p * w).sum((-1, -2))[..., None]).to(torch.bfloat16)
    back = lambda t: t.transpose(0, 1).unsqueeze(1)
    return back(exact), lse.unsqueeze(0), back(rounded)


@pytest.mark.parametrize("Sq,Sk,Hq,Hk,causal", [(1024, 1024, 4, 2, True), (300, 2000, 3, 1, False)])
@pytest.mark.parametrize("kind", ["std3", "std6", "rising", "spike"])
def test_attention_forward_is_as_exact_as_the_running_maximum_allows(kind, Sq, Sk, Hq, Hk, causal):
    """Against 64 bits, the forward is no further off than what the rounding of probabilities below the running maximum and of the
    result costs (computed beside it; 3 % for the 32-bit arithmetic and for sums in another order)."""
    from dhellam_b200.ops.attention import attn_fwd
    q, k, v = _peaked_scores(kind, Sq, Sk, Hq, Hk)
    scale = 1.0 / math.sqrt(128)
    out, lse = attn_fwd(q, k, v, causal, scale)
    exact, exact_lse, rounded = _running_maximum_reference(q, k, v, causal, scale)
    off = lambda t: ((t.double() - exact).norm() / exact.norm()).item()
    assert off(out) < 1.03 * off(rounded), (off(out), off(rounded))
    assert (lse.double() - exact_lse).abs().max().item() < 1e-4 * (1 + exact_lse.abs().max().item())


@pytest.mark.parametrize("scale", [0.0, -0.05])
def test_attention_with_a_scale_that_is_not_positive(scale):
    """Masked keys stay masked whatever the sign of the scale: with 0 every visible key weighs the same.  Ragged and causal, so
    that there are masked keys in the last tile of the keys and on the diagonal."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd
    S, d = 200, 128
    q, k, v, do = bf(S, 2, 2, d), bf(S, 2, 1, d), bf(S, 2, 1, d), bf(S, 2, 2, d)
    cpu = lambda *ts: [t.cpu().float() for t in ts]
    for causal in (True, False):
        o, lse = attn_fwd(q, k, v, causal, scale)
        oref, lref = attn_fwd(*cpu(q, k, v), causal, scale)
        assert rel(o, oref) < 1e-2 and rel(lse, lref) < 1e-3
        grads = attn_bwd(do, q, k, v, o, lse, causal, scale)
        refs = attn_bwd(*cpu(do, q, k, v), oref, lref, causal, scale)
        for a, r in zip(grads, refs):
            assert (a.cpu().float() - r).norm() <= 2e-2 * r.norm()       # dq and dk are zero at scale 0


@pytest.mark.parametrize("budget", [1, 5, 24, 100])
def test_attention_sm_budget_gives_identical_results(budget):
    """With an SM budget the work items of the attention kernels are cut into consecutive launches of at most that many CTAs;
    every tile computes exactly what it computes without a budget."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd
    Sq, B, Hq, Hk, d = 1024, 2, 4, 2, 128
    qkv = bf(Sq, B, Hq + 2 * Hk, d)
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hk], qkv[:, :, Hq + Hk:]
    do = bf(Sq, B, Hq, d)
    scale = 1.0 / math.sqrt(d)
    o0, l0 = attn_fwd(q, k, v, True, scale)
    g0 = attn_bwd(do, q, k, v, o0, l0, True, scale)
    o1, l1 = attn_fwd(q, k, v, True, scale, sm_budget=budget)
    g1 = attn_bwd(do, q, k, v, o1, l1, True, scale, sm_budget=budget)
    torch.cuda.synchronize()
    assert torch.equal(o0, o1) and torch.equal(l0, l1)
    for a, b in zip(g0, g1):
        assert torch.equal(a, b)


def test_varlen_api_with_equal_lengths_matches_the_fixed_length_entry_points():
    """``pymha_varlen_fwd / bwd`` on a packed batch of equal-length sequences against the fixed-length entry points on contiguous
    [s, b, h, d] copies."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd, pymha_varlen_bwd, pymha_varlen_fwd
    b, s, hq, hk, d = 3, 256, 4, 2, 128
    cu = torch.arange(0, (b + 1) * s, s, dtype=torch.int32, device=DEV)
    q, k, v, do = bf(b * s, hq, d), bf(b * s, hk, d), bf(b * s, hk, d), bf(b * s, hq, d)
    scale = 1.0 / math.sqrt(d)
    out, lse = pymha_varlen_fwd(q, k, v, cu, cu, s, s, 0.0, scale, True)
    dq, dk, dv = pymha_varlen_bwd(do, q, k, v, out, lse, cu, cu, s, s, 0.0, scale, True)
    sb = lambda t: t.view(b, s, t.shape[1], d).permute(1, 0, 2, 3).contiguous()
    o2, l2 = attn_fwd(sb(q), sb(k), sb(v), True, scale)
    g2 = attn_bwd(sb(do), sb(q), sb(k), sb(v), o2, l2, True, scale)
    assert torch.equal(sb(out), o2) and torch.equal(lse, l2)
    for a, r in zip((dq, dk, dv), g2):
        assert rel(sb(a), r) < 1e-3


@pytest.mark.parametrize("Sq,Sk,Hq,Hk,causal", [(300, 300, 4, 2, True), (300, 300, 3, 1, True), (129, 400, 2, 2, False),
                                                (400, 129, 6, 2, True), (128, 128, 2, 1, True)])
def test_attention_forward_is_the_same_however_tiles_share_ctas(Sq, Sk, Hq, Hk, causal):
    """One tile per CTA (as these sizes run by themselves) and two heads or two row tiles per CTA (with an SM budget that has no room
    for a CTA each), dense and packed: bitwise the same."""
    from dhellam_b200.ops.attention import attn_fwd, pymha_varlen_fwd
    q, k, v = bf(Sq, 2, Hq, 128), bf(Sk, 2, Hk, 128), bf(Sk, 2, Hk, 128)
    o, lse = attn_fwd(q, k, v, causal)
    for budget in (1, 5):
        o2, lse2 = attn_fwd(q, k, v, causal, sm_budget=budget)
        assert torch.equal(o, o2) and torch.equal(lse, lse2)
    pack = lambda t, last: torch.cat([t[:, 0], t[:last, 1]])      # the second sequence is 37 rows shorter
    cq, ck = [0, Sq, 2 * Sq - 37], [0, Sk, 2 * Sk - 37]
    packed = pack(q, Sq - 37), pack(k, Sk - 37), pack(v, Sk - 37)
    out, lse3 = pymha_varlen_fwd(*packed, cq, ck, Sq, Sk, is_causal=causal)
    assert torch.equal(out[:Sq], o[:, 0]) and torch.equal(lse3[0], lse[0])
    for budget in (1, 5):
        out2, lse4 = pymha_varlen_fwd(*packed, cq, ck, Sq, Sk, is_causal=causal, math_sm_count=budget)
        assert torch.equal(out, out2) and torch.equal(lse3, lse4)


@pytest.mark.parametrize("n,m", [(2, 2), (17, 5), (2000, 2096), (2000, 2097)])
def test_offsets_on_the_device_are_read_as_they_are(n, m):
    """Up to the capacity of the pinned buffer in one read, beyond it one by one; int64 and strided tensors too."""
    from dhellam_b200.ops.attention import _offset_pair
    a, b = torch.arange(n, dtype=torch.int32) * 3, torch.arange(m, dtype=torch.int32) * 5
    for x, y in ((a.cuda(), b.cuda()), (a.cuda().long(), b.cuda()), (torch.stack([a, a], 1).cuda()[:, 0], b.cuda()), (a, b.cuda())):
        assert _offset_pair(x, y) == (a.tolist(), b.tolist())


@pytest.mark.parametrize("hq,hk", [(4, 2), (3, 1), (2, 2)])
@pytest.mark.parametrize("ql,kl,causal", [([1, 127, 128, 129, 300], None, True), ([130, 64, 257], [130, 200, 513], True),
                                          ([65, 0, 256], [40, 7, 300], False), ([17] * 150, None, True)])
def test_packed_attention_against_fp32_sequence_by_sequence(ql, kl, causal, hq, hk):
    """Ragged batches in one launch (and, with 150 sequences, in two): tiles that end inside a sequence, an empty
    sequence, more keys than queries, odd and even groups; the tolerances are those of the dense test above (bf16
    probabilities and outputs).  One sequence holds NaN: nothing of it may reach its neighbours."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd, pymha_varlen_bwd, pymha_varlen_fwd
    kl, d = kl or ql, 128
    off = lambda n: [sum(n[:i]) for i in range(len(n) + 1)]
    cq, ck = off(ql), off(kl)
    q, k, v, do = bf(cq[-1], hq, d), bf(ck[-1], hk, d), bf(ck[-1], hk, d), bf(cq[-1], hq, d)
    sick = 2                                               # between two healthy ones (or the last)
    for t, c in ((q, cq), (k, ck), (v, ck), (do, cq)):
        t[c[sick]:c[sick + 1]] = float("nan")
    out, lse = pymha_varlen_fwd(q, k, v, cq, ck, max(ql), max(kl), is_causal=causal)
    dq, dk, dv = pymha_varlen_bwd(do, q, k, v, out, lse, cq, ck, max(ql), max(kl), is_causal=causal)
    assert lse.shape == (len(ql), hq, max(ql))
    cpu = lambda t, c, i: t[c[i]:c[i + 1]].unsqueeze(1).float().cpu()
    got, want = [[] for _ in range(5)], [[] for _ in range(5)]
    for i in range(len(ql)):
        assert (lse[i, :, ql[i]:] == float("-inf")).all()
        if ql[i] == 0:                                     # keys that no query sees have no gradient
            assert not dk[ck[i]:ck[i + 1]].any() and not dv[ck[i]:ck[i + 1]].any()
        if i == sick or ql[i] == 0:
            continue
        qi, ki, vi, di = cpu(q, cq, i), cpu(k, ck, i), cpu(v, ck, i), cpu(do, cq, i)
        o, l = attn_fwd(qi, ki, vi, causal)
        grads = attn_bwd(di, qi, ki, vi, o, l, causal)
        mine = (cpu(out, cq, i), lse[i:i + 1, :, :ql[i]].cpu(), cpu(dq, cq, i), cpu(dk, ck, i), cpu(dv, ck, i))
        for a, b, x, y in zip(got, want, mine, (o, l) + tuple(grads)):
            a.append(x.flatten())
            b.append(y.flatten())
    for name, a, b, tol in zip(("out", "lse", "dq", "dk", "dv"), got, want, (1e-2, 1e-3, 2e-2, 2e-2, 2e-2)):
        assert rel(torch.cat(a), torch.cat(b)) < tol, (name, rel(torch.cat(a), torch.cat(b)))


@pytest.mark.parametrize("Sq,Sk", [(300, 40), (200, 130), (600, 129)])
@pytest.mark.parametrize("packed", [False, True], ids=["dense", "packed"])
def test_causal_queries_before_the_first_key(Sq, Sk, packed):
    """More queries than keys, aligned at the end: the first Sq - Sk rows see no key (zeros, statistics of -inf, no gradient), in
    whole tiles and in part of one; the others are the square problem of the last Sk rows."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd, pymha_varlen_bwd, pymha_varlen_fwd
    q, k, v, do = bf(Sq, 1, 4, 128), bf(Sk, 1, 2, 128), bf(Sk, 1, 2, 128), bf(Sq, 1, 4, 128)
    if packed:                                             # between two other sequences
        sq, sk = [70, Sq, 131], [70, Sk, 131]
        off = lambda n: [sum(n[:i]) for i in range(len(n) + 1)]
        cq, ck, mid_q, mid_k = off(sq), off(sk), slice(70, 70 + Sq), slice(70, 70 + Sk)
        around = lambda t: torch.cat([bf(70, *t.shape[2:]), t[:, 0], bf(131, *t.shape[2:])])
        Q, K_, V, DO = around(q), around(k), around(v), around(do)
        out, lse = pymha_varlen_fwd(Q, K_, V, cq, ck, max(sq), max(sk))
        dq, dk, dv = pymha_varlen_bwd(DO, Q, K_, V, out, lse, cq, ck, max(sq), max(sk))
        o, dq, dk, dv = (t[s].unsqueeze(1) for t, s in ((out, mid_q), (dq, mid_q), (dk, mid_k), (dv, mid_k)))
        lse = lse[1:2, :, :Sq]
    else:
        o, lse = attn_fwd(q, k, v, True)
        dq, dk, dv = attn_bwd(do, q, k, v, o, lse, True)
    n = Sq - Sk
    assert not o[:n].any() and not dq[:n].any() and (lse[:, :, :n] == float("-inf")).all()
    qc, kc, vc, dc = (t.float().cpu() for t in (q[n:], k, v, do[n:]))
    oref, lref = attn_fwd(qc, kc, vc, True)
    grads = attn_bwd(dc, qc, kc, vc, oref, lref, True)
    assert rel(o[n:], oref) < 1e-2 and rel(lse[:, :, n:], lref) < 1e-3
    for a, b in zip((dq[n:], dk, dv), grads):
        assert rel(a, b) < 2e-2


def test_packed_batch_of_several_launches_equals_the_dense_kernels():
    """More than 768 tiles and more than 128 sequences: cut into several launches, each tile as the dense kernels compute it."""
    from dhellam_b200.ops.attention import attn_bwd, attn_fwd, pymha_varlen_bwd, pymha_varlen_fwd
    lengths, hq, hk, d = [1000] * 100 + [130] * 60, 2, 1, 128
    cu = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    q, k, v, do = bf(cu[-1], hq, d), bf(cu[-1], hk, d), bf(cu[-1], hk, d), bf(cu[-1], hq, d)
    out, lse = pymha_varlen_fwd(q, k, v, cu, cu, 1000, 1000)
    grads = pymha_varlen_bwd(do, q, k, v, out, lse, cu, cu, 1000, 1000)
    for first, n, s in ((0, 100, 1000), (100, 60, 130)):
        rows = slice(cu[first], cu[first + n])
        sb = lambda t: t[rows].view(n, s, t.shape[1], d).permute(1, 0, 2, 3)
        o, l = attn_fwd(sb(q), sb(k), sb(v), True)
        assert torch.equal(sb(out), o) and torch.equal(lse[first:first + n, :, :s], l)
        assert (lse[first:first + n, :, s:] == float("-inf")).all()
        for a, b in zip(grads, attn_bwd(sb(do), sb(q), sb(k), sb(v), o, l, True)):
            assert rel(sb(a), b) < 1e-3                    # the heads of a KV head may be divided otherwise: sums in another order


def test_packed_attention_with_operands_of_different_lengths():
    """Operands may hold rows past the last sequence, each as many as it likes."""
    from dhellam_b200.ops.attention import pymha_varlen_bwd, pymha_varlen_fwd
    cu, n = [0, 200, 333], 333
    q, k, v, do = bf(n + 3, 4, 128), bf(n, 2, 128), bf(n + 130, 2, 128), bf(n + 1, 4, 128)
    long_out, long_lse = pymha_varlen_fwd(q, k, v, cu, cu, 200, 200)
    longs = (long_out, long_lse, *pymha_varlen_bwd(do, q, k, v, long_out, long_lse, cu, cu, 200, 200))
    out, lse = pymha_varlen_fwd(q[:n], k, v[:n], cu, cu, 200, 200)
    shorts = (out, lse, *pymha_varlen_bwd(do[:n], q[:n], k, v[:n], out, lse, cu, cu, 200, 200))
    for i, (a, b) in enumerate(zip(longs, shorts)):
        assert torch.equal(a if i == 1 else a[:n], b)


@pytest.mark.parametrize("R,T,smoothing", [(1, 1, 0.0), (1, 257, 0.1), (4, 1000, 0.0), (8, 33, 0.1)])
def test_ce_combine_against_the_composed_form(R, T, smoothing):
    """Statistics of 1 to 8 ranks -> loss and log-sum-exp; same fp32 arithmetic as the PyTorch composition (CPU), so 1e-6."""
    from dhellam_b200.ops.loss import ce_combine_stats
    stats = torch.randn(R, T, 4) * 3
    stats[..., 1] = stats[..., 1].exp()
    got = ce_combine_stats(stats.cuda(), smoothing, 4096)
    want = ce_combine_stats(stats, smoothing, 4096)
    for g, w in zip(got, want):
        assert rel(g, w) < 1e-6


def test_ce_combine_leaves_to_the_composed_form_what_only_that_handles():
    """Gradients (reverse and forward), a map over the statistics, no rank at all, no sums of logits, another stride: as on the CPU."""
    from dhellam_b200.ops.loss import ce_combine_stats
    stats, tangent = torch.rand(2, 5, 4) + 0.5, torch.randn(2, 5, 4)

    def answers(dev):
        s, t = stats.to(dev), tangent.to(dev)
        leaf = s.clone().requires_grad_()
        loss, lse = ce_combine_stats(leaf)
        (loss.sum() + 2 * lse.sum()).backward()
        yield leaf.grad
        yield from torch.func.jvp(ce_combine_stats, (s,), (t,))[1]
        yield from torch.func.vmap(ce_combine_stats)(torch.stack([s, s + 1]))
        yield from ce_combine_stats(s[:, :, :3].contiguous())
        yield from ce_combine_stats(s[:, ::2])
        with pytest.raises((IndexError, RuntimeError)):
            ce_combine_stats(s[:0])

    for got, want in zip(answers(DEV), answers("cpu")):
        assert rel(got, want) < 1e-6


def test_bounded_wait_reports_timeout_without_hanging():
    """A flag that nobody sets: the device-side wait gives up after its (short) budget and
    the host reads the status word; the context stays usable."""
    from dhellam_b200 import kernels as K
    from dhellam_b200.runtime.signals import probe_flag_wait
    st = probe_flag_wait(expect=1, budget_cycles=200000)
    assert st.code == 2 and st.extra == 1
    x = torch.ones(4, device=DEV)
    assert float(x.sum()) == 4.0
    assert K.read_status().code == 0


def test_communication_wait_entry_point_gives_up_after_its_budget():
    """The real wait in front of a consumer of gathered rows (``dh_wait_counters``) on counters that
    nothing raises, with a budget of about a millisecond: the kernel gives up, the status word says
    "flag timeout" at that site, and the context stays usable.  No peer is involved."""
    from ctypes import c_int, c_int64, c_uint, c_void_p
    from dhellam_b200 import kernels as K
    counters = torch.zeros(16, dtype=torch.int32, device=DEV)
    fn = K.proto("dh_wait_counters", [c_void_p, c_int, c_uint, c_int64, c_void_p])
    K.check(fn(counters.data_ptr(), 16, 3, 2_000_000, K.stream_ptr(None)), "dh_wait_counters")
    st = K.read_status(clear=True)
    assert st.code == 2 and st.where == 641 and st.extra == 3, (st.code, st.where, st.extra)
    counters.fill_(3)                          # the same wait succeeds at once when the counters are there
    K.check(fn(counters.data_ptr(), 16, 3, 2_000_000, K.stream_ptr(None)), "dh_wait_counters")
    assert K.read_status().code == 0
    assert float(torch.ones(4, device=DEV).sum()) == 4.0


def test_device_resident_moe_exchange_and_grouped_gemms():
    """Plan -> dispatch -> grouped expert GEMMs -> combine on one GPU (ep = 1) against plain PyTorch: the
    routing sizes never reach the host on the device path, the reference below sorts on the host."""
    from types import SimpleNamespace
    from dhellam_b200.ops.moe_native import DeviceMoE
    E, k, h, f, T = 4, 2, 512, 256, 300
    cfg = SimpleNamespace(num_experts=E, moe_top_k=k, hidden_size=h)
    ps = SimpleNamespace(ep=1, ep_rank=0, ep_group=None)
    dev = DeviceMoE(ps, cfg, None, torch.device(DEV), T)
    x = bf(T, h)
    logits = torch.randn(T, E, device=DEV)
    topi = logits.topk(k, dim=-1).indices.to(torch.int32).contiguous()
    gates = torch.softmax(torch.randn(T, k, device=DEV), -1).contiguous()
    plan = dev.plan(topi)
    slot, _ = dev.dispatch(plan, x, "xe", record=True)
    xe = dev.landed("xe", slot)
    torch.cuda.synchronize()
    offs, rows_e = plan.offs.cpu().tolist(), plan.rows_e.cpu().tolist()
    flat = topi.reshape(-1).cpu()
    assert int(plan.overflow) == 0 and all(o % 256 == 0 for o in offs)
    for e in range(E):
        idx = torch.nonzero(flat == e).squeeze(1)              # stable order of the copies of expert e
        assert rows_e[e] == idx.numel()
        got = xe[offs[e]:offs[e] + rows_e[e]].cpu()
        assert torch.equal(got, x.cpu()[idx // k]), e
        assert float(xe[offs[e] + rows_e[e]:offs[e + 1]].abs().max() if offs[e + 1] > offs[e] + rows_e[e] else 0.0) == 0.0
    w1 = bf(E, 2 * f, h, scale=0.05)
    w2 = bf(E, h, f, scale=0.05)
    z = dev.grouped_nt(xe, w1, plan)
    a = dev.swiglu_fwd(z, plan)
    y, yslot = dev.output_buffer("y")
    dev.grouped_nt(a, w2, plan, out=y)
    dev.publish("y", yslot)
    out, copies = dev.combine(plan, "y", yslot, gates=gates, keep_copies=True)
    torch.cuda.synchronize()
    # reference: per token, per choice
    xf = x.float()
    ref = torch.zeros(T, h, device=DEV)
    for j in range(k):
        for e in range(E):
            m = topi[:, j] == e
            if m.any():
                zz = (xf[m] @ w1[e].float().t()).to(torch.bfloat16).float()
                aa = (torch.nn.functional.silu(zz[:, :f]) * zz[:, f:]).to(torch.bfloat16).float()
                yy = (aa @ w2[e].float().t()).to(torch.bfloat16).float()
                ref[m] += gates[m, j:j + 1] * yy
    assert rel(out, ref) < 1e-2, rel(out, ref)
    # backward products on the same plan
    d_y = torch.zeros_like(y)
    for e in range(E):
        d_y[offs[e]:offs[e] + rows_e[e]] = bf(rows_e[e], h)
    d_a = dev.grouped_nn(d_y, w2, plan)
    g2 = torch.ones(E, h, f, device=DEV)
    dev.grouped_tn_acc(d_y, a, g2, plan)
    torch.cuda.synchronize()
    for e in range(E):
        lo, hi = offs[e], offs[e] + rows_e[e]
        assert rel(d_a[lo:hi], d_y[lo:hi].float() @ w2[e].float()) < 5e-3
        assert rel(g2[e], 1 + d_y[lo:hi].float().t() @ a[lo:hi].float()) < 1e-3
    # the pull without gates is the plain sum over a token's copies
    s2, sslot = dev.output_buffer("dxe")
    s2.copy_(y)
    dev.publish("dxe", sslot)
    summed, _ = dev.combine(plan, "dxe", sslot)
    assert rel(summed, copies.float().view(T, k, h).sum(1)) < 1e-2
