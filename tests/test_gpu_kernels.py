"""Numerics of every sm_100a kernel against a plain PyTorch fp32 reference of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from matrix_fsdp_b200.ops import kernels
    return kernels


def _rand(*shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(dtype)


def _rel_err(got, ref):
    got, ref = got.float(), ref.float()
    return ((got - ref).norm() / ref.norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("shape", [(256, 512, 128), (384, 640, 320), (4096, 2048, 2048), (200, 72, 136)])
def test_gemm_majors(K, a_mn, b_mn, shape):
    M, N, Kd = shape
    torch.manual_seed(0)
    a = _rand(M, Kd)
    b = _rand(N, Kd)
    ref = a.float() @ b.float().t()
    a_in = a.t().contiguous() if a_mn else a
    b_in = b.t().contiguous() if b_mn else b
    out = K.gemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn)
    K.check_status()
    assert _rel_err(out, ref) < 1e-2
    # forcing the narrow tile must agree too
    out2 = K.gemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn, force_bn=128)
    K.check_status()
    assert _rel_err(out2, ref) < 1e-2


@pytest.mark.parametrize("a_mn", [False, True])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("shape", [(512, 512, 256), (384, 320, 200), (1024, 2304, 512), (4096, 2048, 2048), (136, 72, 64)])
def test_gemm_cta_pair_kernel(K, a_mn, b_mn, shape):
    """The two-CTA (cta_group::2) kernel: 256 x 256 tiles over a cluster of two, every operand-major form, ragged
    edges (rows / columns / reduce length that do not fill a tile), and the scale / add epilogue."""
    M, N, Kd = shape
    torch.manual_seed(M + N)
    a, b, c = _rand(M, Kd), _rand(N, Kd), _rand(M, N)
    ref = a.float() @ b.float().t()
    a_in = a.t().contiguous() if a_mn else a
    b_in = b.t().contiguous() if b_mn else b
    out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
    K.gemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn, out=out, force_bn=2)
    K.check_status()
    assert torch.isfinite(out.float()).all()
    assert _rel_err(out, ref) < 1e-2
    out2 = K.gemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn, cin=c, alpha=0.5, beta=2.0, force_bn=2)
    K.check_status()
    assert _rel_err(out2, 0.5 * ref + 2.0 * c.float()) < 1e-2
    # repeated launches (barrier phases, tensor-memory alloc / free across launches) stay correct
    for _ in range(3):
        out3 = K.gemm(a_in, b_in, a_mn_major=a_mn, b_mn_major=b_mn, force_bn=2)
    assert torch.equal(out3, out)


def test_gemm_alpha_beta_cin(K):
    torch.manual_seed(1)
    a, b, c = _rand(512, 256), _rand(384, 256), _rand(512, 384)
    ref = 0.5 * (a.float() @ b.float().t()) + 2.0 * c.float()
    out = K.gemm(a, b, cin=c, alpha=0.5, beta=2.0)
    K.check_status()
    assert _rel_err(out, ref) < 1e-2


def test_gemm_strided_views(K):
    torch.manual_seed(2)
    big = _rand(512, 1024)
    a = big[:, 256:512]            # row stride 1024, K = 256
    b = _rand(128, 256)
    out_big = torch.zeros(512, 512, device="cuda", dtype=torch.bfloat16)
    out = out_big[:, 128:256]
    K.gemm(a, b, out=out)
    K.check_status()
    assert _rel_err(out, a.float() @ b.float().t()) < 1e-2
    assert out_big[:, :128].abs().sum() == 0 and out_big[:, 256:].abs().sum() == 0


def test_grouped_gemm_m_and_k(K):
    torch.manual_seed(3)
    G, N, Kd = 4, 256, 192
    rows = [128, 0, 256, 128]
    tile_group = []
    for g, r in enumerate(rows):
        tile_group += [g] * (r // 128)
    tile_group.append(-1)  # a padding tile that is skipped
    Mtot = 128 * len(tile_group)
    a = _rand(Mtot, Kd)
    w = _rand(G, N, Kd)
    tg = torch.tensor(tile_group, dtype=torch.int32, device="cuda")
    out = torch.zeros(Mtot, N, device="cuda", dtype=torch.bfloat16)
    K.grouped_gemm_m(a, w, tg, out=out)
    K.check_status()
    for t, g in enumerate(tile_group):
        sl = slice(t * 128, (t + 1) * 128)
        if g < 0:
            assert out[sl].abs().sum() == 0
        else:
            assert _rel_err(out[sl], a[sl].float() @ w[g].float().t()) < 1e-2
    # dgrad form: B stored [G, K(reduce), N]
    dy = _rand(Mtot, N)
    dx = torch.zeros(Mtot, Kd, device="cuda", dtype=torch.bfloat16)
    K.grouped_gemm_m(dy, w, tg, b_mn_major=True, out=dx)
    K.check_status()
    for t, g in enumerate(tile_group):
        if g >= 0:
            sl = slice(t * 128, (t + 1) * 128)
            assert _rel_err(dx[sl], dy[sl].float() @ w[g].float()) < 1e-2
    # wgrad form
    offs = [0]
    for r in rows:
        offs.append(offs[-1] + r)
    go = torch.tensor(offs, dtype=torch.int32, device="cuda")
    dw = K.grouped_gemm_k(dy[: offs[-1]], a[: offs[-1]], go, G)
    K.check_status()
    for g in range(G):
        ref = dy[offs[g]:offs[g + 1]].float().t() @ a[offs[g]:offs[g + 1]].float()
        if rows[g] == 0:
            assert dw[g].abs().sum() == 0
        else:
            assert _rel_err(dw[g], ref) < 1e-2


@pytest.mark.parametrize("H", [256, 2048, 4096, 5120])
def test_rmsnorm(K, H):
    torch.manual_seed(4)
    x, w = _rand(300, H), (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    y, rstd = K.rmsnorm_fwd(x, w, 1e-5)
    xf = x.float().requires_grad_(True)
    wf = w.float().requires_grad_(True)
    ref = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    assert _rel_err(y, ref) < 1e-2
    dy, dres = _rand(300, H), _rand(300, H)
    ref.backward(dy.float())
    dx, dw = K.rmsnorm_bwd(dy, x, w, rstd, dres=dres)
    assert _rel_err(dx, xf.grad + dres.float()) < 1e-2
    assert _rel_err(dw, wf.grad) < 1e-2


def test_rope_roundtrip_and_reference(K):
    torch.manual_seed(5)
    B, S, nH, D = 2, 64, 4, 128
    ld = 3 * nH * D
    buf = _rand(B * S, ld)
    orig = buf.clone()
    inv = 1.0 / (10000.0 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    ang = torch.arange(S, device="cuda").float()[:, None] * inv[None]
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    K.rope_(buf, cos, sin, S, 0, 2 * nH, D)  # q and k heads
    q = orig[:, : 2 * nH * D].float().view(B, S, 2 * nH, D)
    x1, x2 = q[..., : D // 2], q[..., D // 2:]
    c, s = cos[None, :, None, :], sin[None, :, None, :]
    ref = torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).view(B * S, -1)
    assert _rel_err(buf[:, : 2 * nH * D], ref) < 1e-2
    assert torch.equal(buf[:, 2 * nH * D:], orig[:, 2 * nH * D:])
    K.rope_(buf, cos, sin, S, 0, 2 * nH, D, backward=True)
    assert _rel_err(buf, orig) < 2e-2


def test_swiglu(K):
    torch.manual_seed(6)
    T, F = 257, 688
    gu = _rand(T, 2 * F)
    guf = gu.float().requires_grad_(True)
    ref = torch.nn.functional.silu(guf[:, :F]) * guf[:, F:]
    h = K.swiglu_fwd(gu)
    assert _rel_err(h, ref) < 1e-2
    dh = _rand(T, F)
    ref.backward(dh.float())
    dgu = K.swiglu_bwd(dh, gu)
    assert _rel_err(dgu, guf.grad) < 1e-2


@pytest.mark.parametrize("V", [1024, 32000])
def test_cross_entropy(K, V):
    torch.manual_seed(7)
    rows = 130
    logits = _rand(rows, V, scale=2.0)
    tgt = torch.randint(0, V, (rows,), device="cuda")
    tgt[3] = -100
    lf = logits.float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(lf, tgt, ignore_index=-100, reduction="none")
    n_valid = (tgt != -100).sum().item()
    (ref.sum() / n_valid).backward()
    work = logits.clone()
    loss = K.cross_entropy_(work, tgt, 1.0 / n_valid)
    assert torch.allclose(loss, ref, atol=2e-2, rtol=1e-2)
    assert _rel_err(work, lf.grad) < 2e-2
    # the same with the scale read from device memory, and through the masked-target functional path
    work2 = logits.clone()
    scale_dev = torch.full((1,), 1.0 / n_valid, device="cuda")
    loss2 = K.cross_entropy_(work2, tgt, scale_dev)
    assert torch.equal(loss2, loss) and torch.equal(work2, work)
    from matrix_fsdp_b200.ops import functional as OF

    lg = logits.clone().requires_grad_(True)
    out = OF.fused_cross_entropy(lg * 1.0, tgt, ignore_index=-100)
    assert abs(float(out) - float(ref.sum() / n_valid)) < 2e-2
    out.backward()
    assert _rel_err(lg.grad, lf.grad) < 2e-2


@pytest.mark.parametrize("gdtype", [torch.bfloat16, torch.float32])
def test_adamw_flat_matches_torch(K, gdtype):
    torch.manual_seed(8)
    n = 100003
    p0 = torch.randn(n, device="cuda")
    p = p0.clone()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    lp = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    ref_p = torch.nn.Parameter(p0.clone())
    opt = torch.optim.AdamW([ref_p], lr=3e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    for step in range(1, 4):
        g = torch.randn(n, device="cuda").to(gdtype)
        ref_p.grad = g.float() * 0.5
        opt.step()
        K.adamw_flat_(p, m, v, g, lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1,
                      step=step, grad_scale=0.5, p_lp=lp)
    assert torch.allclose(p, ref_p.detach(), atol=1e-6, rtol=1e-5)
    assert torch.equal(lp, p.bfloat16())


def test_sgd_and_muon_elementwise(K):
    torch.manual_seed(9)
    n = 5000
    p0, g = torch.randn(n, device="cuda"), torch.randn(n, device="cuda")
    p, mom = p0.clone(), torch.zeros(n, device="cuda")
    ref = torch.nn.Parameter(p0.clone())
    opt = torch.optim.SGD([ref], lr=0.1, momentum=0.9, weight_decay=0.01)
    for i in range(2):
        ref.grad = g.clone()
        opt.step()
        K.sgd_flat_(p, mom, g, lr=0.1, momentum=0.9, weight_decay=0.01, first_step=(i == 0))
    assert torch.allclose(p, ref.detach(), atol=1e-6, rtol=1e-5)
    # Muon stage 1: lerp momentum + Nesterov + norm
    rows, cols = 96, 160
    buf = torch.randn(rows * cols, device="cuda")
    gm = torch.randn(rows * cols, device="cuda")
    ref_buf = buf.clone().lerp_(gm, 1 - 0.95)
    ref_u = gm.lerp(ref_buf, 0.95)
    u = torch.empty(rows * cols, device="cuda", dtype=torch.bfloat16)
    ss = torch.zeros(1, device="cuda")
    K.muon_momentum(buf, gm, u, ss, 0.95, 1.0, True)
    assert torch.allclose(buf, ref_buf, atol=1e-6)
    assert _rel_err(u, ref_u) < 1e-2
    assert abs(ss.item() - u.float().pow(2).sum().item()) / ss.item() < 1e-3
    K.muon_normalize_(u, ss)
    assert abs(u.float().norm().item() - 1.0) < 1e-2
    pm = torch.randn(rows, cols, device="cuda")
    pm0 = pm.clone()
    o_t = _rand(cols, rows)
    K.muon_apply_(pm, o_t, rows, cols, True, 0.02, 0.1, 0.03)
    assert torch.allclose(pm, pm0 * (1 - 0.02 * 0.1) - 0.03 * o_t.float().t(), atol=1e-5)


def test_copy_segments_and_cast(K):
    torch.manual_seed(10)
    src = torch.arange(10000, device="cuda", dtype=torch.float32).bfloat16()
    dst = torch.zeros(12000, device="cuda", dtype=torch.bfloat16)
    so = torch.tensor([0, 1001, 5000], device="cuda", dtype=torch.int64)
    do = torch.tensor([8, 3003, 9001], device="cuda", dtype=torch.int64)
    ln = torch.tensor([1000, 777, 2999], device="cuda", dtype=torch.int64)
    K.copy_segments(src, dst, so, do, ln, 2999)
    ref = torch.zeros_like(dst)
    for s, d, l in zip(so.tolist(), do.tolist(), ln.tolist()):
        ref[d:d + l] = src[s:s + l]
    assert torch.equal(dst, ref)
    f = torch.randn(4099, device="cuda")
    b = torch.empty(4099, device="cuda", dtype=torch.bfloat16)
    K.cast_f32_bf16(f, b)
    assert torch.equal(b, f.bfloat16())


def test_gemm_with_fused_gather_single_gpu():
    """The all-gather-fused GEMM with its copy jobs reading from a second local buffer: rows of B
    arrive through the kernel's gather warps while tiles are computed."""
    from types import SimpleNamespace

    from matrix_fsdp_b200.ops import kernels as K

    torch.manual_seed(0)
    M, N, Kd, bn = 1024, 1536, 512, 256
    a = (torch.randn(M, Kd, device="cuda") * 0.1).bfloat16()
    src = (torch.randn(N, Kd, device="cuda") * 0.1).bfloat16()       # stands in for the peers' shards
    b = torch.zeros(N, Kd, device="cuda", dtype=torch.bfloat16)
    b[:300] = src[:300]                                              # some rows are already local
    nblocks = (N + bn - 1) // bn
    jobs, need = [], [0] * nblocks
    row = 300
    while row < N:
        blk = row // bn
        end = min(N, (blk + 1) * bn, row + 100)
        jobs.append((src.data_ptr() + row * Kd * 2, b.data_ptr() + row * Kd * 2, (end - row) * Kd * 2, blk))
        need[blk] += 1
        row = end
    dev = "cuda"
    first = [sum(need[:i]) for i in range(nblocks)]                  # jobs above are generated in block order
    plan = SimpleNamespace(
        b_ptr=b.data_ptr(), bn=bn, njobs=len(jobs), budget_ns=int(2e9), rotate=2,
        first=torch.tensor(first, dtype=torch.int32, device=dev),
        src=torch.tensor([j[0] for j in jobs], dtype=torch.int64, device=dev),
        dst=torch.tensor([j[1] for j in jobs], dtype=torch.int64, device=dev),
        nbytes=torch.tensor([j[2] for j in jobs], dtype=torch.int32, device=dev),
        flag_idx=torch.tensor([j[3] for j in jobs], dtype=torch.int32, device=dev),
        need=torch.tensor(need, dtype=torch.int32, device=dev),
        flags=torch.zeros(2 * nblocks, dtype=torch.int32, device=dev))
    out = K.gemm_ag(a, b, plan)
    torch.cuda.synchronize()
    K.check_status()
    assert torch.equal(b, src)
    ref = a.float() @ src.float().t()
    assert (out.float() - ref).abs().max().item() < 2e-2
    # a second call with the rows in place and no jobs is a plain GEMM
    plan.njobs, plan.need = 0, torch.zeros(nblocks, dtype=torch.int32, device=dev)
    out2 = K.gemm_ag(a, b, plan)
    torch.cuda.synchronize()
    assert torch.equal(out2, out)


@pytest.mark.parametrize("T,V,H", [(1000, 517, 256), (8192, 32000, 2048), (300, 40, 1024)])
def test_embedding_backward_matches_fp32(K, T, V, H):
    """Sum of the output-gradient rows of equal ids: against an fp32 index_add, with heavy duplicates, ids outside
    the vocabulary, accumulation into an existing gradient, and run-to-run bitwise equality."""
    torch.manual_seed(T + V)
    dy = _rand(T, H)
    ids = torch.randint(0, V, (T,), device="cuda")
    ids[: T // 4] = ids[0]                      # one id that occurs T/4 times
    ids[-1] = -1                                # an id that is not in the vocabulary contributes nothing
    valid = ids >= 0
    ref = torch.zeros(V, H, device="cuda").index_add_(0, ids[valid], dy[valid].float())
    out = torch.full((V, H), float("nan"), device="cuda", dtype=torch.bfloat16)
    K.embedding_bwd(dy, ids, out)
    assert torch.isfinite(out.float()).all()
    assert _rel_err(out, ref) < 5e-3
    again = torch.empty_like(out)
    K.embedding_bwd(dy, ids, again)
    assert torch.equal(out, again)
    prev = _rand(V, H)
    acc = prev.clone()
    K.embedding_bwd(dy, ids, acc, accumulate=True)
    assert _rel_err(acc, ref + prev.float()) < 5e-3
    untouched = torch.ones(V, dtype=torch.bool, device="cuda")
    untouched[ids[valid]] = False
    assert torch.equal(acc[untouched], prev[untouched])


def test_embedding_function_gradient_matches_torch(K):
    from matrix_fsdp_b200.ops import functional as OF

    torch.manual_seed(3)
    w = torch.nn.Parameter(_rand(1024, 512))
    w_ref = torch.nn.Parameter(w.detach().clone())
    ids = torch.randint(0, 1024, (4, 96), device="cuda")
    up = _rand(4, 96, 512)
    OF.embedding(ids, w, w).backward(up)
    torch.nn.functional.embedding(ids, w_ref).backward(up)
    assert w.grad is not None and w.grad.shape == w_ref.grad.shape
    assert _rel_err(w.grad, w_ref.grad.float()) < 5e-3


def test_grouped_gemms_on_cta_pairs(K):
    """M-grouped GEMM with the caller's promise of 256-row groups, and K-grouped GEMM with 256-row outputs: both
    run the two-CTA kernel and must match fp32."""
    torch.manual_seed(11)
    G, N, Kd = 3, 384, 320
    rows = [256, 512, 256]
    tile_group = torch.tensor(sum(([g] * (r // 128) for g, r in enumerate(rows)), []), dtype=torch.int32, device="cuda")
    a, w, c = _rand(sum(rows), Kd), _rand(G, N, Kd), _rand(sum(rows), N)
    out = torch.full((sum(rows), N), float("nan"), device="cuda", dtype=torch.bfloat16)
    K.grouped_gemm_m(a, w, tile_group, out=out, cin=c, alpha=1.0, beta=0.5, groups_of_256_rows=True)
    K.check_status()
    r0 = 0
    for g, r in enumerate(rows):
        ref = a[r0:r0 + r].float() @ w[g].float().t() + 0.5 * c[r0:r0 + r].float()
        assert _rel_err(out[r0:r0 + r], ref) < 1e-2, g
        r0 += r
    # MN-major B (the aX + BX product of Newton-Schulz)
    wt = w.transpose(1, 2).contiguous()
    out2 = K.grouped_gemm_m(a, wt, tile_group, b_mn_major=True, groups_of_256_rows=True)
    K.check_status()
    r0 = 0
    for g, r in enumerate(rows):
        assert _rel_err(out2[r0:r0 + r], a[r0:r0 + r].float() @ w[g].float().t()) < 1e-2, g
        r0 += r
    # K-grouped, 512-row outputs
    kk, M2, N2 = 192, 512, 320
    a2, b2 = _rand(G * kk, M2), _rand(G * kk, N2)
    offsets = torch.arange(G + 1, dtype=torch.int32, device="cuda") * kk
    o3 = K.grouped_gemm_k(a2, b2, offsets, G)
    K.check_status()
    ref3 = torch.bmm(a2.view(G, kk, M2).float().transpose(1, 2), b2.view(G, kk, N2).float())
    assert _rel_err(o3, ref3) < 1e-2


@pytest.mark.parametrize("n,shift", [(1, 0), (7, 0), (8, 0), (4099, 0), (4096, 1), (4096, 4), (1 << 20, 0)])
def test_cast_bf16_f32(K, n, shift):
    """Every bf16 value has the same fp32 value: exact, with and without 16-byte aligned bases."""
    src = torch.randn(n + shift, device="cuda").bfloat16()[shift:]
    dst = torch.empty(n + shift, device="cuda")[shift:]
    K.cast_bf16_f32(src, dst)
    assert torch.equal(dst, src.float())


@pytest.mark.parametrize("n,with_lp,aligned", [(5, True, True), (1024, True, True), (1001, False, True), (1000, True, False)])
def test_adamw_of_parameters_outside_units(n, with_lp, aligned):
    """One fused launch per parameter against the torch-op update (fp32, terms of one sum in another order: 1e-6),
    whose path unaligned views keep."""
    from matrix_fsdp_b200.optim.flat import FlatShardedAdamW, _adamw_reference_

    torch.manual_seed(0)
    base = torch.randn(n + 1, device="cuda")
    p = torch.nn.Parameter(base[0 if aligned else 1:][:n])
    lp = torch.zeros(n, device="cuda", dtype=torch.bfloat16)
    opt = FlatShardedAdamW([p], lr=1e-2, betas=(0.9, 0.95), weight_decay=0.1)
    if with_lp:
        opt._low_precision_of = lambda _: lp
    want, m, v = p.detach().clone(), torch.zeros_like(p.data), torch.zeros_like(p.data)
    for step in (1, 2):
        p.grad = torch.randn(n, device="cuda")
        _adamw_reference_(want, m, v, p.grad, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step,
                          grad_scale=1.0)
        opt.step()
        assert (p.detach() - want).abs().max() <= 1e-6 * want.abs().max()
        assert (id(p) in opt.lp_written) == (with_lp and aligned)
        if with_lp and aligned:
            assert torch.equal(lp, p.detach().bfloat16())


@pytest.mark.parametrize("T,V,H,ids", [(1, 8, 8, "one"), (300, 5000, 264, "all the same"), (3000, 4097, 72, "few"), (4096, 4096, 2056, "uniform")])
def test_embedding_backward_orders_positions(K, T, V, H, ids):
    """Ids that occur once, up to and beyond the 256 positions that a block sorts, and not at all: the same bits every
    time, within one bf16 rounding of the 64-bit sums plus fp32 rounding of n terms."""
    g = torch.Generator(device="cuda").manual_seed(T)
    t = dict(zip(("one", "all the same", "few", "uniform"),
                 (lambda: torch.full((T,), V - 1), lambda: torch.full((T,), 7), lambda: torch.randint(0, 9, (T,)) * 455,
                  lambda: torch.randint(0, V, (T,)))))[ids]().to("cuda", torch.int64)
    dy = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    outs = [K.embedding_bwd(dy, t, torch.full((V, H), float("nan"), device="cuda", dtype=torch.bfloat16)) for _ in range(3)]
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    want = torch.zeros(V, H, dtype=torch.float64, device="cuda").index_add_(0, t, dy.double())
    size = torch.zeros(V, H, dtype=torch.float64, device="cuda").index_add_(0, t, dy.double().abs())
    assert ((outs[0].double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -23 * T * size).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,shift,f", [(1, 0, 0.5), (7, 0, -3.0), (4103, 0, 0.3), (4096, 1, 0.3), (4096, 0, 1.0), (3 << 20, 0, 0.7)])
def test_scale_and_sum_of_squares(K, n, shift, f, dtype):
    """One fp32 product and one rounding per element: exact against the same in torch.  The sum of n squares in fp32,
    a few hundred terms per thread: 1e-5."""
    x = torch.randn(n + shift, device="cuda").to(dtype)[shift:]
    s = torch.tensor(f, device="cuda")
    total, want = x.double().pow(2).sum(), (x.float() * s).to(dtype)
    assert (K.sumsq(x).double() - total).abs() <= 1e-5 * total
    assert torch.equal(K.scale_(x, s), want)


@pytest.mark.parametrize("rows,V,pad", [(1, 8, 0), (5, 1016, 8), (700, 1032, 0), (149, 4104, 0), (450, 16392, 0), (300, 32760, 8), (297, 49152, 0)])
def test_cross_entropy_block_sizes(K, rows, V, pad):
    """Every block size, vectors that do not divide the block, row pitches above V; ignored targets, -inf logits in
    whole threads' shares.  Loss: fp32 sums (1e-5); gradient: one bf16 rounding."""
    torch.manual_seed(rows)
    logits = (3 * torch.randn(rows, V + pad, device="cuda")).bfloat16()
    logits[:, V // 2:] -= 2.0
    if V > 64:
        logits[rows // 2, 8:V - 8] = -math.inf
    target = torch.randint(0, V, (rows,), device="cuda")
    target[rows // 2] = 0
    if rows > 2:
        target[1] = -100
    x = logits[:, :V].double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(x, target, ignore_index=-100, reduction="none")
    (grad,) = torch.autograd.grad(want.sum() * 0.25, x)
    tail = logits[:, V:].clone()
    loss = K.cross_entropy_(logits[:, :V], target, 0.25)
    K.check_status()
    assert (loss.double() - want).abs().max() <= 1e-5 * max(1.0, want.abs().max().item())
    assert ((logits[:, :V].double() - grad).abs() <= 2 ** -8 * grad.abs() + 1e-7).all()
    assert torch.equal(logits[:, V:], tail)


@pytest.mark.parametrize("rows", [1, 7, 9, 1185, 2500])
@pytest.mark.parametrize("H", [8, 264, 520, 1032, 2056, 4104, 8192])
def test_rmsnorm_rows_and_widths(K, rows, H):
    """One, two and four warps per row with remainders, fewer rows than a block takes, one and several trips.  Bounds: one
    bf16 rounding per element (2^-8) of values whose fp32 terms are a few rounding errors off."""
    torch.manual_seed(rows + H)
    x, w = _rand(rows, H), (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    dy, dres = _rand(rows, H), _rand(rows, H)
    y, rstd = K.rmsnorm_fwd(x, w, 1e-5)
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    ref = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    ref.backward(dy.double())
    assert _rel_err(y, ref) < 2 ** -8 and torch.allclose(rstd.double(), torch.rsqrt(x.double().pow(2).mean(-1) + 1e-5), rtol=1e-5)
    for res in (dres, None):
        old = torch.randn(H, device="cuda").bfloat16()
        acc = old.clone()
        dx, dw = K.rmsnorm_bwd(dy, x, w, rstd, dres=res, dw_out=acc, accumulate_dw=res is None)
        assert _rel_err(dx, xd.grad + (res.double() if res is not None else 0)) < 2 ** -7
        assert _rel_err(acc, wd.grad + (old.double() if res is None else 0)) < 2 ** -7
        assert dw is acc


@pytest.mark.parametrize("M,N,Kd,shift,pitch", [(200, 72, 64, 0, 72), (256, 264, 128, 0, 272), (300, 320, 64, 3, 331), (513, 1000, 192, 8, 1016)])
def test_gemm_adds_cin_of_any_pitch(K, M, N, Kd, shift, pitch):
    """Whole 64-column chunks by vectors read ahead, the right edge and rows off the 16-byte grid element by element, and
    Cin that is the output itself.  Bound: one bf16 rounding of an fp32 sum."""
    torch.manual_seed(M)
    a, b = _rand(M, Kd, scale=Kd ** -0.5), _rand(N, Kd)
    c = torch.randn(M * pitch + shift, device="cuda").bfloat16()[shift:].as_strided((M, N), (pitch, 1))
    want = 0.5 * (a.double() @ b.double().t()) - 2.0 * c.double()
    for force in (0, 2, 128, 256):
        out = K.gemm(a, b, cin=c, alpha=0.5, beta=-2.0, force_bn=force)
        assert _rel_err(out, want) < 2 ** -8, force
    inplace = c.contiguous()
    K.gemm(a, b, cin=inplace, out=inplace, alpha=0.5, beta=-2.0)
    assert _rel_err(inplace, want) < 2 ** -8
    K.check_status()


@pytest.mark.parametrize("factor", [0.5, 1.0])
def test_scaled_cross_entropy_is_walked_once(factor):
    """The gradient lies in the logits buffer and takes the upstream factor there: the first walk is right (two bf16
    roundings), a second over a kept graph is refused."""
    from matrix_fsdp_b200.ops import functional as OF

    torch.manual_seed(0)
    logits = _rand(65, 1000).requires_grad_(True)
    target = torch.randint(0, 1000, (65,), device="cuda")
    loss = OF.fused_cross_entropy(logits * 1, target) * factor
    (grad,) = torch.autograd.grad(loss, logits, retain_graph=True)
    x = logits.detach().double().requires_grad_(True)
    (want,) = torch.autograd.grad(torch.nn.functional.cross_entropy(x, target) * factor, x)
    assert ((grad.double() - want).abs() <= 2 ** -7 * want.abs() + 1e-9).all()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(loss, logits)


def test_adamw_records_the_low_precision_copy_for_autograd():
    from matrix_fsdp_b200.optim.flat import FlatShardedAdamW

    p = torch.nn.Parameter(torch.randn(64, device="cuda"))
    p.grad = torch.randn(64, device="cuda")
    shard = torch.zeros(128, device="cuda", dtype=torch.bfloat16)
    opt = FlatShardedAdamW([p], lr=1e-2)
    opt._low_precision_of = lambda _: shard[64:]
    version = shard._version
    opt.step()
    assert torch.equal(shard[64:], p.detach().bfloat16()) and shard._version > version


def _adamw_64(p, m, v, g, step, lr, beta1, beta2, eps, weight_decay):
    m.mul_(beta1).add_(g, alpha=1 - beta1)
    v.mul_(beta2).addcmul_(g, g, value=1 - beta2)
    p.mul_(1 - lr * weight_decay).sub_(lr / (1 - beta1 ** step) * m / ((v / (1 - beta2 ** step)).sqrt() + eps))


@pytest.mark.parametrize("route", ["outside units", "flat", "reduction"])
@pytest.mark.parametrize("betas", [(0.9, 0.95), (0.9, 0.999), (0.0, 0.99999)])
@pytest.mark.parametrize("first", [1, 1000])
def test_adamw_constants_and_rounding(K, route, betas, first):
    """Three steps from step ``first`` against 64 bits, on each way into the update.  Moments: a handful of fp32 roundings
    a step (the smallest ones, below the normal range, to two units of their spacing outside units; the other kernels
    flush them); the distance covered by the parameter: the same (approximate root and quotients: 4 units in the last
    place more), plus 2.5 * 2^-24 of the parameter itself per step (decay factor, its product, the sum)."""
    import ctypes as C

    from matrix_fsdp_b200.ops import lib
    from matrix_fsdp_b200.optim.flat import FlatShardedAdamW
    from matrix_fsdp_b200.parallel import peer  # noqa: F401  (its entries' signatures)

    torch.manual_seed(first)
    n, hp = 4099, dict(lr=1e-3, eps=1e-8, weight_decay=0.1)
    p0 = torch.randn(n, device="cuda")
    m0, v0 = 1e-3 * torch.randn(n, device="cuda"), 1e-6 * torch.rand(n, device="cuda")
    if first == 1:
        m0.zero_(), v0.zero_()
    p, m, v = torch.nn.Parameter(p0.clone()), m0.clone(), v0.clone()
    want = [t.double() for t in (p0, m0, v0)]
    opt = FlatShardedAdamW([p], betas=betas, **hp)
    opt.state[p] = dict(step=torch.tensor(float(first - 1)), exp_avg=m, exp_avg_sq=v)
    seg = torch.tensor([0, 0, n], device="cuda")
    for step in range(first, first + 3):
        p.grad = 1e-3 * torch.randn(n, device="cuda")
        p.grad[:32] = 1e-20
        if route == "outside units":
            opt.step()
        elif route == "flat":
            K.adamw_flat_(p.data, m, v, p.grad, beta1=betas[0], beta2=betas[1], step=step, **hp)
        else:
            # one rank reducing its own gradient: no peer to wait for
            status = K.status_word()
            rc = lib.load(required=True).mfsdp_rs_pull_adamw(
                (C.c_ulonglong * 1)(p.grad.data_ptr()), 1, 0, seg.data_ptr(), seg[1:].data_ptr(), seg[2:].data_ptr(), 1, n, 0,
                1.0, p.data_ptr(), m.data_ptr(), v.data_ptr(), None, hp["lr"], *betas, hp["eps"], hp["weight_decay"], step,
                status.data_ptr(), torch.cuda.current_stream().cuda_stream)
            assert rc == 0
        _adamw_64(*want, p.grad.double(), step, beta1=betas[0], beta2=betas[1], **hp)
    K.check_status()
    assert ((m.double() - want[1]).abs() <= 1e-6 * want[1].abs() + 3 * 2 ** -24 * 3e-3).all()
    tiny = 6 * 2 ** -149 if route == "outside units" else 3 * 2 ** -126
    assert ((v.double() - want[2]).abs() <= 1e-6 * want[2] + tiny).all()
    moved = (want[0] - p0.double()).abs()
    assert ((p.detach().double() - want[0]).abs() <= 2e-6 * moved + 4 * 2 ** -23 * p0.double().abs().clamp_min(2 ** -8)).all()


def test_rmsnorm_of_no_rows(K):
    """An empty batch goes through both directions; it adds nothing to the weight's gradient."""
    from matrix_fsdp_b200.ops import functional as OF

    x, w = torch.empty(0, 264, device="cuda", dtype=torch.bfloat16), _rand(264)
    y, rstd = K.rmsnorm_fwd(x, w, 1e-5)
    assert y.shape == x.shape and rstd.shape == (0,)
    dx, dw = K.rmsnorm_bwd(y, x, w, rstd)
    assert dx.shape == x.shape and torch.equal(dw, torch.zeros_like(w))
    old = w.clone()
    K.rmsnorm_bwd(y, x, w, rstd, dw_out=old, accumulate_dw=True)
    assert torch.equal(old, w)
    x.requires_grad_(True), w.requires_grad_(True)
    gx, gw = torch.autograd.grad(OF.rms_norm(x, w).sum(), (x, w))
    assert gx.shape == x.shape and torch.equal(gw, torch.zeros_like(w))


@pytest.mark.parametrize("rows", [1, 3, 150])
@pytest.mark.parametrize("H", [8200, 12296, 16384])
def test_rmsnorm_forward_of_the_widest_rows(K, rows, H):
    """Eight warps per row, up to the last width that a CTA's registers hold; wider rows are refused."""
    torch.manual_seed(rows + H)
    x, w = _rand(rows, H), (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    y, rstd = K.rmsnorm_fwd(x, w, 1e-5)
    want = torch.rsqrt(x.double().pow(2).mean(-1) + 1e-5)
    assert torch.allclose(rstd.double(), want, rtol=1e-5)
    assert _rel_err(y, x.double() * want[:, None] * w.double()) < 2 ** -8


def test_rmsnorm_refuses_rows_wider_than_a_block_holds(K):
    x, w = _rand(2, 16392), _rand(16392)
    with pytest.raises(RuntimeError):
        K.rmsnorm_fwd(x, w, 1e-5)


@pytest.mark.parametrize("where", ["current stream", "second stream", "captured"])
def test_dependent_launches_keep_stream_order(K, where):
    """Kernels that may start before their predecessor has ended wait for it before they touch memory: a chain whose
    buffers are freed behind each launch (the next kernel writes into what its predecessor still reads, if it is early)
    gives the bits of the same chain with a synchronisation after every launch."""
    from matrix_fsdp_b200.ops import attention as A

    torch.manual_seed(0)
    B, S, nH, F = 2, 200, 2, 328
    H, T, V = nH * 128, B * S, 1000
    x, dy = torch.empty(T, H, device="cuda", dtype=torch.bfloat16), _rand(T, H)
    w = (1 + 0.1 * torch.randn(H, device="cuda")).bfloat16()
    qkv_w, o_w, gu_w, d_w, head = (_rand(n, k, scale=k ** -0.5) for n, k in ((3 * H, H), (H, H), (2 * F, H), (H, F), (V, H)))
    angles = torch.randn(S, 64, device="cuda")
    cos, sin = angles.cos(), angles.sin()
    target = torch.randint(0, V, (T,), device="cuda")

    def chain(after=lambda: None):
        def run(fn, *args, **kw):
            out = fn(*args, **kw)
            after()
            return out

        y, rstd = run(K.rmsnorm_fwd, x, w, 1e-5)
        qkv = run(K.gemm, y, qkv_w)
        del y
        run(K.rope_, qkv, cos, sin, S, 0, 2 * nH, 128)
        att, lse = run(A.attention_fwd, qkv, B, S, nH, 128)
        h = run(K.gemm, att, o_w, cin=x, beta=1.0)
        gu = run(K.gemm, h, gu_w)
        act = run(K.swiglu_fwd, gu)
        dgu = run(K.swiglu_bwd, act, gu)
        del gu
        out = run(K.gemm, act, d_w, cin=h, beta=1.0)
        del act
        logits = run(K.gemm, out, head)
        loss = run(K.cross_entropy_, logits, target, 1.0 / T)
        dout = run(K.gemm, logits, head, b_mn_major=True)
        del logits
        dqkv = run(A.attention_bwd, dout, qkv, att, lse, B, S, nH, 128)
        del qkv, att, lse
        dx, dw = run(K.rmsnorm_bwd, dy, x, w, rstd, dres=dout)
        return loss, dgu, out, dqkv, dx, dw

    stream = torch.cuda.Stream() if where != "current stream" else torch.cuda.current_stream()
    if where == "captured":
        x.copy_(_rand(T, H))
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            chain()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = chain()
    for _ in range(10):
        x.copy_(_rand(T, H))
        want = chain(torch.cuda.synchronize)
        if where == "captured":
            graph.replay()
        else:
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                got = chain()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    K.check_status()


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("n,H", [(257, 8), (261, 2056), (262, 72), (512, 2048), (513, 4104)])
def test_embedding_backward_of_a_frequent_id(K, n, H, accumulate):
    """More positions of one id than a block sorts: whole and partial lists of 256, remainders of the copies in flight,
    column ranges that leave threads idle.  The fp32 sum in the order of the positions, bit for bit."""
    torch.manual_seed(n)
    ids = torch.full((2 * n,), 3, device="cuda")
    ids[1::2] = torch.randint(4, 40, (n,), device="cuda")
    dy, old = _rand(2 * n, H), _rand(41, H)
    out = old.clone()
    K.embedding_bwd(dy, ids, out, accumulate=accumulate)
    want = old[3].float() if accumulate else torch.zeros(H, device="cuda")
    for row in dy[0::2].float():
        want = want + row
    assert torch.equal(out[3], want.bfloat16())
    total = torch.zeros(41, H, dtype=torch.float64, device="cuda").index_add_(0, ids, dy.double())
    if accumulate:
        total += old.double()
    assert _rel_err(out, total) < 2 ** -8


@pytest.mark.parametrize("rows,H", [(14300, 264), (14208, 512), (7105, 520), (7104, 1024), (7110, 1032), (7104, 1536), (3553, 1544),
                                    (3552, 2048), (3560, 2056), (3552, 3072), (2664, 3080), (2665, 4096), (1777, 4104),
                                    (1776, 6144), (1030, 6152)])
def test_rmsnorm_bwd_with_several_blocks_per_sm(K, rows, H):
    """Row counts from which two or three CTAs share an SM, at both ends of each kernel's widths, and one that keeps a
    single CTA.  Bounds as in test_rmsnorm_rows_and_widths."""
    test_rmsnorm_rows_and_widths(K, rows=rows, H=H)


@pytest.mark.parametrize("H", [256, 264, 768, 776, 1544, 3072, 3080, 6144, 6152, 10240, 10248, 14336, 14344])
def test_rmsnorm_forward_vectors_per_lane(K, H):
    """Both sides of the widths at which a lane takes one vector more, or a row more warps."""
    test_rmsnorm_forward_of_the_widest_rows(K, rows=37, H=H)
