"""tcgen05 causal attention against an fp32 PyTorch reference of the same op."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(qkv, B, S, nH, hd):
    H = nH * hd
    q, k, v = (qkv[:, i * H:(i + 1) * H].float().view(B, S, nH, hd).transpose(1, 2) for i in range(3))
    s = (q @ k.transpose(-1, -2)) / math.sqrt(hd)
    mask = torch.ones(S, S, dtype=torch.bool, device=qkv.device).tril()
    s = s.masked_fill(~mask, float("-inf"))
    lse = torch.logsumexp(s, dim=-1)
    o = torch.softmax(s, dim=-1) @ v
    return o.transpose(1, 2).reshape(B * S, H), lse


@pytest.mark.parametrize("B,S,nH", [(1, 128, 1), (2, 256, 2), (1, 1024, 4), (2, 384, 3), (1, 200, 2)])
def test_attention_fwd_matches_fp32(B, S, nH):
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    assert A.fwd_available(), "attention kernel missing from the kernel library"
    torch.manual_seed(0)
    hd = 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    torch.cuda.synchronize()
    K.check_status()
    ref_o, ref_lse = _ref(qkv, B, S, nH, hd)
    assert torch.isfinite(out).all()
    assert (out.float() - ref_o).abs().max().item() < 3e-2
    assert (lse - ref_lse).abs().max().item() < 2e-3


def test_attention_fwd_large_scores_rescale():
    """Scores that grow along the key axis force the lazy O rescale to fire."""
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    torch.manual_seed(1)
    B, S, nH, hd = 1, 512, 2, 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    ramp = torch.linspace(0.2, 3.0, S, device="cuda").repeat(B)[:, None]
    qkv[:, nH * hd:2 * nH * hd] = (qkv[:, nH * hd:2 * nH * hd].float() * ramp).bfloat16()
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    torch.cuda.synchronize()
    K.check_status()
    ref_o, ref_lse = _ref(qkv, B, S, nH, hd)
    assert (out.float() - ref_o).abs().max().item() < 4e-2
    assert (lse - ref_lse).abs().max().item() < 5e-3


@pytest.mark.parametrize("B,S,nH", [(1, 128, 1), (2, 256, 2), (1, 1024, 2), (2, 384, 3), (1, 200, 2), (2, 130, 1)])
def test_attention_bwd_matches_fp32(B, S, nH):
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    assert A.bwd_available(), "attention backward kernel missing from the kernel library"
    torch.manual_seed(2)
    hd = 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    dout = torch.randn(B * S, nH * hd, device="cuda", dtype=torch.bfloat16)
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    dqkv = A.attention_bwd(dout, qkv, out, lse, B, S, nH, hd)
    torch.cuda.synchronize()
    K.check_status()
    ref_in = qkv.float().requires_grad_(True)
    ref_o, _ = _ref(ref_in, B, S, nH, hd)
    (ref_g,) = torch.autograd.grad(ref_o, ref_in, dout.float())
    assert torch.isfinite(dqkv).all()
    err = (dqkv.float() - ref_g).abs().max().item()
    assert err < 6e-2 * max(1.0, ref_g.abs().max().item() / 4), err
    rel = (dqkv.float() - ref_g).norm() / ref_g.norm()
    assert rel.item() < 2e-2, rel.item()


@pytest.mark.parametrize("B,S,nH,heads", [(1, 1, 150, (0, 149)), (2, 100, 80, (3, 79)), (1, 128, 150, (0, 7)), (1, 129, 80, (0, 79)),
                                          (2, 255, 40, (1, 39)), (1, 257, 50, (0, 49)), (1, 385, 40, (2, 39)),
                                          (3, 1333, 16, (0, 15)), (1, 8192, 20, (0, 15, 16, 19))])
def test_attention_fwd_two_tiles_per_block(B, S, nH, heads):
    """Grids of more than 148 query tiles, which take the kernel with two of them per block from two tiles per row on: a
    lone tile, a second tile of one row, odd and even tile counts, and a last group of heads that is not full.  Bounds as
    for the other kernel."""
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    assert (S + 127) // 128 * B * nH > 148
    torch.manual_seed(0)
    hd = 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    K.check_status()
    assert torch.isfinite(out).all() and torch.isfinite(lse).all()
    for b in range(B):
        for h in heads:
            one = torch.cat([qkv[b * S:(b + 1) * S, (i * nH + h) * hd:(i * nH + h + 1) * hd] for i in range(3)], dim=1)
            ref_o, ref_lse = _ref(one, 1, S, 1, hd)
            assert (out[b * S:(b + 1) * S, h * hd:(h + 1) * hd].float() - ref_o).abs().max().item() < 3e-2
            assert (lse[b, h] - ref_lse[0, 0]).abs().max().item() < 2e-3


def test_attention_fwd_two_tiles_rescale():
    """Scores that grow along the key axis, in steps that force the rescaling of O in some warps and not in others."""
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    torch.manual_seed(1)
    B, S, nH, hd = 1, 700, 32, 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    ramp = torch.linspace(0.2, 6.0, S, device="cuda")[:, None]
    qkv[:, nH * hd:2 * nH * hd] = (qkv[:, nH * hd:2 * nH * hd].float() * ramp).bfloat16()
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    K.check_status()
    ref_o, ref_lse = _ref(qkv, B, S, nH, hd)
    assert (out.float() - ref_o).abs().max().item() < 4e-2
    assert (lse - ref_lse).abs().max().item() < 5e-3


@pytest.mark.parametrize("B,S,nH,heads", [(1, 1, 3, (0, 2)), (2, 127, 2, (0, 1)), (1, 129, 2, (1,)), (2, 1000, 3, (0, 2)),
                                          (1, 8192, 17, (0, 15, 16))])
def test_attention_bwd_tiles_and_head_groups(B, S, nH, heads):
    """One row, both sides of a tile edge, batches whose last tile reads the next one's rows, and more heads than one
    group of the block order.  Bound: bf16 inputs, P and dS of products with fp32 sums, 1e-2 in the 2-norm."""
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    torch.manual_seed(2)
    hd = 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    dout = torch.randn(B * S, nH * hd, device="cuda", dtype=torch.bfloat16)
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    dqkv = A.attention_bwd(dout, qkv, out, lse, B, S, nH, hd)
    K.check_status()
    assert torch.isfinite(dqkv).all()
    for b in range(B):
        for h in heads:
            cols = [slice((i * nH + h) * hd, (i * nH + h + 1) * hd) for i in range(3)]
            one = torch.cat([qkv[b * S:(b + 1) * S, c] for c in cols], dim=1).float().requires_grad_(True)
            ref_o, _ = _ref(one, 1, S, 1, hd)
            (ref,) = torch.autograd.grad(ref_o, one, dout[b * S:(b + 1) * S, h * hd:(h + 1) * hd].float())
            got = torch.cat([dqkv[b * S:(b + 1) * S, c] for c in cols], dim=1).float()
            for i in range(3):
                g, w = got[:, i * hd:(i + 1) * hd], ref[:, i * hd:(i + 1) * hd]
                # with one row P is 1 and dS cancels: the rounding of dO and O remains, 2^-8 of their products
                floor = 2 ** -7 * one[:, :].norm() if S == 1 else 0.0
                assert (g - w).norm() <= 1e-2 * w.norm() + floor, (b, h, i)


@pytest.mark.parametrize("B,S,nH,two", [(2, 1000, 10, False), (2, 1000, 11, True), (1, 8100, 3, False), (1, 8100, 4, True),
                                        (150, 1, 1, False), (2, 129, 38, True)])
def test_attention_fwd_on_both_sides_of_the_line(B, S, nH, two):
    """One or two query tiles per block: 185 + tiles key tiles per query tile, more than a wave of tiles, more than one
    tile per row.  Bounds as for either kernel."""
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    nt = (S + 127) // 128
    assert (nt > 1 and nt * B * nH > 148 and B * nH * (nt + 1) > 185 + nt) == two
    torch.manual_seed(S)
    hd = 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    out, lse = A.attention_fwd(qkv, B, S, nH, hd)
    K.check_status()
    for b, h in ((0, 0), (B - 1, nH - 1)):
        one = torch.cat([qkv[b * S:(b + 1) * S, (i * nH + h) * hd:(i * nH + h + 1) * hd] for i in range(3)], dim=1)
        ref_o, ref_lse = _ref(one, 1, S, 1, hd)
        assert (out[b * S:(b + 1) * S, h * hd:(h + 1) * hd].float() - ref_o).abs().max().item() < 3e-2
        assert (lse[b, h] - ref_lse[0, 0]).abs().max().item() < 2e-3


@pytest.mark.parametrize("B,S,nH", [(3, 200, 2), (5, 64, 16), (2, 1000, 11), (4, 129, 40)])
def test_sequences_do_not_reach_into_each_other(B, S, nH):
    """Infinities and NaN in the other sequences of a batch leave the first one's results as they are, bit for bit, although
    its last tile ends behind its last row (one tile per block and two, both directions)."""
    from matrix_fsdp_b200.ops import attention as A
    from matrix_fsdp_b200.ops import kernels as K

    torch.manual_seed(S)
    hd = 128
    qkv = torch.randn(B * S, 3 * nH * hd, device="cuda", dtype=torch.bfloat16)
    dout = torch.randn(B * S, nH * hd, device="cuda", dtype=torch.bfloat16)

    def first():
        out, lse = A.attention_fwd(qkv, B, S, nH, hd)
        return out[:S], lse[0], A.attention_bwd(dout, qkv, out, lse, B, S, nH, hd)[:S]

    want = first()
    qkv[S:], dout[S:] = math.inf, math.nan
    assert all(torch.equal(a, b) for a, b in zip(first(), want))
    K.check_status()


@pytest.mark.parametrize("S", [31, 32, 33, 64, 65, 97, 161, 1023, 1024])
def test_attention_bwd_parts_that_do_not_count(S):
    """Rows short enough that whole 32 x 32 parts of a tile are left out: both sides of a part's edge, and of the row count
    from which they are computed and masked.  Bound as for the other sizes."""
    test_attention_bwd_tiles_and_head_groups(B=2, S=S, nH=3, heads=(0, 2))
