"""GPU parity of the tcgen05 attention forward (through the C-ABI) against the float64 softmax oracle.
Tolerance: rel. Frobenius <= 4e-3 for bf16 (P and O rounded to bf16), 1e-3 for f16; max abs error reported."""
import numpy as np
import pytest
import torch

from oracle import attn_oracle as ao
from oracle import gemm_oracle as go

pytestmark = pytest.mark.gpu


def _ops():
    from lightly_trian_quant_b200 import ops

    return ops


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 128, 1), (2, 77, 2), (1, 300, 3), (2, 1605, 2), (1, 1805, 1)])
def test_attn_vs_oracle(dtype, shape):
    ops = _ops()
    B, N, H = shape
    g = torch.Generator().manual_seed(N)
    qkv = torch.randn(3, B, N, H, 64, generator=g)
    qkv[0] *= 2.0          # sharper softmax
    qkv = qkv.to(dtype)
    out = ops.attn_fwd(qkv.cuda())
    ops.check_device_error()
    assert out.shape == (B, N, H * 64) and out.dtype == dtype
    ref = ao.attn_ref(qkv.float().numpy())
    err = go.rel_fro(out.float().cpu().numpy(), ref)
    assert err < (4e-3 if dtype == torch.bfloat16 else 1e-3), err


def test_attn_massive_activation_rows():
    """a few key rows with very large norm (the cls / register tokens of DINOv3): softmax stays finite and exact."""
    ops = _ops()
    B, N, H = 1, 517, 2
    g = torch.Generator().manual_seed(1)
    qkv = torch.randn(3, B, N, H, 64, generator=g)
    qkv[1, :, :5] *= 30
    qkv[0, :, 100:110] *= 10
    qkv = qkv.to(torch.bfloat16)
    out = ops.attn_fwd(qkv.cuda())
    ops.check_device_error()
    assert torch.isfinite(out).all()
    ref = ao.attn_ref(qkv.float().numpy())
    assert go.rel_fro(out.float().cpu().numpy(), ref) < 6e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attn_logits_growing_along_the_keys(dtype):
    """the key norm grows with the key index, so for most rows later key tiles hold far larger logits than the running
    maximum of the earlier ones (by more than 2^15 in the exponent domain for many of them, by less for others): the rows
    that have to raise their maximum late and rescale O, and the rows that do not, in the same warp."""
    ops = _ops()
    B, N, H = 1, 453, 2
    g = torch.Generator().manual_seed(7)
    qkv = torch.randn(3, B, N, H, 64, generator=g)
    qkv[0] *= 1.5
    qkv[1] *= (0.2 + torch.arange(N).float() / 30.0).view(1, N, 1, 1)
    qkv[0, :, ::3] *= 0.05                                  # every third query row stays flat: no rescale there
    qkv = qkv.to(dtype)
    out = ops.attn_fwd(qkv.cuda())
    ops.check_device_error()
    assert torch.isfinite(out).all()
    ref = ao.attn_ref(qkv.float().numpy())
    err = go.rel_fro(out.float().cpu().numpy(), ref)
    assert err < (6e-3 if dtype == torch.bfloat16 else 2e-3), err


def test_attn_permutation_of_keys_is_neutral():
    """size-independent property: permuting the keys (and values with them) leaves O unchanged up to rounding."""
    ops = _ops()
    B, N, H = 1, 1605, 4
    g = torch.Generator().manual_seed(2)
    qkv = torch.randn(3, B, N, H, 64, generator=g).to(torch.bfloat16).cuda()
    perm = torch.randperm(N, generator=g).cuda()
    o1 = ops.attn_fwd(qkv)
    qkv2 = qkv.clone()
    qkv2[1] = qkv[1][:, perm]
    qkv2[2] = qkv[2][:, perm]
    o2 = ops.attn_fwd(qkv2.contiguous())
    ops.check_device_error()
    assert go.rel_fro(o2.float().cpu().numpy(), o1.float().cpu().numpy()) < 4e-3


@pytest.mark.parametrize("fmt", ["mx8", "nv4", "mx4"])
def test_attn_fused_quantise_out(fmt):
    """attention with the output quantisation fused in: bit-exact against the oracle quantiser applied to the bf16
    output of the unfused kernel (same arithmetic up to the final rounding), scales in the blocked layout."""
    import numpy as np

    from oracle import quant_oracle as qo

    ops = _ops()
    B, N, H = 2, 333, 4
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(3, B, N, H, 64, generator=g).to(torch.bfloat16).cuda()
    o = ops.attn_fwd(qkv).view(B * N, H * 64)
    on = o.float().cpu().numpy()
    out = ops.ActBuf(B * N, H * 64, fmt, device="cuda")
    ts = None
    if fmt == "nv4":
        ts = qo.nv4_ts(on) * np.float32(2.0)
        out.ts.copy_(torch.from_numpy(ts))
    ops.attn_fwd_quant(qkv, out)
    ops.check_device_error()
    eq, es, _ = qo.quantize(on, fmt, ts)
    assert np.array_equal(out.q.cpu().numpy(), eq)
    assert np.array_equal(out.sf.cpu().numpy(), qo.to_blocked(es).reshape(-1))


@pytest.mark.parametrize("B,N,H", [(1, 1, 1), (40, 1, 16), (40, 64, 16), (3, 65, 2), (40, 128, 9), (2, 129, 3), (1, 192, 2), (20, 193, 16), (1, 257, 5), (2, 95, 3), (40, 96, 16), (2, 97, 3), (20, 191, 16),
                                   (1, 289, 2)])
def test_attn_tile_edges_and_items_shorter_than_the_pipeline(B, N, H):
    """token counts around the 96-key (its 32-key pieces) and 128-query tiles, and items of one to three key tiles in a CTA that works through
    several: S runs ahead of the softmax across item boundaries."""
    ops = _ops()
    g = torch.Generator().manual_seed(B + N)
    qkv = (torch.randn(3, B, N, H, 64, generator=g) * 1.5).to(torch.bfloat16)
    out = ops.attn_fwd(qkv.cuda())
    ops.check_device_error()
    err = go.rel_fro(out.float().cpu().numpy(), ao.attn_ref(qkv.float().numpy()))
    assert err < 4e-3, err


@pytest.mark.parametrize("fmt", ["mx8", "nv4", "mx4"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,N,H", [(1, 1, 2), (40, 64, 16), (2, 95, 4), (40, 96, 16), (2, 97, 2), (2, 129, 4), (1, 192, 2), (20, 193, 16), (1, 261, 12), (1, 289, 2)])
def test_attn_fused_quantise_out_at_tile_edges(fmt, dtype, B, N, H):
    """the codes and scales of the fused output around the 96-key and 128-query tiles, and where a CTA works through several items, are those that
    the row quantiser makes of the 16-bit output."""
    ops = _ops()
    g = torch.Generator(device="cuda").manual_seed(B + N)
    qkv = (torch.randn(3, B, N, H, 64, generator=g, device="cuda") * 1.5).to(dtype)
    o = ops.attn_fwd(qkv).view(B * N, H * 64)
    fused, rows = ops.ActBuf(B * N, H * 64, fmt, device="cuda"), ops.ActBuf(B * N, H * 64, fmt, device="cuda")
    if fmt == "nv4":
        for buf in (fused, rows):
            buf.ts.fill_(float(o.float().abs().max()) / 2688.0 * 2)
    ops.attn_fwd_quant(qkv, fused)
    ops.quant_rows(o, rows)
    ops.check_device_error()
    assert torch.equal(fused.q, rows.q) and torch.equal(fused.sf, rows.sf)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lo,N", [(64, 96), (64, 300), (96, 300), (288, 300)])
def test_attn_larger_logits_behind_the_first_keys(dtype, lo, N):
    """keys lo .. lo + 31 hold far larger logits than those before (more than 2^15 in the exponent domain): behind the first 64 keys, whose
    maximum the rows start with, inside the first key tile (no O to rescale yet), and in the following tiles."""
    ops = _ops()
    g = torch.Generator().manual_seed(lo + N)
    qkv = torch.randn(3, 3, N, 2, 64, generator=g)
    qkv[1, :, lo:lo + 32] *= 12
    qkv[0, :, ::4] *= 0.05                                  # rows that stay flat
    qkv = qkv.to(dtype)
    out = ops.attn_fwd(qkv.cuda())
    ops.check_device_error()
    assert torch.isfinite(out).all()
    err = go.rel_fro(out.float().cpu().numpy(), ao.attn_ref(qkv.float().numpy()))
    assert err < (4e-3 if dtype == torch.bfloat16 else 1e-3), err


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attn_one_key_far_above_the_maximum(dtype):
    """ONE key whose logit exceeds the running maximum by 0 .. 418 in the exponent domain (1.4 more from query row to query row), in every place
    of a group of 8 keys, behind the first 64 keys of the first tile and in later tiles: whichever way its exponential is taken, and
    wherever that would overflow or wrap, the row has to find its maximum."""
    ops = _ops()
    places = [*range(64, 72), 90, 95, *range(96, 104), 197, 198, 294, 295, 296, 299]
    B, N = len(places), 300
    g = torch.Generator().manual_seed(11)
    qkv = torch.randn(3, B, N, 1, 64, generator=g)
    qkv[0, ..., :2] = (torch.arange(N) * 1.4 / (32 * 0.125 * 1.4427)).view(1, N, 1, 1) / 2
    qkv[1, ..., :2] = 0
    for b, p in enumerate(places):
        qkv[1, b, p] = 0
        qkv[1, b, p, 0, :2] = 32                            # q . k = 1.4 * row * 8 / log2(e)
    qkv = qkv.to(dtype)
    out = ops.attn_fwd(qkv.cuda()).cpu()
    ops.check_device_error()
    assert torch.isfinite(out).all()
    ref = ao.attn_ref(qkv.float().numpy())
    bound = 4e-3 if dtype == torch.bfloat16 else 1e-3
    for b, p in enumerate(places):
        err = go.rel_fro(out[b].float().numpy(), ref[b])
        assert err < bound, (p, err)


def test_attn_a_key_that_is_no_number():
    """a NaN in one key, in every place of a group of 8 keys, makes every row of its head NaN, as the softmax of the oracle does."""
    ops = _ops()
    B, N = 24, 300
    qkv = torch.randn(3, B, N, 2, 64, generator=torch.Generator().manual_seed(13)).to(torch.bfloat16)
    for b in range(B):
        qkv[1, b, (64, 96, 200)[b // 8] + b % 8, 0, 5] = float("nan")
    out = ops.attn_fwd(qkv.cuda()).cpu().view(B, N, 2, 64)
    ops.check_device_error()
    assert out[:, :, 0].isnan().all() and torch.isfinite(out[:, :, 1]).all()


def test_attn_outputs_at_16_byte_alignment():
    """outputs that are 16- but not 32-byte aligned take the narrower stores: the same bits."""
    ops = _ops()
    B, N, H = 2, 200, 2
    qkv = torch.randn(3, B, N, H, 64, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    ref = ops.attn_fwd(qkv)
    off = torch.empty(B * N * H * 64 + 8, dtype=torch.bfloat16, device="cuda")[8:].view(B, N, H * 64)
    assert off.data_ptr() % 32 == 16
    assert torch.equal(ops.attn_fwd(qkv, out=off), ref)
    for fmt in ("mx8", "nv4", "mx4"):
        outs = []
        for shift in (0, 16):
            q = ops.ActBuf(B * N, H * 64, fmt, device="cuda")
            if fmt == "nv4":
                q.ts.fill_(0.002)
            q.q = torch.empty(q.q.numel() + shift, dtype=q.q.dtype, device="cuda")[shift:].view_as(q.q)
            assert q.q.data_ptr() % 32 == shift
            ops.attn_fwd_quant(qkv, q)
            outs.append(q)
        assert torch.equal(outs[0].q, outs[1].q) and torch.equal(outs[0].sf, outs[1].sf), fmt
    ops.check_device_error()
