"""GPU: the 16-bit operands of the decode kernel's products against float64: softmax weights and rebuilt keys are
hi + lo pairs, whatever V's type and wherever the running reference maximum stands."""
import math

import pytest
import torch

from util import load_pkg

pkg = load_pkg()
pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# every key is (x, 0, ...) with x and the query exact in 16 bits, so a logit is x * q exactly and only the weights round
@pytest.mark.parametrize("dh,grp,page", [(128, 4, 16), (64, 4, 32), (128, 8, 16), (64, 3, 128)])
@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("v_dtype", [torch.float16, torch.bfloat16])
def test_weights_carry_16_bits(dh, grp, page, late, v_dtype):
    Hkv, ctx = 2, 600 if late else 40
    tiers = pkg.TierSet(dh, (pkg.TierSpec(1, 16, 1),))
    cb = torch.zeros(Hkv, dh // 16, 2, 16)
    cb[:, :, 0, 0] = cb[:, :, 1, 1] = 1.0
    g = torch.Generator().manual_seed(dh + grp)
    x = torch.randint(0, 505, (ctx,), generator=g).double() / 64        # below 2^7.9 of the smallest weight
    if late:  # the large ones come after the reference maximum was taken, and stay below the step that moves it
        x[:-10] = 0
    K = torch.zeros(ctx, Hkv, dh)
    K[:, :, 0] = x[:, None].float()
    V = torch.randn(ctx, Hkv, dh, generator=g).to(v_dtype)
    q = torch.zeros(1, Hkv * grp, dh)
    q[0, :, 0] = 2.0 ** -(torch.arange(Hkv * grp) % 3).float()
    lists = pkg.build_page_lists(torch.ones(1, Hkv, ctx, dtype=torch.uint8, device=DEV), tiers, page, radius_fmt=pkg.RADIUS_F16)
    cache = pkg.encode_pages(K.to(DEV), V.to(DEV), lists, tiers.pack_codebooks([cb]).to(DEV), tiers,
                             radius_fmt=pkg.RADIUS_F16, v_dtype=v_dtype)
    got = pkg.decode_paged(q.to(DEV), cache, None, sm_scale=math.log(2.0), out_dtype=torch.float32).double().cpu()[0]
    p = torch.exp2(x[None] * q[0, :, 0].double()[:, None])
    p = p / p.sum(1, keepdim=True)
    v = V.double().permute(1, 0, 2).repeat_interleave(grp, 0)            # [Hq, ctx, dh]
    want = torch.einsum("ht,htd->hd", p, v)
    # bf16 hi + lo: 2^-17 relative per weight; the logits' scale (log2(e) ln 2 in fp32) and ex2 add a few 2^-22
    bound = 2.0 ** -16 * torch.einsum("ht,htd->hd", p, v.abs())
    assert ((got - want).abs() <= bound).all(), ((got - want).abs() / bound).max()


@pytest.mark.parametrize("dh,page,radius_fmt", [(128, 16, 0), (64, 16, 0), (128, 64, 1)])
def test_keys_are_rounded_not_truncated(dh, page, radius_fmt):
    """rms error of a logit over rms(q) rms(k) sqrt(dh): hi truncated, lo rounded to bf16 gives 0.64 * 2^-17 over normal
    keys, both truncated 1.28 * 2^-17 (and a bias towards zero)"""
    Hkv, grp, ctx = 2, 4, 4000
    tiers = pkg.TierSet(dh, pkg.REFERENCE_TIERS[:1])
    g = torch.Generator().manual_seed(page)
    cb = torch.randn(Hkv, dh // 16, 64, 16, generator=g)
    K = torch.randn(ctx, Hkv, dh, generator=g)
    q = torch.randint(0, 2, (1, Hkv * grp, dh), generator=g).float() * 2 - 1
    lists = pkg.build_page_lists(torch.ones(1, Hkv, ctx, dtype=torch.uint8, device=DEV), tiers, page, radius_fmt=radius_fmt)
    packed = tiers.pack_codebooks([cb]).to(DEV)
    cache = pkg.encode_pages(K.to(DEV), K.to(DEV), lists, packed, tiers, radius_fmt=radius_fmt)
    codes = pkg.encode_codes(K.to(DEV), packed, tiers)                   # r, theta per (head, token, group)
    r, th = codes.r[0].double(), codes.theta[0].long()
    if radius_fmt == 1:
        r = r.half().double()
    else:  # int8 codes, one scale per page and group: pages hold consecutive tokens here
        pad = torch.nn.functional.pad(r, (0, 0, 0, -ctx % page)).view(Hkv, -1, page, dh // 16)
        scale = pad.amax(2, keepdim=True).float()
        code = torch.round(pad.float() / scale * 127.0)
        # the kernel's own fp32 order: scale * fl(1 / 127), times the code
        r = ((scale * torch.tensor(1.0 / 127.0)) * code).double().view(Hkv, -1, dh // 16)[:, :ctx]
    k = (cb.double().to(DEV)[torch.arange(Hkv, device=DEV)[:, None, None], torch.arange(dh // 16, device=DEV), th]
         * r[..., None]).float().double().reshape(Hkv, ctx, dh)          # centroid * radius is one fp32 product
    logits = torch.zeros(1, Hkv * grp, lists.max_blocks * page, device=DEV)
    pkg.decode_paged(q.to(DEV), cache, None, sm_scale=0.125 / math.log2(math.e), logits_out=logits)
    assert not cache.status.item()
    got = logits[0].view(Hkv, grp, -1)[:, :, :ctx].double() * (math.log2(math.e) / 0.125)
    want = torch.einsum("hgd,htd->hgt", q.double().to(DEV).view(Hkv, grp, dh), k)
    err = (got - want).pow(2).mean().sqrt() / (k.pow(2).mean() * dh).sqrt()
    assert err.item() <= 0.9 * 2.0 ** -17, err.item() * 2 ** 17
