"""Hybrid entry points of the C ABI that the training operator itself no longer calls: sampled up product
and dense-form weight gradients, against 64-bit products on the stored pattern.

Bounds: a stored R is one bf16 rounding of an fp32 sum, at most 2^-8 of the value (half an ulp of 8
significant bits) plus 1e-5 of the sum of magnitudes;
T is the exact bf16 product of stored values.  A weight gradient is one bf16 rounding of an fp32 sum:
1.7e-3 in the 2-norm, with the order of summation below that.
"""
import pytest
import torch

from sparser_faster_llms_b200 import _lib, synthetic, twell

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def pattern(m, d, h, cf):
    ffn = synthetic.make_ffn(d, h, seed=m + h, density=0.05, device=DEV)
    x = synthetic.make_tokens(m, d, seed=m, device=DEV)
    slab = twell.matmul_sparse(x, ffn.gate, compression_factor=cf).view(torch.int32)
    words = slab.view(m, h // 256, 256 // cf)
    counts = words[:, :, 0]
    w = 256 // cf
    stored = torch.arange(1, w, device=DEV)[None, None] <= counts.clamp(0, w - 1)[:, :, None]
    rows = torch.arange(m, device=DEV)[:, None, None].expand_as(stored)[stored]
    cols = (words[:, :, 1:] & 0xFFFF)[stored].long()
    return ffn, x, slab, stored, rows, cols


def values(slab, stored):
    words = slab.view(*stored.shape[:2], -1)[:, :, 1:]
    return ((words >> 16) & 0xFFFF)[stored].to(torch.int16).view(torch.bfloat16)


@pytest.mark.parametrize("m,d,h,cf", [(1, 256, 256, 8), (77, 512, 1024, 4), (300, 1024, 768, 2)])
def test_sampled_up_product(m, d, h, cf):
    ffn, x, p, stored, rows, cols = pattern(m, d, h, cf)
    r, t = torch.empty_like(p), torch.empty_like(p)
    l1 = torch.empty(m, device=DEV)
    nnz, drop = (torch.empty(m, dtype=torch.int32, device=DEV) for _ in range(2))
    _lib.call("b200_hybrid_sddmm_fwd", DEV, x.data_ptr(), ffn.up.data_ptr(), p.data_ptr(), r.data_ptr(),
              t.data_ptr(), l1.data_ptr(), nnz.data_ptr(), drop.data_ptr(), m, d, h, cf)
    xr, kr = x.double()[rows], ffn.up.double()[cols]
    ref, size = (xr * kr).sum(1), (xr * kr).abs().sum(1)
    got = values(r, stored)
    assert bool(((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * size).all())
    assert torch.equal(values(t, stored), got * values(p, stored))
    counts = p.view(*stored.shape[:2], -1)[:, :, 0]
    assert torch.equal(nnz, counts.sum(1).int())
    assert torch.equal(drop, (counts - (256 // cf - 1)).clamp_min(0).sum(1).int())
    want = torch.zeros(m, device=DEV).index_add_(0, rows, values(t, stored).float().abs())
    assert torch.allclose(l1, want, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("m,d,h,cf", [(1, 256, 256, 8), (190, 512, 1024, 4), (2100, 256, 768, 2)])
def test_dense_form_weight_gradient(m, d, h, cf):
    ffn, x, p, stored, rows, cols = pattern(m, d, h, cf)
    lib = _lib.load_library()
    ws = torch.empty(lib.b200_hybrid_wgrad_workspace_bytes(m, d, h), dtype=torch.uint8, device=DEV)
    dense = torch.zeros(m, h, device=DEV, dtype=torch.float64)
    dense[rows, cols] = values(p, stored).double()
    want = dense.T @ x.double()
    for reuse in (0, 1):
        out = torch.empty(h, d, dtype=torch.bfloat16, device=DEV)
        _lib.call("b200_hybrid_wgrad_dense", DEV, p.data_ptr(), x.data_ptr(), out.data_ptr(), m, d, h,
                  cf, reuse, ws.data_ptr(), ws.numel())
        assert ((out.double() - want).norm() / want.norm()).item() < 2.5e-3
    assert lib.b200_twell_hybrid_status() == 0
