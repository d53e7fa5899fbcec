"""High precision outside bf16's range: hidden values are carried as bf16 terms on the tensor cores, so
infinite ones and finite ones above the largest bf16 must come out as from an fp32 product.

A few tokens activate a neuron of their own whose gate and up values are powers of two: one hidden
value of 2^128 - 2^117 (finite in fp32, rounds to infinity in bf16) with a down row scaled by 2^-100,
one that overflows fp32 with a down row of +-1.  Reference: the oracle's slabs with fp64 products.
Bound: one rounding of y to bf16 (8 significant bits: half an ulp is at most 2^-8 of the value), and
1e-3 for fp32 sums of some 180 terms of order 1.
"""
import pytest
import torch

from oracle import ffn_oracle as fo, twell_format as tf
from sparser_faster_llms_b200 import _lib, synthetic, twell

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("m", [300, 4200])  # gathered, and as three bf16 terms
def test_hidden_values_outside_the_range_of_bf16(m):
    d, h = 2048, 8192
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=31)
    big, inf = torch.arange(3, m, 29), torch.arange(5, m, 29)
    x[:, 1:4] = 0
    gate[:, 1:4] = 0
    for j, feature, up_value in ((40, 1, 2.0 ** 64), (500, 3, 2.0 ** 100)):
        gate[j], up[j] = 0, 0
        gate[j, feature], up[j, feature] = 2.0 ** 64, up_value
    up[40, 1], up[40, 2] = 2.0 ** 64, -2.0 ** 53
    x[:, 2] = 1
    up[torch.arange(h) != 40, 2] = 0
    x[big, 1], x[inf, 3] = 1, 1
    sign = torch.where(torch.arange(d) % 3 == 0, -1.0, 1.0)
    down[40], down[500] = (sign * 2.0 ** -100).bfloat16(), sign.bfloat16()

    mod = twell.TwELLGatedMLP(9400, gate.to(DEV), up.to(DEV), down.to(DEV), highest_precision=True)
    y = mod(x.to(DEV)).cpu()
    assert _lib.load_library().b200_twell_hybrid_status() == 0
    slab = tf.pack_preactivations(fo.gate_preactivation(x, gate).numpy(), 8)
    rows = torch.cat([big[:8], inf[:8], big[-4:], inf[-4:], torch.tensor([0, 1, m - 1])]).unique()
    g = torch.from_numpy(tf.unpack_to_dense(slab[rows.numpy()], h, 8, strict=False)).double()
    hid = g * (x[rows].double() @ up.double().T)
    assert (hid[:, 40].abs() > torch.finfo(torch.bfloat16).max).sum() >= 8
    hid = hid.float().double()  # 2^164 overflows
    for r, hr in zip(rows.tolist(), hid):
        if torch.isinf(hr).any():
            assert torch.equal(y[r].double(), sign.double() * float("inf")), r
        else:
            ref = hr @ down.double()
            err = (y[r].double() - ref).abs()
            assert bool((err <= 2.0 ** -8 * ref.abs() + 1e-3).all()), (r, float(err.max()))
    mod.destroy()
