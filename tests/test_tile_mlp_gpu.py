"""Fused MLPs on one-SM tiles: edges of the 128-token tiles and of their copies' boxes, both neuron and column
widths, every split of the second product, overflowed slabs, a gate bias, the result over the input.  Inputs,
oracle and bounds of ``test_pair_gemm_gpu`` (the products are dense: y is rounded once)."""
import pytest
import torch

from oracle import ffn_oracle as fo, twell_format as tf
from sparser_faster_llms_b200 import _lib, synthetic, twell
from test_pair_gemm_gpu import DEV, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,d,h", [(33, 2048, 5632), (40, 2048, 8192), (37, 256, 2048), (127, 768, 2304), (128, 4096, 4352),
                                   (129, 1024, 8192), (256, 4096, 2048), (257, 2048, 5632),
                                   (511, 512, 4096), (512, 1024, 4608), (80, 2048, 16384)])
@pytest.mark.parametrize("cf,gated", [(8, True), (2, True), (8, False)])
def test_tile_form(m, d, h, cf, gated):
    assert run_case(m, d, h, cf=cf, gated=gated) > 0


@pytest.mark.parametrize("m,d,h,gated,hp", [(39, 2048, 8192, True, False), (79, 2048, 11008, True, False),
                                            (95, 4096, 16384, False, False), (95, 2048, 8192, True, True),
                                            (63, 4096, 16384, True, True), (257, 2048, 8192, True, True),
                                            (300, 2048, 11008, True, True)])
def test_wide_layers_gather_below_their_lines(m, d, h, gated, hp):
    """The tiles stream all of up and down, which a few dozen tokens of low density do not touch."""
    assert run_case(m, d, h, gated=gated, hp=hp) == 0


@pytest.mark.parametrize("m,h", [(40, 2048), (300, 4096), (130, 16384)])
@pytest.mark.parametrize("gated", [True, False])
def test_values_past_a_slab_leave_the_product(m, h, gated):
    run_case(m, 512, h, gated=gated, dense=True)


@pytest.mark.parametrize("h", [4096, 11008])
def test_bias_and_result_over_the_input(h):
    m, d = 100, 1024
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=3)
    bias = torch.randint(-2, 3, (h,)).float() / 4
    run_case(m, d, h, bias=bias)
    args = [t.to(DEV) for t in (gate, up, down)]
    y = twell.TwELLGatedMLP(9400, *args)(x.to(DEV))
    z = x.to(DEV)
    assert twell.TwELLGatedMLP(9401, *args, inplace=True)(z) is z
    assert torch.equal(y, z)
    assert _lib.load_library().b200_twell_hybrid_status() == 0


@pytest.mark.parametrize("m,h", [(130, 2304), (300, 4096)])
def test_routed_rows_keep_their_positives(m, h):
    """A routed call of this size: rows with an overflowed slab up to the capacity equal the dense formula,
    all others the plain call, bit for bit."""
    d, cap = 512, 16
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=9)
    x[::5, 0] = -0.5
    args = [t.to(DEV) for t in (gate, up, down)]
    plain, routed = twell.TwELLGatedMLP(9402, *args), twell.TwELLGatedMLP(9403, *args)
    routed.enable_dense_route(nnz_threshold=h, dense_cap=cap, min_tokens=128)
    y0, y1 = plain(x.to(DEV)).cpu(), routed(x.to(DEV)).cpu()
    hot = torch.nonzero(torch.arange(m) % 5 == 0).flatten()
    assert routed.dense_route_counters()["dense_rows"] == cap
    taken = torch.zeros(m, dtype=torch.bool)
    taken[hot[:cap]] = True
    assert torch.equal(y0[~taken], y1[~taken])
    p = torch.relu(x.double() @ gate.double().T).bfloat16().double()
    u = (x.double() @ up.double().T).bfloat16().double()
    ref = ((p * u).bfloat16().double() @ down.double())[taken]
    assert ((y1.double()[taken] - ref).norm() / ref.norm()).item() < 2e-3  # y rounded once


@pytest.mark.parametrize("m,d,h", [(33, 1024, 2048), (48, 2048, 5632), (128, 4096, 16384), (257, 1024, 8192),
                                   (160, 512, 11008), (777, 256, 4352), (4095, 2048, 2304)])
@pytest.mark.parametrize("cf,dense", [(8, False), (2, False), (8, True)])
def test_high_precision_with_gathered_down_product(m, d, h, cf, dense):
    """fp32 hidden values in the slots of the slabs, from one-SM tiles and from pairs of SMs."""
    assert run_case(m, d, h, cf=cf, hp=True, dense=dense) > 0


@pytest.mark.parametrize("m,d,h", [(17, 256, 8960), (32, 1024, 16384), (33, 256, 256), (64, 2048, 8192),
                                   (128, 768, 2304), (129, 512, 4352), (256, 4096, 8192)])
@pytest.mark.parametrize("cf", [8, 4])
def test_pack_form(m, d, h, cf):
    """Slabs alone, both neuron widths, bit for bit on the exact inputs; a row past the slab's capacity keeps
    its true count."""
    x, gate, _, _ = synthetic.dyadic_case(m, d, h, seed=m)
    x[::7, 0] = -0.5
    want = tf.pack_preactivations(fo.gate_preactivation(x, gate).numpy(), cf)
    packed = twell.allocate_packed_output(m, h, device=DEV, compression_factor=cf)
    xg, gg = x.to(DEV), gate.to(DEV)
    _lib.call("b200_twell_pack", torch.device(DEV), xg.data_ptr(), gg.data_ptr(), None, packed.data_ptr(),
              m, d, h, cf)
    torch.cuda.synchronize()
    assert (packed.cpu().view(torch.int32).numpy().view("uint32") == want).all()
    assert _lib.load_library().b200_twell_pack_tc_status() == 0


@pytest.mark.parametrize("m,d,h", [(40, 2048, 5632), (100, 2048, 8192), (128, 4096, 4096), (256, 1024, 4096),
                                   (100, 2048, 9216)])
@pytest.mark.parametrize("gated", [True, False])
def test_gate_sums_are_those_of_the_pack(m, d, h, gated):
    """N(0, 1) tokens and N(0, 0.02) weights, whose sums depend on their order: the slabs of a fused call are
    those of the pack of its size.  The error of a running sum grows with its length, and so does the share of
    stored values that are not the rounded 64-bit ones: with four ranges of D it is 0.36 to 0.46 D / 2^18,
    with one range 1.1 to 1.4 D / 2^18 (D 1024 to 4096)."""
    f = synthetic.make_ffn(d, h, seed=m, density=0.02, device=DEV, generate_on_device=True)
    gen = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn(m, d, generator=gen, device=DEV)
    x[:, 0] = 1.0
    x = x.bfloat16()
    want = torch.zeros(m, h // 8, dtype=torch.uint32, device=DEV)
    _lib.call("b200_twell_pack", torch.device(DEV), x.data_ptr(), f.gate.data_ptr(), None, want.data_ptr(), m,
              d, h, 8)
    got, out = torch.zeros_like(want), torch.empty_like(x)
    if h <= 9472:  # the same four ranges of D, by a kernel that gives each to a CTA
        _lib.call("b200_twell_pack_select", torch.device(DEV), x.data_ptr(), f.gate.data_ptr(), None,
                  got.data_ptr(), m, d, h, 8, 8)
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
        got.zero_()
    flags = (0, _lib.FLAG_HIGH_PRECISION) if gated else (0,)
    for flag in flags:
        need = _lib.load_library().b200_twell_mlp_scratch_bytes(m, d, h, int(gated), flag)
        scratch = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
        ws = _lib.workspace(torch.device(DEV))
        if gated:
            _lib.call("b200_twell_gated_mlp_scratch", torch.device(DEV), x.data_ptr(), f.gate.data_ptr(), None,
                      f.up.data_ptr(), f.down.data_ptr(), got.data_ptr(), out.data_ptr(), m, d, h, 8, flag, *ws,
                      scratch.data_ptr(), need)
        else:
            _lib.call("b200_twell_mlp_scratch", torch.device(DEV), x.data_ptr(), f.gate.data_ptr(),
                      f.down.data_ptr(), got.data_ptr(), out.data_ptr(), m, d, h, 8, 2, *ws, scratch.data_ptr(),
                      need)
        torch.cuda.synchronize()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    z = x.double() @ f.gate.double().T
    word = want.view(torch.int32).view(m, h // 256, 32)
    slot = torch.arange(1, 32, device=DEV)
    live = slot <= word[..., :1].clamp(max=31)
    rows = torch.arange(m, device=DEV)[:, None, None].expand_as(live)[live]
    col = (word[..., 1:] & 0xFFFF)[live].long()
    value = (word[..., 1:] & -65536)[live].view(torch.float32)
    off = (value != z[rows, col].bfloat16().float()).float().mean().item()
    assert off < d / 2 ** 18, off


@pytest.mark.parametrize("m,d,h", [(100, 2048, 8192), (100, 4096, 4096), (250, 2048, 8192), (128, 4096, 16384),
                                   (250, 768, 8192), (400, 2048, 11008), (600, 4096, 8192), (777, 2048, 8192)])
def test_high_precision_hidden_values_against_64_bits(m, d, h):
    """N(0, 1) tokens and N(0, 0.02) weights, one-SM tiles and pairs of SMs.  A tensor core's running sum loses
    some 2^-26 of itself with every 16 k-values, so ranges of at most 512 of them keep the fp32 hidden values
    within 32 x 2^-26 = 4.8e-7 (measured 2.4e-7 to 4.8e-7); one range over D 2048 is off by 2.1e-6, two by
    1.0e-6."""
    f = synthetic.make_ffn(d, h, seed=m, density=0.02, device=DEV, generate_on_device=True)
    gen = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn(m, d, generator=gen, device=DEV)
    x[:, 0] = 1.0
    x = x.bfloat16()
    packed, out = torch.zeros(m, h // 8, dtype=torch.uint32, device=DEV), torch.empty_like(x)
    need = _lib.load_library().b200_twell_mlp_scratch_bytes(m, d, h, 1, _lib.FLAG_HIGH_PRECISION)
    assert need > 0
    scratch = torch.empty(need, dtype=torch.uint8, device=DEV)
    _lib.call("b200_twell_gated_mlp_scratch", torch.device(DEV), x.data_ptr(), f.gate.data_ptr(), None,
              f.up.data_ptr(), f.down.data_ptr(), packed.data_ptr(), out.data_ptr(), m, d, h, 8,
              _lib.FLAG_HIGH_PRECISION, *_lib.workspace(torch.device(DEV)), scratch.data_ptr(), need)
    torch.cuda.synchronize()
    word = packed.view(torch.int32).view(m, h // 256, 32)
    live = torch.arange(1, 32, device=DEV) <= word[..., :1].clamp(max=31)
    rows = torch.arange(m, device=DEV)[:, None, None].expand_as(live)[live]
    col = (word[..., 1:] & 0xFFFF)[live].long()
    g = (word[..., 1:] & -65536)[live].view(torch.float32).double()
    got = scratch[:m * h // 8 * 4].view(torch.float32).view(m, h // 256, 32)[..., 1:][live].double()
    want = g * (x.double() @ f.up.double().T)[rows, col]
    rel = ((got - want).norm() / want.norm()).item()
    assert rel < 7e-7, rel
