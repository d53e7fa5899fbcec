"""Fused MLPs on the paired tensor-core GEMM: both sides of every line of the dispatch and the edges of
the 256-row tiles, the split last wave and the slabs' capacity.

Inputs on a dyadic grid make every fp32 sum exact, so slabs must be bit-exact and the hidden
values equal the oracle's; outputs are compared with the exact product of those hidden values.
Bound: y is rounded to bf16 once (relative 2^-9 at most, 1.7e-3 in the 2-norm for values spread
over a binade); in mixed precision u and h are rounded to bf16 as in the oracle, so nothing else
differs except fp32 summation order (below 1e-5).  Where the call gathers without scratch, each product of
the down projection is rounded to bf16 as well: twice that variance more, 3e-3.  Where the device chooses the
gathers of a call with few entries, u and h stay in fp32 as in high precision.
"""
import pytest
import torch

from oracle import ffn_oracle as fo, twell_format as tf
from sparser_faster_llms_b200 import _lib, synthetic, twell

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REL = 2.0e-3
REL_GATHER = 4.0e-3


def hidden_of(x, up, slab, h, cf, hp):
    """Exact hidden values of the stored entries; rounded where the mixed mode rounds."""
    p = torch.from_numpy(tf.unpack_to_dense(slab, h, cf, strict=False)).double()
    if up is None:
        return p
    u = x.double() @ up.double().T
    return p * u if hp else (p * u.bfloat16().double()).bfloat16().double()


def run_case(m, d, h, cf=8, hp=False, gated=True, bias=None, dense=False, sparse=False,
             seed=0, fp32_products=False):
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=seed + m + d + h)
    if dense:  # a few rows with far more positives than a slab holds
        x[::7, 0] = -0.5
    if sparse:  # the shift moves from two to three standard deviations: about 0.2 % positives
        x[:, 0] = 1.5
    z = fo.gate_preactivation(x, gate)
    if bias is not None:
        z = z + bias
    want = tf.pack_preactivations(z.numpy(), cf)
    lib = _lib.load_library()
    flags = _lib.FLAG_HIGH_PRECISION if hp else 0
    need = lib.b200_twell_mlp_scratch_bytes(m, d, h, int(gated), flags)
    xg, gg, ug, dg = (t.to(DEV) for t in (x, gate, up, down))
    bg = None if bias is None else bias.to(DEV)
    packed = twell.allocate_packed_output(m, h, device=DEV, compression_factor=cf)
    out = torch.empty_like(xg)
    scratch = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    ws = _lib.workspace(torch.device(DEV))
    if gated:
        _lib.call("b200_twell_gated_mlp_scratch", torch.device(DEV), xg.data_ptr(), gg.data_ptr(),
                  _lib.ptr(bg), ug.data_ptr(), dg.data_ptr(), packed.data_ptr(), out.data_ptr(),
                  m, d, h, cf, flags, *ws, scratch.data_ptr(), need)
    else:
        _lib.call("b200_twell_mlp_scratch", torch.device(DEV), xg.data_ptr(), gg.data_ptr(),
                  dg.data_ptr(), packed.data_ptr(), out.data_ptr(), m, d, h, cf, 2, *ws,
                  scratch.data_ptr(), need)
    torch.cuda.synchronize()
    assert lib.b200_twell_hybrid_status() == 0
    got = packed.cpu().view(torch.int32).numpy().view("uint32")
    assert (got == want).all()
    rows = sorted({0, 1, 127, 128, 255, 256, 257, m // 2, m - 129, m - 2, m - 1} & set(range(m)))
    hid = hidden_of(x[rows], up if gated else None, want[rows], h, cf, hp or fp32_products)
    ref = hid @ down.double()
    rel = ((out[rows].double().cpu() - ref).norm() / ref.norm()).item()
    assert rel < (REL if need else REL_GATHER), rel
    # counters of the split last wave are back at zero
    view = [t for t in _lib._WORKSPACES.values() if t.data_ptr() == ws[0]][0]
    torch.cuda.synchronize()
    assert int(view[:16384].view(torch.int32).abs().sum()) == 0
    return need


@pytest.mark.parametrize("m,d,h", [(160, 2048, 8192), (320, 1024, 2048), (96, 4096, 11008),
                                   (255, 2048, 8192), (257, 2048, 8192), (777, 2048, 5632),
                                   (1025, 768, 11008), (2304, 512, 2304)])
@pytest.mark.parametrize("cf", [8, 2])
def test_gated_dense_form(m, d, h, cf):
    assert run_case(m, d, h, cf=cf) > 0


@pytest.mark.parametrize("m,d,h", [(4352, 2048, 5632), (9001, 2048, 4352)])
@pytest.mark.parametrize("kind", ["sparse", "plain", "dense"])
def test_large_calls_below_the_choice_run_dense(m, d, h, kind):
    assert run_case(m, d, h, dense=kind == "dense", sparse=kind == "sparse") > 0


@pytest.mark.parametrize("m,d,h,gated,cf", [(6145, 2048, 8192, True, 8), (6400, 2048, 8192, True, 2),
                                            (6500, 1536, 11008, True, 8), (6145, 2048, 8192, False, 8)])
@pytest.mark.parametrize("kind", ["sparse", "plain", "dense"])
def test_device_side_choice_of_the_up_and_down_form(m, d, h, gated, cf, kind):
    """From 1.5 x 2^36 multiply-adds on (gated: rows that L2 holds): the gathers at 0.2 % positives, with fp32
    products, the dense form at the 2 % of the dyadic case and when every seventh row overflows.  The two
    differ in where u and h are rounded, so the bound of one rounding tells which has run."""
    assert run_case(m, d, h, cf=cf, gated=gated, dense=kind == "dense", sparse=kind == "sparse",
                    fp32_products=kind == "sparse") > 0


@pytest.mark.parametrize("m,d,h", [(4096, 2048, 8192), (8192, 1024, 8192)])
@pytest.mark.parametrize("kind", ["sparse", "plain", "dense"])
def test_high_precision_form(m, d, h, kind):
    assert run_case(m, d, h, hp=True, dense=kind == "dense", sparse=kind == "sparse") > 0


@pytest.mark.parametrize("m,d,h", [(320, 2048, 8192), (700, 1024, 4096), (3000, 512, 2048)])
@pytest.mark.parametrize("kind", ["sparse", "plain", "dense"])
def test_non_gated_form(m, d, h, kind):
    run_case(m, d, h, gated=False, dense=kind == "dense", sparse=kind == "sparse")


@pytest.mark.parametrize("offset", [0, 1])
def test_gate_bias_of_any_alignment(offset):
    h = 4096
    b = (torch.randint(-2, 3, (h + offset,)).float() / 4)[offset:]
    bias = torch.empty(h + 4, device=DEV)[offset:offset + h].copy_(b.to(DEV))
    assert bias.data_ptr() % 16 == (4 * offset) % 16
    m, d = 300, 2048
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=5)
    want = tf.pack_preactivations((fo.gate_preactivation(x, gate) + b).numpy(), 8)
    packed = twell.allocate_packed_output(m, h, device=DEV)
    xg, gg = x.to(DEV), gate.to(DEV)  # held: a freed copy's memory would serve the next one
    _lib.call("b200_twell_pack", torch.device(DEV), xg.data_ptr(), gg.data_ptr(), bias.data_ptr(),
              packed.data_ptr(), m, d, h, 8)
    torch.cuda.synchronize()
    assert (packed.cpu().view(torch.int32).numpy().view("uint32") == want).all()


def test_rows_beyond_the_dense_capacity_stay_lossy():
    """The routed form with fewer slots than overflowed rows: later rows equal the plain module's."""
    m, d, h = 600, 2048, 4096
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=9)
    x[::5, 0] = -0.5
    args = [t.to(DEV) for t in (gate, up, down)]
    plain, routed = twell.TwELLGatedMLP(9300, *args), twell.TwELLGatedMLP(9301, *args)
    routed.enable_dense_route(nnz_threshold=h, dense_cap=40, min_tokens=128)
    y0, y1 = plain(x.to(DEV)).cpu(), routed(x.to(DEV)).cpu()
    c = routed.dense_route_counters()
    assert c["dense_rows"] == 40 and c["lossy_rows_left_sparse"] == c["qualified_rows"] - 40 > 0
    hot = torch.arange(m) % 5 == 0
    taken = torch.zeros(m, dtype=torch.bool)
    taken[torch.nonzero(hot).flatten()[:40]] = True
    assert torch.equal(y0[~taken], y1[~taken])
    ref = fo.dense_ffn(x, gate, up, down)
    err = (y1.double() - ref.double()).norm(dim=1) / ref.double().norm(dim=1)
    assert err[taken].max() < 1.5e-2 and err[hot & ~taken].max() > 0.1
    plain.destroy()
    routed.destroy()


@pytest.mark.parametrize("m,h,hp,gated", [(400, 2304, False, False), (1000, 2048, False, False),
                                          (8192, 2048, True, True)])
@pytest.mark.parametrize("kind", ["plain", "dense"])
def test_last_wave_cut_along_k(m, h, hp, gated, kind):
    """64 k-steps: the tiles of the last wave are cut in four (18 tiles) or two (32 and 34) ranges, whose sums
    the warps that arrive last add; gate values and the dense operand come out of the sums."""
    assert run_case(m, 4096, h, hp=hp, gated=gated, dense=kind == "dense") > 0


@pytest.mark.parametrize("gated", [True, False])
def test_a_captured_call_chooses_anew_at_every_replay(gated):
    m, d, h = 6145, 2048, 8192
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=21)
    g, u, dn = (t.to(DEV) for t in (gate, up, down))
    mod = twell.TwELLGatedMLP(9310, g, u, dn) if gated else twell.TwELLMLP(9310, g, dn)
    dense = x.to(DEV)
    sparse = dense.clone()
    sparse[:, 0] = 1.5
    buf = sparse.clone()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(stream):
        want = [mod(sparse), mod(dense)]  # also the workspace of this stream
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            out = mod(buf)
        for new, y in ((dense, want[1]), (sparse, want[0]), (dense, want[1])):
            buf.copy_(new)
            graph.replay()
            stream.synchronize()
            assert torch.equal(out, y)
    mod.destroy()
