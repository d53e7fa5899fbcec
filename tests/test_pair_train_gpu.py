"""Training operator on the paired tensor-core GEMM: token counts around the 256-row tiles, every slab
width, overflowed rows within and beyond the tail's capacity, l1 gradient on and off.

Reference: the same function in 64 bits on the pattern the forward stored (tail rows: on every
positive).  Bound: out is rounded at R, T and out, a gradient at P or R, dT, dR / dU and the
result, each relative 1.7e-3 in the 2-norm (bf16, values spread over a binade): 3.3e-3 for four
independent roundings, doubled.
"""
import pytest
import torch

from sparser_faster_llms_b200 import _lib, sparse_ops, synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REL = 6.6e-3


@pytest.fixture(scope="module", autouse=True)
def ops():
    sparse_ops.register_ops()
    yield
    torch.ops.sparse_ops_config.set_ell_width_regular(128)
    torch.ops.sparse_ops_config.set_tail_rows_regular(2048)


def rel(a, b):
    a, b = a.double().flatten(), b.double().flatten()
    return ((a - b).norm() / b.norm()).item()


def run_case(m, d, h, density, width=128, tail=2048, coeff=0.3, hot=0):
    torch.ops.sparse_ops_config.set_ell_width_regular(width)
    torch.ops.sparse_ops_config.set_tail_rows_regular(tail)
    ffn = synthetic.make_ffn(d, h, seed=m + d, density=density, skew_sigma=0.5, device=DEV)
    x = synthetic.make_tokens(m, d, seed=m + 1, device=DEV)
    if hot:
        x[::hot, 0] = 0.2
    gout = synthetic.make_tokens(m, d, seed=m + 2, fold_bias=False, device=DEV)
    leaves = [x.view(1, m, d).requires_grad_(), *(t.requires_grad_() for t in (ffn.gate, ffn.up, ffn.down))]
    out, l0, l1, P, R, T = torch.ops.sparse_ops.ff_forward_gated(*leaves)
    roots, seeds = [out], [gout.view_as(out)]
    if coeff:
        roots.append(l1)
        seeds.append(torch.full((), coeff * m, device=DEV))
    got = torch.autograd.grad(roots, leaves, seeds)
    torch.cuda.synchronize()
    assert _lib.load_library().b200_twell_hybrid_status() == 0

    cf = sparse_ops.compression_factor()
    w = 256 // cf
    words = P.view(m, h // 256, w)
    counts = words[:, :, 0]
    flagged = (counts < 0).any(1)
    stored = torch.arange(1, w, device=DEV)[None, None] <= counts.clamp(0, w - 1)[:, :, None]
    rows = torch.arange(m, device=DEV)[:, None, None].expand_as(stored)[stored]
    cols = (words[:, :, 1:] & 0xFFFF)[stored].long()
    mask = torch.zeros(m, h, dtype=torch.bool, device=DEV)
    mask[rows, cols] = True
    x64, g64, k64, v64 = (t.detach().double().reshape(-1, d).requires_grad_() for t in leaves)
    z = x64 @ g64.T
    mask = torch.where(flagged[:, None], z.detach() > 0, mask)
    t64 = (x64 @ k64.T) * z * mask
    ref_out, ref_l1 = t64 @ v64, t64.abs().sum() / m
    ref = torch.autograd.grad([ref_out, ref_l1], [x64, g64, k64, v64],
                              [gout.double(), torch.tensor(float(coeff * m), device=DEV).double()])
    assert rel(out.detach(), ref_out.detach()) < REL
    assert abs(l1.item() - ref_l1.item()) < 1e-3 * ref_l1.item()
    true = (counts & 0x7FFFFFFF).sum().item() / m
    assert abs(l0.item() - true) < 1e-5 * true
    for a, b, name in zip(got, ref, ("dX", "dG", "dK", "dV")):
        assert rel(a, b) < REL, (name, rel(a, b))
    # R and T carry P's columns and, entry by entry, T = R * P
    for s in (R, T):
        sw = s.view(m, h // 256, w)
        assert torch.equal(sw[:, :, 0], counts)
        assert torch.equal((sw[:, :, 1:] & 0xFFFF)[stored], (words[:, :, 1:] & 0xFFFF)[stored])
    val = lambda s: ((s.view(m, h // 256, w)[:, :, 1:] >> 16) & 0xFFFF)[stored].to(  # noqa: E731
        torch.int16).view(torch.bfloat16)
    assert torch.equal(val(T), val(R) * val(P))
    return flagged.sum().item(), int(((counts > w - 1).any(1)).sum())


@pytest.mark.parametrize("m,d,h", [(1, 256, 256), (63, 512, 768), (129, 1024, 4096), (257, 256, 2048),
                                   (999, 1024, 4096), (1025, 768, 1280), (5000, 1024, 2048)])
@pytest.mark.parametrize("width", [64, 128, 512])
def test_token_counts_and_slab_widths(m, d, h, width):
    run_case(m, d, h, 0.03, width=width)


def test_without_l1_gradient():
    run_case(300, 512, 1024, 0.05, coeff=0.0)


@pytest.mark.parametrize("m", [70, 700])
def test_overflowed_rows_within_and_beyond_the_tail(m):
    taken, left = run_case(m, 512, 2048, 0.03, hot=9)
    assert taken == (m + 8) // 9 and left == 0
    taken, left = run_case(m, 512, 2048, 0.03, hot=9, tail=5)
    assert taken == 5 and left == (m + 8) // 9 - 5
    taken, left = run_case(m, 512, 2048, 0.03, hot=9, tail=0)
    assert taken == 0 and left == (m + 8) // 9


@pytest.mark.parametrize("width,density", [(64, 0.1), (128, 0.2), (512, 0.05), (512, 0.35)])
def test_entry_counts_around_the_words_fetched_ahead(width, density):
    """Means of 26 / 51 / 13 / 90 entries per 256-neuron tile: more than the 16 slab words that
    are fetched ahead, a few of them only, and (first two) full slabs with overflowed rows."""
    run_case(97, 256, 768, density, width=width)


@pytest.mark.parametrize("m", [300, 1100])
def test_last_wave_cut_along_k(m):
    """64 k-steps and more: 16 tiles of gate, R / T and dT in four ranges each; 80 tiles of dX, the last
    six in four."""
    run_case(m, 4096, 2048, 0.03)
