"""Fused MLPs whose hidden matrix is held for a part of the tokens at a time: full chunks and a shorter
last one whose tiles are cut along k, next to a guard region that no launch may touch.

Same references and bounds as ``test_pair_gemm_gpu``: dyadic inputs, bit-exact slabs, outputs against
the exact product of the oracle's hidden values.
"""
import pytest
import torch

from oracle import ffn_oracle as fo, twell_format as tf
from sparser_faster_llms_b200 import _lib, synthetic, twell
from test_pair_gemm_gpu import REL, hidden_of

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
GUARD = 32 << 20


@pytest.mark.parametrize("m,d,h,max_rows,gated,hp", [
    (640, 2048, 8192, 256, True, False), (1111, 1024, 4096, 512, True, False),
    (700, 1024, 4096, 300, False, False), (4200, 2048, 8192, 1792, True, True)])
def test_chunks_of_a_call(m, d, h, max_rows, gated, hp):
    flags = _lib.FLAG_HIGH_PRECISION if hp else 0
    lib = _lib.load_library()
    need = lib.b200_twell_mlp_scratch_bytes_chunked(m, d, h, int(gated), flags, max_rows)
    assert 0 < need < m * h * 2 * (3 if hp else 1) + GUARD
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=m + d)
    want = tf.pack_preactivations(fo.gate_preactivation(x, gate).numpy(), 8)
    xg, gg, ug, dg = (t.to(DEV) for t in (x, gate, up, down))
    packed = twell.allocate_packed_output(m, h, device=DEV)
    out = torch.empty_like(xg)
    scratch = torch.full((need + GUARD,), 0x5A, dtype=torch.uint8, device=DEV)
    ws = _lib.workspace(DEV)
    if gated:
        _lib.call("b200_twell_gated_mlp_chunked", DEV, xg.data_ptr(), gg.data_ptr(), None,
                  ug.data_ptr(), dg.data_ptr(), packed.data_ptr(), out.data_ptr(), m, d, h, 8,
                  flags, *ws, scratch.data_ptr(), need, max_rows)
    else:
        _lib.call("b200_twell_mlp_chunked", DEV, xg.data_ptr(), gg.data_ptr(), dg.data_ptr(),
                  packed.data_ptr(), out.data_ptr(), m, d, h, 8, 2, *ws, scratch.data_ptr(), need,
                  max_rows)
    torch.cuda.synchronize()
    assert lib.b200_twell_hybrid_status() == 0
    assert (packed.cpu().view(torch.int32).numpy().view("uint32") == want).all()
    assert bool((scratch[need:] == 0x5A).all())
    rows = [0, max_rows // 256 * 256 - 1, max_rows // 256 * 256, m // 2, m - 129, m - 1]
    ref = hidden_of(x[rows], up if gated else None, want[rows], h, 8, hp) @ down.double()
    assert ((out[rows].double().cpu() - ref).norm() / ref.norm()).item() < REL


@pytest.mark.parametrize("offset", [16, 48, 240])
@pytest.mark.parametrize("m,hp", [(160, False), (4096, True)])
def test_scratch_of_any_16_byte_alignment(m, hp, offset):
    """Less than one wave of down tiles (sums written 32 bytes at a time), and several waves."""
    d, h, flags = 2048, 8192, _lib.FLAG_HIGH_PRECISION if hp else 0
    need = _lib.load_library().b200_twell_mlp_scratch_bytes(m, d, h, 1, flags)
    x, *weights = synthetic.dyadic_case(m, d, h, seed=m)
    xg, gg, ug, dg = (t.to(DEV) for t in (x, *weights))
    packed = twell.allocate_packed_output(m, h, device=DEV)
    scratch = torch.full((need + 512,), 0x5A, dtype=torch.uint8, device=DEV)
    outs = []
    for off in (0, offset):
        outs.append(torch.empty_like(xg))
        _lib.call("b200_twell_gated_mlp_scratch", DEV, xg.data_ptr(), gg.data_ptr(), None,
                  ug.data_ptr(), dg.data_ptr(), packed.data_ptr(), outs[-1].data_ptr(), m, d, h, 8,
                  flags, *_lib.workspace(DEV), scratch.data_ptr() + off, need)
    torch.cuda.synchronize()
    assert _lib.load_library().b200_twell_hybrid_status() == 0
    assert torch.equal(outs[0], outs[1])
    assert bool((scratch[need + offset:] == 0x5A).all())


@pytest.mark.parametrize("m,d,h,gated,hp", [(160, 2048, 8192, True, False), (400, 4096, 2304, False, False),
                                            (4096, 2048, 8192, True, True)])
def test_without_a_workspace_no_tile_is_cut(m, d, h, gated, hp):
    """Calls whose tiles are cut along k when there are counters for it, here without a workspace."""
    flags = _lib.FLAG_HIGH_PRECISION if hp else 0
    need = _lib.load_library().b200_twell_mlp_scratch_bytes(m, d, h, int(gated), flags)
    assert need > 0
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=m + h)
    want = tf.pack_preactivations(fo.gate_preactivation(x, gate).numpy(), 8)
    xg, gg, ug, dg = (t.to(DEV) for t in (x, gate, up, down))
    packed = twell.allocate_packed_output(m, h, device=DEV)
    out = torch.empty_like(xg)
    scratch = torch.empty(need, dtype=torch.uint8, device=DEV)
    if gated:
        _lib.call("b200_twell_gated_mlp_scratch", DEV, xg.data_ptr(), gg.data_ptr(), None,
                  ug.data_ptr(), dg.data_ptr(), packed.data_ptr(), out.data_ptr(), m, d, h, 8,
                  flags, None, 0, scratch.data_ptr(), need)
    else:
        _lib.call("b200_twell_mlp_scratch", DEV, xg.data_ptr(), gg.data_ptr(), dg.data_ptr(),
                  packed.data_ptr(), out.data_ptr(), m, d, h, 8, 2, None, 0, scratch.data_ptr(), need)
    torch.cuda.synchronize()
    assert _lib.load_library().b200_twell_hybrid_status() == 0
    assert (packed.cpu().view(torch.int32).numpy().view("uint32") == want).all()
    rows = [0, 127, 128, m // 2, m - 1]
    ref = hidden_of(x[rows], up if gated else None, want[rows], h, 8, hp) @ down.double()
    assert ((out[rows].double().cpu() - ref).norm() / ref.norm()).item() < REL


@pytest.mark.parametrize("m,d,h,cf,hp", [(40, 2048, 8192, 8, False), (300, 1024, 4096, 4, False),
                                         (100, 2048, 8192, 8, True), (100, 2048, 8192, 2, True),
                                         (777, 2048, 8192, 8, True), (777, 1024, 4352, 4, True)])
def test_scratch_of_one_compression_factor(m, d, h, cf, hp):
    """One-SM tiles, and fp32 hidden values in the slots of the slabs: nothing is written past the size."""
    flags = _lib.FLAG_HIGH_PRECISION if hp else 0
    need = _lib.load_library().b200_twell_mlp_scratch_bytes(m, d, h, 1, flags | _lib.scratch_cf(cf))
    assert need == (m * h // cf * 4 if hp else 2 * m * h)
    x, *weights = synthetic.dyadic_case(m, d, h, seed=m)
    x[::5, 0] = -0.5
    gate, up, down = weights
    want = tf.pack_preactivations(fo.gate_preactivation(x, gate).numpy(), cf)
    xg, gg, ug, dg = (t.to(DEV) for t in (x, *weights))
    packed = twell.allocate_packed_output(m, h, device=DEV, compression_factor=cf)
    out = torch.empty_like(xg)
    scratch = torch.full((need + GUARD,), 0x5A, dtype=torch.uint8, device=DEV)
    _lib.call("b200_twell_gated_mlp_scratch", DEV, xg.data_ptr(), gg.data_ptr(), None, ug.data_ptr(),
              dg.data_ptr(), packed.data_ptr(), out.data_ptr(), m, d, h, cf, flags, *_lib.workspace(DEV),
              scratch.data_ptr(), need)
    torch.cuda.synchronize()
    assert (packed.cpu().view(torch.int32).numpy().view("uint32") == want).all()
    assert bool((scratch[need:] == 0x5A).all())
    ref = hidden_of(x, up, want, h, cf, hp) @ down.double()
    assert ((out.double().cpu() - ref).norm() / ref.norm()).item() < REL
