"""Contraction of a few tokens with very different numbers of stored entries in one call: every token is spread
over as many clusters as its own entries are worth (one, four at most, all).  Inputs, oracle and the gather bound of
``test_pair_gemm_gpu``."""
import pytest
import torch

from oracle import ffn_oracle as fo, twell_format as tf
from sparser_faster_llms_b200 import _lib, synthetic, twell
from test_pair_gemm_gpu import DEV, REL_GATHER, hidden_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,d,h", [(2, 2048, 8192), (5, 1024, 8192), (10, 2048, 8192), (18, 256, 8192),
                                   (3, 4096, 8192), (8, 4096, 4096)])
@pytest.mark.parametrize("cf", [8, 2])
def test_tokens_with_few_and_many_entries(m, d, h, cf):
    x, gate, up, down = synthetic.dyadic_case(m, d, h, seed=m + d)
    shift = [0.5, 1.3, 1.0, 3.0, 0.25]  # none to some tenths of the neurons
    for i in range(m):
        x[i, 0] = shift[i % len(shift)]
    want = tf.pack_preactivations(fo.gate_preactivation(x, gate).numpy(), cf)
    stored = want.reshape(m, h // 256, -1)[:, :, 0].clip(max=256 // cf - 1).sum(1)
    assert stored.min() <= 128 and stored.max() > 320
    xg, gg, ug, dg = (t.to(DEV) for t in (x, gate, up, down))
    packed = twell.allocate_packed_output(m, h, device=DEV, compression_factor=cf)
    ws = _lib.workspace(torch.device(DEV))
    outs = []
    for _ in range(2):
        out = torch.empty_like(xg)
        _lib.call("b200_twell_gated_mlp", torch.device(DEV), xg.data_ptr(), gg.data_ptr(), None, ug.data_ptr(),
                  dg.data_ptr(), packed.data_ptr(), out.data_ptr(), m, d, h, cf, 0, *ws)
        torch.cuda.synchronize()
        outs.append(out.cpu())
    assert torch.equal(*outs)
    assert (packed.cpu().view(torch.int32).numpy().view("uint32") == want).all()
    ref = hidden_of(x, up, want, h, cf, False) @ down.double()
    err = (outs[0].double() - ref).norm() / ref.norm()
    assert err.item() < REL_GATHER
    view = [t for t in _lib._WORKSPACES.values() if t.data_ptr() == ws[0]][0]
    assert int(view[:16384].view(torch.int32).abs().sum()) == 0  # arrival counters at rest
