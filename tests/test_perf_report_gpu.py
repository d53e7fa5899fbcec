"""SPARSE_ENABLE_PERF_PROFILING: the report has the parts of a training step as well as its totals."""
import pytest
import torch

from sparser_faster_llms_b200 import sparse_ops, synthetic

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_parts_of_a_step(monkeypatch, capsys):
    sparse_ops.register_ops()
    monkeypatch.setattr(sparse_ops, "_PERF_ENABLED", True)
    torch.ops.sparse_ops_perf.reset_stats()
    ffn = synthetic.make_ffn(512, 2048, seed=3, density=0.03, device=DEV)
    x = synthetic.make_tokens(700, 512, seed=4, device=DEV).view(1, 700, 512)
    leaves = [t.requires_grad_() for t in (x, ffn.gate, ffn.up, ffn.down)]
    for _ in range(3):
        out = torch.ops.sparse_ops.ff_forward_gated(*leaves)[0]
        torch.autograd.grad(out, leaves, torch.ones_like(out))
    torch.ops.sparse_ops_perf.print_report()
    report = capsys.readouterr().out
    for total, parts in (("ff_forward_gated_total", sparse_ops._FORWARD_PARTS),
                         ("ff_backward_gated_total", sparse_ops._BACKWARD_PARTS)):
        assert total in report and all(p in report for p in parts)
        for i in range(3):
            times = [sparse_ops._PERF[p][i] for p in parts]
            assert min(times) > 0 and sum(times) <= sparse_ops._PERF[total][i]
    torch.ops.sparse_ops_perf.reset_stats()
