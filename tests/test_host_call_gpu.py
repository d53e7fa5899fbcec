"""The native host side of eager calls: it serves the plain case with the same bits, and leaves everything
else to the Python path, whose errors stay."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from sparser_faster_llms_b200 import synthetic, twell

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def weights(d=512, h=2048, seed=1):
    return [t.to(DEV) for t in synthetic.dyadic_case(4, d, h, seed=seed)[1:]]


@pytest.fixture
def served(monkeypatch):
    """What the native side answered, call by call."""
    log, real = [], twell._host_call.call
    monkeypatch.setattr(twell, "_host_call", type("H", (), {"call": staticmethod(
        lambda *a: log.append(real(*a)) or log[-1])}))
    return log


@pytest.mark.parametrize("m", [1, 20, 33, 300])
@pytest.mark.parametrize("kind", ["gated", "hp", "plain", "bias"])
def test_native_and_python_paths_agree(served, monkeypatch, m, kind):
    g, u, dn = weights()
    x = synthetic.dyadic_case(m, 512, 2048, seed=2)[0].to(DEV)
    mod = (twell.TwELLMLP(9500, u, dn) if kind == "plain" else
           twell.TwELLGatedMLP(9500, g, u, dn, highest_precision=kind == "hp"))
    if kind == "bias":
        mod.set_gate_bias(torch.full((2048,), 0.25, device=DEV))
    y = mod(x)
    assert served == [0]
    monkeypatch.setattr(twell, "_host_call", None)
    assert torch.equal(y, mod(x))


def test_other_cases_take_the_python_path(served):
    g, u, dn = weights()
    mod = twell.TwELLGatedMLP(9501, g, u, dn)
    x = torch.zeros(40, 512, dtype=torch.bfloat16, device=DEV)
    y = mod(x)
    with pytest.raises(RuntimeError, match="expected scalar type"):
        mod(x.float())
    with pytest.raises(ValueError, match="contiguous"):
        mod(torch.zeros(512, 40, dtype=torch.bfloat16, device=DEV).t())
    with pytest.raises(ValueError, match=r"must all be \[2048, 256\]"):
        mod(torch.zeros(40, 256, dtype=torch.bfloat16, device=DEV))

    class Names(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Names():
        assert torch.equal(mod(x), y)
    assert served == [0, None, None, None, None]
    mod.enable_dense_route(min_tokens=4)  # routed calls are not asked about
    mod(x)
    assert len(served) == 5


@pytest.mark.parametrize("splits", [1 << 70, (1 << 70) + 2, -1])
def test_numbers_beyond_a_long_are_left_to_the_python_path(served, monkeypatch, splits):
    """ctypes passes the low 32 bits of a split count, and 0 and -1 are refused."""
    _, u, dn = weights()
    x = torch.zeros(40, 512, dtype=torch.bfloat16, device=DEV)
    twell.create_d2t_layer(9502, u)

    def outcome():
        try:
            return twell.run_mlp_layer(9502, x, dn, splits)
        except ValueError as e:
            return str(e)

    native = outcome()
    assert served == ([None] if splits > 1 << 62 else [-1])
    monkeypatch.setattr(twell, "_host_call", None)
    python = outcome()
    assert type(native) is type(python)
    assert torch.equal(native, python) if isinstance(python, torch.Tensor) else native == python
    twell.destroy_d2t_layer(9502)
