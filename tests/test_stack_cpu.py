"""Which modules GraphedFFNStack hands the tensor they write; every other one is called as it is."""
import torch
from torch.nn.modules import module

from sparser_faster_llms_b200 import stack, twell


def gated(cls=twell.TwELLGatedMLP, **kw):
    w = torch.zeros(256, 256, dtype=torch.bfloat16)
    return cls(9500, w, w, w, **kw)


def test_only_unchanged_modules_write_into_the_result():
    writes = stack.GraphedFFNStack._writes_into
    w = torch.zeros(256, 256, dtype=torch.bfloat16)
    assert writes(gated()) and writes(twell.TwELLMLP(9501, w, w))
    assert not writes(gated(inplace=True))
    assert not writes(torch.nn.Linear(4, 4))

    class Scaled(twell.TwELLGatedMLP):  # takes part of the forward from the base class
        _entry = {(False, False): lambda *a, **k: None}

    class Doubled(twell.TwELLGatedMLP):
        def __call__(self, x):
            return 2 * super().__call__(x)

    assert not writes(gated(Scaled)) and not writes(gated(Doubled))
    replaced = gated()
    replaced.forward = lambda x: x
    assert not writes(replaced)


def test_hooks_of_a_module_and_of_all_modules_are_kept():
    writes = stack.GraphedFFNStack._writes_into
    mod = gated()
    for register in (mod.register_forward_hook, mod.register_forward_pre_hook,
                     module.register_module_forward_hook, module.register_module_forward_pre_hook):
        handle = register(lambda *args: None)
        assert not writes(mod)
        handle.remove()
        assert writes(mod)
