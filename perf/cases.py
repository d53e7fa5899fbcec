"""The work that users of this package have it do, as cases that can be timed and compared.

Three kinds of call cover the public entry points of one GPU:

* ``layer``  one forward of a module (:class:`twell.TwELLGatedMLP`, :class:`twell.TwELLMLP`),
  launched eagerly: what a model whose MLPs were swapped runs, once per layer and forward pass;
* ``stack``  one step of :class:`stack.GraphedFFNStack`: the sparse FFNs of a whole decoder at a
  decode batch, input from and results to pinned host memory, replayed as a CUDA graph;
* ``train``  ``torch.ops.sparse_ops.ff_forward_gated`` and its autograd backward, with the
  package's default settings: the hybrid training step of one layer.

Shapes (d_model x d_ff) are those of the repository's configurations: 1024 x 4096 (0.5B),
2048 x 5632 and 2048 x 8192 (1.5B, the two the reference's kernels take), 2048 x 11008 (2B
prefill), 4096 x 16384 (kernel sweep).  Weights are ~N(0, 0.02) and tokens ~N(0, 1), the gate
density is set by the per-neuron shift of :mod:`synthetic` (folded into token feature 0), neuron
rates uniform or log-normal.  ``mixed`` tokens have a density of their own: Beta(2, 60), and 5 %
of them between 20 and 40 %.
"""
import itertools
import math

import torch

from sparser_faster_llms_b200 import sparse_ops, stack, synthetic, twell

_LAYER = dict(kind="layer", m=1, d=2048, h=8192, density=0.02, skew=1.0, gated=True, hp=False,
              cf=8, inplace=False, shared=False, route="off", mixed=False)
_STACK = dict(kind="stack", m=1, layers=28, d=2048, h=8192, density=0.02, skew=1.0)
_TRAIN = dict(kind="train", b=8, s=2048, d=1024, h=4096, density=0.01, skew=1.0)

_SHAPES = [(1024, 4096), (2048, 5632), (2048, 8192), (2048, 11008), (4096, 16384)]


def listed():
    return [
        # interactive decode of one sequence, the model's layers called one by one
        dict(_LAYER, name="layer 1 token", m=1, shared=True),
        # a small ragged batch of a server, the narrower FFN of the 1.5B shape
        dict(_LAYER, name="layer 37 tokens", m=37, h=5632, shared=True),
        # a short prompt through a 0.5B layer (the single-layer configuration)
        dict(_LAYER, name="layer 256 tokens", m=256, d=1024, h=4096, skew=0.0),
        # a prompt of odd length, fp32 products and 63 entries per slab
        dict(_LAYER, name="layer 777 tokens hp cf4", m=777, hp=True, cf=4),
        # a non-gated MLP over a batch of prompts
        dict(_LAYER, name="mlp 3000 tokens", m=3000, gated=False),
        # one 2048-token prompt, in place, one slab buffer for all layers
        dict(_LAYER, name="layer 2048 tokens", m=2048, inplace=True, shared=True),
        # the kernel-sweep layer at a chunk of a prefill
        dict(_LAYER, name="layer 4096 tokens wide", m=4096, d=4096, h=16384, density=0.01),
        # a large prefill whose tokens differ in density, dense rows on the tensor cores
        dict(_LAYER, name="prefill 16384 mixed", m=16384, h=11008, density=0.03, skew=0.0,
             route="rows", mixed=True),
        # decode steps of the 28-layer 1.5B shape: one sequence, and a serving batch
        dict(_STACK, name="decode stack 1", m=1),
        dict(_STACK, name="decode stack 32", m=32),
        # the training step of a 0.5B layer: a full global batch, and a small ragged one
        dict(_TRAIN, name="train 8x2048"),
        dict(_TRAIN, name="train 3x333", b=3, s=333, density=0.02),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_once(rng):
    density = math.exp(rng.uniform(math.log(0.005), math.log(0.05)))
    skew = rng.choice([0.0, 1.0])
    kind = rng.choice(["layer"] * 6 + ["stack"] * 2 + ["train"] * 2)
    if kind == "stack":
        return dict(_STACK, m=_log_int(rng, 1, 32), h=rng.choice([5632, 8192]),
                    density=min(density, 0.03), skew=skew)
    if kind == "train":
        d, h = rng.choice([(1024, 4096), (1024, 4096), (2048, 5632)])
        return dict(_TRAIN, b=rng.randint(1, 8), s=_log_int(rng, 33, 2048), d=d, h=h,
                    density=min(density, 0.03), skew=skew)
    d, h = rng.choice(_SHAPES)
    case = dict(_LAYER, m=_log_int(rng, 1, 16384), d=d, h=h, density=density, skew=skew)
    form = rng.random()
    if form < 0.15:
        case.update(gated=False)
    elif form < 0.30:
        case.update(hp=True)
    elif form < 0.45:
        case.update(cf=rng.choice([4, 2]))
    elif form < 0.65:
        case.update(m=_log_int(rng, 256, 16384), skew=0.0, route="rows", mixed=True)
    case.update(inplace=rng.random() < 0.25, shared=rng.random() < 0.5)
    return case


def _cost(case):
    """Multiply-adds of the call with every product taken densely, all layers."""
    m = case["b"] * case["s"] * 3 if case["kind"] == "train" else case["m"]
    return m * case["d"] * case["h"] * case.get("layers", 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw_once(rng)
        if _cost(case) <= most:
            return case


# ---------------------------------------------------------------------------------------------
_NUMBERS = itertools.count(1)  # layer numbers: the package keeps one entry for each


def _ffn(case, seed):
    return synthetic.make_ffn(case["d"], case["h"], seed=seed, density=case["density"],
                              skew_sigma=case["skew"], device="cuda", generate_on_device=True)


def _mixed_rates(m, seed):
    """Gate density of each of ``m`` tokens of a mixed prefill."""
    gen = torch.Generator().manual_seed(seed)

    def gamma(shape):  # Marsaglia and Tsang's method (shape >= 1), with a generator of its own
        out, dd = torch.empty(0, dtype=torch.float64), shape - 1.0 / 3.0
        while out.numel() < m:
            z = torch.randn(2 * m + 64, generator=gen, dtype=torch.float64)
            u = torch.rand(2 * m + 64, generator=gen, dtype=torch.float64)
            v = (1.0 + z / math.sqrt(9.0 * dd)).clamp_min(1e-12) ** 3
            ok = torch.log(u) < 0.5 * z * z + dd - dd * v + dd * torch.log(v)
            out = torch.cat([out, (dd * v)[ok]])
        return out[:m]

    a, b = gamma(2.0), gamma(60.0)
    rho = a / (a + b)
    dense = torch.rand(m, generator=gen) < 0.05
    rho = torch.where(dense, 0.2 + 0.2 * torch.rand(m, generator=gen, dtype=torch.float64), rho)
    return rho.clamp(1e-4, 0.49)


def _tokens(m, case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(m, case["d"], generator=gen, device="cuda")
    if case.get("mixed"):
        # feature 0 scales the per-neuron shift (gate[:, 0]) to the token's own density
        q = torch.special.ndtri(1.0 - _mixed_rates(m, seed))
        base = torch.special.ndtri(torch.tensor(1.0 - case["density"], dtype=torch.float64))
        x[:, 0] = (q / base).float().cuda()
    else:
        x[:, 0] = 1.0
    return x.to(torch.bfloat16)


def _module(case, ffn):
    number = next(_NUMBERS)
    if not case.get("gated", True):
        return twell.TwELLMLP(number, ffn.gate, ffn.down, inplace=case["inplace"],
                              preallocate_shared_hidden_state=case["shared"])
    cf = case.get("cf", 8)
    mod = twell.TwELLGatedMLP(number, ffn.gate, ffn.up, ffn.down,
                              inplace=case.get("inplace", False),
                              preallocate_shared_hidden_state=case.get("shared", False),
                              highest_precision=case.get("hp", False), compression_factor=cf,
                              flex_kernels=cf != 8)
    if case.get("route") == "rows":
        mod.enable_dense_route(nnz_threshold=case["h"] // 64, dense_cap=case["m"],
                               min_tokens=128)
    return mod


@torch.no_grad()
def prepare(case, seed):
    if case["kind"] == "stack":
        mods = [_module(case, _ffn(case, seed * 1000 + n)) for n in range(case["layers"])]
        runner = stack.GraphedFFNStack(mods, case["m"])
        x = _tokens(case["layers"] * case["m"], case, seed + 1)
        runner.x_host.copy_(x.view(runner.x_host.shape))
        return {"runner": runner}
    ffn = _ffn(case, seed)
    if case["kind"] == "train":
        sparse_ops.register_ops()
        b, s, d = case["b"], case["s"], case["d"]
        gen = torch.Generator(device="cuda").manual_seed(seed + 2)
        grad = (torch.randn(b, s, d, generator=gen, device="cuda") / d).to(torch.bfloat16)
        leaves = [_tokens(b * s, case, seed + 1).view(b, s, d), ffn.gate, ffn.up, ffn.down]
        return {"leaves": [t.requires_grad_() for t in leaves], "grad": grad,
                "l1_coeff": torch.full((), 3e-4 / d, device="cuda")}
    x = _tokens(case["m"], case, seed + 1)
    if not case["inplace"]:
        return {"mod": _module(case, ffn), "x": x}
    # an in-place call replaces the residual branch it is given: a program's next call comes
    # with new activations in the same buffer
    return {"mod": _module(case, ffn), "x": torch.empty_like(x), "next": x}


def run(state):
    if "runner" in state:
        runner = state["runner"]
        return runner.run(runner.x_host)
    if "leaves" in state:
        leaves = state["leaves"]
        out, l0, l1, _, _, _ = torch.ops.sparse_ops.ff_forward_gated(*leaves)
        grads = torch.autograd.grad([out, l1], leaves, [state["grad"], state["l1_coeff"]])
        return [out.detach(), l0, l1.detach(), *grads]
    with torch.no_grad():
        if "next" in state:
            state["x"].copy_(state["next"])
        return state["mod"](state["x"])


def _active(case, m):
    """Expected stored gate entries per token and expected distinct active neurons of ``m``."""
    h = case["h"]
    if case.get("mixed"):
        rho = _mixed_rates(m, 1)
        return h * float(rho.mean()), h * (1.0 - math.exp(float(torch.log1p(-rho).sum())))
    rates = synthetic.neuron_rates(h, case["density"], case["skew"],
                                   torch.Generator().manual_seed(1))
    return float(rates.sum()), float((1.0 - (1.0 - rates) ** m).sum())


def work(case):
    d, h = case["d"], case["h"]
    if case["kind"] == "train":
        m = case["b"] * case["s"]
        nnz, union = _active(case, m)
        # forward: gate product dense, up and down on its pattern; backward: the seven products
        # dT = g V^T, dX = dR K + dU G, dK, dG, dV (and none for the gate) on the pattern
        flops = 2.0 * m * d * h + 2.0 * m * nnz * d * (2 + 6)
        # X, g, G and the active rows of K and V in; out, dX and the three gradients out
        return {"bytes": 2.0 * (4 * m * d + d * h + 2 * union * d + 3 * d * h), "flops": flops}
    m, layers = case["m"], case.get("layers", 1)
    nnz, union = _active(case, m)
    products = 2 if case.get("gated", True) else 1
    return {"bytes": layers * 2.0 * (d * h + products * union * d + 2 * m * d),
            "flops": layers * (2.0 * m * d * h + 2.0 * products * m * nnz * d)}


def tolerance(case):
    # Measured against the same functions in 64 bits on the stored pattern, with every result
    # rounded to bf16 (1.7e-3 by itself): training 3.3e-3 to 3.9e-3 and single gradients up to
    # 0.25 of the root mean square; forward with products and hidden values rounded to bf16
    # 3.1e-3 to 3.7e-3 and up to 0.034; with fp32 products 1.7e-3 and up to 0.004.
    if case["kind"] == "train":
        return {"rel": 1.4e-2, "max": 0.95}
    return {"rel": 6e-3, "max": 0.03} if case.get("hp") else {"rel": 1.4e-2, "max": 0.14}
