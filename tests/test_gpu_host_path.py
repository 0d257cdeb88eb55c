"""The native host path beside autograd's other machinery: what a user's program may put around a training call."""
import pytest
import torch
import torch.utils.checkpoint

import elsa_b200 as E
from elsa_b200.attention_bwd import twopass_attention_qkvpacked

pytestmark = pytest.mark.gpu

ENTRIES = ["packed", "op"]


def _problem(entry, n=130, dtype=torch.float16, bias=True, b=2, h=3, d=64):
    """(inputs, bias or None, grad_out), no gradients asked for yet"""
    gen = torch.Generator(device="cuda").manual_seed(n)

    def normal(*shape, dtype=dtype):
        return torch.randn(shape, generator=gen, device="cuda").to(dtype)

    inputs = [normal(b, n, 3, h, d)] if entry == "packed" else [normal(b, h, n, d) for _ in range(3)]
    return inputs, normal(h, n, n, dtype=torch.float32) if bias else None, normal(b, h, n, d)


def _call(entry, inputs, bias, **kwargs):
    return (twopass_attention_qkvpacked if entry == "packed" else E.twopass_attention_train)(*inputs, bias=bias, **kwargs)


def _leaves(inputs, bias):
    inputs = [t.detach().requires_grad_(True) for t in inputs]
    return inputs, None if bias is None else bias.detach().requires_grad_(True)


def _gradients(entry, inputs, bias, grad_out):
    inputs, bias = _leaves(inputs, bias)
    out = _call(entry, inputs, bias)
    return torch.autograd.grad(out, inputs + ([] if bias is None else [bias]), grad_out)


def _assert_same(got, want):
    # (dQ and summed bias gradients are added in arrival order; an element read from a wrong place gives errors of order 1)
    for g, w in zip(got, want):
        assert g.shape == w.shape and g.dtype == w.dtype
        assert (g.double() - w.double()).norm() <= 1e-3 * w.double().norm()


def _by_size(t):
    return torch.empty(t.size(), dtype=t.dtype, device=t.device).copy_(t)


def _off_alignment(t):
    return torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].copy_(t.reshape(-1)).view(t.shape)


def _transposed(t):
    return t.transpose(-1, -2).contiguous().transpose(-1, -2) if t.dim() > 1 else t.clone()


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("n,dtype", [(49, torch.float16), (130, torch.float16), (130, torch.float32)])
@pytest.mark.parametrize("hook", ["offload", "by_size", "off_alignment", "transposed"])
def test_saved_tensors_may_come_back_in_another_layout(entry, n, dtype, hook):
    inputs, bias, grad_out = _problem(entry, n, dtype)
    want = _gradients(entry, inputs, bias, grad_out)
    if hook == "offload":
        hooks = torch.autograd.graph.save_on_cpu(pin_memory=True)
    else:
        pack = {"by_size": _by_size, "off_alignment": _off_alignment, "transposed": _transposed}[hook]
        hooks = torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t)
    with hooks:
        got = _gradients(entry, inputs, bias, grad_out)
    _assert_same(got, want)


@pytest.mark.parametrize("entry", ENTRIES)
def test_a_saved_tensor_of_another_kind_is_refused(entry):
    inputs, bias, grad_out = _problem(entry)
    for unpack in (lambda t: t.float(), lambda t: t.cpu(), lambda t: t[..., :1]):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            leaves, b = _leaves(inputs, bias)
            out = _call(entry, leaves, b)
        with pytest.raises(RuntimeError):
            torch.autograd.grad(out, leaves, grad_out)


@pytest.mark.parametrize("entry", ENTRIES)
def test_checkpoint_whose_first_saved_tensor_is_the_attentions(entry):
    lin = torch.nn.Linear(64, 3 * 2 * 32, device="cuda", dtype=torch.float16)

    def block(x):
        qkv = lin(x).view(x.shape[0], x.shape[1], 3, 2, 32)
        return _call(entry, [qkv] if entry == "packed" else qkv.permute(2, 0, 3, 1, 4).unbind(0), None)

    x = torch.randn(2, 100, 64, device="cuda", dtype=torch.float16, requires_grad=True)
    want = block(x)
    grad_out = torch.randn_like(want)
    want = torch.autograd.grad(want, [x, lin.weight, lin.bias], grad_out)
    got = torch.autograd.grad(torch.utils.checkpoint.checkpoint(block, x, use_reentrant=False), [x, lin.weight, lin.bias], grad_out)
    _assert_same(got, want)


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("which", ["first", "last", "bias"])
def test_forward_mode_is_refused_not_dropped(entry, which):
    inputs, bias, _ = _problem(entry)
    with torch.autograd.forward_ad.dual_level():
        if which == "bias":
            bias = torch.autograd.forward_ad.make_dual(bias, torch.ones_like(bias))
        else:
            i = 0 if which == "first" else -1
            inputs[i] = torch.autograd.forward_ad.make_dual(inputs[i], torch.ones_like(inputs[i]))
        with pytest.raises(NotImplementedError):
            _call(entry, inputs, bias)


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("grad", [False, True])
def test_a_traced_training_call_follows_its_inputs(entry, grad):
    inputs, _, _ = _problem(entry, bias=False)
    if grad:
        inputs, _ = _leaves(inputs, None)
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(lambda *x: _call(entry, x, None), tuple(inputs), check_trace=False)
        other = [t * 0.5 + 0.1 for t in inputs]
        _assert_same([traced(*other)], [_call(entry, other, None)])


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("form", ["leaf", "matrix", "heads", "batch"])
def test_a_bias_changed_before_the_backward_is_found(entry, form):
    inputs, bias, grad_out = _problem(entry)
    inputs, leaf = _leaves(inputs, bias)
    with torch.no_grad():
        bias = {"leaf": leaf, "matrix": leaf[0], "heads": leaf, "batch": leaf[None]}[form]
    out = _call(entry, inputs, bias if form == "leaf" else bias.detach())
    with torch.no_grad():
        leaf.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, inputs, grad_out)


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("which", ["input", "out"])
def test_an_input_or_output_changed_before_the_backward_is_found(entry, which):
    inputs, bias, grad_out = _problem(entry)
    inputs, bias = _leaves(inputs, bias)
    out = _call(entry, inputs, bias)
    with pytest.raises(RuntimeError):
        with torch.no_grad():
            (inputs[-1] if which == "input" else out).mul_(2)
        torch.autograd.grad(out, inputs, grad_out)


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("form", ["heads", "expanded", "transposed"])
def test_a_bias_alone_may_require_a_gradient(entry, dtype, form):
    inputs, bias, grad_out = _problem(entry)
    bias = bias.to(dtype)
    if form == "transposed":
        bias = bias.mT
    leaf = bias.detach().requires_grad_(True)
    used = leaf[None].expand(2, -1, -1, -1) if form == "expanded" else leaf
    got, = torch.autograd.grad(_call(entry, inputs, used), leaf, grad_out)
    want = _gradients(entry, inputs, bias.contiguous().float(), grad_out)[-1].to(dtype)
    _assert_same([got], [want])


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("with_bias", [False, True])
def test_backward_under_compiled_autograd(entry, with_bias):
    from torch._dynamo import compiled_autograd
    for n in (130, 70):
        inputs, bias, grad_out = _problem(entry, n, bias=with_bias)
        want = _gradients(entry, inputs, bias, grad_out)
        for _ in range(2):
            leaves, b = _leaves(inputs, bias)
            out = _call(entry, leaves, b)
            with compiled_autograd._enable(torch.compile(backend="eager")):
                (out * 2).backward(grad_out / 2)
            _assert_same([t.grad for t in leaves + ([b] if with_bias else [])], want)


def _infer(inputs, bias, **kwargs):
    return E.twopass_attention(*inputs, bias=bias, **kwargs)


@pytest.mark.parametrize("entry", ENTRIES + ["infer"])
def test_keywords_are_checked_in_the_order_of_the_general_path(entry):
    call = _infer if entry == "infer" else lambda *a, **kw: _call(entry, *a, **kw)
    layout = "packed" if entry == "packed" else "op"
    # an empty sequence is answered before the keywords are looked at
    empty = [torch.empty((2, 0, 3, 3, 64) if entry == "packed" else (2, 3, 0, 64), device="cuda") for _ in range(1 if entry == "packed" else 3)]
    assert call(empty, None, phase1_warps=3).shape == (2, 3, 0, 64)
    inputs, _, _ = _problem(layout, bias=False)
    with pytest.raises(ValueError, match="must have shape"):
        call([t[0] for t in inputs], None, phase1_warps=3)
    with pytest.raises(ValueError, match="phase1_warps"):
        call(inputs, None, phase1_warps=3)
    with pytest.raises(ValueError, match="algorithm"):
        call(inputs, None, algorithm="other")
    with pytest.raises(TypeError, match="nope"):
        call(inputs, None, nope=1)
    _assert_same([call(inputs, None, block_n=1 << 70, q_chunk_size=1 << 70)], [call(inputs, None)])


@pytest.mark.parametrize("entry", ENTRIES)
def test_operators_work_without_the_host_path(entry, monkeypatch):
    from elsa_b200 import _lib
    inputs, bias, grad_out = _problem(entry)
    want = [_call(entry, inputs, bias), *_gradients(entry, inputs, bias, grad_out)]
    monkeypatch.setattr(_lib, "_host_module", None)
    monkeypatch.setattr(_lib, "_host_tried", True)
    _assert_same([_call(entry, inputs, bias), *_gradients(entry, inputs, bias, grad_out)], want)
    if entry == "op":
        _assert_same([_infer(inputs, bias)], want[:1])


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("native", [True, False])
def test_biased_gradients_repeat_when_torch_is_asked_for_it(entry, native, monkeypatch):
    from elsa_b200 import _lib
    if not native:
        monkeypatch.setattr(_lib, "_host_module", None)
        monkeypatch.setattr(_lib, "_host_tried", True)
    inputs, bias, grad_out = _problem(entry, n=700, b=1)     # (b = 1: the bias gradient is not summed over anything)
    loose = _gradients(entry, inputs, bias, grad_out)
    torch.use_deterministic_algorithms(True)
    try:
        first, *rest = (_gradients(entry, inputs, bias, grad_out) for _ in range(6))
    finally:
        torch.use_deterministic_algorithms(False)
    for again in rest:
        assert all(torch.equal(a, b) for a, b in zip(first, again))
    _assert_same(first, loose)


@pytest.mark.parametrize("entry", ENTRIES)
@pytest.mark.parametrize("n,dtype", [(49, torch.float16), (130, torch.bfloat16), (130, torch.float32)])
def test_under_a_dispatch_mode_the_general_path_agrees(entry, n, dtype):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Passing(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    inputs, bias, grad_out = _problem(entry, n, dtype)
    want = [_call(entry, inputs, bias), *_gradients(entry, inputs, bias, grad_out)]
    with Passing():
        got = [_call(entry, inputs, bias), *_gradients(entry, inputs, bias, grad_out)]
    _assert_same(got, want)
