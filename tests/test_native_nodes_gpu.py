"""The native autograd nodes give the values of the Python nodes, and leave to those every call that is not plain."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def leaf(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16).requires_grad_()


def both(native, python, inputs):
    """Outputs and gradients of the two routes for the same inputs and upstream gradients."""
    results = []
    for fn in (native, python):
        outs = fn(*inputs)
        outs = outs if isinstance(outs, tuple) else (outs,)
        torch.manual_seed(1)
        ups = [torch.randn_like(o) for o in outs]
        grads = torch.autograd.grad(outs, inputs, ups)
        results.append([o.detach() for o in outs] + list(grads))
    return results


CASES = {
    "linear": lambda F, A: (F.linear, F._Linear.apply, [leaf(3, 50, 72), leaf(40, 72)]),
    "rmsnorm": lambda F, A: (F.rmsnorm, lambda x, w: F._RMSNorm.apply(x, w, 1e-5), [leaf(5, 256), leaf(256)]),
    "add_rmsnorm": lambda F, A: (F.add_rmsnorm, lambda x, r, w: F._AddRMSNorm.apply(x, r, w, 1e-5),
                                 [leaf(2, 9, 768), leaf(2, 9, 768), leaf(768)]),
    "swiglu": lambda F, A: (F.swiglu, F._SwiGLU.apply, [leaf(7, 2 * 24)]),
    "attention": lambda F, A: (A.attention, lambda q, k, v: A._Attention.apply(q, k, v, None),
                               [leaf(2, 70, 4, 64), leaf(2, 70, 2, 64), leaf(2, 70, 2, 64)]),
}


@pytest.mark.parametrize("name", CASES)
def test_native_and_python_nodes_agree(name):
    """Same kernels on the same operands: equal bit for bit."""
    from torchft_b200.ops import attention as A
    from torchft_b200.ops import functional as F

    torch.manual_seed(0)
    native, python, inputs = CASES[name](F, A)
    out = native(*inputs)
    node = (out[0] if isinstance(out, tuple) else out).grad_fn
    assert not isinstance(node, torch.autograd.function.BackwardCFunction)  # the base of every Python node
    for a, b in zip(*both(native, python, inputs)):
        assert torch.equal(a, b)


def test_calls_that_stay_with_the_python_nodes():
    from torchft_b200.ops import _native
    from torchft_b200.ops import functional as F

    m = _native.module()
    x, w = leaf(16, 64), leaf(32, 64)
    assert m.linear(x, w) is not None
    wide = torch.zeros(16, 128, device=DEV, dtype=torch.bfloat16)
    odd = torch.zeros(16 * 64 + 1, device=DEV, dtype=torch.bfloat16)[1:].view(16, 64)
    marked, marked_norm = leaf(32, 64), leaf(256)
    for weight in (marked, marked_norm):
        weight.main_grad = torch.zeros_like(weight)
    for a, b in ((wide[:, :64], w), (odd, w), (x.float(), w), (x.cpu(), w), (x, marked), (leaf(16, 60), leaf(32, 60)), (x[:0], w)):
        assert m.linear(a, b) is None
    assert m.rmsnorm(leaf(4, 264), leaf(264), 1e-5) is None  # a width that the kernel has no split for
    rows = leaf(4, 256)
    assert m.rmsnorm(rows, marked_norm, 1e-5) is None and m.add_rmsnorm(rows, rows, marked_norm, 1e-5) is None
    assert m.swiglu(leaf(4, 24)) is None
    torch.manual_seed(0)
    strided = torch.randn(16, 128, device=DEV).to(torch.bfloat16)[:, ::2]
    assert m.linear(strided, w) is None
    with torch.no_grad():  # inference is plain
        assert m.linear(x, w).grad_fn is None

    seen = []

    def transformed(x_):
        seen.append(m.linear(x_, w.detach()) is None and m.linear(x.detach(), w.detach()) is None)
        return x_.sum()

    torch.func.grad(transformed)(x.detach())
    assert seen == [True]
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x))
        assert m.linear(dual, w) is None
    with pytest.raises(F._lib.KernelError):
        F.linear(leaf(16, 60), leaf(32, 60))


def test_saved_tensor_hooks_and_late_gradient_buffers():
    from torchft_b200.ops import functional as F

    torch.manual_seed(0)
    x, w = leaf(16, 64), leaf(32, 64)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.to(DEV)):
        y = F.linear(x, w)
    dy = torch.randn_like(y)
    dx, dw = torch.autograd.grad(y, (x, w), dy)
    assert torch.Size((16, 64)) in packed and torch.Size((32, 64)) in packed
    ref = F._Linear.apply(x, w)
    rx, rw = torch.autograd.grad(ref, (x, w), dy)
    assert torch.equal(dx, rx) and torch.equal(dw, rw)

    # buffers that an engine gives to the weights between forward and backward receive the gradients
    n = leaf(256)
    x, w = leaf(16, 256), leaf(32, 256)
    y = F.linear(F.rmsnorm(x, n), w)
    for p in (w, n):
        p.main_grad = torch.full_like(p, float("nan"))
    y.backward(dy)
    assert w.grad is None and n.grad is None
    assert torch.isfinite(w.main_grad).all() and w.main_grad_initialized
    want = dy.float().t() @ F.rmsnorm(x, n.detach().clone()).detach().float()
    assert (w.main_grad.float() - want).norm() < 8e-3 * want.norm()  # one rounding of the sum to bf16


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("name", ["linear", "rmsnorm", "add_rmsnorm"])
def test_gradient_buffers_under_saved_tensor_hooks(name, late):
    """What the hooks unpack is a copy without the weight's attributes: the gradient goes to the weight's buffer all the same,
    given to it before the forward pass or after it."""
    from torchft_b200.ops import attention as A
    from torchft_b200.ops import functional as F

    torch.manual_seed(0)
    fn, _, inputs = CASES[name](F, A)
    w = inputs[-1]
    out = fn(*inputs)
    out = out[0] if isinstance(out, tuple) else out
    dy = torch.randn_like(out)
    (want,) = torch.autograd.grad(out, (w,), dy)
    buffer = torch.full_like(w, float("nan"))
    if not late:
        w.main_grad = buffer
    with torch.autograd.graph.save_on_cpu():
        out = fn(*inputs)
    w.main_grad = buffer
    (out[0] if isinstance(out, tuple) else out).backward(dy)
    assert w.grad is None and w.main_grad_initialized
    assert torch.equal(buffer, want)


@pytest.mark.parametrize("shape", [(16, 64), (64, 64), (32, 128), (32, 32), (2048,)])
def test_a_weight_replaced_between_the_passes_is_refused(shape):
    """The sizes of the backward products come from the gradient and every operand is held against them."""
    from torchft_b200.ops import functional as F

    x, w = leaf(16, 64), leaf(32, 64)
    y = F.linear(x, w)
    w.data = torch.zeros(shape, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        y.backward(torch.ones_like(y))
    n = leaf(256)
    y = F.rmsnorm(leaf(4, 256), n)
    n.data = torch.ones(512, device=DEV, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError):
        y.backward(torch.ones_like(y))


def at_odd_address(t):
    flat = torch.full((t.numel() + 1,), float("nan"), device=t.device, dtype=t.dtype)
    view = flat[1:].view(t.shape)
    view.copy_(t.detach())
    return view


def in_wider_rows(t):
    wide = torch.full((*t.shape[:-1], t.shape[-1] + 8), float("nan"), device=t.device, dtype=t.dtype)
    wide[..., : t.shape[-1]] = t.detach()
    return wide[..., : t.shape[-1]]


@pytest.mark.parametrize("unpack", [at_odd_address, in_wider_rows, lambda t: t.detach().transpose(0, -1).contiguous().transpose(0, -1)],
                         ids=["odd_address", "wider_rows", "transposed"])
@pytest.mark.parametrize("name", CASES)
def test_saved_tensors_of_another_layout(name, unpack):
    """A hook may give back the values in any layout and at any address: the gradients are the same bit for bit."""
    from torchft_b200.ops import attention as A
    from torchft_b200.ops import functional as F

    torch.manual_seed(0)
    fn, _, inputs = CASES[name](F, A)
    results = []
    for hook in (lambda t: t.detach(), unpack):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, hook):
            outs = fn(*inputs)
        outs = outs if isinstance(outs, tuple) else (outs,)
        torch.manual_seed(1)
        results.append(torch.autograd.grad(outs, inputs, [unpack(torch.randn_like(o)) for o in outs]))
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("unpack", [lambda t: t.float() if t.dtype == torch.bfloat16 else t.double(), lambda t: t.detach()[..., :-1],
                                    lambda t: t.cpu()], ids=["dtype", "size", "device"])
@pytest.mark.parametrize("name", CASES)
def test_saved_tensors_of_another_kind_are_refused(name, unpack):
    from torchft_b200.ops import attention as A
    from torchft_b200.ops import functional as F

    fn, _, inputs = CASES[name](F, A)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        out = fn(*inputs)
    out = out[0] if isinstance(out, tuple) else out
    with pytest.raises(RuntimeError, match="saved-tensor hook"):
        torch.autograd.grad(out, inputs, torch.randn_like(out), allow_unused=True)


def test_checkpointed_plain_layers():
    """Recomputation stops early by an exception out of a hook, in the middle of a native node's forward pass."""
    from torch.utils.checkpoint import checkpoint

    from torchft_b200.ops import functional as F

    torch.manual_seed(0)
    x, n, w13, w2 = leaf(16, 256), leaf(256), leaf(128, 256, scale=0.1), leaf(256, 64, scale=0.1)

    def block(x_):
        return F.linear(F.swiglu(F.linear(F.rmsnorm(x_, n), w13)), w2)

    dy = torch.randn(16, 256, device=DEV).to(torch.bfloat16)
    want = torch.autograd.grad(block(x), (x, n, w13, w2), dy)
    got = torch.autograd.grad(checkpoint(block, x, use_reentrant=False), (x, n, w13, w2), dy)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("name", CASES)
def test_exceptions_of_hooks_keep_their_type(name):
    from torchft_b200.ops import attention as A
    from torchft_b200.ops import functional as F

    class Unwilling(Exception):
        pass

    def refuse(t):
        raise Unwilling("hook")

    fn, _, inputs = CASES[name](F, A)
    with torch.autograd.graph.saved_tensors_hooks(refuse, lambda t: t), pytest.raises(Unwilling):
        fn(*inputs)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, refuse):
        out = fn(*inputs)
    with pytest.raises(Unwilling):
        (out[0] if isinstance(out, tuple) else out).sum().backward()


def test_the_interpreter_lock_is_free_during_launches():
    """In place of every kernel's entry stands the question whether this thread holds the lock: 1 is an error, 0 success."""
    from torchft_b200.ops import _lib, _native
    from torchft_b200.ops import attention as A
    from torchft_b200.ops import functional as F

    entries = {name: ctypes.cast(getattr(_lib.lib(), name), ctypes.c_void_p).value for name in _native._ENTRIES}
    others = (_lib.KernelError, _native._status_address, F._weight_gradient, F._main_grad_target)
    holds = ctypes.cast(ctypes.pythonapi.PyGILState_Check, ctypes.c_void_p).value
    sizes = ("tft_gemm2_workspace", "tft_rmsnorm_bwd_parts")
    m = _native.module()
    calls = [(fn, inputs) for fn, _, inputs in (case(F, A) for case in CASES.values())]
    calls.append((F.cross_entropy, [leaf(33, 1000), torch.randint(1000, (33,), device=DEV)]))
    m.setup({name: at if name in sizes else holds for name, at in entries.items()}, *others)
    try:
        for fn, inputs in calls:
            out = fn(*inputs)
            (out[0] if isinstance(out, tuple) else out).sum().backward()
    finally:
        m.setup(entries, *others)


def test_cross_entropy_matches_the_python_node():
    from torchft_b200.ops import functional as F

    torch.manual_seed(0)
    logits, targets = torch.randn(33, 1000, device=DEV).to(torch.bfloat16), torch.randint(1000, (33,), device=DEV)
    got = []
    for fn in (F.cross_entropy, lambda z, t: F._CrossEntropy.apply(z, t, None)):
        z = logits.clone().requires_grad_()
        loss = fn(z, targets)
        loss.backward()
        got.append((loss.detach(), z.grad))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
