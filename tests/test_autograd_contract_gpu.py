"""What the native entry points refuse, as the torch.autograd.Function classes behind them do: forward-mode tangents, and
second derivatives (a backward under create_graph runs, a derivative through its gradients raises)."""
import pytest
import torch

from helpers import dfw_inputs, lfw_inputs, to_dev

pytestmark = pytest.mark.gpu


def _call(which, dev):
    """(function, differentiable arguments, further arguments, upstream gradients)"""
    from t2fw_b200.functional_dfw import DFWFunction
    from t2fw_b200.functional_fused import LFWFusedFunction
    from t2fw_b200.functional_lfw import LFWFunction

    if which == "lfw":
        *ins, go, gs = to_dev(lfw_inputs(2, 70, 64, 64, "sigmoid", 0.3, 11), torch.float16, dev)
        return LFWFunction, ins, [], [go, gs]
    if which == "dfw":
        *ins, go, gs = to_dev(dfw_inputs(2, 70, 64, 64, "scaled", 0.3, 12), torch.float16, dev)
        return DFWFunction, ins, [], [go, gs]
    g = torch.Generator().manual_seed(13)
    qkvg, state = torch.randn(2, 70, 4 * 128, generator=g), torch.randn(4, 64, 64, generator=g)
    go, gs = torch.randn(2, 70, 128, generator=g), torch.randn(4, 64, 64, generator=g)
    ins = [t.half().to(dev) for t in (qkvg, state, go, gs)]
    return LFWFusedFunction, ins[:2], [2], ins[2:]


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("which", ["lfw", "dfw", "fused"])
def test_forward_mode_is_refused(cuda, which, grad):
    import torch.autograd.forward_ad as fw

    fn, ins, rest, _ = _call(which, cuda)
    for i in range(len(ins)):
        with fw.dual_level(), torch.set_grad_enabled(grad):
            args = list(ins)
            args[i] = fw.make_dual(ins[i], torch.ones_like(ins[i]))
            with pytest.raises(NotImplementedError, match="jvp"):
                fn.apply(*args, *rest)
        fn.apply(*ins, *rest)      # outside the level the same tensors are plain again


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("which", ["lfw", "dfw", "fused"])
def test_second_derivative_raises(cuda, which, native):
    fn, ins, rest, up = _call(which, cuda)
    if not native:      # a subclass takes torch.autograd.Function.apply and torch.ops
        fn = type("Sub", (fn,), {})
    leaves = [t.clone().requires_grad_(True) for t in ins]
    first = torch.autograd.grad(fn.apply(*leaves, *rest), leaves, up)
    # constant upstream gradients: the dependence on the inputs is through the saved tensors alone
    again = torch.autograd.grad(fn.apply(*leaves, *rest), leaves, up, create_graph=True)
    for a, b in zip(first, again):
        assert torch.equal(a, b) and b.requires_grad
    with pytest.raises(RuntimeError, match="not implemented"):
        torch.autograd.grad(again[0].float().sum() + leaves[0].float().square().sum(), leaves[0])
    # and through the upstream gradients
    up = [t.clone().requires_grad_(True) for t in up]
    again = torch.autograd.grad(fn.apply(*leaves, *rest), leaves, up, create_graph=True)
    with pytest.raises(RuntimeError, match="not implemented"):
        torch.autograd.grad(again[-1].float().sum(), up[0])


@pytest.mark.parametrize("n_head", [0, -1, 3, 1 << 70, (1 << 56) + 2])
def test_impossible_head_counts_are_refused_alike(cuda, n_head):
    """The class's assertion, also for numbers that a C integer, or their product with the row length, does not hold."""
    fn, ins, _, _ = _call("fused", cuda)
    with pytest.raises(AssertionError):
        fn.apply(*ins, n_head)
