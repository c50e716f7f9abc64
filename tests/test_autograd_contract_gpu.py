"""What the native entry points refuse, as the torch.autograd.Function classes behind them do."""
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
