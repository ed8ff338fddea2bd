"""A training step that fails (an empty batch, an error of the library) is not counted: the next one
takes the moments' corrections of the step it is."""
import types

import pytest

from xyce_b200 import _native
from xyce_b200.surrogate import N_IN, N_OUT, AdamConfig, SurrogateMLP

torch = pytest.importorskip("torch")


def network(rc):
    net = SurrogateMLP.__new__(SurrogateMLP)
    net.torch, net.dev, net.step_count = torch, "cpu", 4
    net.T, net.sq = torch.zeros(8, N_OUT), torch.zeros(8)
    seen = []

    def step(args, stream):
        seen.append(args._obj.adam.bias_corr1)
        return rc

    net.k = types.SimpleNamespace(lib=types.SimpleNamespace(xd_mlp_train_step=step), stream=lambda: None)
    net._load_inputs = lambda X: (len(X), 8)
    net._train_args = _native.XdMlpTrainArgs
    return net, seen


def test_failed_steps_are_not_counted():
    net, seen = network(-3)
    with pytest.raises(_native.NativeError):
        net.train_step(torch.zeros(3, N_IN), torch.zeros(3, N_OUT), AdamConfig())
    with pytest.raises(ZeroDivisionError):
        net.train_step(torch.zeros(0, N_IN), torch.zeros(0, N_OUT), AdamConfig())
    assert net.step_count == 4 and len(seen) == 1
    net, seen = network(0)
    net.train_step(torch.zeros(3, N_IN), torch.zeros(3, N_OUT), AdamConfig(beta1=0.5))
    assert net.step_count == 5 and seen == [1 - 0.5 ** 5]
