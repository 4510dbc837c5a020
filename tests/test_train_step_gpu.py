"""Training steps that the fused call is not for run layer by layer, as before it was there.

The layers' loss and bias gradients are summed with atomics, so two runs differ in the last
bits: weights are compared to 1e-5, as the fused step's are with the layers'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(ctx, n=3000):
    import torch

    from delta_b200.learned import labelled
    from delta_b200.scenarios import narrowphase_pairs

    a, b, _, _ = narrowphase_pairs(n, seed=3)
    X, T, valid = labelled(ctx, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    return X, T, valid, int(valid.sum().item())


def _same(one, ref):
    assert np.max(np.abs(one.params.cpu().numpy() - ref.params.cpu().numpy())) <= 1e-5
    assert one.steps == ref.steps == 2


def _layers(model, X, T, valid, nv):
    for _ in range(2):
        model.forward(X)
        model.backward(X, T, valid, nv)
        model.adam()


def test_a_models_own_update_is_called():
    """A subclass whose adam also decays the weights."""
    from delta_b200.learned import WarmStartMLP
    from delta_b200.narrowphase import Context

    class Decaying(WarmStartMLP):
        def adam(self, *args, **kw):
            super().adam(*args, **kw)
            self.params.mul_(0.99)

    ctx = Context(0)
    X, T, valid, nv = _rows(ctx)
    one, ref = Decaying.load(ctx), Decaying.load(ctx)
    _layers(ref, X, T, valid, nv)
    for _ in range(2):
        one.train_step(X, T, valid, nv)
    ctx.synchronize()
    _same(one, ref)
    ctx.close()


def test_an_engine_set_through_the_library_is_followed():
    """delta_mlp_set_engine without learned.set_engine: the step runs on mma.sync."""
    from delta_b200._lib import check, lib
    from delta_b200.learned import ENGINES, WarmStartMLP
    from delta_b200.narrowphase import Context

    ctx = Context(0)
    check(lib().delta_mlp_set_engine(ctx.handle, ENGINES["mma"]))
    X, T, valid, nv = _rows(ctx, 200)
    one, ref = WarmStartMLP.load(ctx), WarmStartMLP.load(ctx)
    _layers(ref, X, T, valid, nv)
    for _ in range(2):
        one.train_step(X, T, valid, nv)
    ctx.synchronize()
    _same(one, ref)
    ctx.close()


def test_a_step_that_fails_is_not_counted():
    from delta_b200._lib import DeltaError
    from delta_b200.learned import WarmStartMLP
    from delta_b200.narrowphase import Context

    class Nothing:
        @staticmethod
        def data_ptr():
            return None  # refused on the host

    ctx = Context(0)
    X, T, _, nv = _rows(ctx, 200)
    model = WarmStartMLP.load(ctx)
    with pytest.raises(DeltaError):
        model.train_step(X, T, Nothing, nv)
    assert model.steps == 0
    ctx.close()
