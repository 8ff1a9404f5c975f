"""What the loss module launches around its step: the learned scalars made in the publish launch, the kept summands, and the
backward pass in one launch, each against the torch operations it stands for, bit for bit."""
import math

import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka, MatryoshkaSigmoidLoss
from scalingcontrasts_b200._ext import native, stream_handle

pytestmark = pytest.mark.gpu


def _module(rows=128, hidden=256, **changes):
    return MatryoshkaSigmoidLoss(rows, hidden, ladder=Matryoshka((64, hidden)), spec=LossSpec("pairs"), device="cuda", **changes)


def _embeddings(rows=128, hidden=256, dtype=torch.bfloat16):
    generator = torch.Generator(device="cuda").manual_seed(1)
    values = torch.nn.functional.normalize(torch.randn(rows, hidden, device="cuda", generator=generator), dim=1)
    return values.to(dtype).requires_grad_()


@pytest.mark.parametrize("count", [8, 2048, 2056, 148 * 8 * 256 * 8 + 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("upstream", [1.0, -0.3, 0.0, float("inf"), float("nan")])
def test_scaling_the_gradients_in_one_launch(count, dtype, upstream):
    gradient = torch.randn(count, device="cuda").to(torch.bfloat16)
    factor, summands = torch.tensor(upstream, device="cuda"), torch.randn(12, device="cuda")
    out = torch.full((count,), 7.0, dtype=dtype, device="cuda")
    by_scale, by_bias = torch.empty((), device="cuda"), torch.empty((), device="cuda")
    native().scale_gradients(gradient.data_ptr(), factor.data_ptr(), summands.data_ptr(), out.data_ptr(), dtype == torch.float32,
                             by_scale.data_ptr(), by_bias.data_ptr(), count, stream_handle())
    expected = (gradient * factor.to(torch.bfloat16)).to(dtype)
    assert torch.equal(out.nan_to_num(9.0), expected.nan_to_num(9.0))
    assert torch.equal(torch.stack([by_scale, by_bias]).nan_to_num(9.0), (summands[[2, 1]] * factor).nan_to_num(9.0))


def test_learned_scalars_are_torch_exp():
    """Over the range a log scale takes, and past both ends of float32's exponential."""
    block = _embeddings().detach()
    module, out = _module(), torch.empty(2, device="cuda")
    for value in torch.cat([torch.linspace(-8.0, 8.0, 97), torch.tensor([-200.0, 100.0])]).tolist():
        scale, bias = torch.tensor(value, device="cuda"), torch.tensor(-value, device="cuda")
        module.engine._publish(block, None, (scale, bias, out))
        assert torch.equal(out, torch.stack([scale.exp(), bias]))
        assert not module.engine.loss.sums.any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_backward_in_one_launch_and_through_torch_agree(dtype):
    """With ``create_graph`` the backward pass is made of torch operations that can be differentiated again."""
    module, embeddings = _module(init_logit_scale=math.log(7.0), init_logit_bias=-3.0), _embeddings(dtype=dtype)
    inputs = [embeddings, module.logit_scale, module.logit_bias]
    plain = torch.autograd.grad(module(embeddings) * 0.7, inputs)
    graphed = torch.autograd.grad(module(embeddings) * 0.7, inputs, create_graph=True)
    assert all(a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b) for a, b in zip(plain, graphed))
    weight = torch.tensor(0.7, device="cuda", requires_grad=True)
    first = torch.autograd.grad(module(embeddings) * weight, module.logit_bias, create_graph=True)[0]
    second = torch.autograd.grad(first, weight)[0]
    assert torch.equal(second, module.last_summands[1])


def test_a_module_whose_scalars_are_not_float32():
    module, embeddings = _module(), _embeddings()
    expected = module(embeddings).detach()
    half = _module().to(torch.bfloat16)
    half.logit_scale.data = half.logit_scale.data.double().fill_(math.log(10.0))
    half.logit_bias.data = half.logit_bias.data.double().fill_(-10.0)
    half._scalars = half._scalars.float()
    assert torch.equal(half(embeddings).detach(), expected)


def test_the_loss_is_the_callers_own():
    module, embeddings = _module(), _embeddings()
    first = module(embeddings)
    kept = (first.item(), module.last_summands.clone())
    first += 1.0  # changes neither the kept summands nor anything the next step reads
    second = module(embeddings)
    assert second.item() == kept[0] and first.item() == pytest.approx(kept[0] + 1.0)
    assert torch.equal(module.last_summands, kept[1])
