"""The loss module's backward pass under the forms of differentiation that torch offers, each against plain backward passes."""
import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka, MatryoshkaSigmoidLoss

pytestmark = pytest.mark.gpu

ROWS, HIDDEN = 256, 256


def _module(**changes):
    return MatryoshkaSigmoidLoss(ROWS, HIDDEN, ladder=Matryoshka((64, HIDDEN)), spec=LossSpec("pairs"), device="cuda", **changes)


def _embeddings(seed=1, dtype=torch.bfloat16):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    values = torch.nn.functional.normalize(torch.randn(ROWS, HIDDEN, device="cuda", generator=generator), dim=1)
    return values.to(dtype).requires_grad_()


def _inputs(module, embeddings):
    return [embeddings, module.logit_scale, module.logit_bias]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("batched", ["is_grads_batched", "vmap"])
def test_a_batch_of_upstream_gradients(dtype, batched):
    """A batch of vector-Jacobian products in one call holds what as many single ones hold."""
    module, embeddings = _module(), _embeddings(dtype=dtype)
    inputs, loss = _inputs(module, embeddings), module(embeddings)
    upstream = torch.tensor([1.0, -0.3, 0.0, 7.0], device="cuda")
    single = [torch.autograd.grad(loss, inputs, u, retain_graph=True) for u in upstream]

    def product(u, **changes):
        return torch.autograd.grad(loss, inputs, u, retain_graph=True, **changes)

    together = product(upstream, is_grads_batched=True) if batched == "is_grads_batched" else torch.vmap(product)(upstream)
    for position, value in enumerate(together):
        expected = torch.stack([one[position] for one in single])
        assert value.dtype == expected.dtype and torch.equal(value, expected)


def test_a_lazily_negated_upstream_gradient():
    """A real view of a conjugate keeps its sign in a flag beside the memory."""
    module, embeddings = _module(), _embeddings()
    inputs, loss = _inputs(module, embeddings), module(embeddings)
    negated = torch.view_as_complex(torch.tensor([0.0, 0.5], device="cuda")).conj().imag
    assert negated.is_neg() and float(negated) == -0.5
    for one, other in zip(torch.autograd.grad(loss, inputs, negated, retain_graph=True),
                          torch.autograd.grad(loss, inputs, torch.tensor(-0.5, device="cuda"))):
        assert torch.equal(one, other)


@pytest.mark.parametrize("cast", [torch.bfloat16, torch.float16, torch.float64])
def test_a_module_cast_to_another_type(cast):
    """The kernels' two scalars stay float32 words whatever the module's parameters become, and when these come back."""
    module, embeddings = _module(init_logit_scale=2.0, init_logit_bias=-3.0), _embeddings()  # exact in every type
    expected = [module(embeddings).detach().clone()] + [g.clone() for g in torch.autograd.grad(module(embeddings), _inputs(module, embeddings))]
    for kind in (cast, torch.float32):
        module.to(kind)
        assert module.logit_scale.dtype == kind and module._scalars.dtype == torch.float32 and module._scalars.numel() == 2
        loss = module(embeddings)
        gradients = torch.autograd.grad(loss, _inputs(module, embeddings))
        assert torch.equal(loss.detach(), expected[0]) and torch.equal(gradients[0], expected[1])
        assert torch.equal(gradients[1], expected[2].to(kind)) and torch.equal(gradients[2], expected[3].to(kind))
