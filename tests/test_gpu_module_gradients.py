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


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_two_forwards_before_a_backward(dtype, graphs):
    """Each forward's gradients are its own, also when another forward, or a step of the engine, comes before the backward."""
    module = _module()
    module.engine.use_graphs = graphs
    first, second = _embeddings(1, dtype), _embeddings(2, dtype)
    expected = [torch.autograd.grad(module(x), _inputs(module, x)) for x in (first, second)]
    for _ in range(3):  # of a captured step: in line, captured, replayed
        a, b = module(first), module(second)
        module.engine.step(_embeddings(3).detach())
        gradients = torch.autograd.grad(a + 2.0 * b, [first, second, module.logit_scale, module.logit_bias])
        assert torch.equal(gradients[0], expected[0][0]) and torch.equal(gradients[1], 2.0 * expected[1][0])
        for value, one, other in zip(gradients[2:], expected[0][1:], expected[1][1:]):
            assert torch.equal(value, one + 2.0 * other)


@pytest.mark.parametrize("graphs", [False, True])
def test_the_promise_of_a_bare_backward(graphs):
    """``unit_upstream`` hands the row gradients on as they are; with captured steps these lie in the engine's one buffer, and a
    backward that comes after the next step is refused instead of handing on that step's."""
    module, first, second = _module(), _embeddings(1), _embeddings(2)
    expected = [torch.autograd.grad(module(x), x)[0] for x in (first, second)]
    module.unit_upstream, module.engine.use_graphs = True, graphs
    for _ in range(3):
        for x, gradient in zip((first, second), expected):
            assert torch.equal(torch.autograd.grad(module(x), x)[0], gradient)
    late, _ = module(first), module(second)
    if graphs:
        with pytest.raises(RuntimeError, match="overwritten by a later step"):
            torch.autograd.grad(late, first)
    else:
        assert torch.equal(torch.autograd.grad(late, first)[0], expected[0])
