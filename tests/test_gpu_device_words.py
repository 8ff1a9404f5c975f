"""What the kernels take by address as float32 words (the scalars, a learned log scale and bias, the span to clear): anything else
is refused on the host, or goes the way through torch."""
import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka, MatryoshkaSigmoidLoss, StreamedLoss
from scalingcontrasts_b200.ops.streamed_loss import BlockNorms, compute_block_norms
from scalingcontrasts_b200.parallel.box import BoxLoss

pytestmark = pytest.mark.gpu

ROWS, LADDER = 128, Matryoshka((64, 256))
# more words than the kernels touch: on code without the checks these calls stay inside their tensors
BAD = {"half": lambda: torch.zeros(8, dtype=torch.float16, device="cuda"), "double": lambda: torch.zeros(8, dtype=torch.float64, device="cuda"),
       "strided": lambda: torch.zeros(8, device="cuda")[::2], "host": lambda: torch.zeros(8)}


def _rows():
    generator = torch.Generator(device="cuda").manual_seed(1)
    return torch.nn.functional.normalize(torch.randn(ROWS, LADDER.hidden, device="cuda", generator=generator), dim=1).bfloat16()


def _word(value):
    return torch.tensor(value, device="cuda")


@pytest.mark.parametrize("kind", list(BAD))
def test_words_of_another_kind_are_refused(kind):
    rows, norms = _rows(), BlockNorms(LADDER.count, ROWS, device="cuda")
    good = (_word(1.0), _word(-1.0), torch.zeros(2, device="cuda"))
    for position in range(3):
        learned = list(good)
        learned[position] = BAD[kind]()
        with pytest.raises(ValueError, match="float32|must lie on"):
            compute_block_norms(rows, LADDER, norms, learned=tuple(learned))
    with pytest.raises(ValueError, match="float32|must lie on"):
        compute_block_norms(rows, LADDER, norms, clear=BAD[kind]())
    loss = StreamedLoss(ROWS, LADDER.hidden, LADDER, LossSpec("pairs"), "cuda")
    loss.begin(rows)
    with pytest.raises(ValueError, match="float32|must lie on"):
        loss.score(rows, rows, 0, 0, 10.0, -10.0, ROWS, scalars=BAD[kind]())


def test_too_few_words_and_no_place_for_them_are_refused():
    rows, engine = _rows(), BoxLoss(ROWS, LADDER.hidden, LADDER, LossSpec("pairs"), None, "cuda")
    with pytest.raises(ValueError, match="at least 2"):
        engine.step(rows, scalars=torch.zeros(1, device="cuda"))
    with pytest.raises(ValueError, match="at least 2"):
        engine.step(rows, scalars=torch.zeros(1, device="cuda"), learned=(_word(1.0), _word(-1.0)))
    with pytest.raises(ValueError, match="both must be given"):
        engine.step(rows, learned=(_word(1.0), _word(-1.0)))
    expected = engine.step(rows, 10.0, -10.0)[1].clone()
    for scalars in (torch.tensor([10.0, -10.0], device="cuda"), torch.tensor([10.0, -10.0]).pin_memory()):
        assert torch.equal(engine.step(rows, scalars=scalars)[1], expected)


def test_a_log_scale_that_is_no_single_word():
    """Two values cannot be a scale; one value in a vector, on the host or negated lazily can."""
    def module(scale):
        made = MatryoshkaSigmoidLoss(ROWS, LADDER.hidden, ladder=LADDER, spec=LossSpec("pairs"), device="cuda")
        made.logit_scale = torch.nn.Parameter(scale)
        return made(_rows()).detach()

    expected = module(_word(2.0))
    with pytest.raises(RuntimeError):
        module(torch.tensor([2.0, 1.0], device="cuda"))
    negated = torch.view_as_complex(torch.tensor([0.0, -2.0], device="cuda")).conj().imag
    for scale in (torch.tensor([2.0], device="cuda"), torch.tensor(2.0), negated):
        assert torch.equal(module(scale), expected)
