"""The forward kernel's forms of the cell math (series for easy and near negatives, the general form, cells scored apart on
the diagonal, cells on the cosine floor) at every ladder length, and what the kernels around it do at their edges."""
import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka, StreamedLoss
from scalingcontrasts_b200.cpu.streamed import CpuStreamedLoss

pytestmark = pytest.mark.gpu

LADDERS = {
    1: (256,), 2: (112, 256), 3: (64, 176, 320), 4: (16, 208, 576, 832), 5: (48, 96, 192, 384, 768),
    6: (32, 48, 128, 208, 272, 320), 7: (16, 32, 64, 128, 256, 272, 512), 8: (16, 32, 48, 96, 176, 256, 400, 448),
}


def _rows(rows, hidden, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    values = torch.randn(rows, hidden, device="cuda", generator=generator)
    values[1::2] = 0.6 * values[0::2] + 0.8 * values[1::2]  # partners are alike, so that positives matter
    return torch.nn.functional.normalize(values, dim=1).to(torch.bfloat16)


def _relative(measured, expected):
    return float((measured.double() - expected.double()).norm() / expected.double().norm().clamp_min(1e-30))


# Series and general form agree with the exact functions to about 1e-7 relative; the summands add up to rows * columns such
# terms in float32, the gradient leaves through bfloat16 gradient cubes and a bfloat16 store (2^-9 each, at random).
SUMMAND_TOLERANCE, GRADIENT_TOLERANCE = 2e-5, 8e-3


def _absolute_sums(blocks, ladder, spec, beta, bias):
    """Sums over all cells, in float64, of |d loss / d bias| and |d loss / d log scale|, without the weight 1 / live: what the
    signed sums' rounding errors are measured against."""
    queries, rows = blocks[0].double(), blocks[0].shape[0]
    candidates = torch.cat(blocks).double()
    numbers = torch.arange(rows, device="cuda")[:, None]
    columns = torch.arange(candidates.shape[0], device="cuda")[None, :]
    own, positive = numbers == columns, torch.zeros(rows, candidates.shape[0], dtype=torch.bool, device="cuda")
    if spec.pairs:
        positive |= (numbers ^ 1) == columns
    if spec.diagonal == "own":
        positive |= own
    mask = ~own if spec.diagonal == "skip" else torch.ones_like(own)
    sums = torch.zeros(2, dtype=torch.float64, device="cuda")
    for end in ladder.ends:
        cosine = torch.nn.functional.normalize(queries[:, :end], dim=1) @ torch.nn.functional.normalize(candidates[:, :end], dim=1).T
        logit = beta * torch.where(own, 1.0, cosine)
        cell = mask * torch.sigmoid(torch.where(positive, -1.0, 1.0) * (logit + bias))
        sums += torch.stack([cell.sum(), (cell * logit.abs()).sum()])
    return sums


@pytest.mark.parametrize("beta,bias", [(10.0, -10.0), (10.0, -6.0), (20.0, -3.0), (1.0, 2.0)])
@pytest.mark.parametrize("spec", [LossSpec("self"), LossSpec("pairs"), LossSpec("pairs", "skip")], ids=lambda s: f"{s.positives}-{s.diagonal}")
@pytest.mark.parametrize("prefixes", sorted(LADDERS))
def test_forms_of_the_cell_math_against_float64(prefixes, spec, beta, bias):
    ladder = Matryoshka(LADDERS[prefixes])
    rows, hidden = (128 if prefixes % 2 else 384), ladder.hidden
    blocks = [_rows(rows, hidden, seed) for seed in (1, 2)]
    reference = CpuStreamedLoss(rows, hidden, ladder, spec, torch.float64, "cuda")
    reference.begin(blocks[0])
    for index, block in enumerate(blocks):
        reference.score(blocks[0], block, 0, index * rows, beta, bias, 2 * rows)
    expected, expected_summands = reference.finish(blocks[0], torch.empty(rows, hidden, dtype=torch.float64, device="cuda"))
    absolute = _absolute_sums(blocks, ladder, spec, beta, bias)
    for fused in ([False, True] if prefixes <= 6 else [False]):
        loss = StreamedLoss(rows, hidden, ladder, spec, "cuda", fused=fused)
        for scratch in (loss.query_gradient, loss.row_accumulators, loss.partials, loss.similarity_gradients):
            scratch.fill_(float("nan"))  # a step starts from whatever is there
        for _ in range(2):
            loss.begin(blocks[0])
            for index, block in enumerate(blocks):
                loss.score(blocks[0], block, 0, index * rows, beta, bias, 2 * rows)
            gradient, summands = loss.finish(blocks[0])
        loss.check()
        assert _relative(summands[:3], expected_summands[:3]) < SUMMAND_TOLERANCE
        assert _relative(summands[4:], expected_summands[4:]) < SUMMAND_TOLERANCE
        # each by itself: the losses are sums of positive terms, the two scalar gradients of signed ones
        losses = [0] + list(range(4, 4 + prefixes))
        assert torch.allclose(summands[losses].double(), expected_summands[losses].double(), rtol=SUMMAND_TOLERANCE, atol=0.0)
        assert ((summands[1:3].double() - expected_summands[1:3].double()).abs() <= SUMMAND_TOLERANCE * absolute / (2 * rows)).all()
        assert _relative(gradient, expected) < GRADIENT_TOLERANCE


@pytest.mark.parametrize("prefixes", [1, 4, 8])
def test_every_cosine_on_the_floor(prefixes):
    """Rows so short that every product of inverse norms is past the floor: cosines and gradients are exactly zero."""
    ladder = Matryoshka(LADDERS[prefixes])
    rows, hidden = 128, ladder.hidden
    queries, candidates = (_rows(rows, hidden, seed) * 2.0 ** -7 for seed in (3, 4))
    loss = StreamedLoss(rows, hidden, ladder, LossSpec("self"), "cuda")
    loss.begin(queries)
    loss.score(queries, candidates, 0, rows, 10.0, -10.0, 2 * rows)
    gradient, summands = loss.finish(queries)
    loss.check()
    assert not gradient.any()
    per_prefix = rows * torch.nn.functional.softplus(torch.tensor(-10.0, dtype=torch.float64)) / 2
    assert torch.allclose(summands[4:4 + prefixes].double().cpu(), per_prefix.expand(prefixes), rtol=1e-5)


def test_a_step_without_blocks_is_zero():
    ladder = Matryoshka(LADDERS[5])
    queries = _rows(128, ladder.hidden, 5)
    loss = StreamedLoss(128, ladder.hidden, ladder, LossSpec("self"), "cuda")
    loss.begin(queries)
    loss.score(queries, queries, 0, 0, 10.0, -10.0, 128)
    loss.finish(queries)
    loss.begin(queries)
    gradient, summands = loss.finish(queries)
    assert not gradient.any() and not summands.any()


@pytest.mark.parametrize("fused", [False, True])
def test_row_accumulators_between_blocks(fused):
    """Read in mid-step the accumulators hold what was scored so far."""
    ladder = Matryoshka(LADDERS[5])
    rows, hidden = 256, ladder.hidden
    blocks = [_rows(rows, hidden, seed) for seed in (6, 7, 8)]
    loss = StreamedLoss(rows, hidden, ladder, LossSpec("pairs"), "cuda", fused=fused)
    reference = CpuStreamedLoss(rows, hidden, ladder, LossSpec("pairs"), torch.float64, "cuda")
    loss.begin(blocks[0]), reference.begin(blocks[0])
    for index, block in enumerate(blocks):
        loss.score(blocks[0], block, 0, index * rows, 10.0, -10.0, 3 * rows)
        reference.score(blocks[0], block, 0, index * rows, 10.0, -10.0, 3 * rows)
        if index != 1:
            assert _relative(loss.row_accumulators[0], reference.row_bias_grad) < SUMMAND_TOLERANCE
            assert _relative(loss.row_accumulators[2:7], reference.row_loss) < SUMMAND_TOLERANCE
            assert _relative(loss.row_accumulators[7:], reference.self_coefficients) < 10 * SUMMAND_TOLERANCE  # signed terms
    loss.finish(blocks[0])


@pytest.mark.parametrize("rows,slots,offset", [(128, 1, 0), (128, 9, 0), (384, 70, 0), (132, 8, 0), (130, 5, 0), (128, 3, 1)])
def test_fold_of_the_partials(rows, slots, offset):
    """Whole vectors, ragged rows and buffers that start off a 16-byte boundary."""
    from scalingcontrasts_b200._ext import native

    quantities = 4
    generator = torch.Generator(device="cuda").manual_seed(slots)
    storage = torch.randn(slots * quantities * rows + 1, device="cuda", generator=generator)
    partials = storage[offset:offset + slots * quantities * rows]
    sums = torch.ones(quantities, rows, device="cuda")
    native().fold_partials(partials.data_ptr(), sums.data_ptr(), rows, slots, quantities, torch.cuda.current_stream().cuda_stream)
    expected = 1.0 + partials.view(slots, quantities, rows).double().sum(dim=0)
    assert torch.allclose(sums.double(), expected, rtol=0.0, atol=slots * 4 * 2.0 ** -23)


@pytest.mark.parametrize("rows,hidden", [(64, 64), (192, 832), (37, 128)])
def test_norms_and_their_maxima(rows, hidden):
    from scalingcontrasts_b200._ext import native

    block = torch.randn(rows, hidden, device="cuda").to(torch.bfloat16)
    ends = [16, hidden // 2 // 16 * 16, hidden]
    inverse = torch.full((3, rows), float("nan"), device="cuda")
    maxima = torch.full((3, max(1, rows // 64)), float("nan"), device="cuda")
    copy = torch.zeros_like(block)
    native().prefix_norms(block.data_ptr(), copy.data_ptr(), inverse.data_ptr(), maxima.data_ptr() if rows % 64 == 0 else 0, rows, hidden,
                          ends, torch.cuda.current_stream().cuda_stream)
    expected = torch.stack([block.double()[:, :end].norm(dim=1).reciprocal() for end in ends])
    assert torch.allclose(inverse.double(), expected, rtol=2e-6)
    assert torch.equal(copy, block)
    if rows % 64 == 0:
        assert torch.equal(maxima, inverse.view(3, rows // 64, 64).amax(dim=2))


@pytest.mark.parametrize("rows_q,ends", [(3200, [48, 96, 192, 384, 768]), (4096, [64, 128, 256, 512, 1024]), (4736, [16, 208, 576, 832])])
def test_backward_with_two_ctas_to_a_multiprocessor(rows_q, ends):
    """Launches of more than one CTA per multiprocessor and at most two: 128-channel tiles with half the ring. Float32 sums
    of bfloat16 products against the same in float64; 192 candidates, so the half ring wraps."""
    from scalingcontrasts_b200._ext import native

    ext, hidden, rows_c = native(), ends[-1], 192
    tiles, ctas = ext.backward_plan(rows_q, ends, 1, 148)
    assert 148 < ctas <= 296 and max(t[2] for t in tiles) <= 128
    generator = torch.Generator(device="cuda").manual_seed(9)
    cube = (torch.randn(len(ends), rows_q, rows_c, device="cuda", generator=generator) * 0.1).to(torch.bfloat16)
    candidates = torch.randn(rows_c, hidden, device="cuda", generator=generator).to(torch.bfloat16)
    gradient = torch.ones(rows_q, hidden, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    ext.backward(cube.data_ptr(), 0, gradient.data_ptr(), status.data_ptr(), rows_q, rows_c, hidden, ends, 1, 0.5, 2 * 10 ** 9,
                 torch.cuda.current_stream().cuda_stream, candidates.data_ptr())
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    begins = [0] + ends[:-1]
    expected = 0.5 * torch.cat([cube[b].double() @ candidates.double()[:, begins[b]:ends[b]] for b in range(len(ends))], dim=1)
    assert _relative(gradient, expected + 1.0) < 1e-5
