"""GPU: a step's sums live on the device and follow the stream: ``begin`` clears them, every ``score`` adds to them, whether it
is launched or replayed, and reading them launches nothing."""
import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka, StreamedLoss
from scalingcontrasts_b200._ext import native

pytestmark = pytest.mark.gpu

LADDER = Matryoshka((48, 96, 192, 384, 768))
ROWS = 256


def _rows(seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    return torch.nn.functional.normalize(torch.randn(ROWS, LADDER.hidden, device="cuda", generator=generator), dim=1).bfloat16()


def _loss(fused):
    return StreamedLoss(ROWS, LADDER.hidden, LADDER, LossSpec("pairs"), "cuda", fused=fused)


def _score(loss, queries, block):
    loss.score(queries, block, 0, ROWS, 10.0, -10.0, 4 * ROWS)


def _relative(measured, expected):
    return float((measured.double() - expected.double()).norm() / expected.double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("before,replays", [(0, 1), (0, 3), (1, 2)])
def test_a_captured_block_replays_between_begin_and_finish(fused, before, replays):
    """Captured as a step's first or second block, replayed once or more often in a step begun and finished eagerly."""
    loss, queries, block = _loss(fused), _rows(1), _rows(2)
    loss.begin(queries)
    for _ in range(before + replays):
        _score(loss, queries, block)
    expected = [value.clone() for value in loss.finish(queries)]

    loss.begin(queries)
    for _ in range(before):
        _score(loss, queries, block)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _score(loss, queries, block)
    loss.finish(queries)

    for _ in range(2):
        loss.begin(queries)
        for _ in range(before):
            _score(loss, queries, block)
        for _ in range(replays):
            graph.replay()
        gradient, summands = loss.finish(queries)
        loss.check()
        assert summands.any() and torch.equal(summands, expected[1])  # every block adds, in stream order
        if fused:  # its gradient repeats to float32 rounding, which may move a bfloat16 result by one step of 2^-8
            assert _relative(gradient, expected[0]) < 2.0 ** -8
        else:
            assert torch.equal(gradient, expected[0])


@pytest.mark.parametrize("fused", [False, True])
def test_sums_read_in_mid_step_follow_the_step(fused):
    """Zero after ``begin``, and a tensor held from before shows every block, also one scored on another stream; reading
    launches nothing, so it cannot race with that stream."""
    loss, queries, block = _loss(fused), _rows(3), _rows(4)
    held, gradient = loss.row_accumulators, loss.query_gradient
    loss.begin(queries)
    _score(loss, queries, block)
    loss.finish(queries)
    once, once_gradient = held.clone(), gradient.clone()
    assert once.any() and once_gradient.any()

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    loss.begin(queries, stream=side)
    side.synchronize()
    assert not held.any() and not gradient.any()
    for blocks in (1, 2):
        loss.score(queries, block, 0, ROWS, 10.0, -10.0, 4 * ROWS, stream=side)
        launched = native().launch_count()
        assert loss.row_accumulators.data_ptr() == held.data_ptr()
        assert native().launch_count() == launched
        side.synchronize()
        assert torch.equal(held, blocks * once)  # each block adds the same fold, and doubling is exact
        assert _relative(gradient, blocks * once_gradient) < 1e-6
    loss.finish(queries, stream=side)
    side.synchronize()
    loss.check()


@pytest.mark.parametrize("rows,candidate_rows,ends,tiles_per_run", [
    (128, 128, (64,), 2),                                # one CTA, four records: half of the fold's chains are empty
    (128, 640, (48, 96, 192, 384, 768), 1),              # forty records
    (384, 1152, (16, 32, 48, 96, 176, 256, 400, 448), 2),  # thirty-six: the chains' lengths differ
    (2944, 1408, (16, 208, 576, 832), 1),                # more sums than the launch's warps take in one pass
    (4096, 512, (256,), 2),
    (9600, 256, (16, 32, 48, 96, 176, 256, 400, 448), 4),  # two row blocks to a CTA, the last one alone
])
def test_fold_in_the_backward_launch(rows, candidate_rows, ends, tiles_per_run):
    """The records' fold rides in the backward launch, or is a launch of its own where that launch is split: the same bits."""
    ladder = Matryoshka(ends)
    generator = torch.Generator(device="cuda").manual_seed(5)
    queries, *blocks = (torch.nn.functional.normalize(torch.randn(n, ladder.hidden, device="cuda", generator=generator), dim=1).bfloat16()
                        for n in (rows, candidate_rows, candidate_rows))
    sums = []
    for split in (1, 2):
        loss = StreamedLoss(rows, ladder.hidden, ladder, LossSpec("pairs"), "cuda", candidate_rows=candidate_rows,
                            tiles_per_run=tiles_per_run, backward_split=split)
        loss.partials.fill_(float("nan"))
        loss.begin(queries)
        for index, block in enumerate(blocks):
            loss.score(queries, block, 0, rows + index * candidate_rows, 10.0, -10.0, rows)
        loss.check()
        sums.append((loss.row_accumulators.clone(), loss.query_gradient.clone()))
        loss.finish(queries)
    assert torch.equal(sums[0][0], sums[1][0]) and sums[0][0].isfinite().all() and sums[0][0][0].all()
    assert _relative(sums[0][1], sums[1][1]) < 1e-6  # float32 sums, of a split launch in no fixed order
