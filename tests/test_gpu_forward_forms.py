"""The forward kernel's forms (one CTA per tile, pairs of CTAs, pairs without anything of the diagonal) at the sizes and places where the
choice between them, or a tile of theirs, ends: each block against float64, own copies and partners inside, beside and astride."""
import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka, StreamedLoss
from scalingcontrasts_b200._ext import native, stream_handle
from scalingcontrasts_b200.cpu.streamed import CpuStreamedLoss

pytestmark = pytest.mark.gpu

# As for the forms of the cell math: the functions are good to about 1e-7, sums of rows * columns terms in float32; the gradient leaves
# through bfloat16 cubes and a bfloat16 store.
SUMMAND_TOLERANCE, GRADIENT_TOLERANCE = 2e-5, 8e-3


def _rows(rows, hidden, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    values = torch.randn(rows, hidden, device="cuda", generator=generator)
    values[1::2] = 0.6 * values[0::2] + 0.8 * values[1::2]
    return torch.nn.functional.normalize(values, dim=1).to(torch.bfloat16)


def _check(queries, block, ladder, spec, query_base, candidate_base, beta=10.0, bias=-10.0):
    rows, hidden = queries.shape
    live = rows + block.shape[0]
    loss = StreamedLoss(rows, hidden, ladder, spec, "cuda", candidate_rows=block.shape[0])
    for scratch in (loss.partials, loss.similarity_gradients):
        scratch.fill_(float("nan"))
    loss.begin(queries)
    loss.score(queries, block, query_base, candidate_base, beta, bias, live)
    gradient, summands = loss.finish(queries)
    loss.check()
    reference = CpuStreamedLoss(rows, hidden, ladder, spec, torch.float64, "cuda")
    reference.begin(queries)
    reference.score(queries, block, query_base, candidate_base, beta, bias, live)
    expected, sums = reference.finish(queries, torch.empty(rows, hidden, dtype=torch.float64, device="cuda"))
    assert float((gradient.double() - expected).norm() / expected.norm()) < GRADIENT_TOLERANCE
    assert torch.allclose(summands[4:4 + ladder.count].double(), sums[4:4 + ladder.count].double(), rtol=SUMMAND_TOLERANCE, atol=0.0)


@pytest.mark.parametrize("rows,candidates", [(1152, 1024), (1280, 1024), (128, 9472), (128, 9600), (2432, 512), (1152, 1152),
                                             (4736, 5248)])  # the last: runs of two tiles, 41 tiles to a strip
@pytest.mark.parametrize("prefixes", [1, 4, 5, 8])
def test_both_sides_of_one_wave(rows, candidates, prefixes):
    """148 tiles of 64 candidates go to single CTAs, more to pairs or to a walk over the tiles."""
    ladder = Matryoshka(tuple(64 * (k + 1) for k in range(prefixes)))
    queries, block = _rows(rows, ladder.hidden, 1), _rows(candidates, ladder.hidden, 2)
    for base in (0, 128 * 1024):
        _check(queries, block, ladder, LossSpec("pairs"), 0, base)


@pytest.mark.parametrize("ends", [(64, 128, 256, 384, 512, 768), (64, 128, 256, 384, 512, 704), (96, 192, 384, 768, 1536), (96, 192, 384, 768, 1472),
                                  (64, 128, 192, 256, 320, 448, 512), (64, 128, 192, 256, 320, 384, 448), (320, 640), (320, 576), (320,), (256,)])
@pytest.mark.parametrize("base", [0, 1])
def test_both_sides_of_the_lines_for_blocks_with_own_copies(ends, base):
    """Channels and bands at which a block that holds the rows' own copies changes from single CTAs to pairs."""
    ladder = Matryoshka(ends)
    queries, block = _rows(1280, ladder.hidden, 10), _rows(1280, ladder.hidden, 11)
    _check(queries, block, ladder, LossSpec("pairs"), 0, base)


@pytest.mark.parametrize("spec", [LossSpec("self"), LossSpec("pairs"), LossSpec("pairs", "skip")], ids=lambda s: f"{s.positives}-{s.diagonal}")
@pytest.mark.parametrize("query_base,candidate_base", [(0, 0), (1536, 0), (0, 1536), (0, 1535), (1535, 0), (1537, 0), (0, 1537), (1, 1537),
                                                       (1537, 1), (3, 0), (0, 17), (1520, 0), (64, 0)])
def test_own_copies_and_partners_wherever_they_lie(spec, query_base, candidate_base):
    """Blocks side by side hold no own copies; where a number is odd a partner can be just across the border."""
    ladder = Matryoshka((48, 160, 256))
    queries, block = _rows(1536, ladder.hidden, 3), _rows(1536, ladder.hidden, 4)
    _check(queries, block, ladder, spec, query_base, candidate_base)


@pytest.mark.parametrize("prefixes", [1, 3, 5, 6, 8])
@pytest.mark.parametrize("rows_c", [64, 192, 1088])
def test_an_odd_number_of_64_candidates(prefixes, rows_c):
    """The native launch takes candidates in 64s, which single CTAs score: what lies behind the cube and the norms is neither read into
    the sums nor written."""
    ext, rows_q, ladder = native(), 256, Matryoshka(tuple(64 * (k + 1) for k in range(prefixes)))
    hidden = ladder.hidden
    queries, block = _rows(rows_q, hidden, 5), _rows(rows_c, hidden, 6)
    quantities, slots = ext.forward_quantities(prefixes), ext.forward_partial_slots(rows_c, 1)
    f32 = dict(dtype=torch.float32, device="cuda")

    def norms(values):
        inverse, largest = torch.empty(prefixes, values.shape[0], **f32), torch.empty(prefixes, values.shape[0] // 64, **f32)
        ext.prefix_norms(values.data_ptr(), 0, inverse.data_ptr(), largest.data_ptr(), values.shape[0], hidden, list(ladder.ends), stream_handle())
        return inverse, largest

    (q_inverse, _), (c_inverse, c_largest) = norms(queries), norms(block)
    cube = torch.full((prefixes * rows_q * rows_c + 4096,), 7.0, dtype=torch.bfloat16, device="cuda")
    partials = torch.full((slots * quantities * rows_q + 4096,), 7.0, **f32)
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    ext.forward(queries=queries.data_ptr(), candidates=block.data_ptr(), q_inv=q_inverse.data_ptr(), c_inv=c_inverse.data_ptr(),
                c_tile_max=c_largest.data_ptr(), cube=cube.data_ptr(), partials=partials.data_ptr(), status=status.data_ptr(), rows_q=rows_q,
                rows_c=rows_c, hidden=hidden, ends=list(ladder.ends), tiles_per_run=1, beta=10.0, bias=-10.0, weight=1.0, scalars=0,
                query_base=0, candidate_base=0, spec_code=LossSpec("pairs").code(), budget_ns=10 ** 9, pull_src0=0, pull_dst0=0,
                pull_bytes0=0, pull_src1=0, pull_dst1=0, pull_bytes1=0, sms=148, stream=stream_handle())
    torch.cuda.synchronize()
    assert not status.any() and (cube[-4096:] == 7.0).all() and (partials[-4096:] == 7.0).all()
    rows = torch.arange(rows_q, device="cuda")[:, None]
    columns = torch.arange(rows_c, device="cuda")[None, :]
    losses = partials[:-4096].view(slots, quantities, rows_q).double().sum((0, 2))[2:2 + prefixes]
    for k, end in enumerate(ladder.ends):
        cosine = torch.nn.functional.normalize(queries[:, :end].double(), dim=1) @ torch.nn.functional.normalize(block[:, :end].double(), dim=1).T
        logits = 10.0 * torch.where(rows == columns, 1.0, cosine) - 10.0
        signs = torch.where(((rows ^ 1) == columns) | ((rows == columns) & (LossSpec("pairs").diagonal == "own")), 1.0, -1.0)
        expected = torch.nn.functional.softplus(-signs * logits).sum()
        assert float(losses[k]) == pytest.approx(float(expected), rel=SUMMAND_TOLERANCE)


@pytest.mark.parametrize("rows_q,rows_c", [(256, 64), (256, 1088), (1152, 1088), (1280, 1088), (1280, 1024)])
@pytest.mark.parametrize("prefixes,candidate_base", [(1, 0), (4, 64), (5, 0), (5, 4096), (8, 0), (8, 4096)])
def test_the_cube_and_the_records_at_odd_and_even_numbers_of_64_candidates(rows_q, rows_c, prefixes, candidate_base):
    """Every gradient of the cube against float64, and exactly as many records as there are runs, column groups and rows. An odd number
    of 64 candidates has none of 128: single CTAs take it, on and off the diagonal."""
    ext, ladder = native(), Matryoshka(tuple(64 * (k + 1) for k in range(prefixes)))
    hidden, quantities, slots = ladder.hidden, ext.forward_quantities(prefixes), ext.forward_partial_slots(rows_c, 1)
    assert slots == 4 * (rows_c // 64)
    queries, block = _rows(rows_q, hidden, 8), _rows(rows_c, hidden, 9)
    f32 = dict(dtype=torch.float32, device="cuda")
    inverse = []
    for values in (queries, block):
        inverse.append((torch.empty(prefixes, values.shape[0], **f32), torch.empty(prefixes, values.shape[0] // 64, **f32)))
        ext.prefix_norms(values.data_ptr(), 0, inverse[-1][0].data_ptr(), inverse[-1][1].data_ptr(), values.shape[0], hidden,
                         list(ladder.ends), stream_handle())
    cube = torch.full((prefixes, rows_q, rows_c), float("nan"), dtype=torch.bfloat16, device="cuda")
    partials = torch.full((slots, quantities, rows_q), float("nan"), **f32)
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    ext.forward(queries=queries.data_ptr(), candidates=block.data_ptr(), q_inv=inverse[0][0].data_ptr(), c_inv=inverse[1][0].data_ptr(),
                c_tile_max=inverse[1][1].data_ptr(), cube=cube.data_ptr(), partials=partials.data_ptr(), status=status.data_ptr(),
                rows_q=rows_q, rows_c=rows_c, hidden=hidden, ends=list(ladder.ends), tiles_per_run=1, beta=10.0, bias=-10.0, weight=1.0,
                scalars=0, query_base=0, candidate_base=candidate_base, spec_code=LossSpec("pairs").code(), budget_ns=10 ** 9,
                pull_src0=0, pull_dst0=0, pull_bytes0=0, pull_src1=0, pull_dst1=0, pull_bytes1=0, sms=148, stream=stream_handle())
    torch.cuda.synchronize()
    assert not status.any() and partials.isfinite().all()
    rows, columns = torch.arange(rows_q, device="cuda")[:, None], candidate_base + torch.arange(rows_c, device="cuda")[None, :]
    own, signs = rows == columns, torch.where((rows ^ 1) == columns, 1.0, -1.0)  # a row's own copy moves no dot product
    below = torch.zeros(rows_q, rows_c, dtype=torch.float64, device="cuda")
    for k in reversed(range(prefixes)):
        end = ladder.ends[k]
        q, c = queries[:, :end].double(), block[:, :end].double()
        inverses = 1.0 / (q.norm(dim=1)[:, None] * c.norm(dim=1)[None, :])
        logits = 10.0 * (q @ c.T) * inverses - 10.0
        below += torch.where(own, 0.0, -signs * torch.sigmoid(-signs * logits) * 10.0 * inverses)
        # bfloat16 has eight significant bits: rounding to the nearest moves a value by 2^-8 of itself at most, and so the whole
        assert float((cube[k].double() - below).norm() / below.norm()) < 2.0 ** -8


@pytest.mark.parametrize("rows_q,ends", [(4096, [48, 96, 192, 384, 768]), (3584, [64, 112, 1024]), (4864, [1024]), (4096, [32, 272, 1024]),
                                         (3328, [96, 768, 1104]), (4096, [16, 1024]), (4992, [1024])])
@pytest.mark.parametrize("rows_c", [64, 448])
def test_backward_in_pairs_of_ctas(rows_q, ends, rows_c):
    """Launches of more than one round of one-block tiles: pairs, whose UMMAs take channels in steps of 32, and the ones that stay with
    single CTAs (a band of 16, an odd number of row blocks). Float32 sums of bfloat16 products against the same in float64."""
    ext, hidden = native(), ends[-1]
    tiles, ctas = ext.backward_plan(rows_q, ends, 1, 148)
    assert ctas > 148 and all(t[3] == 1 for t in tiles)
    generator = torch.Generator(device="cuda").manual_seed(7)
    cube = (torch.randn(len(ends), rows_q, rows_c, device="cuda", generator=generator) * 0.1).to(torch.bfloat16)
    candidates = torch.randn(rows_c, hidden, device="cuda", generator=generator).to(torch.bfloat16)
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    begins = [0] + ends[:-1]
    expected = 1.0 + 0.5 * torch.cat([cube[b].double() @ candidates.double()[:, begins[b]:ends[b]] for b in range(len(ends))], dim=1)
    outcomes = []
    for _ in range(2):
        gradient = torch.ones(rows_q, hidden, device="cuda")
        ext.backward(cube.data_ptr(), 0, gradient.data_ptr(), status.data_ptr(), rows_q, rows_c, hidden, ends, 1, 0.5, 10 ** 9,
                     stream_handle(), candidates.data_ptr())
        torch.cuda.synchronize()
        assert not status.any()
        # one float32 sum of rows_c products per element: 448 * 2^-24 of the terms' size at most, and one rounding of the whole
        assert float((gradient.double() - expected).norm() / expected.norm()) < 1e-5
        outcomes.append(gradient)
    assert torch.equal(outcomes[0], outcomes[1])


@pytest.mark.parametrize("rows,candidates,ends,candidate_base", [
    (128, 128, (64, 256), 0),                     # single CTAs
    (1280, 1280, (320,), 0),                      # pairs, with own copies
    (1280, 1280, (64, 256), 4096),                # pairs, without
    (4096, 512, (48, 96, 192, 384, 768), 4096),   # the backward in pairs as well
])
def test_a_failure_recorded_before_is_left_at_once(rows, candidates, ends, candidate_base):
    """Kernels that find a failure in the status block score and add nothing, whatever their form, give everything back and leave; once
    the block is clear the same launches work."""
    ladder = Matryoshka(ends)
    queries, block = _rows(rows, ladder.hidden, 12), _rows(candidates, ladder.hidden, 13)
    loss = StreamedLoss(rows, ladder.hidden, ladder, LossSpec("pairs"), "cuda", candidate_rows=candidates)

    def scored():
        loss.begin(queries)
        loss.score(queries, block, 0, candidate_base, 10.0, -10.0, rows + candidates)
        torch.cuda.synchronize()
        return loss.query_gradient.clone(), loss.row_accumulators.clone()

    expected = scored()
    loss.status[0] = 2
    for scratch in (loss.partials, loss.similarity_gradients):
        scratch.fill_(7.0)
    for _ in range(3):
        gradient, accumulators = scored()
        assert not gradient.any() and not accumulators.any()
        assert (loss.partials == 7.0).all() and (loss.similarity_gradients == 7.0).all()
    with pytest.raises(RuntimeError, match="gave up"):
        loss.check()
    loss.status.zero_()
    again = scored()
    loss.check()
    assert torch.equal(again[0], expected[0]) and torch.equal(again[1], expected[1])
