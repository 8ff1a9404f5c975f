"""What a user of this framework has it do on one GPU, as cases for a timing program.

Every case goes through a public entry point: ``StreamedLoss`` (begin / score / finish over one or several candidate
blocks), ``MatryoshkaSigmoidLoss`` (forward and backward of the module, temperature and bias learned), ``BoxLoss`` (the
step of one rank of a box, and one rank of a larger world played on one GPU) and ``ContrastiveTrainer`` (projector, loss,
backward, optimizer, fed from pinned host memory). Sizes are those of the command line modes, the benchmark and the
tests, or lie between them; rows are multiples of 128 and prefix edges multiples of 16, which is what the kernels take.
"""
from __future__ import annotations

import math

import torch

from scalingcontrasts_b200 import ContrastiveTrainer, Domain, LossSpec, Matryoshka, MatryoshkaSigmoidLoss, StreamedLoss
from scalingcontrasts_b200.parallel.box import BoxLoss

IN_FEATURES, MID_FEATURES = 1024, 3072  # the projector of the training benchmark
COST_LIMIT = 72 * 4096 * 4096 * 768     # block rows x rows x channels of the largest listed case


def _case(kind, rows, hidden, ends, blocks=1, positives="self", diagonal="own", beta=10.0, bias=-10.0, dtype="bf16", related=0.0):
    return {"kind": kind, "rows": rows, "hidden": hidden, "ends": ",".join(str(e) for e in ends), "blocks": blocks,
            "positives": positives, "diagonal": diagonal, "beta": beta, "bias": bias, "dtype": dtype, "related": related}


def _halvings(hidden, count):
    return Matryoshka.halvings(hidden, count).ends


def listed():
    pairs = dict(positives="pairs", diagonal="negative")
    named = {
        # The oracle's size: one small block, scored once. Launches and latency are all there is.
        "stream_128": _case("stream", 128, 768, _halvings(768, 5), **pairs),
        # The loss module in somebody's training loop at an everyday batch.
        "module_1024": _case("module", 1024, 768, _halvings(768, 5)),
        # One rank's step of the box mode (publish, barrier, score, finish, all-reduce), replayed as a CUDA graph.
        "box_4096": _case("box", 4096, 768, _halvings(768, 5), **pairs),
        # The width and rows per GPU that the reference publishes its step time at, through the module.
        "module_16384_wide": _case("module", 16384, 1024, _halvings(1024, 5)),
        # One rank of 72 GPUs played on one: 72 blocks of candidates, all but one without own copies.
        "simulate_72x4096": _case("simulate", 4096, 768, _halvings(768, 5), blocks=72),
        # The headline training step, from a pinned host batch to updated weights.
        "train_16384": _case("train", 16384, 768, _halvings(768, 5)),
        # The same training step at a batch where the projector and the host side weigh as much as the loss.
        "train_2048": _case("train", 2048, 768, _halvings(768, 5)),
        # A larger batch streamed through one GPU in three blocks; odd row count, a ladder that is not halvings.
        "stream_ragged_3x2944": _case("stream", 2944, 832, (16, 208, 576, 832), blocks=3, positives="pairs", diagonal="skip"),
        # Learned temperature and bias far from where they start, float32 embeddings, pairs that are alike: the general
        # form of the sigmoid instead of the series for certain negatives.
        "module_learned_3072": _case("module", 3072, 512, _halvings(512, 4), beta=20.0, bias=-3.0, dtype="fp32", related=0.6, **pairs),
        # The memory-saving form of the loss (no gradient cube), two blocks.
        "fused_2x8192": _case("fused", 8192, 768, _halvings(768, 5), blocks=2),
        # The plain sigmoid loss: a single prefix, candidates in four blocks.
        "stream_plain_4x4096": _case("stream", 4096, 1024, (1024,), blocks=4),
        # The deepest ladder the kernels take.
        "stream_deep_2048": _case("stream", 2048, 2048, _halvings(2048, 8), **pairs),
    }
    return [dict(case, name=name) for name, case in named.items()]


def _log_uniform(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng):
    kind = rng.choice(["stream", "stream", "module", "module", "box", "simulate", "train", "fused"])
    rows = 128 * max(1, round(_log_uniform(rng, 128, 16384) / 128))
    if kind == "train":
        hidden = rng.choice([256, 512, 768, 1024])  # the trainer's ladders are halvings
        ends = _halvings(hidden, rng.randint(1, 5))
    elif rng.random() < 0.5:
        hidden = rng.choice([256, 512, 768, 1024])
        ends = _halvings(hidden, rng.randint(1, 5))
    else:
        hidden = 64 * rng.randint(2, 16)
        count = rng.randint(1, 6 if kind == "fused" else 8)
        ends = tuple(sorted(rng.sample(range(16, hidden, 16), min(count - 1, hidden // 16 - 1)))) + (hidden,)
    blocks = 1
    if kind in ("stream", "fused"):
        blocks = rng.randint(1, 4)
    elif kind == "simulate":
        blocks = rng.randint(2, 72)
    most = COST_LIMIT // 2 // (rows * rows * max(hidden, 512))
    blocks = max(1, min(blocks, most))
    positives, diagonal = rng.choice([("self", "own"), ("self", "own"), ("pairs", "negative"), ("pairs", "skip")])
    if kind == "train":
        positives, diagonal = "self", "own"
    beta, bias = rng.choice([(10.0, -10.0), (10.0, -10.0), (5.0, 0.0), (20.0, -3.0), (1.0, 2.0)]) if kind != "train" else (10.0, -10.0)
    dtype = rng.choice(["bf16", "fp32"]) if kind == "module" else "bf16"
    related = rng.choice([0.0, 0.6]) if positives == "pairs" else 0.0
    return _case(kind, rows, hidden, ends, blocks, positives, diagonal, beta, bias, dtype, related)


def _ladder(case):
    return Matryoshka(tuple(int(e) for e in case["ends"].split(",")))


def _embeddings(case, rows, generator):
    """Rows of unit length; with ``related`` above zero, rows 2m and 2m+1 share that much of their variance."""
    values = torch.randn(rows, case["hidden"], device="cuda", generator=generator)
    if case["related"] > 0.0:
        shared = torch.randn(rows // 2, case["hidden"], device="cuda", generator=generator).repeat_interleave(2, dim=0)
        values = math.sqrt(case["related"]) * shared + math.sqrt(1.0 - case["related"]) * values
    values = torch.nn.functional.normalize(values, dim=1)
    return values if case["dtype"] == "fp32" else values.to(torch.bfloat16)


def prepare(case, seed):
    kind, rows, hidden, blocks = case["kind"], case["rows"], case["hidden"], case["blocks"]
    ladder, spec = _ladder(case), LossSpec(case["positives"], case["diagonal"])
    generator = torch.Generator(device="cuda").manual_seed(seed)
    state = {"case": case}
    if kind in ("stream", "fused"):
        state["loss"] = StreamedLoss(rows, hidden, ladder, spec, "cuda", fused=kind == "fused")
        state["blocks"] = [_embeddings(case, rows, generator) for _ in range(blocks)]
    elif kind == "module":
        state["loss"] = MatryoshkaSigmoidLoss(rows, hidden, ladder=ladder, spec=spec, device="cuda",
                                              init_logit_scale=math.log(case["beta"]), init_logit_bias=case["bias"])
        state["embeddings"] = _embeddings(case, rows, generator).requires_grad_()
    elif kind == "box":
        domain = Domain.create(payload_scalars=16, heap_bytes=BoxLoss.heap_bytes(rows, hidden, ladder.count), device="cuda")
        state["engine"] = BoxLoss(rows, hidden, ladder, spec, domain)
        state["engine"].use_graphs = True
        state["embeddings"] = _embeddings(case, rows, generator)
    elif kind == "simulate":
        state["engine"] = BoxLoss(rows, hidden, ladder, spec, None, "cuda")
        state["embeddings"] = _embeddings(case, rows, generator)
    else:
        trainer = ContrastiveTrainer(rows, IN_FEATURES, MID_FEATURES, hidden, ladder.count, spec, device="cuda", seed=seed)
        # A run that is under way: the optimizer has moments and the biases have moved off zero.
        resumed = trainer.state_dict()
        for name, value in resumed["projector"].items():
            if name.endswith("bias"):
                value.normal_(0.0, 0.02, generator=generator)
        for first, second in zip(resumed["optimizer"]["exp_avg"], resumed["optimizer"]["exp_avg_sq"]):
            first.normal_(0.0, 1e-4, generator=generator)
            second.uniform_(1e-8, 1e-7, generator=generator)
        resumed["optimizer"]["steps"] = 1000
        trainer.load_state_dict(resumed)
        batch = torch.randn(rows, IN_FEATURES, device="cuda", generator=generator).to(torch.bfloat16)
        state["trainer"], state["batch"] = trainer, batch.cpu().pin_memory()
    return state


def run(state):
    case = state["case"]
    kind, rows, blocks = case["kind"], case["rows"], case["blocks"]
    if kind in ("stream", "fused"):
        loss, own = state["loss"], state["blocks"][0]
        loss.begin(own)
        for index, block in enumerate(state["blocks"]):
            loss.score(own, block, 0, index * rows, case["beta"], case["bias"], blocks * rows)
        return loss.finish(own)
    if kind == "module":
        loss, embeddings = state["loss"], state["embeddings"]
        embeddings.grad = loss.logit_scale.grad = loss.logit_bias.grad = None
        value = loss(embeddings)
        value.backward()
        return {"loss": value, "prefix_losses": loss.prefix_losses(), "gradient": embeddings.grad,
                "scale_gradient": loss.logit_scale.grad, "bias_gradient": loss.logit_bias.grad}
    if kind == "box":
        gradient, summands = state["engine"].step(state["embeddings"], case["beta"], case["bias"])
        return gradient, summands.clone()  # the engine's are a view of its domain, rewritten by the next step
    if kind == "simulate":
        return state["engine"].simulate(state["embeddings"], blocks, case["beta"], case["bias"])
    trainer = state["trainer"]
    trainer.step(state["batch"])
    parameters = dict(trainer.projector.named_parameters())
    return {"summands": trainer.loss.last_summands, "parameters": {name: p for name, p in parameters.items()},
            "gradients": {name: p.grad for name, p in parameters.items()},
            "scale": trainer.loss.logit_scale, "bias": trainer.loss.logit_bias}


def work(case):
    """Two products of rows x block rows x channels per block (scores, gradient); embeddings in once, gradient out once.
    A training step adds the projector's three products per layer, its batch, and weights, gradients and moments."""
    rows, hidden, blocks = case["rows"], case["hidden"], case["blocks"]
    width = 4 if case["dtype"] == "fp32" else 2
    distinct = blocks if case["kind"] in ("stream", "fused") else 1
    flops = 4.0 * rows * rows * blocks * hidden
    nbytes = (distinct + 1.0) * rows * hidden * width
    if case["kind"] == "train":
        weights = IN_FEATURES * MID_FEATURES + MID_FEATURES * hidden + MID_FEATURES + hidden
        flops += 6.0 * rows * (IN_FEATURES * MID_FEATURES + MID_FEATURES * hidden)
        nbytes = rows * IN_FEATURES * 2.0 + weights * (2 + 2 + 2 + 4 * 4)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Gradients leave in bfloat16 after products with bfloat16 operands: against the same step in float64 they are off by
    2.1e-3 to 3.2e-3 (largest difference 3.5e-2 of the root mean square), the loss and its scalar gradients by 1e-6."""
    return {"rel": 1.2e-2, "max": 1.4e-1}


def _loss_exact(rows, blocks, case):
    """The streamed loss of bfloat16 ``rows`` against ``blocks`` (tensor, first row's number, how often) in float64:
    the gradient of the rows and the twelve summands. An own cell's logit is the scale itself; a cosine whose inverse
    norms' product reaches 100 counts as zero; a cell and its mirror both move the row, hence the factor two."""
    ladder, count = _ladder(case), rows.shape[0]
    live, beta, bias = count * sum(times for _, _, times in blocks), case["beta"], case["bias"]
    q, edges = rows.double(), [0] + list(ladder.ends)
    bands = list(zip(edges[:-1], edges[1:]))

    def inverse_norms(values):
        squares = torch.stack([values[:, a:b].square().sum(1) for a, b in bands]).cumsum(0)
        return torch.where(squares > 0, squares.rsqrt(), torch.zeros_like(squares))

    q_inverse = inverse_norms(q)
    gradient, sums = torch.zeros_like(q), torch.zeros(12, dtype=torch.float64, device=q.device)
    step = 1024
    for block, base, times in blocks:
        c = block.double()
        c_inverse = inverse_norms(c)
        columns = base + torch.arange(c.shape[0], device=q.device)[None, :]
        for first in range(0, count, step):
            part = slice(first, min(first + step, count))
            numbers = torch.arange(part.start, part.stop, device=q.device)[:, None]
            own = numbers == columns
            z, mask = torch.full(own.shape, -1.0, dtype=torch.float64, device=q.device), torch.ones_like(own, dtype=torch.float64)
            if case["positives"] == "pairs":
                z[(numbers ^ 1) == columns] = 1.0
            if case["diagonal"] == "own":
                z[own] = 1.0
            if case["diagonal"] == "skip":
                mask[own] = 0.0
            dots, raws = torch.zeros_like(z), []
            for k, (a, b) in enumerate(bands):
                dots = dots + q[part, a:b] @ c[:, a:b].T
                inverse = q_inverse[k][part, None] * c_inverse[k][None, :]
                floored = inverse >= 100.0
                logit = beta * torch.where(own, 1.0, torch.where(floored, 0.0, dots * inverse))
                s = z * (logit + bias)
                cell = -mask * z * torch.sigmoid(-s) / live
                loss = (mask * torch.nn.functional.softplus(-s)).sum() / live
                sums[[0, 4 + k]] += times * loss
                sums[1] += times * cell.sum()
                sums[2] += times * (cell * logit).sum()
                raws.append(torch.where(own | floored, 0.0, 2.0 * beta * cell * inverse))
                fold = (raws[-1] * dots).sum(1) * q_inverse[k][part].square()
                gradient[part, :b] -= times * fold[:, None] * q[part, :b]
            suffix = torch.zeros_like(z)
            for k in reversed(range(len(bands))):
                a, b = bands[k]
                suffix += raws[k]
                gradient[part, a:b] += times * (suffix @ c[:, a:b])
    return gradient, sums


def _train_exact(case, state):
    """One step of the trainer from the state that ``prepare`` leaves, in float64 from its bfloat16 weights on."""
    trainer, batch = state["trainer"], state["batch"].to("cuda").double()
    names = [name for name, _ in trainer.projector.named_parameters()]
    weights = {name: value.double() for name, value in trainer.projector.state_dict().items()}
    leaves = {name: weights[name].clone().requires_grad_() for name in names}
    hidden = torch.nn.functional.gelu(batch @ leaves["fc1.weight"].T + leaves["fc1.bias"])
    rows = hidden @ leaves["fc2.weight"].T + leaves["fc2.bias"]
    gradient, sums = _loss_exact(rows.detach().to(torch.bfloat16), [(rows.detach().to(torch.bfloat16), 0, 1)], case)
    rows.backward(gradient)
    resumed = trainer.state_dict()["optimizer"]
    values = list(leaves.values()) + [trainer.loss.logit_scale.detach().double(), trainer.loss.logit_bias.detach().double()]
    gradients = [leaf.grad for leaf in leaves.values()] + [sums[2], sums[1]]
    (first, second), count, updated = resumed["betas"], resumed["steps"] + 1, []
    for value, g, m, v in zip(values, gradients, resumed["exp_avg"], resumed["exp_avg_sq"]):
        m, v = first * m.double() + (1 - first) * g, second * v.double() + (1 - second) * g * g
        move = (m / (1 - first ** count)) / ((v / (1 - second ** count)).sqrt() + resumed["eps"])
        updated.append(value.detach() * (1 - resumed["lr"] * resumed["weight_decay"]) - resumed["lr"] * move)
    return {"summands": sums, "parameters": dict(zip(names, updated)), "gradients": dict(zip(names, gradients)),
            "scale": updated[-2], "bias": updated[-1]}


def exact(case, seed):
    kind, count = case["kind"], case["blocks"]
    if kind == "train":
        return _train_exact(case, prepare(case, seed))
    generator = torch.Generator(device="cuda").manual_seed(seed)
    distinct = [_embeddings(case, case["rows"], generator) for _ in range(count if kind in ("stream", "fused") else 1)]
    distinct = [block.to(torch.bfloat16) for block in distinct]
    blocks = [(block, index * case["rows"], 1) for index, block in enumerate(distinct)]
    if kind == "simulate" and count > 1:  # blocks beyond the first hold no own copies and are all alike
        blocks.append((distinct[0], case["rows"], count - 1))
    gradient, sums = _loss_exact(distinct[0], blocks, case)
    if kind == "module":
        ladder = _ladder(case)
        return {"loss": sums[0], "prefix_losses": sums[4:4 + ladder.count], "gradient": gradient,
                "scale_gradient": sums[2], "bias_gradient": sums[1]}
    return gradient, sums
