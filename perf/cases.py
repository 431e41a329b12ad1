"""Performance cases: what a program that trains with this package has it do, on one GPU.

Every case is one call of a public entry point, with the state that a training program has in hand at that moment:

* ``step``      ``soap_step`` on an ordinary step: rotate, Adam in the eigenbasis, rotate back, Gram averages;
* ``refresh``   ``soap_step`` on a step that also refreshes both eigenbases (power iteration + QR, momentum and variance
  carried over), which training does every tenth step;
* ``optimizer`` ``SoapTP.step()`` over the weights of one small decoder layer: many small matrices and vectors, where
  launches and the host count;
* ``embedding`` ``SoapTP.step()`` on a vocabulary-sized matrix, preconditioned on its short side only;
* ``rotate``    the public two-sided rotation, there and back, as programs that compose the ops use it.

A case names its sizes and the gradient's type (``fp32``, or ``bf16`` as mixed-precision training hands it over).
"""
import math

import torch
import torch.distributed as dist

from soap_tp_b200 import soap_step
from soap_tp_b200.ops import rotate_2d_block_cyclic_
from soap_tp_b200.optim import SoapTP

BLOCK, GRID = 128, (1, 1)
BETA, BETA1, BETA2, EPS = 0.95, 0.95, 0.95, 1e-8
SIGMA = 1e-3                    # standard deviation of a gradient's entries
START = 20                      # steps taken before the measured one
NEVER = 10**9                   # refresh interval of the cases that time ordinary steps
LR, DECAY = 3e-3, 0.01
NAMES = ("left_preconditioner", "right_preconditioner", "momentum", "variance")


def listed():
    return [
        # the smallest matrices a user shards or replicates: a router, a small projection.  Launches and host time.
        dict(name="step_256x512", kind="step", rows=256, cols=512, dtype="fp32"),
        # an odd, ragged shape: not a multiple of any tile, and columns that are not 16-byte aligned
        dict(name="step_1000x1501", kind="step", rows=1000, cols=1501, dtype="bf16"),
        # a weight of a model of ordinary width, with the gradients of mixed-precision training
        dict(name="step_2048x5504", kind="step", rows=2048, cols=5504, dtype="bf16"),
        # an attention projection of a decoder of hidden size 4096
        dict(name="step_4096x4096", kind="step", rows=4096, cols=4096, dtype="bf16"),
        # the benchmark's matrix
        dict(name="step_8192x8192", kind="step", rows=8192, cols=8192, dtype="fp32"),
        # the MLP of the same decoder: the longest side that is preconditioned in practice
        dict(name="step_14336x4096", kind="step", rows=14336, cols=4096, dtype="bf16"),
        # refresh steps: the smallest configuration of record, a ragged oblong one, and the benchmark's matrix
        dict(name="refresh_1024x1024", kind="refresh", rows=1024, cols=1024, dtype="fp32"),
        dict(name="refresh_3000x2000", kind="refresh", rows=3000, cols=2000, dtype="bf16"),
        dict(name="refresh_8192x8192", kind="refresh", rows=8192, cols=8192, dtype="fp32"),
        # one decoder layer of hidden size 512: seven matrices and two norms in one optimizer step
        dict(name="optimizer_512_1376", kind="optimizer", rows=512, cols=1376, dtype="fp32"),
        # a quarter of a 128256-word vocabulary, one-sided
        dict(name="embedding_32064x2048", kind="embedding", rows=32064, cols=2048, dtype="bf16"),
        # the composable op
        dict(name="rotate_3072x2048", kind="rotate", rows=3072, cols=2048, dtype="fp32"),
    ]


def _side(rng, low, high):
    """A side, spread over the logarithm of its range: any integer, or a multiple of 64 as widths mostly are."""
    value = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return value if rng.random() < 0.4 else max(64, value // 64 * 64)


def draw(rng):
    kind = rng.choice(("step", "step", "step", "refresh", "refresh", "optimizer", "embedding", "rotate"))
    dtype = rng.choice(("fp32", "bf16"))
    if kind == "step":
        rows = _side(rng, 128, 14336)
        cols = _side(rng, 128, min(14336.0, 14336.0 * 4096 / rows))
    elif kind == "refresh":
        rows, cols = _side(rng, 256, 6144), _side(rng, 256, 6144)
    elif kind == "optimizer":
        rows = rng.randrange(4, 17) * 64
        cols, dtype = rows * rng.randrange(20, 40) // 10, "fp32"
    elif kind == "embedding":
        rows, cols = rng.randrange(16400, 32065), rng.randrange(4, 33) * 64
    else:
        rows, cols, dtype = _side(rng, 128, 6144), _side(rng, 128, 6144), "fp32"
    return dict(kind=kind, rows=rows, cols=cols, dtype=dtype)


# ---- inputs ----------------------------------------------------------------------------------------------------
_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}


def _group():
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _column_major(matrix):
    """The packed buffer of a (1, 1) grid: fp32, column-major."""
    return matrix.to(torch.float32).T.contiguous().T


def _empty(rows, cols):
    return torch.zeros((cols, rows), dtype=torch.float32, device="cuda").T


def _dct_basis(n, gen):
    """A dense orthogonal matrix: cosines with random signs and a random column order."""
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    basis = torch.cos(torch.pi / n * (i[:, None] + 0.5) * i[None, :]).mul_(math.sqrt(2.0 / n))
    basis[:, 0] *= math.sqrt(0.5)
    signs = torch.randint(0, 2, (2, n), generator=gen, device="cuda", dtype=torch.float64) * 2 - 1
    return basis.mul_(signs[0][:, None]).mul_(signs[1])[:, torch.randperm(n, generator=gen, device="cuda")]


def _plain_gram(n, other, gen):
    """A symmetric positive matrix of the size that an average of Gram matrices has (``other`` is the contracted side)."""
    noise = torch.randn(n, n, generator=gen, device="cuda")
    noise = (noise + noise.T).mul_(0.7 * SIGMA * SIGMA * math.sqrt(other) * 0.2)
    noise.diagonal().add_(SIGMA * SIGMA * other)
    return noise


def _separated_problem(n, other, gen):
    """``(P, Q)`` of a refresh, in fp64: a preconditioner and the basis that it is nearly diagonal in.

    The order of the new columns comes from eigenvalue estimates, and their signs from the signs of the pivots.  So that
    both are the same for every correct implementation, the eigenvalues lie in a geometric series (1000 : 1), well above
    what one gradient adds, and the basis is a product of reflectors whose pivots are 0.1 to 0.8 of a column's norm.
    """
    tail = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * 0.7 + 0.1
    tail[-1] = 0.0
    vectors = torch.randn(n, n, generator=gen, device="cuda", dtype=torch.float64).tril_(-1)
    norms = vectors.square().sum(dim=0).clamp_min_(1e-300)
    vectors *= (tail / norms).sqrt()
    vectors.diagonal().fill_(1.0)
    tau = 2.0 / vectors.square().sum(dim=0)
    tau[-1] = 0.0
    basis = torch.linalg.householder_product(vectors, tau)
    del vectors
    values = 30.0 * SIGMA * SIGMA * other * torch.logspace(3, 0, n, device="cuda", dtype=torch.float64)
    moved = torch.randn(n, n, generator=gen, device="cuda", dtype=torch.float64).triu_(1)
    moved = (moved + moved.T).mul_(1e-4).mul_(values.sqrt()[:, None]).mul_(values.sqrt())
    moved.diagonal().add_(values)
    preconditioner = basis @ moved @ basis.T
    preconditioner = (preconditioner + preconditioner.T) * 0.5
    return preconditioner, basis[:, torch.randperm(n, generator=gen, device="cuda")]


def _moments(rows, cols, gen):
    momentum = torch.randn(rows, cols, generator=gen, device="cuda") * (0.3 * SIGMA)
    variance = (torch.rand(rows, cols, generator=gen, device="cuda") + 0.5) * (SIGMA * SIGMA)
    return momentum, variance


def _soap_state(rows, cols, gen, separated):
    if separated:
        left, left_basis = _separated_problem(rows, cols, gen)
        right, right_basis = _separated_problem(cols, rows, gen)
    else:
        left, left_basis = _plain_gram(rows, cols, gen), _dct_basis(rows, gen)
        right, right_basis = _plain_gram(cols, rows, gen), _dct_basis(cols, gen)
    momentum, variance = _moments(rows, cols, gen)
    return dict(left_preconditioner=_column_major(left), right_preconditioner=_column_major(right),
                left_basis=_column_major(left_basis), right_basis=_column_major(right_basis),
                left_work=_empty(rows, rows), right_work=_empty(cols, cols), momentum=_column_major(momentum),
                variance=_column_major(variance), step=START)


def _gradient(rows, cols, dtype, gen):
    return (torch.randn(rows, cols, generator=gen, device="cuda") * SIGMA).to(_DTYPES[dtype])


def _layer_shapes(case):
    """One decoder layer: q, k, v, o, gate, up, down and two norms; ``(shape, tp_shard_dim)``."""
    h, m = case["rows"], case["cols"]
    return [((h, h), 0), ((h // 4, h), 0), ((h // 4, h), 0), ((h, h), 1), ((m, h), 0), ((m, h), 0), ((h, m), 1),
            ((h,), None), ((h,), None)]


def _shapes(case):
    return _layer_shapes(case) if case["kind"] == "optimizer" else [((case["rows"], case["cols"]), 0)]


def _optimizer(case, gen):
    parameters, entries = [], {}
    for index, (shape, shard_dim) in enumerate(_shapes(case)):
        p = torch.nn.Parameter((torch.randn(shape, generator=gen, device="cuda") * 0.02).to(_DTYPES[case["dtype"]]))
        p.grad = (torch.randn(shape, generator=gen, device="cuda") * SIGMA).to(p.dtype)
        if shard_dim is not None:
            p.tp_shard_dim, p.tp_global_shape = shard_dim, shape
        if case["kind"] == "embedding":
            rows, h = shape
            momentum, variance = _moments(rows, h, gen)
            # the engine keeps the transposed moments of a one-sided matrix: h x rows, column-major
            entry = dict(right_preconditioner=_column_major(_plain_gram(h, rows, gen)),
                         right_basis=_column_major(_dct_basis(h, gen)), right_work=_empty(h, h), momentum=momentum.T,
                         variance=variance.T, step=START)
        elif shard_dim is None:
            momentum, variance = _moments(shape[0], 1, gen)
            entry = dict(step=START, exp_avg=momentum[:, 0].clone(), exp_avg_sq=variance[:, 0].clone())
        else:
            entry = _soap_state(shape[0], shape[1], gen, separated=False)
        parameters.append(p)
        entries[index] = entry
    optimizer = SoapTP(parameters, lr=LR, weight_decay=DECAY, precondition_frequency=NEVER)
    saved = optimizer.state_dict()
    saved["state"] = entries
    optimizer.load_state_dict(saved)
    return optimizer, parameters


def prepare(case, seed):
    _group()
    gen = _generator(seed)
    kind, rows, cols = case["kind"], case["rows"], case["cols"]
    if kind in ("optimizer", "embedding"):
        optimizer, parameters = _optimizer(case, gen)
        return dict(case=case, optimizer=optimizer, parameters=parameters)
    if kind == "rotate":
        return dict(case=case, matrix=_column_major(torch.randn(rows, cols, generator=gen, device="cuda")),
                    left=_column_major(_dct_basis(rows, gen)), right=_column_major(_dct_basis(cols, gen)))
    state = _soap_state(rows, cols, gen, separated=kind == "refresh")
    return dict(case=case, gradient=_gradient(rows, cols, case["dtype"], gen), soap=state)


# ---- one pass ----------------------------------------------------------------------------------------------------
def _optimizer_outputs(case, parameters, state_of):
    outputs = {}
    for index, p in enumerate(parameters):
        entry = state_of(p)
        outputs[f"p{index}"] = p.detach()
        for name in NAMES + ("exp_avg", "exp_avg_sq"):
            if name in entry:
                outputs[f"p{index}_{name}"] = entry[name]
    return outputs


def run(state):
    case = state["case"]
    if case["kind"] in ("optimizer", "embedding"):
        optimizer = state["optimizer"]
        optimizer.step()
        return _optimizer_outputs(case, state["parameters"], lambda p: optimizer.state[p])
    shape = (case["rows"], case["cols"])
    if case["kind"] == "rotate":
        rotated = rotate_2d_block_cyclic_(state["matrix"].clone(), state["left"], state["right"], shape, BLOCK, GRID,
                                          direction="forward")
        back = rotate_2d_block_cyclic_(rotated.clone(), state["left"], state["right"], shape, BLOCK, GRID,
                                       direction="backward")
        return dict(rotated=rotated, back=back)
    soap = state["soap"]
    refreshing = case["kind"] == "refresh"
    update = soap_step(state["gradient"], soap, global_shape=shape, shard_dim=0, block_size=BLOCK, process_grid_shape=GRID,
                       preconditioner_beta=BETA, beta1=BETA1, beta2=BETA2, eps=EPS,
                       basis_refresh_interval=1 if refreshing else NEVER)
    outputs = dict(update=update, **{name: soap[name] for name in NAMES})
    if refreshing:
        outputs.update(left_basis=soap["left_basis"], right_basis=soap["right_basis"])
    return outputs


# ---- cost --------------------------------------------------------------------------------------------------------
def _step_work(rows, cols, item):
    """Two two-sided products and two symmetric Gram products; every buffer read (and, if it changes, written) once."""
    flops = 5.0 * rows * cols * (rows + cols)
    moved = item * rows * cols + 4.0 * (5 * rows * cols + 3 * rows * rows + 3 * cols * cols)
    return moved, flops


def work(case):
    item = 2 if case["dtype"] == "bf16" else 4
    rows, cols = case["rows"], case["cols"]
    if case["kind"] == "rotate":
        return dict(bytes=4.0 * (3 * rows * cols + rows * rows + cols * cols), flops=4.0 * rows * cols * (rows + cols))
    if case["kind"] == "embedding":
        # rotate there and back on one side, one symmetric Gram product; the parameter is read and written as well
        return dict(bytes=3.0 * item * rows * cols + 4.0 * (4 * rows * cols + 3 * cols * cols), flops=5.0 * rows * cols * cols)
    if case["kind"] == "optimizer":
        moved = flops = 0.0
        for shape, shard_dim in _shapes(case):
            if shard_dim is None:
                moved += 28.0 * shape[0]
                continue
            more, products = _step_work(shape[0], shape[1], item)
            moved, flops = moved + more + 4.0 * shape[0] * shape[1], flops + products
        return dict(bytes=moved, flops=flops)
    moved, flops = _step_work(rows, cols, item)
    if case["kind"] == "refresh":
        # momentum there and back; P Q, QR and the explicit Q of both sides
        flops += 4.0 * rows * cols * (rows + cols) + (2.0 + 8.0 / 3.0) * (rows**3 + cols**3)
        moved += 4.0 * (rows * rows + cols * cols)
    return dict(bytes=moved, flops=flops)


# ---- what is right -----------------------------------------------------------------------------------------------
def tolerance(case):
    # products of fp32 accuracy; a refresh passes them through a QR factorisation as well
    return {"rel": 4e-5 if case["kind"] == "refresh" else 1e-5}


def _wide(t):
    return t.detach().to(torch.float64)


def _exact_step(gradient, soap, step, refreshing):
    g = _wide(gradient)
    QL, QR = _wide(soap["left_basis"]), _wide(soap["right_basis"])
    L, R, M, V = (_wide(soap[name]) for name in NAMES)
    rotated = QL.T @ g @ QR
    M = BETA1 * M + (1 - BETA1) * rotated
    V = BETA2 * V + (1 - BETA2) * rotated * rotated
    bias1, bias2 = 1 - BETA1**step, 1 - BETA2**step
    update = QL @ ((M / bias1) / ((V / bias2).sqrt() + EPS / math.sqrt(bias2))) @ QR.T
    L = BETA * L + (1 - BETA) * g @ g.T
    R = BETA * R + (1 - BETA) * g.T @ g
    outputs = dict(update=update)
    if refreshing:
        M = QL @ M @ QR.T
        bases, orders = [], []
        for P, Q in ((L, QL), (R, QR)):
            powered = P @ Q
            order = torch.argsort((Q * powered).sum(dim=0), descending=True, stable=True)
            bases.append(torch.linalg.qr(powered[:, order])[0])
            orders.append(order)
        V = V[orders[0]][:, orders[1]]
        M = bases[0].T @ M @ bases[1]
        outputs.update(left_basis=bases[0], right_basis=bases[1])
    outputs.update(zip(NAMES, (L, R, M, V)))
    return outputs


def _exact_optimizer(case, optimizer, parameters):
    expected, values = {}, []
    step = START + 1
    for p in parameters:
        entry, g = optimizer.state[p], _wide(p.grad)
        if case["kind"] == "embedding":
            Q, P, M, V = (_wide(entry[name]) for name in ("right_basis", "right_preconditioner", "momentum", "variance"))
            rotated = Q.T @ g.T
            M = BETA1 * M + (1 - BETA1) * rotated
            V = BETA2 * V + (1 - BETA2) * rotated * rotated
            bias1, bias2 = 1 - BETA1**step, 1 - BETA2**step
            update = (Q @ ((M / bias1) / ((V / bias2).sqrt() + EPS / math.sqrt(bias2)))).T
            made = dict(right_preconditioner=BETA * P + (1 - BETA) * g.T @ g, momentum=M, variance=V)
        elif p.ndim == 1:
            m = 0.9 * _wide(entry["exp_avg"]) + 0.1 * g
            v = 0.95 * _wide(entry["exp_avg_sq"]) + 0.05 * g * g
            update = (m / (1 - 0.9**step)) / ((v / (1 - 0.95**step)).sqrt() + EPS)
            made = dict(exp_avg=m, exp_avg_sq=v)
        else:
            made = _exact_step(p.grad, entry, step, refreshing=False)
            update = made.pop("update")
        values.append(_wide(p) * (1 - LR * DECAY) - LR * update)
        expected[id(values[-1])] = made
    return _optimizer_outputs(case, values, lambda p: expected[id(p)])


def exact(case, seed):
    state = prepare(case, seed)
    if case["kind"] in ("optimizer", "embedding"):
        return _exact_optimizer(case, state["optimizer"], state["parameters"])
    if case["kind"] == "rotate":
        X, left, right = _wide(state["matrix"]), _wide(state["left"]), _wide(state["right"])
        rotated = left.T @ X @ right
        return dict(rotated=rotated, back=left @ rotated @ right.T)
    return _exact_step(state["gradient"], state["soap"], START + 1, case["kind"] == "refresh")
