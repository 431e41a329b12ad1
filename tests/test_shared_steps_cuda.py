"""Ordinary steps of several small parameters in shared launches: value for value the steps that each would take alone."""
import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 40), (64, 64), (5, 3), (130, 70), (130, 70), (257, 300), (640, 129), (1025, 64), (130, 70)]


def _state(rows, cols, seed):
    g = torch.Generator().manual_seed(seed)
    packed = lambda m: m.cuda().T.contiguous().T
    basis = lambda n: packed(torch.linalg.qr(torch.randn(n, n, generator=g))[0])
    spd = lambda n: packed(torch.eye(n) + 0.01 * torch.ones(n, n))
    return dict(left_preconditioner=spd(rows), right_preconditioner=spd(cols), left_basis=basis(rows), right_basis=basis(cols),
                left_work=packed(torch.zeros(rows, rows)), right_work=packed(torch.zeros(cols, cols)),
                momentum=packed(torch.randn(rows, cols, generator=g) * 0.1), variance=packed(torch.rand(rows, cols, generator=g) + 0.1),
                step=4)


def _gradient(rows, cols, seed):
    """Types and layouts in turn; every fourth one has rows so far apart that the rotation takes the mixed form."""
    g = torch.Generator().manual_seed(seed)
    grad = torch.randn(rows, cols, generator=g)
    if seed % 4 == 3:
        grad = grad * torch.logspace(0, -6, rows)[:, None]
    grad = grad.cuda()
    return (grad, grad.to(torch.bfloat16), grad.T.contiguous().T, torch.cat([grad, grad], dim=1)[:, 1:cols + 1])[seed % 4]


@pytest.mark.parametrize("count", [1, 8, 10])
@pytest.mark.parametrize("side_stream", [False, True])
def test_shared_launches_give_each_parameters_own_step(count, side_stream):
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    scalars = dict(beta=0.95, beta1=0.9, beta2=0.95, eps=1e-8)
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    results = []
    for together in (False, True):
        states = [_state(*shape, 3 + i) for i, shape in enumerate(SHAPES[:count])]
        steps = [[_gradient(*shape, 10 * turn + i) for i, shape in enumerate(SHAPES[:count])] for turn in range(2)]
        stream.wait_stream(torch.cuda.default_stream())
        updates = []
        with torch.cuda.stream(stream):
            for gradients in steps:
                if together:
                    assert all(local.shares_launches(state, *shape, 1000) for state, shape in zip(states, SHAPES))
                    updates += local.shared_steps([(grad, state, *shape) for grad, state, shape in zip(gradients, states, SHAPES)],
                                                  **scalars)
                else:
                    updates += [local.soap_step(grad, state, global_shape=shape, interval=1000, implementation="householder",
                                                initializing=False, **scalars)
                                for grad, state, shape in zip(gradients, states, SHAPES)]
        torch.cuda.synchronize()
        results.append((updates, states))
    k.check_status()
    (alone, alone_states), (shared, shared_states) = results
    for a, b in zip(alone, shared):
        assert torch.equal(a, b) and bool(torch.isfinite(a).all())
    for a, b in zip(alone_states, shared_states):
        for name in ("left_preconditioner", "right_preconditioner", "momentum", "variance", "step"):
            assert torch.equal(a[name], b[name]) if torch.is_tensor(a[name]) else a[name] == b[name]


def test_which_steps_share_launches():
    """Not the first one, not one with a refresh, not where a product runs on CTA pairs."""
    from soap_tp_b200.engine import local

    state = dict(left_basis=None, step=8)
    assert local.shares_launches(state, 512, 1376, 10)
    assert not local.shares_launches(dict(left_basis=None, step=9), 512, 1376, 10)
    assert not local.shares_launches({}, 512, 1376, 10)
    assert not local.shares_launches(state, 4096, 4096, 10)
    assert not local.shares_launches(state, 0, 64, 10)


def test_optimizer_steps_small_matrices_together():
    """Seven matrices (two shapes twice) and a vector: state, parameters and step counts as with one optimizer per parameter."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.optim import SoapTP

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    shapes = [(96, 96), (24, 96), (24, 96), (200, 96), (200, 96), (96, 200), (96,)]

    def make():
        g = torch.Generator().manual_seed(0)
        parameters = [torch.nn.Parameter(torch.randn(shape, generator=g).cuda()) for shape in shapes]
        for p in parameters:
            if p.ndim == 2:
                p.tp_shard_dim, p.tp_global_shape = 0, tuple(p.shape)
        return parameters

    together, alone = make(), make()
    options = dict(lr=1e-2, precondition_frequency=3)
    optimizers = [SoapTP(together, **options)], [SoapTP([p], **options) for p in alone]
    before = dict(k.LAUNCH_COUNTS)
    for step in range(6):
        g = torch.Generator().manual_seed(100 + step)
        grads = [torch.randn(shape, generator=g).cuda() for shape in shapes]
        for parameters, some in zip((together, alone), optimizers):
            for p, grad in zip(parameters, grads):
                p.grad = grad
            for optimizer in some:
                optimizer.step()
    torch.cuda.synchronize()
    k.check_status()
    assert k.LAUNCH_COUNTS["apply_updates_kernel"] > before.get("apply_updates_kernel", 0)
    for p, q, own in zip(together, alone, optimizers[1]):
        assert torch.equal(p, q)
        mine, its = optimizers[0][0].state[p], own.state[q]
        assert mine.keys() == its.keys()
        for name in mine:
            assert torch.equal(mine[name], its[name]) if torch.is_tensor(mine[name]) else mine[name] == its[name], name


def _assert_shared_equals_alone(shapes, gradients):
    """Two steps of every parameter, together and one after another; returns the scratch of the shared ones."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    scalars = dict(beta=0.95, beta1=0.9, beta2=0.95, eps=1e-8)
    results = []
    for together in (False, True):
        local.release_workspaces()
        states = [_state(*shape, 3 + i) for i, shape in enumerate(shapes)]
        updates = []
        for turn in range(2):
            grads = [gradients(i, turn) for i in range(len(shapes))]
            if together:
                updates += local.shared_steps([(grad, state, *shape) for grad, state, shape in zip(grads, states, shapes)], **scalars)
            else:
                updates += [local.soap_step(grad, state, global_shape=shape, interval=1000, implementation="householder",
                                            initializing=False, **scalars) for grad, state, shape in zip(grads, states, shapes)]
        torch.cuda.synchronize()
        results.append(updates + [state[name] for state in states for name in local._WRITTEN])
    k.check_status()
    for a, b in zip(*results):
        assert torch.equal(a.nan_to_num(nan=123.0), b.nan_to_num(nan=123.0))
    return [entry for entry in local._WORKSPACES.values() if isinstance(entry, local._Scratch)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("spread", ["graded", "zero row", "zero column"])
def test_steps_in_the_mixed_form_that_have_sides_in_common(dtype, spread):
    """Every one of them converts its own bases, also where another one of the same size is converted in the same launch."""
    shapes = [(64, 64), (160, 64), (64, 160), (64, 64), (160, 64), (192, 192), (64, 192), (192, 64)]

    def gradient(i, turn):
        rows, cols = shapes[i]
        grad = torch.randn(rows, cols, generator=torch.Generator().manual_seed(20 * turn + i))
        if spread == "graded":
            grad *= torch.logspace(0, -6, rows)[:, None]
        elif spread == "zero row":
            grad[rows // 2] = 0.0
        else:
            grad[:, cols // 3] = 0.0
        return grad.to(dtype).cuda()

    scratches = _assert_shared_equals_alone(shapes, gradient)
    assert len(scratches) == len(shapes) and all(int(scratch.wide) == 1 for scratch in scratches)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_gradient_that_is_not_finite_among_others(value, dtype):
    """Its own step is what it would be alone, and so are the others'."""
    shapes = [(64, 64), (160, 64), (130, 70), (64, 160)]

    def gradient(i, turn):
        grad = torch.randn(*shapes[i], generator=torch.Generator().manual_seed(20 * turn + i))
        if i == 1:
            grad[3, 4] = value
        return grad.to(dtype).cuda()

    scratches = _assert_shared_equals_alone(shapes, gradient)
    assert sorted(int(scratch.wide) for scratch in scratches) == [0, 0, 0, 1]
