"""Matrices whose rows or columns differ in size by many orders: their rotations keep as many bits of the small ones as the mixed
form (tf32 values with bf16 corrections) does, row by row and column by column."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _packed(matrix):
    return matrix.float().cuda().T.contiguous().T


def _spread(count, orders, kind):
    """Sizes over `orders` decimal orders: evenly, or one group of small ones among ordinary ones, or some exactly zero."""
    if kind == "even":
        return torch.logspace(0, -orders, count, dtype=torch.float64)
    sizes = torch.ones(count, dtype=torch.float64)
    sizes[count // 3: count // 2] = 0.0 if kind == "zero" else 10.0**-orders
    return sizes


def _gradient(rows, cols, orders, kind, side, seed):
    g = torch.Generator().manual_seed(seed)
    matrix = torch.randn(rows, cols, generator=g, dtype=torch.float64)
    if side in ("rows", "both"):
        matrix *= _spread(rows, orders, kind)[:, None]
    if side in ("columns", "both"):
        matrix *= _spread(cols, orders, kind)
    return matrix


def _bases(gradient, seed):
    """What the preconditioners' eigenbases are for such gradients: nearly aligned with the small rows and columns."""
    left, _, right = torch.linalg.svd(gradient, full_matrices=True)
    return left.float(), right.T.float()


def _mixed_rotation(source, first, second):
    """(source^T first)^T second on mixed planes: the form that pairs replaced."""
    from soap_tp_b200.engine import kernels as k

    planes = lambda m: k.split_planes(m, mixed=True)
    middle = k.Planes.empty(source.shape[1], first.shape[1], "cuda", mixed=True)
    k.gemm(planes(source), planes(first), mode=k.EPI_SPLIT, out_planes=middle)
    out = torch.empty(second.shape[1], first.shape[1], device="cuda").T
    k.gemm(middle, planes(second), out=out)
    return out


def _worst(actual, expected, gradient, left, right):
    """Largest error of a row and of a column of Q_l^T G Q_r, relative to what enters it: the lengths of G's rows (columns) times
    the basis vector's entries, whose rounding no fp32 sum is free of."""
    error = actual.double().cpu() - expected
    rows = (left.double().square().T @ gradient.square().sum(dim=1)).sqrt()
    columns = (right.double().square().T @ gradient.square().sum(dim=0)).sqrt()
    worst = lambda lengths, sizes: float((lengths / sizes.clamp_min(1e-300)).max())
    return worst(error.norm(dim=1), rows), worst(error.norm(dim=0), columns)


CASES = [(orders, kind, side) for orders in (3, 6, 8, 10) for kind in ("even", "group") for side in ("rows", "columns", "both")]
CASES += [(0, "zero", side) for side in ("rows", "columns", "both")]


@pytest.mark.parametrize("rows,cols", [(130, 70), (256, 300)])
@pytest.mark.parametrize("orders,kind,side", CASES)
def test_rotated_gradient_row_by_row_and_column_by_column(rows, cols, orders, kind, side):
    """Momentum with beta1 = 0 is the rotated gradient itself."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    gradient = _gradient(rows, cols, orders, kind, side, seed=rows)
    left, right = _bases(gradient, seed=1)
    g = gradient.float()
    expected = left.double().T @ g.double() @ right.double()
    state = dict(left_preconditioner=_packed(torch.eye(rows)), right_preconditioner=_packed(torch.eye(cols)),
                 left_basis=_packed(left), right_basis=_packed(right), momentum=_packed(torch.zeros(rows, cols)),
                 variance=_packed(torch.ones(rows, cols)), step=3)
    update = local.soap_step(g.cuda(), state, global_shape=(rows, cols), beta=0.9, beta1=0.0, beta2=0.0, eps=1e-30, interval=1000,
                             implementation="householder", initializing=False)
    mixed = _mixed_rotation(g.cuda(), left.cuda(), right.cuda())
    k.check_status()
    worst, bound = (_worst(result, expected, g.double(), left, right) for result in (state["momentum"], mixed))
    assert worst[0] <= 1.05 * bound[0] and worst[1] <= 1.05 * bound[1], (worst, bound)
    assert bool(torch.isfinite(update).all())


@pytest.mark.parametrize("orders,kind,side", [(8, "even", "columns"), (10, "group", "both"), (0, "zero", "rows")])
@pytest.mark.parametrize("rows,cols", [(1, 40), (130, 70), (600, 520), (2304, 2560)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_wide_matrices_take_the_mixed_form_bit_for_bit(orders, kind, side, rows, cols, dtype):
    """Adam's moments and the update of a step, and the public rotation, against the tf32 kernel on the same operands."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    if rows == 1 and side == "rows":
        pytest.skip("a single row has no other beside it")
    g = torch.Generator(device="cuda").manual_seed(rows)
    grad = _gradient(rows, cols, orders, kind, side, seed=2).to(dtype).cuda()
    left, right = (torch.linalg.qr(torch.randn(n, n, generator=g, device="cuda"))[0].T.contiguous().T for n in (rows, cols))
    momentum, variance = (torch.rand(cols, rows, generator=g, device="cuda").T + 0.1 for _ in range(2))
    adam = dict(beta1=0.9, beta2=0.95, eps=1e-8 / (1 - 0.95**4) ** 0.5, bias_correction1=1 - 0.9**4, bias_correction2=1 - 0.95**4)
    m, v = (t.clone(memory_format=torch.preserve_format) for t in (momentum, variance))
    planes = lambda x, turned=False: k.split_planes(x.float(), transpose=turned, mixed=True)
    mixed = lambda depth, width: k.Planes.empty(depth, width, "cuda", mixed=True)
    middle, u = mixed(cols, rows), mixed(rows, cols)
    expected = torch.empty(rows, cols, device="cuda")
    k.gemm(planes(grad), planes(left), mode=k.EPI_SPLIT, out_planes=middle)
    k.gemm(middle, planes(right), mode=k.EPI_ADAM, out_planes=u, momentum=m, variance=v, adam=adam)
    k.gemm(u, planes(left, True), mode=k.EPI_SPLIT, out_planes=middle)
    k.gemm(middle, planes(right, True), mode=k.EPI_ROW_MAJOR, out=expected)

    state = dict(left_preconditioner=_packed(torch.eye(rows)), right_preconditioner=_packed(torch.eye(cols)), left_basis=left,
                 right_basis=right, momentum=momentum, variance=variance, step=3)
    options = dict(global_shape=(rows, cols), beta=0.9, beta1=0.9, beta2=0.95, eps=1e-8, interval=1000,
                   implementation="householder", initializing=False)
    update = local.soap_step(grad, state, **options)
    k.check_status()
    assert torch.equal(state["momentum"], m) and torch.equal(state["variance"], v) and torch.equal(update, expected)

    # an ordinary gradient after a wide one, on the same scratch, and back
    ordinary = torch.randn(rows, cols, generator=g, device="cuda")
    for source in (ordinary, grad.float()):
        for direction in ("forward", "backward"):
            out = source.T.clone(memory_format=torch.contiguous_format).T
            local.rotate(out, left, right, (rows, cols), direction)
            turned = direction == "backward"
            double = [q.double().T if not turned else q.double() for q in (left, right)]
            wanted = (double[0] @ source.double() @ double[1].T).cpu()
            assert float((out.double().cpu() - wanted).norm()) <= 2e-6 * float(wanted.norm())
            if source is not ordinary:
                again = _mixed_rotation(source, *((q.T.contiguous().T if not turned else q.T) for q in (left, right)))
                assert torch.equal(out, again)
    k.check_status()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_infinities_and_nan_stay_in_their_rows_and_columns(value):
    """An infinite or undefined entry reaches the averages of its own row and column and the rotated gradient, nothing else."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    g = torch.Generator().manual_seed(0)
    grad = torch.randn(60, 50, generator=g)
    grad[7, 9] = value
    state = dict(left_preconditioner=_packed(torch.eye(60)), right_preconditioner=_packed(torch.eye(50)),
                 left_basis=_packed(torch.eye(60)), right_basis=_packed(torch.eye(50)), momentum=_packed(torch.zeros(60, 50)),
                 variance=_packed(torch.ones(60, 50)), step=3)
    local.soap_step(grad.cuda(), state, global_shape=(60, 50), beta=0.9, beta1=0.9, beta2=0.95, eps=1e-8, interval=1000,
                    implementation="householder", initializing=False)
    k.check_status()
    finite = torch.isfinite(state["left_preconditioner"]).cpu()
    expected = torch.ones(60, 60, dtype=torch.bool)
    expected[7] = expected[:, 7] = False
    assert torch.equal(finite, expected)
    assert not bool(torch.isfinite(state["momentum"])[7, 9])


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 65), (64, 64), (300, 1000), (5000, 130)])
@pytest.mark.parametrize("layout", ["row", "column"])
def test_the_decision(rows, cols, layout):
    """At the line (2^12 between the largest magnitudes), for zero rows, zero matrices, infinities, and again after each other."""
    from soap_tp_b200.engine import local

    base = torch.full((rows, cols), 1.0, device="cuda")
    inputs = [(base, 0), (base * 0, 0), (base * 1e-30, 0), (base * float("inf"), 1)]
    if rows > 1:
        for factor, wide in ((2.0**-12, 0), (2.0**-13, 1), (0.0, 1)):
            matrix = base.clone()
            matrix[rows // 2] *= factor
            inputs.append((matrix, wide))
    if cols > 1:
        for factor, wide in ((2.0**-12, 0), (2.0**-13, 1), (0.0, 1)):
            matrix = base.clone()
            matrix[:, cols - 1] *= factor
            inputs.append((matrix, wide))
    left, right = local.BasisPlanes(), local.BasisPlanes()
    bases = [torch.eye(n, device="cuda") for n in (rows, cols)]
    left.refresh(bases[0], rows)
    right.refresh(bases[1], cols)
    out = torch.empty(cols, rows, device="cuda").T
    for matrix, wide in inputs + inputs[::-1]:
        source = matrix if layout == "row" else matrix.T.contiguous().T
        local.rotate_matrix(source, left, right, False, out)
        scratch = local._scratch(rows, cols, out.device, 2)
        assert scratch.wide.tolist() == [wide]


@pytest.mark.parametrize("dtype", [torch.float64, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("orders", [0, 9])
def test_bases_of_other_types_are_read_as_what_they_hold(dtype, orders):
    """Also where the rotation reads the basis itself, for its mixed form."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    g = torch.Generator().manual_seed(5)
    matrix = _gradient(150, 90, orders, "even", "rows", seed=8).float()
    bases = [torch.linalg.qr(torch.randn(n, n, generator=g))[0].to(dtype) for n in (150, 90)]
    results = []
    for held in (bases, [b.float() for b in bases]):
        out = _packed(matrix)
        local.rotate(out, held[0].cuda().T.contiguous().T, held[1].cuda().T.contiguous().T, (150, 90), "forward")
        results.append(out)
    k.check_status()
    assert torch.equal(*results)
    expected = bases[0].double().T @ matrix.double() @ bases[1].double()
    assert float((results[0].double().cpu() - expected).norm()) <= 2e-6 * float(expected.norm())
