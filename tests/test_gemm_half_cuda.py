"""The fp16-pair GEMM and its operand planes against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# Both operands carry at least 22 bits and the sums are rounded to nearest in fp32 every 64 of K, so a product is as far from
# fp64 as an fp32 one: the bound of the tf32 kernels' tests.
BOUND = 2e-6


def _rel(actual, expected):
    return float((actual.double().cpu() - expected).norm() / expected.norm())


def _planes(matrix, turned=False):
    from soap_tp_b200.engine import kernels as k

    rows, cols = matrix.shape
    terms = 1 if matrix.dtype == torch.bfloat16 else 2
    planes = k.HalfPlanes.empty(cols if turned else rows, rows if turned else cols, "cuda", terms=terms)
    k.half_planes(matrix, None if turned else planes, planes if turned else None)
    return planes


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 70), (63, 1), (64, 64), (65, 129), (500, 333), (2049, 130)])
@pytest.mark.parametrize("layout", ["row", "column", "offset", "strided"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_planes_of_every_layout(rows, cols, layout, dtype):
    """Both orientations at once, any strides and alignments: what the planes stand for is the source (22 bits; bf16: all)."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(rows + cols)
    values = torch.randn(rows, cols, generator=g) * torch.logspace(-9, 5, cols)      # columns of very different size
    values = values.to(dtype).cuda()
    if layout == "column":
        values = values.T.contiguous().T
    elif layout == "offset":
        values = torch.cat([torch.zeros(rows, 1, dtype=dtype, device="cuda"), values], dim=1)[:, 1:]
    elif layout == "strided":
        values = values.repeat_interleave(2, dim=0).repeat_interleave(3, dim=1)[::2, ::3]
    terms = 1 if dtype == torch.bfloat16 else 2
    plain = k.HalfPlanes.empty(rows, cols, "cuda", terms=terms)
    turned = k.HalfPlanes.empty(cols, rows, "cuda", terms=terms)
    k.half_planes(values, plain, turned)
    x = values.double()
    # a split keeps 2^-23 of an element or 2^-39 of the largest element of its vector, whichever is more
    for planes, matrix in ((plain, x), (turned, x.T)):
        floor = matrix.abs().amax(dim=0, keepdim=True) * 2.0**-39
        bound = floor if terms == 1 else torch.maximum(matrix.abs() * 2.0**-22, floor)
        assert bool(((planes.dense() - matrix).abs() <= bound).all())


def test_planes_of_extreme_values():
    """Zeros, the smallest and largest magnitudes; an infinity or NaN spoils its own vector only."""
    x = torch.zeros(40, 6, device="cuda")
    x[:, 1] = 3e38
    x[:, 2] = 1e-38
    x[7, 3], x[8, 3] = 65504.0, 1e-3
    x[3, 4], x[3, 5] = float("inf"), float("nan")
    dense = _planes(x).dense()
    assert bool((dense[:, 0] == 0).all())
    for column in (1, 2, 3):
        torch.testing.assert_close(dense[:, column], x[:, column].double(), rtol=2.0**-22,
                                   atol=float(x[:, column].max()) * 2.0**-39)
    assert not bool(torch.isfinite(dense[3, 4:]).any())
    assert bool(torch.isfinite(dense[:, :4]).all())


SHAPES = [(1, 1, 1), (8, 8, 8), (33, 1, 5), (64, 128, 256), (65, 129, 127), (200, 130, 70), (128, 257, 300), (1000, 300, 511),
          (4096, 256, 512)]


@pytest.mark.parametrize("K,M,N", SHAPES)
@pytest.mark.parametrize("tiles", [1, 2])
@pytest.mark.parametrize("terms", [(2, 2), (1, 2), (2, 1), (1, 1)])
def test_products_match_fp64(K, M, N, tiles, terms):
    """Edges of tiles and of K, single CTAs and pairs, one- and two-term operands; padding stays untouched."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(K + M + N)
    a, b = torch.randn(K, M, generator=g) * 1e-3, torch.randn(K, N, generator=g)
    a, b = (t.bfloat16() if n == 1 else t for t, n in zip((a, b), terms))
    expected = 0.5 * (a.double().T @ b.double())
    backing = torch.full((N + 1, M + 3), 7.0, device="cuda")
    out = backing.T[:M, :N]
    ap, bp = _planes(a.cuda()), _planes(b.cuda())
    k.gemm_half(ap, bp, out=out, alpha=0.5, tiles=tiles)
    wide = torch.full((M + 1, N + 1), 7.0, device="cuda")
    k.gemm_half(ap, bp, mode=k.EPI_ROW_MAJOR, out=wide[:M, :N], alpha=0.5, tiles=tiles)
    k.check_status()
    assert _rel(out, expected) < BOUND
    assert torch.equal(wide[:M, :N], out)
    assert bool((backing[:, M:] == 7.0).all()) and bool((backing[N:] == 7.0).all())
    assert bool((wide[M:] == 7.0).all()) and bool((wide[:, N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(7, 9, 5), (130, 70, 260), (300, 257, 129), (511, 300, 500)])
@pytest.mark.parametrize("tiles", [1, 2])
def test_chained_products_and_adam(M, N, K, tiles):
    """Planes written by a product (one scale per 128 rows and column), used as the first operand of the next one, with
    rows whose sizes differ by ten orders: every row of the planes to the rounding of its own size, or to 2^-39 of the largest
    row that shares its scale (rotations whose rows ask for more take the mixed form, tests/test_range_cuda.py); the Adam
    epilogue against fp64."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(M)
    a = torch.randn(K, M, generator=g) * torch.logspace(-6, 4, M)
    b = torch.randn(K, N, generator=g)
    c = torch.randn(M, M, generator=g)
    t = k.HalfPlanes.empty(M, N, "cuda", blocked=True)
    k.gemm_half(_planes(a.cuda()), _planes(b.cuda()), mode=k.EPI_SPLIT, out_planes=t, tiles=tiles)
    expected_t = a.double().T @ b.double()
    assert _rel(t.dense(), expected_t) < BOUND
    error = (t.dense().cpu() - expected_t).norm(dim=1)
    for first in range(0, M, k.HALF_SCALE_BLOCK):
        block = slice(first, min(M, first + k.HALF_SCALE_BLOCK))
        floor = 2.0**-39 * expected_t[block].abs().amax(dim=0).norm()
        assert bool((error[block] <= BOUND * expected_t[block].norm(dim=1) + floor).all())
    cp = _planes(c.cuda())
    moments = [torch.randn(M, N, generator=g), torch.rand(M, N, generator=g) + 0.1]
    m, v = (x.cuda().T.contiguous().T for x in moments)
    y = torch.empty(M, N, device="cuda").T
    k.gemm_half(t, cp, out=y, tiles=tiles)                                      # N x M
    assert _rel(y, expected_t.T @ c.double()) < BOUND
    gp = _planes(b.cuda())
    ap = _planes((a * 1e-2).cuda())
    u = k.HalfPlanes.empty(M, N, "cuda", blocked=True)
    adam = dict(beta1=0.9, beta2=0.99, eps=1e-6, bias_correction1=1 - 0.9**3, bias_correction2=1 - 0.99**3)
    k.gemm_half(ap, gp, mode=k.EPI_ADAM, out_planes=u, momentum=m, variance=v, adam=adam, tiles=tiles)
    k.check_status()
    x = 1e-2 * expected_t
    em = 0.9 * moments[0].double() + 0.1 * x
    ev = 0.99 * moments[1].double() + 0.01 * x * x
    eu = (em / adam["bias_correction1"]) / (ev.sqrt() / adam["bias_correction2"] ** 0.5 + 1e-6)
    assert _rel(m, em) < BOUND and _rel(v, ev) < 3 * BOUND and _rel(u.dense(), eu) < 5 * BOUND


@pytest.mark.parametrize("size", [1, 127, 130, 385, 700])
@pytest.mark.parametrize("tiles", [1, 2])
def test_symmetric_average(size, tiles):
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(size)
    a = torch.randn(300, size, generator=g)
    old = torch.randn(size, size, generator=g)
    old = old + old.T
    out = old.cuda().T.contiguous().T
    ap = _planes(a.cuda())
    k.gemm_half(ap, ap, out=out, alpha=0.1, beta=0.9, symmetric=True, tiles=tiles)
    k.check_status()
    assert _rel(out, 0.9 * old.double() + 0.1 * (a.double().T @ a.double())) < BOUND
    assert torch.equal(out, out.T)


def test_no_further_from_fp64_than_the_tf32_forms():
    """At the benchmark's depth: Gaussian operands, and a first operand whose columns are graded over eight orders."""
    from soap_tp_b200.engine import kernels as k

    for grade in (0, 8):
        g = torch.Generator(device="cuda").manual_seed(3)
        a = torch.randn(8192, 512, generator=g, device="cuda") * torch.logspace(0, -grade, 8192, device="cuda")[:, None]
        b = torch.randn(8192, 512, generator=g, device="cuda")
        expected = (a.double().T @ b.double()).cpu()
        errors = {}
        for name, mixed in (("tf32", False), ("mixed", True)):
            out = torch.empty(512, 512, device="cuda").T
            k.gemm(k.split_planes(a, mixed=mixed), k.split_planes(b, mixed=mixed), out=out)
            errors[name] = _rel(out, expected)
        out = torch.empty(512, 512, device="cuda").T
        k.gemm_half(_planes(a), _planes(b), out=out)
        errors["half"] = _rel(out, expected)
        print(errors)
        assert errors["half"] < 1.05 * min(errors.values())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("symmetric", [False, True])
def test_sums_of_squares_are_no_further_from_fp64_than_in_the_mixed_form(dtype, symmetric):
    """On the diagonal of a Gram product every truncated addition errs to the same side; the mixed form is what these products
    ran on before."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randn(8192, 768, generator=g, device="cuda").to(dtype)
    b = a if symmetric else torch.randn(8192, 768, generator=g, device="cuda").to(dtype)
    expected = (a.double().T @ b.double()).cpu()
    mixed, half = (torch.empty(768, 768, device="cuda").T for _ in range(2))
    am, bm = (k.split_planes(t.float(), mixed=True) for t in (a, b))
    k.gemm(am, bm, out=mixed)
    ap = _planes(a)
    k.gemm_half(ap, ap if symmetric else _planes(b), out=half, symmetric=symmetric)
    k.check_status()
    errors = _rel(half, expected), _rel(mixed, expected)
    print(errors)
    assert errors[0] < 1.05 * errors[1]


@pytest.mark.parametrize("depth", [128, 1000, 8192])
@pytest.mark.parametrize("terms", [(2, 2), (1, 2), (2, 1), (1, 1)])
@pytest.mark.parametrize("kind", ["positive", "itself"])
@pytest.mark.parametrize("tiles", [1, 2])
def test_one_sided_sums_are_no_further_from_fp64_than_in_the_mixed_form(depth, terms, kind, tiles):
    """Plain products whose terms do not cancel, as in a rotation along a leading singular vector: every truncated addition errs
    to the same side.  The whole result where all entries are such sums, the diagonal where the second operand is the first."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator(device="cuda").manual_seed(depth)
    a, b = (torch.randn(depth, 384, generator=g, device="cuda") for _ in range(2))
    if kind == "itself":
        b = a
    else:
        a, b = a.abs(), b.abs()
    a, b = (t.bfloat16() if count == 1 else t for t, count in zip((a, b), terms))
    expected = (a.double().T @ b.double()).cpu()
    mixed, half = (torch.empty(384, 384, device="cuda").T for _ in range(2))
    k.gemm(*(k.split_planes(t.float(), mixed=True) for t in (a, b)), out=mixed)
    k.gemm_half(_planes(a), _planes(b), out=half, tiles=tiles)
    k.check_status()
    if kind == "itself":
        mixed, half, expected = mixed.diagonal(), half.diagonal(), expected.diagonal()
    assert _rel(half, expected) < 1.05 * _rel(mixed, expected)


@pytest.mark.parametrize("size", [130, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_sided_chains_are_no_further_from_fp64_than_in_the_mixed_form(size, dtype):
    """Two products in a row, the first one's result as scaled planes: positive operands, and a rotation of a matrix into its own
    singular vectors."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator(device="cuda").manual_seed(size)
    x, q, w = (torch.rand(size, size, generator=g, device="cuda") + 0.1 for _ in range(3))
    left, _, right = torch.linalg.svd((x - 0.6).double())
    for source, first, second in ((x, q, w), (x - 0.6, left.float(), right.T.float())):
        source = source.to(dtype)
        expected = ((source.double().T @ first.double()).T @ second.double()).cpu()
        middle = k.Planes.empty(size, size, "cuda", mixed=True)
        mixed, half = (torch.empty(size, size, device="cuda").T for _ in range(2))
        k.gemm(k.split_planes(source.float(), mixed=True), k.split_planes(first, mixed=True), mode=k.EPI_SPLIT, out_planes=middle)
        k.gemm(middle, k.split_planes(second, mixed=True), out=mixed)
        middle = k.HalfPlanes.empty(size, size, "cuda", blocked=True)
        k.gemm_half(_planes(source), _planes(first), mode=k.EPI_SPLIT, out_planes=middle)
        k.gemm_half(middle, _planes(second), out=half)
        k.check_status()
        assert _rel(half, expected) < 1.05 * _rel(mixed, expected)


@pytest.mark.parametrize("sizes", [(-60, -60), (-62, -50), (-110, 0), (-75, 25), (25, -75), (60, 58), (100, 20), (20, 100)])
@pytest.mark.parametrize("mode", ["store", "split", "row", "average"])
def test_operands_near_the_limits_of_fp32(sizes, mode):
    """Powers of two on either operand change no bit of a product as long as the result is a normal number."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(6)
    a, b = torch.randn(100, 140, generator=g), torch.randn(100, 150, generator=g)
    plain, scaled = [], []
    for results, (down_a, down_b) in ((plain, (0, 0)), (scaled, sizes)):
        ap, bp = _planes((a * 2.0**down_a).cuda()), _planes((b * 2.0**down_b).cuda())
        if mode == "split":
            out = k.HalfPlanes.empty(140, 150, "cuda", blocked=True)
            k.gemm_half(ap, bp, mode=k.EPI_SPLIT, out_planes=out)
            results.append(out.dense())
        elif mode == "row":
            out = torch.empty(140, 150, device="cuda")
            k.gemm_half(ap, bp, mode=k.EPI_ROW_MAJOR, out=out)
            results.append(out.double())
        elif mode == "store":
            out = torch.empty(150, 140, device="cuda").T
            k.gemm_half(ap, bp, out=out)
            results.append(out.double())
        else:
            out = torch.empty(140, 140, device="cuda").T
            k.gemm_half(ap, ap, out=out, symmetric=True)
            results.append(out.double())
    k.check_status()
    exponent = 2 * sizes[0] if mode == "average" else sum(sizes)
    if not -124 < exponent < 120:
        pytest.skip("the result is not a normal number")
    assert _rel(plain[0], (a.double().T @ (a if mode == "average" else b).double())) < BOUND
    expected = plain[0] * 2.0**exponent
    # entries of a product that fall below the smallest normal number round there
    assert bool((scaled[0] - expected).abs().max() <= 2.0**-148)
    assert _rel(scaled[0], expected.cpu()) < 1e-6


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (64, 61), (65, 130), (130, 333), (257, 1500)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("turned", [False, True])
def test_sources_read_sixteen_bytes_at_a_time(rows, cols, dtype, turned):
    """A ragged matrix in a buffer whose pitch is aligned is read by 16 bytes, its last elements one by one, and nothing past it:
    the same planes as from a copy that is read element by element."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(rows * cols)
    height, width = (cols, rows) if turned else (rows, cols)
    buffer = torch.full((height, -(-width // 16) * 16), float("nan"), dtype=dtype, device="cuda")
    buffer[:, :width] = torch.randn(height, width, generator=g).to(dtype).cuda()
    apart = torch.full((height, 2 * width + 1), float("nan"), dtype=dtype, device="cuda")
    apart[:, 1::2] = buffer[:, :width]
    planes = []
    for source in (buffer[:, :width], apart[:, 1::2]):
        source = source.T if turned else source
        terms = 1 if dtype == torch.bfloat16 else 2
        both = k.HalfPlanes.empty(rows, cols, source.device, terms=terms), k.HalfPlanes.empty(cols, rows, source.device, terms=terms)
        k.half_planes(source, *both)
        planes.append(both)
    for a, b in zip(*planes):
        assert torch.equal(a.dense(), b.dense()) and bool(torch.isfinite(a.dense()).all())
        assert torch.equal(a.scale, b.scale)
