"""Operand planes of the tf32 forms: every layout, type and window, in one or both orientations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tf32(x):
    """Round to nearest (ties away) to 11 significant bits, as the planes' high part is."""
    bits = x.view(torch.int32)
    return ((bits + 0x1000) & ~0x1FFF).view(torch.float32)


def _layout(values, layout):
    rows, cols = values.shape
    if layout == "column":
        return values.T.contiguous().T
    if layout == "offset":
        return torch.cat([torch.zeros(rows, 1, dtype=values.dtype, device="cuda"), values], dim=1)[:, 1:]
    if layout == "strided":
        return values.repeat_interleave(2, dim=0).repeat_interleave(3, dim=1)[::2, ::3]
    return values


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 70), (63, 1), (64, 64), (65, 129), (330, 257)])
@pytest.mark.parametrize("layout", ["row", "column", "offset", "strided"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mixed", [False, True])
def test_both_orientations_are_exact(rows, cols, layout, dtype, mixed):
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(rows + cols)
    x = _layout(torch.randn(rows, cols, generator=g).to(dtype).cuda(), layout)
    plain, turned = k.Planes.empty(rows, cols, "cuda", mixed=mixed), k.Planes.empty(cols, rows, "cuda", mixed=mixed)
    k.split_planes_both(x, plain, turned)
    single = k.split_planes(x, transpose=True, mixed=mixed)
    for planes, matrix in ((plain, x.float()), (turned, x.float().T), (single, x.float().T)):
        high = _tf32(matrix.contiguous())
        assert torch.equal(planes.hi[: planes.cols, : planes.depth].T, high)
        if mixed:
            hb, lb = planes.halves()
            assert torch.equal(hb.T, matrix.bfloat16().float()) and torch.equal(lb.T, (matrix - high).bfloat16().float())
            tail = planes.hl.view(max(1, planes.cols), -1, 2, 32).permute(0, 2, 1, 3).reshape(max(1, planes.cols), 2, -1)
            assert bool((tail[:, :, planes.depth:] == 0).all())          # the products rely on zeros past the depth
        else:
            assert torch.equal(planes.lo[: planes.cols, : planes.depth].T, matrix - high)


@pytest.mark.parametrize("depth,cols", [(1, 3), (7, 5), (63, 64), (64, 65), (129, 2)])
def test_windows_leave_their_surroundings_alone(depth, cols):
    from soap_tp_b200.engine import kernels as k

    whole = k.Planes.empty(200, 80, "cuda")
    whole.hi.fill_(7.0), whole.lo.fill_(7.0)
    x = torch.randn(depth, cols, device="cuda")
    k.split_planes(x, out=whole.sub(4, 3, depth, cols))
    inside = torch.zeros(80, 200, dtype=torch.bool, device="cuda")
    inside[3:3 + cols, 4:4 + depth] = True
    for plane in (whole.hi, whole.lo):
        assert bool((plane[:, :200][~inside] == 7.0).all())
    assert torch.equal((whole.hi + whole.lo)[3:3 + cols, 4:4 + depth], x.T)
