"""A refresh whose launches are all issued while the device is still busy with something else."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(384, 256), (1024, 1100)])
def test_refreshes_issued_far_ahead_of_the_device(rows, cols):
    """The waits between the thread blocks of a panel are bounded in device time: none may run out because launches queued up
    behind one another, and the results are those of refreshes that the host waited for."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    g = torch.Generator().manual_seed(rows)
    gradients = [torch.randn(rows, cols, generator=g).cuda() for _ in range(4)]
    options = dict(global_shape=(rows, cols), beta=0.9, beta1=0.9, beta2=0.95, eps=1e-8, interval=1, implementation="householder")
    filler = torch.randn(8192, 8192, device="cuda")
    results = []
    for ahead in (False, True):
        packed = lambda m, n: torch.zeros(n, m, device="cuda").T
        state = dict(left_preconditioner=packed(rows, rows), right_preconditioner=packed(cols, cols), left_basis=packed(rows, rows),
                     right_basis=packed(cols, cols), left_work=packed(rows, rows), right_work=packed(cols, cols),
                     momentum=packed(rows, cols), variance=packed(rows, cols))
        local.soap_step(gradients[0], state, initializing=True, **options)
        torch.cuda.synchronize()
        if ahead:
            for _ in range(6):
                filler @ filler                      # some 100 ms of fp32 products: the host is done long before them
        for gradient in gradients[1:]:
            update = local.soap_step(gradient, state, initializing=False, **options)
            if not ahead:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        k.check_status()
        results.append((update, state))
    assert torch.equal(results[0][0], results[1][0])
    for name in ("left_basis", "right_basis", "momentum", "variance"):
        assert torch.equal(results[0][1][name], results[1][1][name])


@pytest.mark.parametrize("rows,cols", [(100, 100), (384, 256), (257, 640), (1024, 1100)])
@pytest.mark.parametrize("graded", [False, True])
@pytest.mark.parametrize("side_stream", [False, True])
def test_update_beside_the_factorisations(rows, cols, graded, side_stream, monkeypatch):
    """The step's update and the momentum's way out of the old bases run beside the factorisations, or before them (as with stage
    timers): the same values, also where the rotations read the old bases themselves (rows far apart: the mixed form)."""
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    g = torch.Generator().manual_seed(rows + cols)
    gradients = [torch.randn(rows, cols, generator=g).cuda() for _ in range(3)]
    if graded:
        gradients = [gradient * torch.logspace(0, -6, rows, device="cuda")[:, None] for gradient in gradients]
    options = dict(global_shape=(rows, cols), beta=0.9, beta1=0.9, beta2=0.95, eps=1e-8, interval=1, implementation="householder")
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    results = []
    for apart in (False, True):
        packed = lambda m, n: torch.zeros(n, m, device="cuda").T
        state = dict(left_preconditioner=packed(rows, rows), right_preconditioner=packed(cols, cols), left_basis=packed(rows, rows),
                     right_basis=packed(cols, cols), left_work=packed(rows, rows), right_work=packed(cols, cols),
                     momentum=packed(rows, cols), variance=packed(rows, cols))
        stream.wait_stream(torch.cuda.default_stream())
        with torch.cuda.stream(stream):
            local.soap_step(gradients[0], state, initializing=True, **options)
            monkeypatch.setattr(local.TIMER, "enabled", apart)
            updates = [local.soap_step(gradient, state, initializing=False, **options) for gradient in gradients[1:]]
            monkeypatch.setattr(local.TIMER, "enabled", False)
        torch.cuda.synchronize()
        k.check_status()
        results.append((updates, state))
    for a, b in zip(results[0][0], results[1][0]):
        assert torch.equal(a, b)
    for name in ("left_preconditioner", "left_basis", "right_basis", "momentum", "variance"):
        assert torch.equal(results[0][1][name], results[1][1][name])
