"""The natively issued ordinary step against the same step composed launch by launch: the same kernels on the same operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _state(rows, cols, seed):
    g = torch.Generator().manual_seed(seed)
    packed = lambda m: m.cuda().T.contiguous().T
    basis = lambda n: packed(torch.linalg.qr(torch.randn(n, n, generator=g))[0])
    spd = lambda n: packed(torch.eye(n) + 0.01 * torch.ones(n, n))
    return dict(left_preconditioner=spd(rows), right_preconditioner=spd(cols), left_basis=basis(rows), right_basis=basis(cols),
                left_work=packed(torch.zeros(rows, rows)), right_work=packed(torch.zeros(cols, cols)),
                momentum=packed(torch.randn(rows, cols, generator=g) * 0.1), variance=packed(torch.rand(rows, cols, generator=g) + 0.1),
                step=4)


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 40), (5, 3), (130, 70), (257, 300), (640, 129)])
@pytest.mark.parametrize("kind", ["fp32", "bf16", "fp16", "turned", "offset"])
@pytest.mark.parametrize("side_stream", [False, True])
def test_native_step_is_the_composed_one(rows, cols, kind, side_stream, monkeypatch):
    from soap_tp_b200.engine import kernels as k
    from soap_tp_b200.engine import local

    g = torch.Generator().manual_seed(9)
    options = dict(global_shape=(rows, cols), beta=0.95, beta1=0.9, beta2=0.95, eps=1e-8, interval=1000,
                   implementation="householder", initializing=False)
    results = []
    gradients = []
    for _ in range(2):
        grad = torch.randn(rows, cols, generator=g).cuda()
        if kind in ("bf16", "fp16"):
            grad = grad.to(torch.bfloat16 if kind == "bf16" else torch.float16)
        elif kind == "turned":
            grad = grad.T.contiguous().T
        elif kind == "offset":
            grad = torch.cat([grad, grad], dim=1)[:, 1:cols + 1]
        gradients.append(grad)
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for composed in (False, True):
            monkeypatch.setattr(local.TIMER, "enabled", composed)
            state = _state(rows, cols, 3)
            stream.wait_stream(torch.cuda.default_stream())
            updates = [local.soap_step(grad, state, **options) for grad in gradients]
            results.append((updates, state))
    monkeypatch.setattr(local.TIMER, "enabled", False)
    torch.cuda.synchronize()
    k.check_status()
    (native, native_state), (composed, composed_state) = results
    for a, b in zip(native, composed):
        assert torch.equal(a, b) and bool(torch.isfinite(a).all())
    for name in ("left_preconditioner", "right_preconditioner", "momentum", "variance", "step"):
        a, b = native_state[name], composed_state[name]
        assert torch.equal(a, b) if torch.is_tensor(a) else a == b
