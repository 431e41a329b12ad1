"""What the optimizer hands to the native calls when small parameters share launches, with these calls recorded instead of made."""
import pytest
import torch

from soap_tp_b200.engine import kernels as k
from soap_tp_b200.engine import local

SCALARS = dict(beta=0.95, beta1=0.9, beta2=0.95, eps=1e-8)


class Handle:
    """Stands for a native object."""

    def __init__(self, *arguments):
        pass


@pytest.fixture
def groups(monkeypatch):
    """The steps of every shared launch, as `steady_steps` receives them."""
    made = []
    monkeypatch.setattr(local, "_WORKSPACES", {})
    monkeypatch.setattr(local, "_CONTEXTS", type(local._CONTEXTS)())
    for name in ("RotationScratch", "BasisOperands"):
        monkeypatch.setattr(k._C, name, Handle)
    monkeypatch.setattr(k._C, "half_planes", lambda *arguments: None)
    monkeypatch.setattr(k._C, "steady_steps", lambda calls, *tail: made.append(calls))
    monkeypatch.setattr(k, "MIXED_CORRECTIONS", True)
    monkeypatch.setattr(k, "_stream", lambda: 0)
    monkeypatch.setattr(k, "status_word", lambda device: torch.zeros(4, dtype=torch.int32))
    monkeypatch.setattr(local, "_side_stream", lambda device, home: home)
    return made


def _state(rows, cols):
    packed = lambda m, n: torch.zeros(n, m).T
    return dict(left_preconditioner=packed(rows, rows), right_preconditioner=packed(cols, cols), left_basis=packed(rows, rows),
                right_basis=packed(cols, cols), left_work=packed(rows, rows), right_work=packed(cols, cols),
                momentum=packed(rows, cols), variance=packed(rows, cols), step=4)


def _tensors(holder):
    if torch.is_tensor(holder):
        return [holder]
    if isinstance(holder, (list, tuple)):
        return [tensor for each in holder for tensor in _tensors(each)]
    if isinstance(holder, (k.Planes, k.HalfPlanes, local._Scratch)):
        return [tensor for each in vars(holder).values() for tensor in _tensors(each)]
    return []


@pytest.mark.parametrize("shapes", [
    [(64, 64), (160, 64), (64, 160), (64, 64), (160, 64), (64, 160), (160, 160), (64, 32)],
    [(48, 32), (32, 48)] * 4,
    [(16, 8 * i) for i in range(1, 9)],
    [(8 * i, 16) for i in range(1, 9)],
    [(24, 24)] * 8,
])
@pytest.mark.parametrize("dtypes", [(torch.float32,), (torch.float32, torch.bfloat16)])
def test_steps_that_share_launches_write_no_scratch_of_each_other(groups, shapes, dtypes):
    """A decoder layer's matrices have sides in common, and all of them may take the mixed form, which writes their bases too."""
    parameters = [(torch.zeros(shape, dtype=dtypes[i % len(dtypes)]), _state(*shape), *shape) for i, shape in enumerate(shapes)]
    local.shared_steps(parameters, **SCALARS)
    by_handle = {id(entry.native): entry for entry in local._WORKSPACES.values() if isinstance(entry, local._Scratch)}
    group, = groups
    storages = [{tensor.untyped_storage().data_ptr() for tensor in _tensors(by_handle[id(call[0])])} for call in group]
    assert len(storages) == len(shapes) and all(len(mine) > 10 for mine in storages)
    for i, mine in enumerate(storages):
        for theirs in storages[:i]:
            assert mine.isdisjoint(theirs)


@pytest.fixture
def optimizer(groups, monkeypatch):
    """Makes an optimizer whose small matrices share launches, and records which of them are updated."""
    import torch.distributed as dist

    from soap_tp_b200 import optim

    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    applied = []
    monkeypatch.setattr(optim, "_apply", lambda pairs, lr, decay: applied.extend(p for p, _ in pairs))
    monkeypatch.setattr(optim.SoapTP, "_shares_launches", staticmethod(
        lambda p, state, plan, group: local.shares_launches(state, *plan["global_shape"], group["precondition_frequency"])))
    monkeypatch.setattr(k, "poll_status", lambda device: None)

    def make(parameters, **options):
        made = optim.SoapTP(parameters, **options)
        for p in parameters:
            p.grad = torch.zeros_like(p)
            made.state[p] = _state(*p.shape)
        return made

    yield make, applied
    dist.destroy_process_group()


@pytest.mark.parametrize("count,fails", [(20, 1), (20, 2), (9, 1), (20, None)])
def test_updates_are_applied_launch_by_launch(groups, optimizer, monkeypatch, count, fails):
    """No more of them wait than a launch takes, and where a later launch fails every state that has advanced was applied."""
    make, applied = optimizer
    parameters = [torch.nn.Parameter(torch.zeros(16, 24)) for _ in range(count)]
    soap = make(parameters, precondition_frequency=1000)
    waiting = []

    def launch(calls, *tail):
        if len(waiting) == fails:
            raise torch.OutOfMemoryError("out of memory")
        waiting.append(sum(len(group) for group in groups) + len(calls) - len(applied))
        groups.append(calls)

    monkeypatch.setattr(k._C, "steady_steps", launch)
    if fails is None:
        soap.step()
        assert len(applied) == count
    else:
        with pytest.raises(torch.OutOfMemoryError):
            soap.step()
    assert max(waiting) <= k._C.STEP_GROUP
    for p in parameters:
        assert (soap.state[p]["step"] == 5) == any(p is other for other in applied)


def test_as_many_steps_are_collected_as_one_launch_takes():
    from soap_tp_b200 import optim

    assert optim.SHARED_STEPS == k._C.STEP_GROUP


def test_a_parameter_that_a_group_holds_twice(groups, optimizer, monkeypatch):
    """It takes one step after the other: never two in one launch, and the second one is a refresh where its count says so."""
    from soap_tp_b200 import optim

    make, applied = optimizer
    p, q = (torch.nn.Parameter(torch.zeros(16, 24)) for _ in range(2))
    refreshed = []

    def refresh(gradient, state, **options):
        refreshed.append(int(state["step"]) + 1)
        state["step"] += 1
        return torch.zeros(16, 24)

    monkeypatch.setattr(optim, "soap_step", refresh)
    with pytest.warns(UserWarning, match="duplicate"):
        soap = make([p, q, p, q, p], precondition_frequency=7)
    soap.step()
    assert [len(calls) for calls in groups] == [2, 2] and refreshed == [7]
    assert soap.state[p]["step"] == 7 and soap.state[q]["step"] == 6
    assert len(applied) == 5


@pytest.mark.parametrize("interval", [0, -1, -7])
def test_an_interval_that_is_refused_stays_refused(groups, optimizer, interval):
    make, applied = optimizer
    p = torch.nn.Parameter(torch.zeros(16, 24))
    soap = make([p], precondition_frequency=5)
    soap.param_groups[0]["precondition_frequency"] = interval
    with pytest.raises(ValueError, match="must be positive"):
        soap.step()
    assert groups == [] and applied == [] and soap.state[p]["step"] == 4
