"""State buffers that the single-GPU kernels cannot write through their addresses are refused before anything is launched."""
import pytest
import torch

from soap_tp_b200.engine import local

ROWS, COLS = 6, 4


def _state():
    packed = lambda m, n: torch.zeros(n, m).T
    return dict(left_preconditioner=packed(ROWS, ROWS), right_preconditioner=packed(COLS, COLS), left_basis=packed(ROWS, ROWS),
                right_basis=packed(COLS, COLS), left_work=packed(ROWS, ROWS), right_work=packed(COLS, COLS),
                momentum=packed(ROWS, COLS), variance=packed(ROWS, COLS), step=1)


def _step(state, interval=1000):
    return local.soap_step(torch.zeros(ROWS, COLS), state, global_shape=(ROWS, COLS), beta=0.9, beta1=0.9, beta2=0.9, eps=1e-8,
                           interval=interval, implementation="householder", initializing=False)


@pytest.mark.parametrize("name", ["momentum", "variance", "left_preconditioner", "right_preconditioner"])
@pytest.mark.parametrize("spoil,what", [
    (lambda t: t.contiguous(), "column-major"), (lambda t: t.bfloat16(), "float32"), (lambda t: t.double(), "float32"),
    (lambda t: t[:-1], "smaller"), (lambda t: t[:, :-1], "smaller"), (lambda t: t.flatten(), "shape"),
    (lambda t: t[:1].expand(t.shape), "column-major"),
])
@pytest.mark.parametrize("interval", [1, 1000])
def test_other_buffers_are_refused(name, spoil, what, interval):
    state = _state()
    state[name] = spoil(state[name])
    with pytest.raises(ValueError, match=f"{name}.*{what}|{what}.*{name}"):
        _step(state, interval)
    assert state["step"] == 1


def test_buffers_with_padding_are_taken():
    state = _state()
    state["momentum"] = torch.zeros(COLS + 2, ROWS + 3).T[:ROWS, :COLS]
    local._check_state(state, ROWS, COLS)
    local._check_state(dict(state, momentum=torch.zeros(COLS + 2, ROWS + 3).T), ROWS, COLS)


@pytest.mark.parametrize("rows,cols", [(1, 5), (5, 1), (1, 1)])
def test_vectors_have_no_order(rows, cols):
    state = {name: torch.zeros(m, n) for name, m, n in (("momentum", rows, cols), ("variance", rows, cols),
                                                        ("left_preconditioner", rows, rows), ("right_preconditioner", cols, cols))}
    if max(rows, cols) > 1:
        name = "left_preconditioner" if rows > 1 else "right_preconditioner"
        state[name] = state[name].T.contiguous().T
    local._check_state(state, rows, cols)
