"""Averages that bases are derived from: the public op and the engine form the same ones, bit for bit, so that a step composed
from the ops (tracing, injected bindings) derives the bases that the engine's own step derives."""
import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu
BLOCK, GRID = 128, (1, 1)


@pytest.fixture
def one_rank():
    started = not dist.is_initialized()
    if started:
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    yield
    if started:
        dist.destroy_process_group()


@pytest.mark.parametrize("rows,cols", [(5, 3), (130, 70), (257, 300)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_op_forms_the_engines_averages(one_rank, rows, cols, dtype):
    from soap_tp_b200 import ops, soap_step

    g = torch.Generator().manual_seed(rows)
    gradients = [torch.randn(rows, cols, generator=g).to(dtype).cuda() for _ in range(2)]
    state, averages = {}, [torch.zeros(n, n, device="cuda").T for n in (rows, cols)]
    updates = (ops.update_left_preconditioner_2d_block_cyclic_, ops.update_right_preconditioner_2d_block_cyclic_)
    for grad in gradients:                            # the first call and a refresh step
        soap_step(grad, state, global_shape=(rows, cols), shard_dim=0, block_size=BLOCK, process_grid_shape=GRID,
                  preconditioner_beta=0.9, basis_refresh_interval=1, basis_implementation="householder")
        for average, update in zip(averages, updates):
            update(grad, average, 0.9, BLOCK, GRID, shard_dim=0)
        assert torch.equal(averages[0], state["left_preconditioner"][:rows, :rows])
        assert torch.equal(averages[1], state["right_preconditioner"][:cols, :cols])
