"""Parameter updates in one pass against the tensor operations that they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1,), (7,), (512,), (3, 5), (64, 130), (1025, 33)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("decay", [0.0, 0.01])
@pytest.mark.parametrize("offset", [0, 1])
def test_apply_is_value_for_value_the_tensor_operations(shape, dtype, decay, offset):
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(sum(shape))
    count = int(torch.tensor(shape).prod())
    values = (torch.randn(count + offset, generator=g) * 0.02).to(dtype).cuda()
    p = values[offset:].view(shape)
    update = torch.randn(count + offset, generator=g).cuda()[offset:].view(shape)
    expected = p.clone()
    if decay:
        expected.mul_(1.0 - 3e-3 * decay)
    expected.add_(update.to(dtype), alpha=-3e-3)
    version = p._version
    assert k.apply_update(p, update, 1.0 - 3e-3 * decay, 3e-3)
    assert torch.equal(p, expected) and p._version > version


def test_apply_leaves_other_tensors_to_the_caller():
    from soap_tp_b200.engine import kernels as k

    p = torch.ones(4, 6, device="cuda")
    assert not k.apply_update(p.double(), torch.ones(4, 6, device="cuda"), 1.0, 0.1)
    assert not k.apply_update(p, torch.ones(6, 4, device="cuda").T, 1.0, 0.1)
    assert not k.apply_update(p[:, ::2], torch.ones(4, 3, device="cuda"), 1.0, 0.1)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_adamw_matches_fp64(shape, dtype):
    """A few fp32 roundings in each of m, v and the update; bf16 parameters round once or twice more (2^-8 each)."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(1)
    p = (torch.randn(shape, generator=g) * 0.02).to(dtype).cuda()
    grad = torch.randn(shape, generator=g).to(dtype).cuda()
    m, v = torch.randn(shape, generator=g).cuda() * 0.1, torch.rand(shape, generator=g).cuda() + 0.1
    em = 0.9 * m.double() + 0.1 * grad.double()
    ev = 0.95 * v.double() + 0.05 * grad.double() ** 2
    bias1, bias2, keep, lr = 1 - 0.9**3, 1 - 0.95**3, 1 - 3e-5, 3e-3
    ep = p.double() * keep - lr * (em / bias1) / ((ev / bias2).sqrt() + 1e-8)
    assert k.adamw_update(p, grad, m, v, 0.9, 0.95, bias1, bias2, 1e-8, keep, lr)
    torch.testing.assert_close(m.double(), em, rtol=1e-6, atol=1e-7)
    torch.testing.assert_close(v.double(), ev, rtol=1e-6, atol=1e-7)
    bound = dict(rtol=2e-6, atol=1e-8) if dtype == torch.float32 else dict(rtol=2.0**-7, atol=lr * 2.0**-6)
    torch.testing.assert_close(p.double(), ep, **bound)


@pytest.mark.parametrize("beta1", [0.0, 0.3, 0.5, 0.9])
def test_adamw_average_is_lerp_for_every_beta(beta1):
    """Also where the old average is far above the gradient: beta1 = 0 leaves the gradient itself."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(2)
    grad = torch.randn(1000, generator=g).cuda()
    m = (torch.randn(1000, generator=g) * torch.logspace(-3, 9, 1000)).cuda()
    p, v = torch.zeros(1000, device="cuda"), torch.ones(1000, device="cuda")
    expected = m.clone().lerp_(grad, 1.0 - beta1)
    assert k.adamw_update(p, grad, m, v, beta1, 0.95, 1.0, 1.0, 1e-8, 1.0, 0.1)
    assert torch.equal(m, expected)
    if beta1 == 0.0:
        assert torch.equal(m, grad)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("count", [2, 16, 17])
def test_apply_several_at_once(dtype, count):
    """More parameters than a launch takes, aligned and not, empty ones, and two that share memory (one after the other)."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(count)
    flat = torch.randn(40000, generator=g).to(dtype).cuda()
    sizes = [0, 1, 5, 512, 1025, 3000][:count] + [777] * max(0, count - 6)
    starts = [sum(sizes[:i]) for i in range(count)]
    parameters = [flat[a:a + n] for a, n in zip(starts, sizes)] + [flat[100:900]]
    pairs = [(p, torch.randn(p.numel(), generator=g).cuda()) for p in parameters]
    expected = flat.clone()
    for (a, n), (_, update) in zip(list(zip(starts, sizes)) + [(100, 800)], pairs):
        expected[a:a + n].mul_(0.99).add_(update.to(dtype), alpha=-3e-3)
    assert k.apply_updates(pairs, 0.99, 3e-3) == []
    assert torch.equal(flat, expected)


def test_what_a_shared_update_does_not_take_comes_back_untouched():
    """Parameters of both types and tensors that the kernel does not take, mixed: exactly these are returned."""
    from soap_tp_b200.engine import kernels as k

    g = torch.Generator().manual_seed(2)
    values = lambda *shape: torch.randn(*shape, generator=g).cuda()
    taken = [(values(*shape).to(dtype), values(*shape)) for shape in ((7, 5), (33,), (64, 130)) for dtype in (torch.float32, torch.bfloat16)]
    refused = [(values(4, 6).double(), values(4, 6)), (values(4, 6), values(6, 4).T), (values(4, 6)[:, ::2], values(4, 3)),
               (values(4, 6), values(4, 6).bfloat16())]
    pairs = [pair for four in zip(refused, taken) for pair in four] + taken[len(refused):]
    before = [p.clone() for p, _ in refused]
    expected = []
    for p, update in taken:
        expected.append(p.clone())
        expected[-1].mul_(0.99).add_(update.to(p.dtype), alpha=-0.1)
    left = k.apply_updates(pairs, 0.99, 0.1)
    assert [id(p) for p, _ in left] == [id(p) for p, _ in refused]
    assert all(torch.equal(p, old) for (p, _), old in zip(refused, before))
    assert all(torch.equal(p, new) for (p, _), new in zip(taken, expected))
