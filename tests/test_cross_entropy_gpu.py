"""Cross entropy kernel and the fused vocabulary head: edges of the row walk, masked columns, every way to differentiate."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v", [8, 264, 4096, 32768, 49152, 49160, 131080])
@pytest.mark.parametrize("masked", [False, True])
def test_loss_and_gradient_of_logits(v, masked):
    from system_lab_b200.ops import cuda
    g = torch.Generator(device="cuda").manual_seed(v)
    rows = 5
    x = (4 * torch.randn(rows, v, generator=g, device="cuda")).bfloat16()
    tgt = torch.randint(0, v, (rows,), generator=g, device="cuda")
    if masked:                                   # most columns carry no probability, the first ones among them
        keep = torch.rand(v, generator=g, device="cuda") < 0.1
        keep[tgt] = True
        x[:, ~keep] = float("-inf")
    ref = x.double()
    loss = torch.logsumexp(ref, -1).sub(ref.gather(1, tgt[:, None]).squeeze(1)).sum()
    grad = torch.softmax(ref, -1)
    grad[torch.arange(rows), tgt] -= 1
    alone = torch.zeros(1, device="cuda")
    cuda.call("slab_ce_fwd", x, tgt, alone, rows, v, cuda.stream())
    assert torch.equal(x.double(), ref)          # the loss alone leaves the logits as they are
    both = torch.zeros(1, device="cuda")
    cuda.call("slab_ce_fwd_bwd", x, tgt, both, rows, v, 0.5, cuda.stream())
    # fp32 exponentials (2 ulp) and sums: 1e-5 of the loss, and a bf16 rounding (2^-9) of the gradient
    for got in (alone, both):
        assert abs(float(got) - float(loss)) <= 1e-5 * abs(float(loss)) + 1e-5
    assert bool(((x.double() - 0.5 * grad).abs() <= 2 ** -8 * (0.5 * grad).abs() + 1e-6).all())


def _head(n, h, v):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, h, generator=g, device="cuda").bfloat16().requires_grad_(True)
    w = (0.05 * torch.randn(v, h, generator=g, device="cuda")).bfloat16().requires_grad_(True)
    return x, w, torch.randint(0, v, (n,), generator=g, device="cuda")


@pytest.mark.parametrize("factor", [1.0, 0.37])
@pytest.mark.parametrize("chunk", [64, 8192])
def test_head_gradients_by_every_route(factor, chunk):
    from system_lab_b200.ops import cuda
    x, w, t = _head(130, 128, 320)

    def loss():
        return cuda.linear_cross_entropy(x, w, t, chunk) * factor

    first = torch.autograd.grad(loss(), [x, w])
    kept = loss()
    one = torch.autograd.grad(kept, [x, w], retain_graph=True)
    two = torch.autograd.grad(kept, [x, w])
    with torch.autograd.graph.saved_tensors_hooks(lambda a: a.clone(), lambda a: a):
        hooked = torch.autograd.grad(loss(), [x, w])
    for got in (one, two, hooked):
        assert all(torch.equal(a, b) for a, b in zip(first, got))
    y = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    ref = torch.autograd.grad(torch.nn.functional.cross_entropy(y[0] @ y[1].t(), t) * factor, list(y))
    # bf16 logits and bf16 logit gradients (2^-9 each) through one more product: 1 % of the gradient's norm
    for a, b in zip(first, ref):
        assert float((a.double() - b).norm() / b.norm()) < 1e-2
    once = loss()
    torch.autograd.grad(once, [x])
    with pytest.raises(RuntimeError):
        torch.autograd.grad(once, [x])


def test_head_gradients_that_are_differentiated_or_come_as_a_batch():
    from system_lab_b200.ops import cuda
    x, w, t = _head(130, 128, 320)
    f = torch.tensor(0.5, device="cuda", requires_grad=True)             # scaling a gradient by it is exact in bf16
    dx, dw = torch.autograd.grad(cuda.linear_cross_entropy(x, w, t), [x, w])
    sx, sw = torch.autograd.grad(cuda.linear_cross_entropy(x, w, t) * f, [x, w], create_graph=True, retain_graph=False)
    assert torch.equal(sx.detach(), dx * 0.5) and torch.equal(sw.detach(), dw * 0.5)
    (df,) = torch.autograd.grad(sx.double().sum() + sw.double().sum(), f)
    want = float(dx.double().sum() + dw.double().sum())
    # the sums over the two gradients are rounded to bf16 (2^-9 each)
    assert abs(float(df) - want) <= 2 ** -8 * float(dx.double().sum().abs() + dw.double().sum().abs())
    bx, bw = torch.autograd.grad(cuda.linear_cross_entropy(x, w, t), [x, w], torch.tensor([1.0, 2.0], device="cuda"),
                                 is_grads_batched=True)
    for got, one in ((bx, dx), (bw, dw)):
        assert torch.equal(got[0], one) and torch.equal(got[1], one * 2)


def test_head_without_gradients_is_the_same_loss():
    from system_lab_b200.ops import cuda
    x, w, t = _head(200, 128, 320)
    with torch.no_grad():
        plain = cuda.linear_cross_entropy(x, w, t, 64)
    assert abs(float(plain) - float(cuda.linear_cross_entropy(x, w, t, 64).detach())) <= 1e-5 * abs(float(plain))
    only = torch.autograd.grad(cuda.linear_cross_entropy(x, w.detach(), t), x)[0]
    assert torch.equal(only, torch.autograd.grad(cuda.linear_cross_entropy(x, w, t), x)[0])
