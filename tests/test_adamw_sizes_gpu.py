"""Flat AdamW where its pieces end: every 128-element block comes out as if it had been updated alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
STATE = {0: torch.float32, 1: torch.bfloat16, 2: torch.float8_e4m3fn}


def _update(p, g, m, v, ms, vs, out, sq, kind, decay_end):
    from system_lab_b200.ops import cuda
    n = p.numel()
    cuda.call("slab_adamw", p, int(p.dtype == torch.bfloat16), g, int(g.dtype == torch.bfloat16), m, v,
              ms if kind == 2 else None, vs if kind == 2 else None, out, None, sq, n, kind, 1e-2, 0.9, 0.95, 1e-8, 0.1,
              1 - 0.9 ** 3, 1 - 0.95 ** 3, decay_end, 0, cuda.stream())


@pytest.mark.parametrize("n", [128, 384, 512, 640, 512 * 7 + 256])
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("pd,gd", [(torch.float32, torch.float32), (torch.float32, torch.bfloat16),
                                   (torch.bfloat16, torch.bfloat16)])
def test_blocks_are_independent(n, kind, pd, gd):
    gen = torch.Generator(device="cuda").manual_seed(n)

    def rand(dtype, size=n):
        return torch.randn(size, generator=gen, device="cuda").to(dtype)

    p, g, m, v = rand(pd), rand(gd), rand(STATE[kind]), rand(torch.float32).abs().to(STATE[kind])
    ms, vs = rand(torch.float32, n // 128).abs() + 0.1, rand(torch.float32, n // 128).abs() + 0.1
    out, sq = torch.zeros(n, device="cuda", dtype=torch.bfloat16), torch.zeros(1, device="cuda")
    decay_end = n // 256 * 128
    alone = [t.clone() for t in (p, g, m, v, ms, vs, out)]
    start, grad, m0, v0 = (t.double() for t in (p, g, m, v))
    _update(p, g, m, v, ms, vs, out, sq, kind, decay_end)
    for b in range(n // 128):
        e, s = slice(128 * b, 128 * b + 128), slice(b, b + 1)
        pp, gg, mm, vv, m1, v1, oo = alone
        _update(pp[e], gg[e], mm[e], vv[e], m1[s], v1[s], oo[e], None, kind, 128 if 128 * b < decay_end else 0)
    for a, b in zip((p, m, v, ms, vs, out), (alone[0], alone[2], alone[3], alone[4], alone[5], alone[6])):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    assert torch.equal(out.float(), p.to(torch.bfloat16).float())
    assert abs(float(sq) - float(grad.square().sum())) <= 1e-5 * float(grad.square().sum())
    if kind == 0:
        m2, v2 = 0.9 * m0 + 0.1 * grad, 0.95 * v0 + 0.05 * grad * grad
        decay = torch.where(torch.arange(n, device="cuda") < decay_end, 1 - 1e-2 * 0.1, 1.0)
        want = start * decay - 1e-2 * (m2 / (1 - 0.9 ** 3)) / ((v2 / (1 - 0.95 ** 3)).sqrt() + 1e-8)
        # fp32 arithmetic with approximate roots and quotients: 1e-5 of the weight and of the step; bf16 weights round (2^-9)
        bound = (2 ** -8 if pd == torch.bfloat16 else 1e-5) * (start.abs() + (want - start).abs()) + 1e-7
        assert bool(((p.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("pd", [torch.float32, torch.bfloat16])
def test_first_step_is_the_same_with_every_kind_of_state(pd):
    """The update is computed in fp32 before the state is rounded, by one function: from zero moments the weights are the
    same bits whether the moments are kept in 32, 16 or 8 bits."""
    n = 128 * 33
    gen = torch.Generator(device="cuda").manual_seed(1)
    g = torch.randn(n, generator=gen, device="cuda").bfloat16()
    start = torch.randn(n, generator=gen, device="cuda").to(pd)
    got = []
    for kind in (0, 1, 2):
        p, m, v = start.clone(), torch.zeros(n, device="cuda").to(STATE[kind]), torch.zeros(n, device="cuda").to(STATE[kind])
        ones = torch.ones(n // 128, device="cuda")
        _update(p, g, m, v, ones, ones.clone(), torch.zeros(n, device="cuda", dtype=torch.bfloat16), None, kind, n // 256 * 128)
        got.append(p)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2]) and not torch.equal(got[0], start)


def test_update_behind_a_reduce_scatter_is_the_flat_one():
    import ctypes
    from system_lab_b200.ops import cuda
    from tests.test_fsdp_comm_gpu import _comms
    world, shard, decay_end = 2, 128 * 20, 128 * 15
    cs = _comms(world, shard * world * 2)
    gen = torch.Generator(device="cuda").manual_seed(2)
    grads = [torch.randn(shard * world, generator=gen, device="cuda").bfloat16() for _ in range(world)]
    p, m = (torch.randn(shard, generator=gen, device="cuda") for _ in range(2))
    v, out = torch.rand(shard, generator=gen, device="cuda"), torch.zeros(shard, device="cuda", dtype=torch.bfloat16)
    flat = [t.clone() for t in (p, m, v, out)]
    meta = []
    for c, g in zip(cs, grads):
        c._ensure(g.numel() * 2)
        slot, ep, ack = c._next()
        c._stage(g, slot, ep, ack)
        meta.append((slot, ep))
    c, (slot, ep) = cs[0], meta[0]
    cuda.call("slab_fsdp_reduce_scatter_adamw", shard, ctypes.addressof(c._ptrs), ctypes.addressof(c._lay), world, 0, slot, ep,
              1.0, p, m, v, out, None, None, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1 - 0.9 ** 3, 1 - 0.95 ** 3, decay_end, c.status,
              c.done, cuda.stream())
    _update(flat[0], grads[0][:shard].float() + grads[1][:shard].float(), flat[1], flat[2], None, None, flat[3], None, 0, decay_end)
    cuda.check_status()
    for a, b in zip((p, m, v, out), flat):
        assert torch.equal(a, b)
