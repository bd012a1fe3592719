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
