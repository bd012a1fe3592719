"""e4m3 quantisers: row lengths around the vector and warp mappings, odd starts, special values."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rounded_to_nearest(q, s, x):
    """Half an e4m3 step: 2^-4 of the value, 2^-10 of the scale near zero.  The kernels multiply by 448 / amax in fp32, whose error
    (2^-20 of the value at most, reciprocal and product) can turn a near-tie only."""
    d = q.double() * s.double()
    assert bool(((d - x.double()).abs() <= x.double().abs() * (2 ** -4 + 2 ** -19) + s.double() * 2 ** -10).all())


@pytest.mark.parametrize("rows,h", [(1, 128), (3, 256), (77, 768), (33, 2880), (129, 7168), (5, 16384), (4, 16512)])
def test_row_and_block_scales(rows, h):
    from system_lab_b200.ops import cuda
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, h, generator=g, device="cuda").bfloat16()
    x[0, :128] = 0
    q, s = cuda.quant_rowwise(x)
    _rounded_to_nearest(q, s[:, None], x)
    assert torch.equal(s, x.abs().amax(-1).float().clamp_min(1e-12) / 448) or \
        bool((s * 448 / x.abs().amax(-1).float() - 1).abs().max() < 1e-6)
    if h % 128 == 0:
        q, s = cuda.quant_1x128(x)
        _rounded_to_nearest(q, s.repeat_interleave(128, -1), x)
        odd = torch.empty(rows * h + 4, device="cuda", dtype=torch.bfloat16)[4:].view(rows, h).copy_(x)   # 8-byte aligned
        qo, so = cuda.quant_1x128(odd)
        assert torch.equal(q.view(torch.uint8), qo.view(torch.uint8)) and torch.equal(s, so)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2048, 100003])
def test_one_scale_gives_the_oracles_bytes(n):
    from system_lab_b200.ops import cuda, reference as ref
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n + 1, generator=g, device="cuda").bfloat16()
    for t in (x[:n], x[1:], torch.zeros_like(x[:n]), x[:n] * 1e30, x[:n] * 1e-30):
        q, s = cuda.quant_tensorwise(t)
        qr, sr = ref.quant_tensorwise(t)
        assert torch.equal(q.view(torch.uint8), qr.view(torch.uint8)) and float(s) == float(sr) and q.shape == qr.shape


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_one_scale_of_special_values(bad):
    from system_lab_b200.ops import cuda, reference as ref
    x = torch.randn(3000, device="cuda").bfloat16()
    x[1234] = bad
    q, s = cuda.quant_tensorwise(x)
    qr, sr = ref.quant_tensorwise(x)
    assert torch.equal(torch.isnan(q.float()), torch.isnan(qr.float()))
    assert torch.equal(q.float().nan_to_num(), qr.float().nan_to_num())
    assert torch.equal(torch.isnan(s), torch.isnan(sr)) and float(s.nan_to_num()) == float(sr.nan_to_num())
