"""Grouped GEMM on pairs of SMs at the sizes where its tiles end: chunks of rows, output blocks, reduction remainders."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(counts, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    cnt = torch.tensor(counts, dtype=torch.int32)
    pad = (cnt + 127) // 128 * 128
    off, rows = torch.cumsum(pad, 0) - pad, max(int(pad.sum()), 128)
    used = torch.zeros(rows, 1, device="cuda")
    for o, c in zip(off.tolist(), counts):
        used[o:o + c] = 1
    a = (torch.randn(rows, k, generator=g, device="cuda") * used).bfloat16()
    dy = (torch.randn(rows, n, generator=g, device="cuda") * used).bfloat16()
    w = (0.05 * torch.randn(len(counts), n, k, generator=g, device="cuda")).bfloat16()
    return a, dy, w, off.int().cuda(), cnt.cuda()


def _close(out, ref, magnitude):
    """bf16 result of an fp32 sum: half a bf16 step of the value (2^-9), doubled for sums that round across a binade, and
    2^-20 of the summed magnitudes for the order of the sum."""
    from system_lab_b200.ops import cuda
    cuda.check_status()
    bound = ref.abs() * 2 ** -8 + magnitude * 2 ** -20 + 1e-30
    assert bool(((out.double() - ref).abs() <= bound).all()), float(((out.double() - ref).abs() / bound).max())


# rows around the 32-row unit, the 256-row chunk and uneven cuts; output columns around the 64-, 128- and 256-wide blocks
SIZES = [([1], 64, 64), ([31, 32, 33], 64, 192), ([255, 256, 257], 192, 128), ([0, 513, 0, 5], 320, 64),
         ([1100, 3], 128, 320), ([700] * 9, 576, 448), ([2] * 400, 64, 128),
         ([60, 0, 300, 90] * 6, 384, 320), ([1, 0, 33, 2] * 128, 64, 64)]


# CTAs a launch may take: all of them (a tile per pair at these sizes), and so few that a pair walks many tiles, which carries the
# ring's and the accumulators' phases, staging buffers and old results over from tile to tile (odd values round down to pairs)
CTAS = [0, 1, 2, 3, 7]


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("counts,n,k", SIZES)
def test_rows_against_64_bits(counts, n, k, ctas):
    from system_lab_b200.ops import cuda
    a, dy, w, off, cnt = _operands(counts, n, k, 1)
    for mode, x, cols in ((0, a, n), (1, dy, k)):
        out = torch.full((x.shape[0], cols), float("nan"), device="cuda", dtype=torch.bfloat16)
        cuda.grouped_gemm_raw(mode, x, w, off, cnt, n, k, out=out, max_ctas=ctas)
        for e, (o, c) in enumerate(zip(off.tolist(), counts)):
            we = w[e].double().t() if mode == 0 else w[e].double()
            _close(out[o:o + c], x[o:o + c].double() @ we, x[o:o + c].double().abs() @ we.abs())
            assert not bool(out[o + c:o + (c + 127) // 128 * 128].any())     # padding rows are zero


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("counts,n,k", SIZES)
def test_weight_gradient_against_64_bits(counts, n, k, ctas):
    from system_lab_b200.ops import cuda
    a, dy, w, off, cnt = _operands(counts, n, k, 2)
    out = torch.full_like(w, float("nan"))
    cuda.grouped_gemm_raw(2, dy, a, off, cnt, n, k, out=out, max_ctas=ctas)
    twice = w.clone()
    cuda.grouped_gemm_raw(2, dy, a, off, cnt, n, k, out=twice, accumulate=True, max_ctas=ctas)
    for e, (o, c) in enumerate(zip(off.tolist(), counts)):
        d, x = dy[o:o + c].double(), a[o:o + c].double()
        _close(out[e], d.t() @ x, d.abs().t() @ x.abs())
        _close(twice[e], w[e].double() + d.t() @ x, w[e].double().abs() + d.abs().t() @ x.abs())


# N just over a multiple of 256 against a wide K: the operands change sides (which the launch's pairs decide), in tiles of 128 and
# of 256 columns of N, with a last one of 64, 192 and 320; K that ends inside a 128- and a 64-wide half of a block
@pytest.mark.parametrize("ctas", [0, 2, 7])
@pytest.mark.parametrize("counts,n,k", [([200], 576, 7168), ([1], 576, 7104), ([130, 0, 33], 576, 2368), ([513, 7], 320, 3136),
                                        ([77] * 5, 832, 4096), ([0, 40], 320, 704)])
def test_weight_gradient_with_exchanged_sides(counts, n, k, ctas):
    from system_lab_b200.ops import cuda
    a, dy, w, off, cnt = _operands(counts, n, k, 6)
    out = torch.full_like(w, float("nan"))
    cuda.grouped_gemm_raw(2, dy, a, off, cnt, n, k, out=out, max_ctas=ctas)
    for e, (o, c) in enumerate(zip(off.tolist(), counts)):
        d, x = dy[o:o + c].double(), a[o:o + c].double()
        _close(out[e], d.t() @ x, d.abs().t() @ x.abs())


@pytest.mark.parametrize("rows", [1, 33, 100, 1021])
def test_one_segment_that_ends_inside_a_tile(rows):
    from system_lab_b200.ops import cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(rows, 192, generator=g, device="cuda").bfloat16()
    w = torch.randn(1, 320, 192, generator=g, device="cuda").bfloat16()
    off, cnt = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((1,), rows, dtype=torch.int32, device="cuda")
    guard = torch.full((rows + 64, 320), 7.0, device="cuda", dtype=torch.bfloat16)
    cuda.grouped_gemm_raw(0, x, w, off, cnt, 320, 192, out=guard[:rows])
    _close(guard[:rows], x.double() @ w[0].double().t(), x.double().abs() @ w[0].double().abs().t())
    assert bool((guard[rows:] == 7).all())
    dw = cuda.grouped_gemm_raw(2, guard[:rows], x, off, cnt, 320, 192)[0]
    _close(dw, guard[:rows].double().t() @ x.double(), guard[:rows].double().abs().t() @ x.double().abs())


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("counts,n,k", [([1], 64, 128), ([31, 0, 257], 192, 256), ([700, 130], 320, 768)])
def test_row_scaled_e4m3(counts, n, k, ctas):
    from system_lab_b200.ops import cuda
    a, _, w, off, cnt = _operands(counts, n, k, 4)
    aq, sa = cuda.quant_rowwise(a)
    wq, sw = cuda.quant_rowwise(w)
    out = cuda.grouped_gemm_fp8_rowwise_raw(aq, sa, wq, sw.contiguous(), off, cnt, max_ctas=ctas)
    for e, (o, c) in enumerate(zip(off.tolist(), counts)):
        x = aq[o:o + c].double() * sa[o:o + c, None].double()
        m = (wq[e].double() * sw[e][:, None].double()).t()
        # the tensor core adds e4m3 products with fewer bits than fp32 (2^-13 of the summed magnitudes at most)
        _close(out[o:o + c], x @ m, (x.abs() @ m.abs()) * 2 ** 7)


class _Arrived:
    """Arrival flags as a dispatcher hands them over: the first ``n`` experts' rows are there, the others never come."""

    def __init__(self, n, experts):
        self.flags = (torch.arange(experts, device="cuda") < n).int().view(1, experts)
        self.world, self.epoch, self.gemm_max_ctas, self.d = 1, 1, 4, self

    def mark_consumed(self):
        pass

    join_side = mark_consumed


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("arrived", [0, 1, 5, 11, 12])
def test_rows_that_never_arrive_end_the_launch(mode, arrived):
    """The wait for the missing rows runs out (20 ms) while the accumulators of the tiles before them are being read out: the
    kernel returns with the status code, what it computed until then is right, and the next launch is healthy."""
    from system_lab_b200.ops import cuda
    n, k, counts = 320, 192, [300] * 12
    a, dy, w, off, cnt = _operands(counts, n, k, 5)
    x = (a, dy)[mode]
    whole = cuda.grouped_gemm_raw(mode, x, w, off, cnt, n, k)
    out = torch.zeros_like(whole)
    cuda.register("slab_moe_set_wait_limit_ms", "l")
    cuda.lib().slab_moe_set_wait_limit_ms(20)
    try:
        cuda.grouped_gemm_raw(mode, x, w, off, cnt, n, k, out=out, ready=_Arrived(arrived, len(counts)))
        torch.cuda.synchronize()
        assert cuda.peek_status() == (0 if arrived == 12 else 5)
    finally:
        cuda.lib().slab_moe_set_wait_limit_ms(60000)
        cuda.clear_status()
    same = (out == whole) | (out == 0)                       # a tile is stored whole or left alone
    assert bool(same.all()) and (arrived < 12 or torch.equal(out, whole))
    assert torch.equal(cuda.grouped_gemm_raw(mode, x, w, off, cnt, n, k), whole)
    cuda.check_status()
