"""Dispatch on one rank: the token-ordered scatter behind both entry points delivers rows, scales, scalars and flags."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,topk,experts,hidden", [(1, 1, 8, 128), (61, 8, 128, 256), (300, 3, 12, 1152), (257, 2, 4, 7168)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("scaled", [False, True])
def test_rows_scales_scalars_and_padding(tokens, topk, experts, hidden, fp8, scaled):
    from system_lab_b200.moe.fused_dispatch import FusedDispatcher
    from system_lab_b200.ops import cuda
    from system_lab_b200.parallel.mesh import single_process_mesh
    g = torch.Generator(device="cuda").manual_seed(tokens)
    d = FusedDispatcher(single_process_mesh(), experts, topk, hidden, tokens, 128, torch.device("cuda", 0), fp8_payload=fp8)
    x = torch.randn(tokens, hidden, generator=g, device="cuda").bfloat16()
    p = torch.rand(tokens, topk, generator=g, device="cuda")
    scale = torch.rand(tokens, topk, generator=g, device="cuda") + 0.5 if scaled else None
    idx = torch.rand(tokens, experts, generator=g, device="cuda").topk(topk, -1).indices.int()
    plan = d.plan(idx)
    rows = (plan.pair_loc & 0xFFFFFF).long().view(tokens, topk)
    want = x[:, None, :] if scale is None else (x.float()[:, None, :] * scale[..., None])
    want = want.expand(tokens, topk, hidden)
    used = int(plan.meta[0])
    for ordered in (True, False):
        buf = d.rows_fp8.view(torch.uint8) if fp8 else d.rows[0].view(torch.int16)
        buf.fill_(1)
        d.scalars[0].fill_(-1)
        if ordered:
            d.scatter_ordered(plan, x, p, 0, scale_in=scale, fp8=fp8).wait()
        else:
            d.wait_rows(0, d.scatter(plan, x, p, 0, scale_in=scale, fp8=fp8))
        cuda.check_status()
        if not fp8:
            assert torch.equal(d.rows[0][rows], want.bfloat16())
        elif scale is None:
            q, s = cuda.quant_1x128(x)
            assert torch.equal(d.rows_fp8.view(torch.uint8)[rows], q.view(torch.uint8)[:, None, :].expand(tokens, topk, hidden))
            assert torch.equal(d.row_scales[rows], s[:, None, :].expand(tokens, topk, hidden // 128))
        else:                                        # half an e4m3 step, and 2^-19 for products and reciprocal in fp32
            unit = d.row_scales[rows].repeat_interleave(128, -1)
            got = d.rows_fp8[rows].float() * unit
            assert bool(((got - want).abs() <= want.abs() * (2 ** -4 + 2 ** -19) + unit * 2 ** -10).all())
        assert torch.equal(d.scalars[0][rows], p)
        free = torch.ones(used, dtype=torch.bool, device="cuda")
        free[rows.reshape(-1)] = False
        assert not bool(buf[:used][free].any()) and not bool(d.scalars[0][:used][free].any())
        assert torch.equal(d.origin[rows].long(), torch.arange(tokens * topk, device="cuda").view(tokens, topk))
        assert not bool(d.chunk_done.any()) and not bool(d.done_counter.any())


@pytest.mark.parametrize("ordered", [False, True])
def test_segments_that_do_not_fit_end_with_the_buffer(ordered):
    """Two ranks whose tokens all pick rank 0's first two experts, 912 padded rows for a buffer of 640: reported, and neither
    rows nor alignment rows land outside the receive region."""
    from system_lab_b200.ops import cuda
    from tests.test_dispatch_gpu import _make
    ds = _make(2, 200, 2, 8, 256, factor=0.25)
    cap = ds[0].capacity
    idx = torch.tensor([0, 1], device="cuda", dtype=torch.int32).repeat(200, 1)
    plans = [d.plan_finish(*p) for d, p in zip(ds, [d.plan_publish(idx) for d in ds])]
    torch.cuda.synchronize()
    assert cap == 640 and cuda.peek_status() == 7
    cuda.clear_status()
    assert plans[0].expert_offsets.tolist() == [0, 512, 640, 640] and plans[0].expert_counts.tolist() == [400, 128, 0, 0]
    outside = [d.ws.buf[d.off["rows1"]:d.off["origin"]] for d in ds]
    for o in outside:
        o.fill_(77)
    x = torch.ones(200, 256, device="cuda", dtype=torch.bfloat16)
    for d, plan in zip(ds, plans):
        if ordered:
            d.scatter_ordered(plan, x, None, 0)
        else:
            d.scatter(plan, x, None, 0)
    torch.cuda.synchronize()
    assert all(bool((o[:d.off["scalars0"] - d.off["rows1"]] == 77).all()) for d, o in zip(ds, outside))
    assert all(bool((o[d.off["out_rows"] - d.off["rows1"]:] == 77).all()) for d, o in zip(ds, outside))
    assert bool((ds[0].rows[0][:400] == 1).all()) and not bool(ds[0].rows[0][400:512].any())
    assert bool((ds[0].rows[0][512:640] == 1).all())
