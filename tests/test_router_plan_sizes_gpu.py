"""Fused router and dispatch plan around the sizes where their kernels change: experts per lane, blocks of pairs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,topk", [(1, 4, 1), (65, 128, 8), (65, 129, 4), (65, 256, 8), (65, 257, 2),
                                                 (33, 512, 8), (2500, 96, 8), (4200, 512, 8)])
@pytest.mark.parametrize("score", ["softmax", "sigmoid"])
def test_selection_gradient_and_plan(tokens, experts, topk, score):
    from system_lab_b200 import ops
    from system_lab_b200.moe.fused_dispatch import FusedDispatcher
    from system_lab_b200.ops import cuda
    from system_lab_b200.parallel.mesh import single_process_mesh
    g = torch.Generator(device="cuda").manual_seed(experts)
    logits = torch.randn(tokens, experts, generator=g, device="cuda").requires_grad_(True)
    w, idx, _ = ops.router_fused(logits, topk, score)
    ref = logits.detach().double().requires_grad_(True)
    scores = torch.softmax(ref, -1) if score == "softmax" else torch.sigmoid(ref)
    order = torch.sort(scores.detach(), -1, descending=True).indices[:, :topk]
    chosen = scores.gather(1, idx.long())
    # the same scores in the same order (an fp32 tie may swap two experts): 1e-6 of the score, from its exponential
    assert bool((chosen.detach() - scores.detach().gather(1, order)).abs().max() < 1e-6)
    wr = chosen / chosen.sum(-1, keepdim=True)
    up = torch.randn(tokens, topk, generator=g, device="cuda")
    (gl,) = torch.autograd.grad(w, logits, up)
    (gr,) = torch.autograd.grad(wr, ref, up.double())
    assert float((w.detach().double() - wr.detach()).abs().max()) < 1e-5
    assert float((gl.double() - gr).abs().max()) < 1e-5 * max(1.0, float(gr.abs().max()))
    d = FusedDispatcher(single_process_mesh(), experts, topk, 128, tokens, 128, torch.device("cuda", 0))
    plan = d.plan(idx)
    cuda.check_status()
    flat = idx.reshape(-1).long()
    counts = torch.bincount(flat, minlength=experts)
    padded = (counts + 127) // 128 * 128
    start, first = torch.cumsum(padded, 0) - padded, torch.cumsum(counts, 0) - counts
    by = torch.argsort(flat, stable=True)
    rows = torch.empty_like(flat)
    rows[by] = start[flat[by]] + torch.arange(flat.numel(), device="cuda") - first[flat[by]]
    assert torch.equal(plan.pair_loc.long(), rows) and torch.equal(plan.perm.long(), by)
    assert torch.equal(plan.expert_offsets.long(), start) and torch.equal(plan.expert_counts.long(), counts)
    assert int(plan.meta[0]) == int(plan.meta[1]) == int(padded.sum())
