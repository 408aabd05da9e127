"""GPU tests of the paths that a group of one rank takes when an op runs in one launch (the virtual-rank tests split every op
into phases): rows that stay on the rank, against the CPU oracle, at the sizes where their loops end."""
import pytest
import torch

import umdk_original_b200 as u
from umdk_original_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
ops = torch.ops.umdk_cam_op_lib
DEV = torch.device("cuda", 0)


def _routing(t, e, k, seed, skip):
    """Distinct experts per token where there are enough of them; every `skip`-th first choice is left out."""
    g = torch.Generator().manual_seed(seed)
    if e >= k:
        idx = torch.rand(t, e, generator=g).argsort(dim=1)[:, :k].contiguous()
    else:
        idx = torch.randint(0, e, (t, k), generator=g)
    if skip:
        idx[::skip, 0] = -1
    return idx, torch.rand(t, k, generator=g), g


def _want(y, plan, idx, w, e, wire):
    """Weighted sums of the rows y (receive order), in k order."""
    if wire == 2:
        y = ref.dequant_int8_1x128(*ref.quant_int8_1x128(y.float()))
    t, k = idx.shape
    rows = torch.zeros(t, k, y.shape[1])
    rows[plan.src[:, 1].long(), plan.src[:, 2].long()] = y[:plan.src.shape[0]].float()
    ok = ((idx >= 0) & (idx < e)).float().unsqueeze(-1)
    acc = torch.zeros(t, y.shape[1])
    for kk in range(k):
        acc = torch.addcmul(acc, rows[:, kk] * ok[:, kk], w[:, kk].unsqueeze(-1))
    return acc


@pytest.mark.parametrize("t,h,e,k,skip", [(1, 128, 1, 1, 0), (3, 640, 6, 2, 2), (149, 1152, 10, 5, 7), (300, 512, 256, 8, 0),
                                          (2500, 256, 601, 16, 3)])
def test_prefill_pair_in_one_launch(t, h, e, k, skip):
    # experts: one, not a multiple of four, more than the threads of a CTA (and odd); more pairs per CTA than threads at t = 2500
    buf = u.Buffer(None, u.CamConfig(num_experts=e, max_tokens=t, hidden=h, topk=k, timeout_ms=2000.0), device=DEV, rank=0,
                   num_ranks=1)
    for it in range(2):  # the second call must not see the first one's rows
        idx, w, g = _routing(t, e, k, seed=t + it, skip=skip if it == 0 else 0)
        x = torch.randn(t, h, generator=g).to(torch.bfloat16)
        plan = ref.plan_dispatch([idx], e)[0]
        n = plan.src.shape[0]
        rx, src, cnt, per_e, _ = ops.moe_dispatch_prefill_quant(x.to(DEV), idx.to(DEV), w.to(DEV), 0, buf.name, 0, 1, 0)
        assert torch.equal(src.cpu().view(-1, 3), plan.src) and torch.equal(cnt.cpu(), plan.recv_count)
        assert torch.equal(per_e.cpu(), plan.per_expert) and torch.equal(rx.cpu(), x[plan.src[:, 1].long()])
        y = torch.randn(n, h, generator=g).to(torch.bfloat16)
        out = ops.moe_combine_prefill(y.to(DEV), idx.to(DEV), w.to(DEV), src.clone(), cnt.clone(), buf.name, 0, 1)
        buf.check()
        want = _want(y, plan, idx, w, e, 0)
        # the kernel adds the same products in the same order with fused multiply-adds; half a bf16 step remains
        assert ((out.cpu().float() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6 * k).all()
    buf.destroy()


@pytest.mark.parametrize("quant,wire", [(0, 0), (2, 2), (3, 2), (4, 0)])
@pytest.mark.parametrize("t,h,e,k,skip", [(1, 128, 1, 1, 0), (5, 1152, 6, 3, 2), (35, 2176, 16, 3, 4), (40, 4224, 32, 8, 3),
                                          (40, 4096, 32, 9, 3), (151, 512, 64, 8, 5), (256, 128, 8, 8, 0),
                                          (257, 128, 16, 8, 3), (1024, 128, 64, 8, 5),
                                          (1025, 128, 64, 8, 7)])
# 8192 pairs: the most the scan of the ids serves; int8 rows of more than 2048 and at least 512 x k: combined in place
def test_low_latency_pair_in_one_launch(t, h, e, k, skip, quant, wire):
    buf = u.Buffer(None, u.CamConfig(num_experts=e, max_tokens=t, hidden=h, topk=k, ll_max_tokens=t, timeout_ms=2000.0),
                   device=DEV, rank=0, num_ranks=1)
    for it in range(2):
        idx, w, g = _routing(t, e, k, seed=7 * t + it, skip=skip if it == 0 else 0)
        idx = idx.to(torch.int32)
        x = torch.randn(t, h, generator=g).to(torch.bfloat16)
        smooth = torch.rand(e, h, generator=g) + 0.5 if quant == 2 else None
        active = torch.arange(t) < t - t // 4
        live = torch.where(active.unsqueeze(1), idx, torch.full_like(idx, -1))
        plan = ref.plan_dispatch([live], e)[0]
        n = plan.src.shape[0]
        d = ops.moe_dispatch_shmem(x.to(DEV), idx.to(DEV), None if smooth is None else smooth.to(DEV), active.to(DEV), 1, 0, e,
                                   1, 0, 0, 0, 0, quant, 0, it, buf.handle)
        rows = x[plan.src[:, 1].long()]
        if quant == 0:
            assert torch.equal(d[0][:n].cpu(), rows)
        elif quant == 2:
            q, s = ref.quant_int8_token(rows.float() * smooth[live[plan.src[:, 1].long(), plan.src[:, 2].long()].long()])
            assert (d[0][:n].cpu().int() - q.int()).abs().max() <= 1  # x * 127 / amax on a rounding boundary
            assert torch.allclose(d[1][:n].cpu(), s, rtol=1e-6)
        else:
            q, s = ref.quant_fp8_1x128(rows, quant == 4)
            assert torch.equal(d[0][:n].cpu().view(torch.uint8), q.view(torch.uint8)) and torch.equal(d[1][:n].cpu(), s)
        assert torch.equal(d[2].cpu(), ref.slots_in_expert(live, e))
        assert torch.equal(d[3].cpu(), plan.per_expert if it else plan.per_expert.cumsum(0))
        assert torch.equal(d[4].cpu(), plan.recv_count) and d[5].tolist() == [0]
        y = torch.randn(d[0].shape[0], h, generator=g).to(torch.bfloat16)
        out = ops.moe_combine_shmem(y.to(DEV), idx.to(DEV), d[2], d[4], w.to(DEV), None, active.to(DEV), None, None, None, None,
                                    1, 0, e, 1, 0, 0, 0, 0, 0, wire, buf.handle, 0, 0)
        buf.check()
        want = _want(y[:n], plan, live, w, e, wire)
        # half a bf16 step; with int8 rows a value on a rounding boundary may also land one step (1 / 127 of its block) apart
        slack = 1e-6 * k + (float(y.abs().max()) / 127 * float(w.max()) if wire else 0.0)
        assert ((out.cpu().float() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()
    buf.destroy()


@pytest.mark.parametrize("t,e,k,r", [(0, 8, 2, 2), (1, 1, 1, 1), (33, 72, 3, 72), (4097, 256, 8, 8), (16384, 64, 16, 4),
                                     (16385, 64, 2, 64)])  # one and two launches
def test_layout_at_its_sizes(t, e, k, r):
    idx = torch.randint(-1, e + 1, (t, k), generator=torch.Generator().manual_seed(t))
    got = ops.get_dispatch_layout(idx.to(DEV), e, r)
    for a, b in zip(got, ref.get_dispatch_layout(idx, e, r)):
        assert torch.equal(a.cpu(), b)


@pytest.mark.parametrize("dtype,offset", [(torch.int64, 0), (torch.int64, 1), (torch.int32, 1)])  # ids off the 16-byte grid
@pytest.mark.parametrize("t,e,k,r", [(4095, 63, 5, 7), (4097, 64, 8, 8), (8192, 256, 8, 8), (8193, 256, 8, 8), (8192, 256, 9, 8),
                                     (100, 72, 8, 9), (31, 1024, 6, 4)])
def test_layout_on_both_sides_of_its_limits(t, e, k, r, dtype, offset):
    flat = torch.randint(-1, e + 1, (t * k + offset,), generator=torch.Generator().manual_seed(t + k)).to(dtype)
    got = ops.get_dispatch_layout(flat.to(DEV)[offset:].view(t, k), e, r)
    for a, b in zip(got, ref.get_dispatch_layout(flat[offset:].view(t, k), e, r)):
        assert torch.equal(a.cpu(), b)


@pytest.mark.parametrize("quant", [0, 2, 3, 4])
@pytest.mark.parametrize("t,h,e,k", [(1, 128, 1, 1), (149, 1408, 5, 3), (512, 256, 32, 8), (513, 256, 32, 8), (592, 384, 7, 2),
                                     (593, 384, 7, 2)])  # 4096 pairs and four tokens per CTA: the most the short form serves
def test_prefill_dispatch_formats_in_one_launch(t, h, e, k, quant):
    buf = u.Buffer(None, u.CamConfig(num_experts=e, max_tokens=t, hidden=h, topk=k, timeout_ms=2000.0), device=DEV, rank=0,
                   num_ranks=1)
    idx, w, g = _routing(t, e, k, seed=3 * t + quant, skip=4)
    x = torch.randn(t, h, generator=g).to(torch.bfloat16)
    plan = ref.plan_dispatch([idx], e)[0]
    n = plan.src.shape[0]
    if n == 0:  # the only pair is the one left out
        idx[0, 0] = 0
        plan = ref.plan_dispatch([idx], e)[0]
        n = 1
    rx, src, cnt, per_e, rs = ops.moe_dispatch_prefill_quant(x.to(DEV), idx.to(DEV), w.to(DEV), buf.capacity, buf.name, 0, 1, quant)
    buf.check()
    rows = x[plan.src[:, 1].long()]
    assert torch.equal(src.cpu().view(-1, 3)[:n], plan.src) and torch.equal(cnt.cpu(), plan.recv_count)
    assert torch.equal(per_e.cpu(), plan.per_expert) and int(buf.native.total_recv()) == n
    if quant == 0:
        assert torch.equal(rx[:n].cpu(), rows)
    elif quant == 2:
        q, s = ref.quant_int8_token(rows)
        assert (rx[:n].cpu().int() - q.int()).abs().max() <= 1  # x * 127 / amax on a rounding boundary
        assert torch.allclose(rs[:n].cpu().reshape(-1), s, rtol=1e-6)
    else:
        q, s = ref.quant_fp8_1x128(rows, quant == 4)
        assert torch.equal(rx[:n].cpu().view(torch.uint8), q.view(torch.uint8)) and torch.equal(rs[:n].cpu(), s)
    stats = buf.stats()
    assert stats["dispatch_calls"] == 1 and stats["rows_routed_to_peer"] == [n]
    buf.destroy()


@pytest.mark.parametrize("t", [9, 700])  # the short form, and the general kernel of a rank alone
def test_receive_overflow_in_one_launch(t):
    e, k, h = 4, 2, 128
    idx, w, g = _routing(t, e, k, seed=t, skip=0)
    cap = t * k - 1
    buf = u.Buffer(None, u.CamConfig(num_experts=e, max_tokens=t, hidden=h, topk=k, capacity=cap, timeout_ms=2000.0), device=DEV,
                   rank=0, num_ranks=1)
    region = buf.native.recv_x(cap, h, 0)
    region.fill_(7.0)
    canary = region.clone()
    x = torch.randn(t, h, generator=g).to(torch.bfloat16)
    per_e = ops.moe_dispatch_prefill_quant(x.to(DEV), idx.to(DEV), w.to(DEV), cap, buf.name, 0, 1, 0)[3]
    with pytest.raises(u.RecvOverflow) as ei:
        buf.check()
    assert ei.value.who == 0 and ei.value.detail == t * k
    assert int(buf.native.total_recv().item()) == 0 and int(per_e.sum().item()) == 0
    assert int(buf.native.expert_offsets(e + 1).abs().sum().item()) == 0
    assert bool((buf.native.send_row(t * k) == -1).all()) and torch.equal(region, canary)
    buf.reset()
    idx[1:] = -1  # after the reset a call that fits goes through
    rx = ops.moe_dispatch_prefill_quant(x.to(DEV), idx.to(DEV), w.to(DEV), 0, buf.name, 0, 1, 0)[0]
    buf.check()
    assert torch.equal(rx.cpu(), x[:1].expand(k, h))
    buf.destroy()
