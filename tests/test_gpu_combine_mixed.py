"""GPU test of a combine that sends and reduces in one launch in a group of more than one rank: the rank's own rows are gathered in
place while the others come through its slots.  Two virtual ranks on one GPU; nothing ever waits for a launch that has not ended:
rank 1 sends, rank 0 does its whole call in one launch (rank 1's flag is up, its own is raised inside the launch), rank 1 reduces."""
import pytest
import torch

import umdk_original_b200 as u
from umdk_original_b200.ops import reference as ref
from umdk_original_b200.parallel import PHASE_COUNT, PHASE_RECV, PHASE_SEND, phases, run_virtual

pytestmark = pytest.mark.gpu
ops = torch.ops.umdk_cam_op_lib
DEV = torch.device("cuda", 0)


def _want(y, plans, idx, w, r, wire):
    """Sums of rank r's tokens over the rows that every rank holds for it (receive order), in k order."""
    t, k = idx.shape
    rows = torch.zeros(t, k, y[0].shape[1])
    for s in range(2):
        v = y[s].float()
        if wire == 2:
            v = ref.dequant_int8_1x128(*ref.quant_int8_1x128(v))
        mine = plans[s].src[:, 0] == r
        rows[plans[s].src[mine, 1].long(), plans[s].src[mine, 2].long()] = v[:plans[s].src.shape[0]][mine]
    acc = torch.zeros(t, y[0].shape[1])
    for kk in range(k):
        acc = torch.addcmul(acc, rows[:, kk], w[:, kk].unsqueeze(-1))
    return acc


def _close(got, want, w, y, k, wire):
    # half a bf16 step; with int8 rows a value on a rounding boundary may also land one step (1 / 127 of its block) apart
    slack = 1e-6 * k + (max(float(v.abs().max()) for v in y) / 127 * float(w.max()) if wire else 0.0)
    assert ((got.cpu().float() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()


def _one_launch_between(fn):
    with phases(PHASE_SEND):
        fn(1)
    out0 = fn(0)
    with phases(PHASE_RECV):
        out1 = fn(1)
    torch.cuda.synchronize()
    return out0, out1


@pytest.mark.parametrize("t,h,e,k,wire", [(1, 128, 2, 1, 0), (37, 640, 8, 3, 0), (37, 640, 8, 3, 2), (37, 2176, 8, 3, 2),
                                          (90, 4224, 16, 8, 2), (90, 1152, 16, 8, 2),
                                          (200, 256, 32, 12, 0), (200, 256, 32, 12, 2)])
def test_low_latency_combine(t, h, e, k, wire):
    bufs = u.Buffer.virtual(2, u.CamConfig(num_experts=e, max_tokens=t, hidden=h, topk=k, ll_max_tokens=t, timeout_ms=2000.0),
                            DEV, name=f"mix{t}_{k}_{wire}_")
    for it in range(2):  # the second call must not see the first one's rows: other routing, some pairs left out
        g = torch.Generator().manual_seed(10 * t + it)
        idx = [torch.rand(t, e, generator=g).argsort(dim=1)[:, :k].to(torch.int32).contiguous() for _ in range(2)]
        if it:
            idx[0][::3, 0] = -1
        w = [torch.rand(t, k, generator=g) for _ in range(2)]
        x = torch.randn(t, h, generator=g).to(torch.bfloat16).to(DEV)
        plans = ref.plan_dispatch(idx, e)
        dk, dw = [i.to(DEV) for i in idx], [v.to(DEV) for v in w]
        d = run_virtual(lambda r: ops.moe_dispatch_shmem(x, dk[r], None, None, 2, r, e, 1, 0, 0, 0, 0, 0, 0, 1, bufs[r].handle), 2,
                        masks=(PHASE_SEND, PHASE_RECV))
        y = [torch.randn(d[r][0].shape[0], h, generator=g).to(torch.bfloat16) for r in range(2)]
        dy = [v.to(DEV) for v in y]
        out = _one_launch_between(lambda r: ops.moe_combine_shmem(dy[r], dk[r], d[r][2], d[r][4], dw[r], None, None, None, None, None,
                                                                  None, 2, r, e, 1, 0, 0, 0, 0, 0, wire, bufs[r].handle, 0, 0))
        for r in range(2):
            bufs[r].check()
            _close(out[r], _want(y, plans, idx[r], w[r], r, wire), w[r], y, k, wire)
    for b in bufs:
        b.destroy()


@pytest.mark.parametrize("t,h,e,k", [(3, 256, 4, 2), (300, 1152, 16, 8), (300, 256, 32, 11)])
def test_prefill_combine(t, h, e, k):
    bufs = u.Buffer.virtual(2, u.CamConfig(num_experts=e, max_tokens=t, hidden=h, topk=k, timeout_ms=2000.0), DEV, name=f"mixp{t}_{k}_")
    for it in range(2):
        g = torch.Generator().manual_seed(20 * t + it)
        idx = [torch.rand(t, e, generator=g).argsort(dim=1)[:, :k].contiguous() for _ in range(2)]
        if it:
            idx[0][::3, 0] = -1
        w = [torch.rand(t, k, generator=g) for _ in range(2)]
        x = torch.randn(t, h, generator=g).to(torch.bfloat16).to(DEV)
        plans = ref.plan_dispatch(idx, e)
        dk, dw = [i.to(DEV) for i in idx], [v.to(DEV) for v in w]
        d = run_virtual(lambda r: ops.moe_dispatch_prefill_quant(x, dk[r], dw[r], bufs[r].capacity, bufs[r].name, r, 2, 0), 2,
                        masks=(PHASE_COUNT, PHASE_SEND, PHASE_RECV))
        src, cnt = [d[r][1].clone() for r in range(2)], [d[r][2].clone() for r in range(2)]
        y = [torch.randn(bufs[r].capacity, h, generator=g).to(torch.bfloat16) for r in range(2)]
        dy = [v.to(DEV) for v in y]
        out = _one_launch_between(lambda r: ops.moe_combine_prefill(dy[r], dk[r], dw[r], src[r], cnt[r], bufs[r].name, r, 2))
        for r in range(2):
            bufs[r].check()
            _close(out[r], _want(y, plans, idx[r], w[r], r, 0), w[r], y, k, 0)
    for b in bufs:
        b.destroy()
