"""GPU tests of Buffers that serve calls of changing sizes, as a decode server's do: what one call sets up must not get in the
way of a larger one seen before."""
import pytest
import torch

import umdk_original_b200 as u
from umdk_original_b200.ops import reference as ref
from umdk_original_b200.parallel import PHASE_RECV, PHASE_SEND, run_virtual

pytestmark = pytest.mark.gpu
ops = torch.ops.umdk_cam_op_lib
DEV = torch.device("cuda", 0)


def _low_latency(buf, t, h, e, k, quant, seed):
    g = torch.Generator().manual_seed(seed)
    idx = torch.rand(t, e, generator=g).argsort(dim=1)[:, :k].to(torch.int32).contiguous()
    x = torch.randn(t, h, generator=g).to(torch.bfloat16)
    plan = ref.plan_dispatch([idx], e)[0]
    d = ops.moe_dispatch_shmem(x.to(DEV), idx.to(DEV), None, None, 1, 0, e, 1, 0, 0, 0, 0, quant, 0, 1, buf.handle)
    buf.check()
    rows, n = x[plan.src[:, 1].long()], plan.src.shape[0]
    assert torch.equal(d[3].cpu(), plan.per_expert) and torch.equal(d[4].cpu(), plan.recv_count)
    if quant == 0:
        assert torch.equal(d[0][:n].cpu(), rows)
    else:
        q, s = ref.quant_fp8_1x128(rows, quant == 4)
        assert torch.equal(d[0][:n].cpu().view(torch.uint8), q.view(torch.uint8)) and torch.equal(d[1][:n].cpu(), s)


@pytest.mark.parametrize("quant", [0, 3])
def test_low_latency_batches_of_changing_size(quant):
    # shared memory of the calls with 256 experts (e4m3): 56, 30 and 56 KB
    bufs = {e: u.Buffer(None, u.CamConfig(num_experts=e, max_tokens=256, hidden=7168, topk=8, ll_max_tokens=256, timeout_ms=2000.0),
                        device=DEV, rank=0, num_ranks=1) for e in (256, 16)}
    for i, (t, e) in enumerate([(256, 256), (8, 256), (256, 256), (1, 16), (256, 256), (256, 16)]):
        _low_latency(bufs[e], t, 7168, e, 8, quant, seed=i)
    for b in bufs.values():
        b.destroy()


def test_low_latency_batch_that_does_not_fit():
    # 65 K pairs need more shared memory than a CTA has: refused on the host, and the next call is not blamed for it
    buf = u.Buffer(None, u.CamConfig(num_experts=16, max_tokens=8192, hidden=128, topk=8, ll_max_tokens=8192, timeout_ms=2000.0),
                   device=DEV, rank=0, num_ranks=1)
    with pytest.raises(RuntimeError, match="does not fit"):
        _low_latency(buf, 8192, 128, 16, 8, 0, seed=0)
    ops.get_dispatch_layout(torch.zeros(4, 2, dtype=torch.int64, device=DEV), 16, 1)
    _low_latency(buf, 8, 128, 16, 8, 0, seed=1)
    buf.destroy()


def test_low_latency_rows_past_the_outputs_are_reported():
    # rank 0 has 2 tokens, so its outputs hold 2 x 2 rows; rank 1 sends it 8 more than that
    tokens, e, h = (2, 8), 2, 128
    bufs = u.Buffer.virtual(2, u.CamConfig(num_experts=e, max_tokens=8, hidden=h, topk=1, ll_max_tokens=8, timeout_ms=2000.0),
                            DEV, name="past_")
    x = [torch.randn(t, h, generator=torch.Generator().manual_seed(t)).to(torch.bfloat16) for t in tokens]
    idx = [torch.zeros(t, 1, dtype=torch.int32, device=DEV) for t in tokens]

    def disp(r):
        return ops.moe_dispatch_shmem(x[r].to(DEV), idx[r], None, None, 2, r, e, 1, 0, 0, 0, 0, 0, 0, 1, bufs[r].handle)

    res = run_virtual(disp, 2, masks=(PHASE_SEND, PHASE_RECV))
    assert res[0][0].shape[0] == 4 and torch.equal(res[0][0].cpu(), torch.cat(x)[:4])
    with pytest.raises(u.CamError) as ei:
        bufs[0].check()
    assert ei.value.who == 5 and ei.value.detail == 10  # the rows there were
    bufs[1].check()
    for b in bufs:
        b.destroy()
