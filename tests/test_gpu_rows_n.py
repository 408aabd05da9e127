"""GPU tests of the grouped GEMM whose rows are the tensor core's N operand (CTA pairs), in its three arithmetics, against the
CPU oracle: expert sizes round the steps of its tiles, weight blocks that do not fill the last tile, short reductions.  The int8
tests run the one-CTA kernel as well, and the last test compares the two on either side of the lines between them."""
import pytest
import test_gpu_gemm_fused as layer_tests
import torch

import umdk_original_b200 as u  # noqa: F401
from umdk_original_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
ops = torch.ops.umdk_cam_op_lib
DEV = torch.device("cuda", 0)

# rows per expert: one; none; a step of 16 or 32 rows, one more; one tile of 128, 224 or 256 rows, one more; several tiles
COUNTS = [[1], [0, 16, 17, 0, 31, 33], [127, 128, 129], [223, 0, 224, 225], [255, 256, 257], [3, 700, 5]]
# (N, K): blocks of 128 weight rows 1, 3, 4, 10; K-blocks 1, 4, 5, 9
SHAPES = [(128, 128), (384, 512), (512, 640), (1280, 1152)]


@pytest.fixture(autouse=True)
def _form(monkeypatch):
    monkeypatch.setenv("UMDK_CAM_GEMM_PAIR", "0")
    monkeypatch.setenv("UMDK_CAM_GEMM_SWAP", "1")


def _fp8_problem(counts, n, k, po2):
    g = torch.Generator().manual_seed(sum(counts) + n + k)
    # rows and weight blocks of very different magnitude, so that a misplaced scale shows
    a = torch.randn(sum(counts), k, generator=g) * torch.exp(torch.randn(sum(counts), 1, generator=g) * 2.0)
    w = torch.randn(len(counts), n // 128, 128, k // 128, 128, generator=g) * 0.05
    w = (w * torch.exp(torch.randn(len(counts), n // 128, 1, k // 128, 1, generator=g))).reshape(len(counts), n, k)
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    return (*ref.quant_fp8_1x128(a, po2), *ref.quant_fp8_128x128(w, po2), off)


def _row_error(got, want):
    return ((got - want).abs() / (want.abs().amax(dim=1, keepdim=True) + 1e-6)).max().item()


@pytest.mark.parametrize("po2", [False, True])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("counts", COUNTS)
def test_plain(counts, n, k, po2):
    p = _fp8_problem(counts, n, k, po2)
    got = ops.grouped_gemm_fp8(*[t.to(DEV) for t in p], po2).cpu().float()
    # both sides round fp32 sums to bf16; sums that differ in their last bits round apart by one step where a tie lies between
    # them, and a bf16 step is at most 2^-7 of the value (8 significant bits), of the row's largest at most
    assert _row_error(got, ops.grouped_gemm_fp8(*p, po2).float()) <= 2.0 ** -7


@pytest.mark.parametrize("po2", [False, True])
@pytest.mark.parametrize("inter,k", [(128, 128), (384, 512), (640, 1152)])
@pytest.mark.parametrize("counts", COUNTS)
def test_swiglu_requant(counts, inter, k, po2):
    p = _fp8_problem(counts, 2 * inter, k, po2)
    q, s = ops.grouped_gemm_fp8_swiglu(*[t.to(DEV) for t in p], po2)
    qc, sc = ops.grouped_gemm_fp8_swiglu(*p, po2)
    got, want = ref.dequant_fp8_1x128(q.cpu(), s.cpu()), ref.dequant_fp8_1x128(qc, sc)
    # a value on a rounding boundary lands one e4m3 step (1/8 of it) apart, a block whose amax / 448 sits on a power of two
    # takes the next scale, which moves its values by at most half a step of the coarser one
    assert _row_error(got, want) <= 0.14
    ratio = s.cpu() / sc
    assert ((ratio - 1).abs() < 1e-4).float().mean() > (0.98 if po2 else 0.999)


@pytest.mark.parametrize("swap", ["0", "1"])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("counts", COUNTS)
def test_int8(counts, n, k, swap, monkeypatch):
    monkeypatch.setenv("UMDK_CAM_GEMM_SWAP", swap)
    g = torch.Generator().manual_seed(sum(counts) + n + k)
    a = torch.randint(-127, 128, (sum(counts), k), generator=g).to(torch.int8)
    w = torch.randint(-127, 128, (len(counts), n, k), generator=g).to(torch.int8)
    a_s, w_s = torch.rand(sum(counts), generator=g) + 0.01, torch.rand(len(counts), n, generator=g) + 0.01
    off = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32)
    p = (a, a_s, w, w_s, off)
    got = ops.grouped_gemm_w8a8(*[t.to(DEV) for t in p]).cpu().float()
    want = ops.grouped_gemm_w8a8(*p).float()
    # exact integers, two fp32 products, one bf16 rounding: at most one bf16 step
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs()).all()


@pytest.mark.parametrize("swap", ["0", "1"])
@pytest.mark.parametrize("world", [1, 2])
def test_int8_layer(world, swap, monkeypatch):
    monkeypatch.setenv("UMDK_CAM_GEMM_SWAP", swap)
    layer_tests.test_fused_moe_w8a8_reference_layout(world)


@pytest.mark.parametrize("e,n,k,rows", [
    (30, 4096, 1536, 3), (31, 4096, 1536, 3),     # 189 and 195 MB of weights
    (31, 3968, 1536, 65), (32, 4096, 1536, 113),  # 6.1 M weights per expert and the full 128-row tiles; past them
    (47, 1024, 6144, 2), (48, 1024, 6144, 2),     # 94 and 96 tiles
    (40, 1536, 3840, 2)])                         # 5.9 M weights per expert
def test_the_choice_changes_no_byte(e, n, k, rows, monkeypatch):
    # int8 sums are exact and the scales are applied in one order, so both forms and the default give the same bytes
    g = torch.Generator(device=DEV).manual_seed(e + n)
    a = torch.randint(-127, 128, (e * rows, k), device=DEV, generator=g).to(torch.int8)
    w = torch.randint(-127, 128, (e, n, k), device=DEV, generator=g, dtype=torch.int8)
    a_s, w_s = torch.rand(e * rows, device=DEV, generator=g) + 0.01, torch.rand(e, n, device=DEV, generator=g) + 0.01
    off = torch.arange(0, e * rows + 1, rows, dtype=torch.int32, device=DEV)
    got = {}
    for swap in ("", "0", "1"):
        monkeypatch.setenv("UMDK_CAM_GEMM_SWAP", swap)
        got[swap] = ops.grouped_gemm_w8a8(a, a_s, w, w_s, off).view(torch.int16)
    assert torch.equal(got[""], got["0"]) and torch.equal(got[""], got["1"])
    last = slice((e - 1) * rows, e * rows)
    want = (a[last].double() @ w[e - 1].double().t()).float() * a_s[last, None] * w_s[e - 1]
    assert torch.equal(got[""][last], want.to(torch.bfloat16).view(torch.int16))
