"""The ways in which the tcgen05 GEMMs cut their work: K slices in clusters, whole tiles and stream-K, with two CTAs per SM, one, and pairs
of them, at the edges of tiles and of the super-blocks that two teams of producers share.

Reference: float64 products with the dequantizer's weights.  Bounds are for the largest difference over the largest result, in roundings u
of the 16-bit type (2^-9 / 2^-11 of a value): a split operand holds the weight, which leaves the rounding of the output, 2 u with the tensor
cores' sums; an ordinary operand is the product of a rounded scale plus a rounded min, rounded again, so three more, independent from
weight to weight: the error of a sum is to the sum as that of one operand, whose scale and min terms are up to twice the weight: 2 u + 6 u."""
import pytest
import torch

from dinoml_v2_b200 import kernels
from dinoml_v2_b200 import synthetic as S

pytestmark = pytest.mark.gpu
TYPES = ["Q4_K", "Q6_K", "Q8_0", "Q5_K", "Q4_0", "Q2_K", "Q3_K", "MXFP4", "NVFP4"]
U = {"bfloat16": 2.0 ** -9, "float16": 2.0 ** -11}
# (m, n, k): two CTAs per SM: slices of 8 / 4 / 3 / 2, whole tiles, stream-K; sixteen warps: slices, whole, stream-K, teams that share
# super-blocks and teams that take turns; pairs: slices of 4 / 2, whole tiles, stream-K with an odd number of tiles
SHAPES = [(9, 130, 4096), (33, 4100, 4096), (64, 11000, 2048), (17, 14400, 2048), (40, 36000, 2048), (16, 20500, 4096),
          (65, 1000, 4096), (128, 520, 14336), (100, 11000, 4096), (100, 9700, 6144), (70, 19500, 4096),
          (129, 300, 4096), (200, 1500, 6144), (250, 4090, 2048), (257, 9000, 4096), (600, 5000, 4096), (300, 19000, 2048)]


def _case(qtype, dtype, m, n, k):
    dev = torch.device("cuda:0")
    w = S.random_blocks_torch(qtype, n, k, m + n, dev)
    x = torch.randn(m, k, device=dev, generator=torch.Generator(device=dev).manual_seed(m)).to(getattr(torch, dtype))
    return x, w, kernels.dequantize_rows(w, qtype, k, "float32").double()


def _close(got, ref, dtype, roundings):
    assert kernels.device_status() == 0
    err = ((got.double() - ref).abs().max() / ref.abs().max()).item()
    assert err <= roundings * U[dtype], err


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("qtype", TYPES)
def test_work_cuts(qtype, dtype):
    for m, n, k in SHAPES if qtype in ("Q4_K", "Q6_K", "Q8_0") else SHAPES[::3]:
        x, w, wd = _case(qtype, dtype, m, n, k)
        bias = torch.randn(n, device=x.device).to(x.dtype)
        ref = x.double() @ wd.T + bias.double()
        y = kernels.gemm_rcr(x, w, qtype, bias, variant="umma")
        _close(y, ref, dtype, 8)
        assert torch.equal(y.view(torch.int16), kernels.gemm_rcr(x, w, qtype, bias, variant="umma").view(torch.int16))      # one order of sums


@pytest.mark.parametrize("m,n,k", [(16, 2048, 4096), (64, 22016, 2048), (100, 1024, 4096), (200, 1024, 4096), (333, 8192, 2048), (300, 19008, 2048)])
def test_gated_cuts(m, n, k):
    x, w, wd = _case("Q4_K", "bfloat16", m, n, k)
    x = (x * k ** -0.5).contiguous()
    both = (x.double() @ wd.T).view(m, n // 16, 2, 8)
    ref = (torch.nn.functional.silu(both[:, :, 0]) * both[:, :, 1]).reshape(m, n // 2)
    _close(kernels.dual_gemm_rcr(x, w, "Q4_K", "silu"), ref, "bfloat16", 8)


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("qtype,k", [("Q6_K", 4352), ("Q8_0", 2080), ("Q4_0", 4128), ("MXFP4", 2880), ("NVFP4", 2880), ("Q3_K", 2560), ("Q2_K", 2816)])
def test_split_cuts(qtype, k, dtype):
    """Ragged weight rows: one to three terms per weight, rings shorter than a super-block."""
    for m, n in ((24, 5000), (64, 2100), (100, 5000), (128, 19500), (129, 1000), (257, 5003), (300, 19000)):
        x, w, wd = _case(qtype, dtype, m, n, k)
        _close(kernels.gemm_rcr(x, w, qtype), x.double() @ wd.T, dtype, 2)


@pytest.mark.parametrize("qtype,m,n,k", [("Q4_K", 16, 100, 256 * 2400), ("Q4_0", 24, 100, 256 * 1200 + 32)])
def test_a_tile_in_more_pieces_than_producer_threads(qtype, m, n, k):
    """One tile of a very long K over all SMs, two CTAs each: 296 pieces, and 256 threads that look after them.  (Ordinary and split operands.)"""
    x, w, wd = _case(qtype, "bfloat16", m, n, k)
    ref = x.double() @ wd.T
    del wd
    variant = "umma" if k % 256 == 0 else "auto"
    results = [kernels.gemm_rcr(x, w, qtype, variant=variant) for _ in range(4)]          # a flag that stayed up would reach the next launch
    for y in results:
        _close(y, ref, "bfloat16", 8)
        assert torch.equal(y.view(torch.int16), results[0].view(torch.int16))


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("qtype,k", [("Q6_K", 2816), ("Q2_K", 2816), ("Q3_K", 2560), ("Q8_0", 2080)])
def test_split_few_weight_tiles_of_many_rows(qtype, k, dtype):
    """More than 128 rows against one to a few weight tiles: several tiles of at most 128 rows instead of pairs, the last of them ragged."""
    for m, n in ((129, 1), (200, 300), (257, 130), (700, 1000), (1025, 512)):
        x, w, wd = _case(qtype, dtype, m, n, k)
        _close(kernels.gemm_rcr(x, w, qtype), x.double() @ wd.T, dtype, 2)


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("k", [256, 512, 1280, 2304])
def test_q8_0_super_blocks_of_teams(k, dtype):
    """A slot holds a whole Q8_0 super-block: one per CTA, which both teams take, odd numbers that they take in turns, laps of rings of four and of two."""
    for m, n in ((16, 129), (64, 20000), (65, 4100), (128, 40000), (129, 130), (260, 20000)):
        x, w, wd = _case("Q8_0", dtype, m, n, k)
        _close(kernels.gemm_rcr(x, w, "Q8_0", variant="umma"), x.double() @ wd.T, dtype, 8)
