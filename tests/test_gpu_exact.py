"""The exact tensor-core GEMM behind the simt family, from three activation rows on: tiles that are not full in either direction, K of one
block up to several super-blocks with a remainder, rows at every 16-byte phase, K cut across a cluster.  Against the float64 product."""
import numpy as np
import pytest
import torch

import oracle
from dinoml_v2_b200 import kernels, synthetic as S
from dinoml_v2_b200.gguf_blocks import QTYPES

pytestmark = pytest.mark.gpu
TDT = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
BOUND = {"float16": 6e-4, "bfloat16": 4e-3, "float32": 2e-6}          # output rounding; float32: the sums


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("qtype,k", [("Q8_0", 288), ("Q6_K", 2816), ("Q4_0", 2880), ("Q2_K", 1280), ("Q3_K", 2560), ("MXFP4", 2848), ("MXFP4", 2880), ("NVFP4", 2880)])
def test_split_operands(qtype, k, dtype):
    """The tcgen05 kernel with split weights: full and last tiles of 128 rows, one and more activation tiles, rows of every residue."""
    dev = torch.device("cuda:0")
    for n, m in ((1, 129), (128, 160), (301, 257), (4099, 24)):
        blocks = S.random_blocks(qtype, n, k, seed=n + k)
        x = torch.from_numpy(S.random_activations(m, k, 7, "float32")).to(dev).to(TDT[dtype])
        bias = torch.randn(n, device=dev).to(TDT[dtype])
        ref = x.double().cpu().numpy() @ oracle.dequantize(blocks, qtype, k).astype(np.float64).T + bias.double().cpu().numpy()
        y = kernels.gemm_rcr(x, torch.from_numpy(blocks).to(dev), qtype, bias)
        assert kernels.device_status() == 0
        _, _, norm = oracle.max_errors(ref, y.float().cpu().numpy())
        assert norm <= BOUND[dtype], (n, m, norm)


@pytest.mark.parametrize("dtype", sorted(TDT))
@pytest.mark.parametrize("qtype", sorted(QTYPES))
def test_edges(qtype, dtype):
    dev = torch.device("cuda:0")
    block = QTYPES[qtype].block_size
    for k in (block, 768, 1280 + (block if block < 256 else 0)):
        for n, m in ((1, 3), (65, 33), (300, 70), (4097, 130)):
            blocks = S.random_blocks(qtype, n, k, seed=n + k)
            x = torch.from_numpy(S.random_activations(m, k, 7, "float32")).to(dev).to(TDT[dtype])
            bias = torch.randn(n, device=dev).to(TDT[dtype])
            ref = x.double().cpu().numpy() @ oracle.dequantize(blocks, qtype, k).astype(np.float64).T + bias.double().cpu().numpy()
            y = kernels.gemm_rcr(x, torch.from_numpy(blocks).to(dev), qtype, bias, variant="simt")
            assert kernels.device_status() == 0
            _, _, norm = oracle.max_errors(ref, y.float().cpu().numpy())
            assert norm <= BOUND[dtype], (k, n, m, norm)


@pytest.mark.parametrize("dtype", sorted(TDT))
@pytest.mark.parametrize("qtype,k", [("Q8_0", 288), ("Q6_K", 2816), ("Q4_0", 2880), ("Q2_K", 1280), ("Q3_K", 2560), ("MXFP4", 2848), ("NVFP4", 2880),
                                     ("Q4_K", 1280), ("Q5_K", 768)])
def test_infinite_and_huge_activations(qtype, k, dtype):
    """Rows with an Inf, a NaN or values near the end of the type's range get what the products give, the other rows what they had."""
    dev = torch.device("cuda:0")
    n = 40
    blocks = S.random_blocks(qtype, n, k, seed=k)
    w = oracle.dequantize(blocks, qtype, k).astype(np.float64)
    largest = float(torch.finfo(TDT[dtype]).max)
    for m, kind in ((3, ""), (9, ""), (40, ""), (130, ""), (131, "infinite"), (132, "tiny")):        # from 130 with 16-bit activations the tcgen05 kernel
        base = torch.from_numpy(S.random_activations(m, k, 41, "float32")).to(dev).to(TDT[dtype])
        if kind == "infinite":                              # every row at one place, beside the ones below
            base[:, 11] = float("inf")
        elif kind == "tiny" and dtype != "float16":
            base *= 1e-34
        x = base.clone()
        x[0, 5], x[1, k - 1], x[2, k // 2] = float("inf"), float("-inf"), float("nan")
        if m > 3:
            x[m - 1, 7] = 1.0 if kind == "infinite" else largest          # largest x weight + Inf x weight is Inf or NaN with the arithmetic's range
            x[m - 2, 9], x[m - 2, 300 % k] = float("inf"), float("-inf")
            x[3] = base[3] * 1e-36 if dtype != "float16" else 0
        xd = x.double().cpu().numpy()
        with np.errstate(all="ignore"):
            ref = (xd[:, None, :] * w[None]).sum(-1)
            ref[np.abs(ref) > largest] *= np.inf               # results beyond the type
        y = kernels.gemm_rcr(x, torch.from_numpy(blocks).to(dev), qtype, variant="simt").double().cpu().numpy()
        assert kernels.device_status() == 0
        assert np.array_equal(np.isnan(y), np.isnan(ref)), m
        assert np.array_equal(np.where(np.isinf(ref), ref, 0), np.where(np.isinf(y), y, 0)), m
        for r in range(m):
            fine = np.isfinite(ref[r])
            if fine.any():
                assert np.abs(y[r][fine] - ref[r][fine]).max() <= BOUND[dtype] * np.abs(ref[r][fine]).max(), (m, r)


D_AT = {"Q8_0": (34, (0,)), "Q6_K": (210, (208,)), "Q4_0": (18, (0,)), "Q2_K": (84, (80, 82)), "Q3_K": (110, (108,))}


@pytest.mark.parametrize("qtype,k", [("Q8_0", 288), ("Q6_K", 2816), ("Q4_0", 2880), ("Q2_K", 1280), ("Q3_K", 2560), ("MXFP4", 2848)])
def test_float16_scales_of_any_size(qtype, k):
    """Block scales that float16 operands do not hold, beside ones that they do, in the tcgen05 kernel with split weights."""
    dev = torch.device("cuda:0")
    n, m = 40, 260
    blocks = S.random_blocks(qtype, n, k, seed=k)
    if qtype == "MXFP4":
        e = blocks[:, ::17]                             # the exponent byte of every block of a row
        for row, byte in enumerate((127 + 11, 127 + 12, 127 + 20, 127 - 23, 127 - 24, 127 - 30)):
            e[row] = byte
        e[6, 3], e[7, 5] = 127 + 14, 127 - 27           # one block of the row
        for row, byte in ((8, 0), (9, 254)):            # blocks whose weights are zero, with any scale
            for col in range(17 * 4, 17 * 6):
                blocks[row, col] = 0 if col % 17 else byte
    else:
        size, offsets = D_AT[qtype]
        for row, d in enumerate((2000.0, 2100.0, 30000.0, 60000.0, 6e-8, 3e-5)):
            for at in offsets:
                for i, byte in enumerate(np.float16(d).tobytes()):
                    blocks[row, at + i::size] = byte
        blocks[6, offsets[0]:offsets[0] + 2] = np.frombuffer(np.float16(50000.0).tobytes(), np.uint8)      # its first block only
    w = oracle.dequantize(blocks, qtype, k).astype(np.float64)
    x = torch.from_numpy(S.random_activations(m, k, 43, "float32")).to(dev)
    x[: m // 2] *= 2.0 ** -14                           # for results of the large scales, and of the small ones
    x[m // 2:] *= 2.0 ** 12
    x = x.half()
    xd = x.double().cpu().numpy()
    ref = xd @ w.T
    y = kernels.gemm_rcr(x, torch.from_numpy(blocks).to(dev), qtype).double().cpu().numpy()
    assert kernels.device_status() == 0
    # float16 rounding of the result, 1e-5 of the products' magnitudes for the sums, half the smallest float16 step
    bound = 2.0 ** -11 * np.abs(ref) + 1e-5 * (np.abs(xd) @ np.abs(w).T) + 2.0 ** -25
    inside = np.abs(ref) + bound < 65504
    assert inside[:, :8].any(axis=0).all()
    assert (np.abs(y[inside] - ref[inside]) <= bound[inside]).all()
    beyond = np.abs(ref) - bound >= 65520
    assert (np.isinf(y[beyond]) & (np.sign(y[beyond]) == np.sign(ref[beyond]))).all()
