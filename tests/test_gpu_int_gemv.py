"""The decode GEMV with byte operands (one and two activation rows) at the sizes where it can go wrong: fewer rows than a tile, a
tile cut between two CTAs, K from one super-block to the lengths that are cut into slices, weight rows that are not 16-byte
multiples, a last super-block that is not full, activations of very different size.  Against the float64 product of the dequantized weights."""
import numpy as np
import pytest
import torch

import oracle
from dinoml_v2_b200 import kernels, synthetic as S

pytestmark = pytest.mark.gpu
TDT = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
BOUND = {"float16": 6e-4, "bfloat16": 4e-3, "float32": 2e-6}          # output rounding; float32: the sums
KS = {"Q4_K": (256, 4096, 20480), "Q5_K": (2304, 14336), "Q6_K": (256, 768, 11008, 20480), "Q8_0": (32, 288, 2048, 14336),
      "Q4_0": (96, 2880, 4096), "Q2_K": (256, 1280, 4096), "Q3_K": (256, 2560, 4096)}


def _check(x, blocks, qtype, k, dtype, dev):
    y = kernels.gemm_rcr(x, torch.from_numpy(blocks).to(dev), qtype)
    assert kernels.device_status() == 0
    ref = x.double().cpu().numpy() @ oracle.dequantize(blocks, qtype, k).astype(np.float64).T
    _, _, norm = oracle.max_errors(ref, y.float().cpu().numpy())
    assert norm <= BOUND[dtype], norm


@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("dtype", sorted(TDT))
@pytest.mark.parametrize("qtype", sorted(KS))
def test_edges(qtype, dtype, m):
    dev = torch.device("cuda:0")
    for k in KS[qtype]:
        for n in (1, 17, 4800 if k <= 4096 else 400):         # 4800: a few tiles more than CTAs
            x = torch.from_numpy(S.random_activations(m, k, 11, "float32")).to(dev).to(TDT[dtype])
            _check(x, S.random_blocks(qtype, n, k, seed=n + k), qtype, k, dtype, dev)


@pytest.mark.parametrize("qtype", ["Q4_K", "Q6_K", "Q8_0"])
def test_range_of_the_activations(qtype):
    """Zeros, tiny and huge values in one row: the digits are relative to the largest of a super-block, results to the largest result."""
    dev = torch.device("cuda:0")
    k, n = 1024, 64
    x = torch.zeros(2, k, device=dev)
    x[0, ::7] = 1e-30
    x[0, 300] = 3.0
    x[1, 256:512] = torch.randn(256, device=dev) * 1e20
    x[1, 600:700] = 1e-3
    _check(x, S.random_blocks(qtype, n, k, seed=5), qtype, k, "float32", dev)
    x[1, 5] = float("inf")
    y = kernels.gemm_rcr(x, torch.from_numpy(S.random_blocks(qtype, n, k, seed=5)).to(dev), qtype)
    assert torch.isfinite(y[0]).all() and not torch.isfinite(y[1]).any()


@pytest.mark.parametrize("dtype", sorted(TDT))
@pytest.mark.parametrize("qtype", sorted(KS))
def test_values_without_planes(qtype, dtype):
    """Infinities, NaN and (where the type has them) values near the ends of its range: what the products give, for each row by itself."""
    dev = torch.device("cuda:0")
    n = 40
    for k in KS[qtype]:
        blocks = S.random_blocks(qtype, n, k, seed=k)
        w = oracle.dequantize(blocks, qtype, k).astype(np.float64)
        variants = ["simt"] + (["stream"] if dtype != "float32" and kernels.variant_supports("stream", qtype, dtype, 2, n, k) else [])
        special = [(3, np.inf), (k - 1, -np.inf), (k // 2, np.nan)]
        if dtype != "float16":
            special += [(5, 1e36), (k - 2, -1e37)]                # times weights below 20: results below 3.4e38
            assert np.abs(w).max() < 20
        base = S.random_activations(2, k, 31, "float32")
        for at, value in special + [(slice(None), 0.0)] + ([(slice(0, 256), 1e-34)] if dtype != "float16" else []):
            x = base.copy()
            x[0, at] = value
            if value == 1e-34:
                x[0] = 1e-34 * base[0]
            for rows in (x[:1], x):
                xt = torch.from_numpy(rows).to(dev).to(TDT[dtype])
                xd = xt.double().cpu().numpy()
                with np.errstate(all="ignore"):
                    ref = (xd[:, None, :] * w[None]).sum(-1)
                for variant in variants:
                    y = kernels.gemm_rcr(xt, torch.from_numpy(blocks).to(dev), qtype, variant=variant).double().cpu().numpy()
                    assert kernels.device_status() == 0
                    assert np.array_equal(np.isnan(y), np.isnan(ref)), (k, at, value, variant)
                    assert np.array_equal(np.where(np.isinf(ref), ref, 0), np.where(np.isinf(y), y, 0)), (k, at, value, variant)
                    for r in range(len(rows)):
                        if np.isfinite(ref[r]).all():
                            largest = np.abs(ref[r]).max()
                            assert np.abs(y[r] - ref[r]).max() <= BOUND[dtype] * largest, (k, at, value, variant, r)


def _zero_weights(blocks, qtype, k, columns):
    """Quants of these columns -> the value that stands for a weight of zero (types without mins)."""
    for col in columns:
        sb, i = col // 256, col % 256
        half, quad, l = i // 128, i % 128 // 32, i % 32
        if qtype == "Q8_0":
            blocks[:, 34 * (col // 32) + 2 + col % 32] = 0
        elif qtype == "Q4_0":
            at, high = 18 * (col // 32) + 2 + col % 16, col % 32 >= 16
            blocks[:, at] = (blocks[:, at] & (0x0F if high else 0xF0)) | (0x80 if high else 0x08)
        elif qtype == "Q6_K":                             # 32 = low nibble 0, high two bits 2
            at = 210 * sb + 64 * half + 32 * (quad & 1) + l
            blocks[:, at] &= 0x0F if quad >= 2 else 0xF0
            at = 210 * sb + 128 + 32 * half + l
            blocks[:, at] = (blocks[:, at] & (0xFF ^ (3 << (2 * quad)))) | (2 << (2 * quad))
        else:                                             # Q3_K: 4 = low bits 0, mask bit 1
            blocks[:, 110 * sb + 32 + 32 * half + l] &= 0xFF ^ (3 << (2 * quad))
            blocks[:, 110 * sb + l] |= 1 << (4 * half + quad)
    return blocks


@pytest.mark.parametrize("dtype", sorted(TDT))
@pytest.mark.parametrize("qtype", ["Q8_0", "Q6_K", "Q4_0", "Q3_K"])
def test_outliers_on_zero_weights(qtype, dtype):
    """Channels whose activations are 2^s times the others' and whose weights are zero: what is left in the result keeps the accuracy that
    it has without them.  One such channel per super-block, or every other one."""
    dev = torch.device("cuda:0")
    n, k = 300, 2048
    for columns in (range(37, k, 256), range(1, k, 2)):
        blocks = _zero_weights(S.random_blocks(qtype, n, k, seed=9), qtype, k, columns)
        w = oracle.dequantize(blocks, qtype, k).astype(np.float64)
        assert not w[:, list(columns)].any() and w.any()
        for s in (4, 6, 7, 8, 10, 12, 15, 20, 26, 40):
            x = S.random_activations(2, k, 12, "float32")
            shrink = 2.0 ** -20 if dtype == "float16" and s > 12 else 1.0        # keeps 2^s times a value in range
            if dtype == "float16" and s > 20:
                continue
            x *= shrink ** 0.5
            x[:, list(columns)] *= 2.0 ** s
            xt = torch.from_numpy(x).to(dev).to(TDT[dtype])
            ref = xt.double().cpu().numpy() @ w.T
            for m in (1, 2):
                for variant in ["simt"] + (["stream"] if kernels.variant_supports("stream", qtype, dtype, m, n, k) else []):
                    y = kernels.gemm_rcr(xt[:m].contiguous(), torch.from_numpy(blocks).to(dev), qtype, variant=variant)
                    assert kernels.device_status() == 0
                    _, _, norm = oracle.max_errors(ref[:m], y.float().cpu().numpy())
                    # float16 results of 2^-10 and less: their spacing is 2^-24 at least
                    floor = 2.0 ** -25 / np.abs(ref[:m]).max() if dtype == "float16" else 0.0
                    assert norm <= BOUND[dtype] + floor, (len(columns), s, m, variant, norm)
