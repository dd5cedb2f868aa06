"""Every form of the dequantizer against the oracle, bit for bit: nine types, three outputs, packed buffers and outputs at each start that
the entry takes, block counts around a thread block's share (8, 16, 32, 64 or 256 blocks), bytes of every value (so scales of infinity and NaN too),
and nothing written outside the output."""
import numpy as np
import pytest
import torch

import oracle
from dinoml_v2_b200 import kernels
from dinoml_v2_b200.gguf_blocks import qtype_of

pytestmark = pytest.mark.gpu

TYPES = ("Q4_K", "Q6_K", "Q8_0", "Q5_K", "Q4_0", "Q3_K", "Q2_K", "MXFP4", "NVFP4")
ALIGN = {"Q4_K": 4, "Q6_K": 2, "Q8_0": 2}
DTYPES = ("float16", "bfloat16", "float32")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("qtype", TYPES)
def test_starts_and_block_counts(qtype, dtype):
    t, td = qtype_of(qtype), getattr(torch, dtype)
    bits = torch.int32 if dtype == "float32" else torch.int16
    rng = np.random.default_rng(len(qtype))
    for blocks in (1, 2, 7, 8, 9, 31, 33, 63, 65, 257):
        raw = rng.integers(0, 256, (blocks, t.block_bytes), dtype=np.uint8)
        number = ~np.isnan(oracle.dequantize(raw, qtype, t.block_size)).reshape(-1)      # which NaN it is depends on the machine that multiplies
        number = torch.from_numpy(number)
        want = oracle.dequantize(raw, qtype, t.block_size, dtype)
        want = torch.from_numpy(np.ascontiguousarray(want).view(np.int32 if dtype == "float32" else np.int16)).reshape(-1)
        for start in (0, 1, 2, 3, 4, 8, 18):
            if start % ALIGN.get(qtype, 1):
                continue
            store = torch.zeros(start + raw.size, dtype=torch.uint8, device="cuda")
            store[start:].copy_(torch.from_numpy(raw).reshape(-1))
            for skip in (0, 16 // td.itemsize):                 # outputs at a 32-byte boundary and 16 bytes past one
                dense = torch.full((skip + want.numel() + 16,), 7.0, dtype=td, device="cuda")
                y = dense[skip:skip + want.numel()].view(blocks, -1)
                kernels.dequantize_rows(store[start:].view(blocks, -1), qtype, t.block_size, dtype, out=y)
                got = y.reshape(-1).view(bits).cpu()
                assert torch.equal(~torch.isnan(y.reshape(-1).cpu()), number)
                assert torch.equal(got[number], want[number])
                assert bool((dense[:skip] == 7).all()) and bool((dense[skip + want.numel():] == 7).all())


def test_behind_kernels_that_write_its_input_and_before_ones_that_read_its_output():
    """The launch may begin before the kernel in front of it has ended: it reads nothing of it before."""
    k, n = 4096, 512
    rng = np.random.default_rng(3)
    packed = [torch.from_numpy(rng.integers(0, 120, (n, k // 256 * 144), dtype=np.uint8)).cuda() for _ in range(4)]
    want = [kernels.dequantize_rows(p, "Q4_K", k, "float32") for p in packed]
    work, out = torch.empty_like(packed[0]), torch.empty(n, k, device="cuda")
    sums = []
    for i in range(40):
        work.copy_(packed[i % 4])
        kernels.dequantize_rows(work, "Q4_K", k, "float32", out=out)
        sums.append(out.clone())
        kernels.dequantize_rows(work, "Q4_K", k, "float32", out=out)
    for i, s in enumerate(sums):
        assert torch.equal(s.view(torch.int32), want[i % 4].view(torch.int32))
    assert torch.equal(out.view(torch.int32), want[39 % 4].view(torch.int32))
