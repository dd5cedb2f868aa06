"""Q4_K dequantization from packed buffers at every start the entry takes: 16-byte loads, word loads, and one block as the smallest."""
import numpy as np
import pytest
import torch

import oracle
from dinoml_v2_b200 import kernels, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("offset", [0, 4, 8, 16])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_start_of_the_packed_buffer(n, offset, dtype):
    blocks = S.random_blocks("Q4_K", n, 256, seed=n)
    store = torch.zeros(offset + blocks.size, dtype=torch.uint8, device="cuda")
    packed = store[offset:]
    packed.copy_(torch.from_numpy(np.ascontiguousarray(blocks).reshape(-1)))
    y = kernels.dequantize_rows(packed.view(n, -1), "Q4_K", 256, dtype)
    ref = torch.from_numpy(oracle.dequantize(blocks, "Q4_K", 256)).to(y.dtype)
    assert torch.equal(y.cpu().view(torch.int16).reshape(-1), ref.view(torch.int16).reshape(-1))
