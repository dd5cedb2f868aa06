"""The tcgen05 kernel's scatter epilogues beside the one that joins K slices in a cluster: whole tiles, and tiles finished after a stream-K reduction,
with two CTAs per SM, one, and pairs of them.  All destinations are local buffers."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

from dinoml_v2_b200 import _native, kernels, synthetic as S   # noqa: E402
from dinoml_v2_b200.gguf_blocks import qtype_of                # noqa: E402

pytestmark = pytest.mark.gpu
BF16 = 6


@pytest.mark.parametrize("m,n,k", [(40, 36000, 2048), (16, 20500, 4096), (100, 17000, 4608), (70, 19500, 4096), (250, 9000, 2048), (300, 19000, 2048)])
def test_scatter_of_whole_and_cut_tiles(m, n, k):
    dev = torch.device("cuda:0")
    w = torch.from_numpy(S.random_blocks("Q4_K", n, k, seed=31)).to(dev)
    x = torch.from_numpy(S.random_activations(m, k, 32, "float32")).to(dev).to(torch.bfloat16)
    want = kernels.gemm_rcr(x, w, "Q4_K", variant="umma")
    dst = [torch.full((m, n), float("nan"), device=dev, dtype=torch.bfloat16) for _ in range(3)]
    peers = (ctypes.c_void_p * 2)(dst[1].data_ptr(), dst[2].data_ptr())
    rc = _native.lib().dinoml_b200_gguf_gemm_rcr_scatter(x.data_ptr(), w.data_ptr(), None, dst[0].data_ptr(), peers, 2, qtype_of("Q4_K").value, BF16, m, n, k, 0,
                                                         torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _native.last_error()
    torch.cuda.synchronize()
    assert kernels.device_status() == 0
    for t in dst:
        assert torch.equal(t.view(torch.int16), want.view(torch.int16))
