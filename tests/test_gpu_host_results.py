"""`Session.run_numpy` results: kept ones stay as they were, dropped ones give their memory back, at each way a result reaches the host
(a copy of at most 64 KB, loans the kernels store into, loans the copy engine fills, copies once the loans are out)."""
import numpy as np
import pytest

import dinoml_v2_b200 as dml
import oracle
from dinoml_v2_b200 import gguf_file, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,m,n", [("float16", 3, 512), ("float16", 9, 8192), ("bfloat16", 9, 8192), ("float32", 5, 4104), ("float16", 260, 8208)])
def test_kept_results(tmp_path, dtype, m, n):
    k = 512
    blocks = S.random_blocks("Q4_K", n, k, 7)
    gguf_file.write_gguf(tmp_path / "w.gguf", {"w": ("Q4_K", (n, k), blocks)})
    spec = dml.trace(dml.nn.Linear(k, n, bias=False, dtype=dtype), inputs={"x": dml.TensorSpec([dml.Dim("m", 1, 512, buckets=(1, 512)), k], dtype)},
                     constants={"weight": dml.gguf_constant(tmp_path / "w.gguf", "w")})
    module = dml.runtime.load(dml.compile(spec, dml.Target("cuda"), tmp_path / "art").path)
    module.load_encoded_constants()
    session = module.create_session()
    np_dtype = np.float16 if dtype == "float16" else np.float32
    xs = [S.random_activations(m, k, 20 + i, "float32").astype(np_dtype) for i in range(8)]
    kept = [session.run_numpy({"x": x})["t0"] for x in xs]
    first = [y.copy() for y in kept]
    again = [session.run_numpy({"x": x})["t0"] for x in reversed(xs)][::-1]       # more than can be lent
    for i, x in enumerate(xs):
        assert kept[i].dtype == np_dtype and kept[i].shape == (m, n) and kept[i].flags.writeable
        assert np.array_equal(kept[i], first[i]) and np.array_equal(again[i], first[i])
    x0 = S.bf16_bits_to_float32(S.float32_to_bf16_bits(xs[0])) if dtype == "bfloat16" else xs[0].astype(np.float32)
    ref = oracle.gemm_quant(x0[:2], blocks, "Q4_K", n, k)
    assert oracle.max_errors(ref, kept[0][:2].astype(np.float32))[2] <= (2e-2 if dtype == "bfloat16" else 1e-3)
    kept[1][...] = 0                                                              # the caller's to write
    del again
    kept = kept[-1:]
    seen = set()
    for _ in range(12):                                                           # a loop that drops its results reuses their memory
        y = session.run_numpy({"x": xs[0]})["t0"]
        seen.add(y.ctypes.data)
        assert np.array_equal(y, first[0])
    assert np.array_equal(kept[0], first[-1])
    if y.nbytes > 65536:                                                          # smaller results are copies, at addresses of malloc's choice
        assert len(seen) <= 8
    session.close()
    module.close()
    assert np.array_equal(y, first[0]) and np.array_equal(kept[0], first[-1])     # results outlive their session
