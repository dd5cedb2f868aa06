"""Replayed session runs whose independent linears are branches of the captured graph: the same bits as launches one after another, on the
session's own stream and on others, with new inputs in the same buffers, and in order where a result is written twice."""
import pytest
import torch

import dinoml_v2_b200 as dml
from dinoml_v2_b200 import synthetic
from dinoml_v2_b200.constant_sources import GGUFConstant

pytestmark = pytest.mark.gpu
H, KV, F = 1024, 256, 2816


class Layer(dml.Module):
    def __init__(self):
        self.q, self.k, self.v = (dml.Parameter([n, H], dtype="bfloat16") for n in (H, KV, KV))
        self.gate, self.up, self.down = dml.Parameter([F, H], dtype="bfloat16"), dml.Parameter([F, H], dtype="bfloat16"), dml.Parameter([H, F], dtype="bfloat16")

    def forward(self, x, y):
        ops = dml.ops
        return [ops.gemm_rcr(x, self.q), ops.gemm_rcr(x, self.k), ops.gemm_rcr(x, self.v), ops.gemm_rcr(ops.dual_gemm_rcr_silu(y, self.gate, self.up), self.down)]


@pytest.fixture(scope="module")
def module(tmp_path_factory):
    shapes = {"q": (H, H), "k": (KV, H), "v": (KV, H), "gate": (F, H), "up": (F, H), "down": (H, F)}
    constants = {name: GGUFConstant.from_blocks(synthetic.random_blocks("Q6_K" if name == "down" else "Q4_K", n, k, seed=i), "Q6_K" if name == "down" else "Q4_K",
                                                (n, k), tensor=name) for i, (name, (n, k)) in enumerate(shapes.items())}
    tokens = dml.Dim("tokens", 1, 256)
    spec = dml.trace(Layer(), inputs={name: dml.TensorSpec([tokens, H], "bfloat16") for name in ("x", "y")}, constants=constants)
    loaded = dml.runtime.load(dml.compile(spec, dml.Target("cuda"), str(tmp_path_factory.mktemp("layer"))).path)
    loaded.load_encoded_constants()
    return loaded


def _inputs(m, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return {name: (torch.randn(m, H, device="cuda", generator=g) * H ** -0.5).bfloat16() for name in ("x", "y")}


def _outputs(module, m):
    return {o["name"]: torch.zeros(m, n, device="cuda", dtype=torch.bfloat16) for o, n in zip(module.metadata["outputs"], (H, KV, KV, H))}


@pytest.mark.parametrize("m", [1, 2, 5, 17, 64, 128, 129])       # the last one is above the row limit: one after another
def test_same_bits_as_in_order(module, m):
    plain, replayed = module.create_session(), module.create_session()
    replayed.set_graph_replay(True)
    x, want, got = _inputs(m, 0), _outputs(module, m), _outputs(module, m)
    for step in range(5):
        fresh = _inputs(m, 10 * m + step)
        for name in x:
            x[name].copy_(fresh[name])
        plain.run_torch(x, want)
        stream = torch.cuda.Stream() if step == 4 else torch.cuda.current_stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            replayed.run_torch(x, got)
        torch.cuda.current_stream().wait_stream(stream)
        torch.cuda.synchronize()
        for name in want:
            assert torch.equal(want[name].view(torch.int16), got[name].view(torch.int16)), (m, step, name)


def test_results_in_one_buffer_keep_their_order(module):
    """k and v written to the same memory: the later one stays, in every run."""
    m = 4
    plain, replayed = module.create_session(), module.create_session()
    replayed.set_graph_replay(True)
    x, want, got = _inputs(m, 3), _outputs(module, m), _outputs(module, m)
    plain.run_torch(x, want)
    names = [o["name"] for o in module.metadata["outputs"]]
    got[names[1]] = got[names[2]]
    for _ in range(20):
        got[names[2]].zero_()
        replayed.run_torch(x, got)
        torch.cuda.synchronize()
        assert torch.equal(want[names[2]].view(torch.int16), got[names[2]].view(torch.int16))
