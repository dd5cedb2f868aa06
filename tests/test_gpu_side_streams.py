"""Graphs with branches on streams of the caller: runs on two streams that nothing orders, and sessions that are dropped right behind their last run,
give the bits of launches one after another."""
import ctypes

import pytest
import torch

import dinoml_v2_b200 as dml
from dinoml_v2_b200 import kernels, synthetic
from dinoml_v2_b200.constant_sources import GGUFConstant

pytestmark = pytest.mark.gpu
K, ROWS = 2048, {"q": 2048, "k": 500, "v": 512}


class Projections(dml.Module):
    """No temporary: runs of one session on different streams share no buffer."""

    def __init__(self):
        self.q, self.k, self.v = (dml.Parameter([n, K], dtype="bfloat16") for n in ROWS.values())

    def forward(self, x):
        return [dml.ops.gemm_rcr(x, w) for w in (self.q, self.k, self.v)]


@pytest.fixture(scope="module")
def module(tmp_path_factory):
    constants = {name: GGUFConstant.from_blocks(synthetic.random_blocks("Q4_K", n, K, seed=i), "Q4_K", (n, K), tensor=name) for i, (name, n) in enumerate(ROWS.items())}
    spec = dml.trace(Projections(), inputs={"x": dml.TensorSpec([dml.Dim("tokens", 1, 256), K], "bfloat16")}, constants=constants)
    loaded = dml.runtime.load(dml.compile(spec, dml.Target("cuda"), str(tmp_path_factory.mktemp("projections"))).path)
    loaded.load_encoded_constants()
    return loaded


def _buffers(module, m, seed):
    """Inputs, results of launches in order, room for other results."""
    x = {"x": torch.randn(m, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).bfloat16()}
    want, got = ({o["name"]: torch.zeros(m, n, device="cuda", dtype=torch.bfloat16) for o, n in zip(module.metadata["outputs"], ROWS.values())} for _ in range(2))
    torch.cuda.synchronize()
    module.create_session().run_torch(x, want)
    return x, want, got


def _same(want, got):
    return all(torch.equal(want[name].view(torch.int16), got[name].view(torch.int16)) for name in want)


@pytest.mark.parametrize("m", [1, 17, 128])
def test_two_streams_that_nothing_orders(module, m):
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    sets = [_buffers(module, m, 40 + i) for i in range(2)]
    session = module.create_session()
    session.set_graph_replay(True)
    for step in range(40):
        for stream, (x, want, got) in zip(streams, sets):
            session.set_stream(stream.cuda_stream)
            session.run_torch(x, got)
    torch.cuda.synchronize()
    assert session.graph_stats() == {"cached_graphs": 2, "graph_launches": 2 * 39}
    assert all(_same(want, got) for _, want, got in sets)
    # the first buffers on the other stream: not the first stream's graph, whose workspaces that stream may be using
    x, want, got = sets[0]
    session.set_stream(streams[1].cuda_stream)
    for step in range(3):
        for t in got.values():
            t.zero_()
        torch.cuda.synchronize()
        session.run_torch(x, got)
        torch.cuda.synchronize()
        assert _same(want, got)
    assert session.graph_stats() == {"cached_graphs": 3, "graph_launches": 2 * 39 + 2} and kernels.device_status() == 0


@pytest.mark.parametrize("m", [1, 17, 128])
def test_session_dropped_behind_its_last_run(module, m):
    x, want, _ = _buffers(module, m, 50)
    streams = [torch.cuda.Stream() for _ in range(3)]
    results = [{name: torch.zeros_like(t) for name, t in want.items()} for _ in range(9)]
    torch.cuda.synchronize()
    for i, got in enumerate(results):
        stream = streams[i % 3]
        session = module.create_session()
        session.set_graph_replay(True)
        session.set_stream(stream.cuda_stream)
        session.run_torch(x, got)
        session.run_torch(x, got)
        with torch.cuda.stream(stream):
            for t in got.values():
                t.zero_()
            torch.cuda._sleep(2_000_000)                        # a millisecond in front of the last run
        session.run_torch(x, got)
        assert session.graph_stats()["graph_launches"] == 2
        del session                                             # the next one gets its workspaces
    torch.cuda.synchronize()
    assert all(_same(want, got) for got in results) and kernels.device_status() == 0


def test_first_pass_makes_no_side_workspaces(module):
    """A pass over new buffers is launched in order: sessions that never replay hold no more memory with replay switched on than without."""
    x, want, got = _buffers(module, 1, 60)

    def taken(replay):
        sessions = [module.create_session() for _ in range(12)]         # more than the sets that the library keeps for new streams
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        for session in sessions:
            session.set_graph_replay(replay)
            session.run_torch(x, got)
            assert _same(want, got)
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]

    plain = taken(False)
    assert taken(True) <= plain + (2 << 20)                             # the driver's granularity; three workspaces a session would be 12 MB


def test_host_runs_of_several_shapes_share_their_sides(module):
    """Host runs have a stream per set of input shapes, and are waited for: their graphs have branches, and one set of side workspaces serves them all."""
    names = [o["name"] for o in module.metadata["outputs"]]
    cases = []
    for m in (1, 5, 17, 64):
        x, want, _ = _buffers(module, m, 70 + m)
        torch.cuda.synchronize()
        cases.append((x["x"].float().cpu().numpy(), {name: want[name].float().cpu() for name in names}))
    session = module.create_session()
    for _ in range(4):
        for x, want in cases:
            got = session.run_numpy({"x": x})
            assert all(torch.equal(torch.from_numpy(got[name]), want[name]) for name in names)
    count = ctypes.c_size_t()
    module._check(session._lib.dino_session_get_branched_graphs(session._handle, ctypes.byref(count)))
    assert count.value == len(cases) and session.graph_stats()["graph_launches"] == 3 * len(cases) and kernels.device_status() == 0
