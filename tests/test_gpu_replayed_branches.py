"""Replayed runs with branches on the session's own stream and on a caller's, ordered behind their inputs, and whether a graph and branches were there."""
import ctypes

import pytest
import torch

from test_gpu_side_by_side import _inputs, _outputs, module  # noqa: F401

pytestmark = pytest.mark.gpu


def _branched_graphs(session):
    count = ctypes.c_size_t()
    session.module._check(session._lib.dino_session_get_branched_graphs(session._handle, ctypes.byref(count)))
    return count.value


@pytest.mark.parametrize("m", [1, 2, 5, 17, 64, 128, 129])       # the last one is above the row limit: one after another
def test_branches_on_own_and_callers_stream(module, m):           # noqa: F811
    plain, replayed = module.create_session(), module.create_session()
    replayed.set_graph_replay(True)
    x, want, got = _inputs(m, 0), _outputs(module, m), _outputs(module, m)
    stream = torch.cuda.Stream()
    for step in range(7):                       # on either stream: an ordinary run, the captured one, replays
        fresh = _inputs(m, 10 * m + step)
        for name in x:
            x[name].copy_(fresh[name])
        if step == 4:
            replayed.set_stream(stream.cuda_stream)
        torch.cuda.synchronize()                # neither session's stream waits for torch's
        plain.run_torch(x, want)
        replayed.run_torch(x, got)
        torch.cuda.synchronize()
        for name in want:
            assert torch.equal(want[name].view(torch.int16), got[name].view(torch.int16)), (m, step, name)
    assert replayed.graph_stats() == {"cached_graphs": 2, "graph_launches": 5}
    assert _branched_graphs(replayed) == (2 if m <= 128 else 0)


def test_results_in_one_buffer_take_no_branches(module):          # noqa: F811
    m = 4
    plain, replayed = module.create_session(), module.create_session()
    replayed.set_graph_replay(True)
    x, want, got = _inputs(m, 3), _outputs(module, m), _outputs(module, m)
    torch.cuda.synchronize()
    plain.run_torch(x, want)
    names = [o["name"] for o in module.metadata["outputs"]]
    got[names[1]] = got[names[2]]
    for _ in range(20):
        got[names[2]].zero_()
        torch.cuda.synchronize()
        replayed.run_torch(x, got)
        torch.cuda.synchronize()
        assert torch.equal(want[names[2]].view(torch.int16), got[names[2]].view(torch.int16))
    assert replayed.graph_stats() == {"cached_graphs": 1, "graph_launches": 19} and _branched_graphs(replayed) == 0
