"""Which launches of a step may start beside the end of another (``csrc/launch.h``), read from a captured step's graph, where such a
dependency is an edge of its own kind."""
import pytest
import torch

from scalingcontrasts_b200 import LossSpec, Matryoshka
from scalingcontrasts_b200.parallel.box import BoxLoss

pytestmark = pytest.mark.gpu


def _edges(work):
    """Per node the kinds of its incoming edges, True where the kernel may start before and waits by itself."""
    runtime = pytest.importorskip("cuda.bindings.runtime")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        work()
    handle = runtime.cudaGraph_t(graph.raw_cuda_graph())
    code, _, _, _, count = runtime.cudaGraphGetEdges_v2(handle)
    assert code == runtime.cudaError_t.cudaSuccess
    code, _, to, data, count = runtime.cudaGraphGetEdges_v2(handle, count)
    assert code == runtime.cudaError_t.cudaSuccess
    programmatic = runtime.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic
    incoming = {}
    for node, edge in zip(to[:count], data[:count]):
        incoming.setdefault(int(node), []).append(edge.type == programmatic)
    return list(incoming.values())


@pytest.mark.parametrize("overlap", [False, True])
def test_what_waits_for_another_stream_waits_for_all_of_it(overlap):
    """With the overlapped backward a launch behind the other stream's (the fold of a block's records among them) starts only when all
    before it is complete; in line nothing waits for another stream, and launches start beside one another's ends."""
    rows, hidden, world = 512, 768, 4
    engine = BoxLoss(rows, hidden, Matryoshka.halvings(hidden, 5), LossSpec("pairs"), None, "cuda", overlap_backward=overlap)
    block = torch.nn.functional.normalize(torch.randn(rows, hidden, device="cuda"), dim=1).bfloat16()
    engine.simulate(block, world)  # loads the kernels
    torch.cuda.synchronize()
    nodes = _edges(lambda: engine.simulate(block, world))
    several = [kinds for kinds in nodes if len(kinds) > 1]
    assert bool(several) == overlap and not any(any(kinds) for kinds in several)
    assert any(kinds == [True] for kinds in nodes)
