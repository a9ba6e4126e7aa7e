"""A captured timed step: between two recorded stage boundaries run the kernels of one stage and
no others, so that an interval is that stage's time."""

import ctypes as C

import pytest
import torch

from gpu_helpers import need_gpu
from test_gpu_columns import _model

pytestmark = pytest.mark.gpu

EVENT_RECORD = 7  # CU_GRAPH_NODE_TYPE_EVENT_RECORD
BOUNDARIES = 256


def _graph(g):
    """Node types and successors of a captured graph."""
    cu = C.CDLL("libcuda.so.1")
    raw, n = C.c_void_p(g.raw_cuda_graph()), C.c_size_t()
    assert cu.cuGraphGetNodes(raw, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(raw, nodes, C.byref(n)) == 0
    assert cu.cuGraphGetEdges(raw, None, None, C.byref(n)) == 0
    a, b = (C.c_void_p * n.value)(), (C.c_void_p * n.value)()
    assert cu.cuGraphGetEdges(raw, a, b, C.byref(n)) == 0
    kinds, after = {}, {x: [] for x in nodes}
    for x in nodes:
        kind = C.c_int()
        assert cu.cuGraphNodeGetType(C.c_void_p(x), C.byref(kind)) == 0
        kinds[x] = kind.value
    for x, y in zip(a, b):
        after[x].append(y)
    return kinds, after


def _reach(start, after):
    seen, todo = set(), [start]
    while todo:
        for y in after[todo.pop()]:
            if y not in seen:
                seen.add(y)
                todo.append(y)
    return seen


@pytest.mark.parametrize("terrain,options", [(0.0, {}), (1500.0, {}), (0.0, {"config_dynamics_split_steps": 1}),
                                             (0.0, {"config_precision": "mixed"})])
def test_stage_intervals_are_disjoint(terrain, options):
    need_gpu()
    model, _ = _model(12, terrain, **options)
    plain, _ = _model(12, terrain, **options)
    events = [torch.cuda.Event(enable_timing=True) for _ in range(BOUNDARIES)]
    for e in events:
        e.record()
    torch.cuda.synchronize()
    handles = (C.c_void_p * BOUNDARIES)(*[e.cuda_event for e in events])
    kinds = (C.c_int32 * BOUNDARIES)()
    args = [C.byref(s) for s in (model.dmesh.struct, model.cstruct, model.state.struct)]
    g, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=stream):
        n = model.lib.mpasg_step_timed(*args, handles, kinds, BOUNDARIES, C.c_void_p(stream.cuda_stream))
    assert 0 < n <= BOUNDARIES
    types, after = _graph(g)
    marks = [x for x, t in types.items() if t == EVENT_RECORD]
    assert len(marks) == n
    before = {x: [] for x in after}
    for x, ys in after.items():
        for y in ys:
            before[y].append(x)
    for x in marks:  # every node runs before the boundary or after it
        assert len(_reach(x, after)) + len(_reach(x, before)) + 1 == len(types)
    g.instantiate()
    g.replay()
    plain.step()
    torch.cuda.synchronize()
    assert min(events[i].elapsed_time(events[i + 1]) for i in range(n - 1)) >= 0.0
    want, got = plain.export(), model.export()
    for k, v in want.items():
        assert torch.equal(got[k], v), k
