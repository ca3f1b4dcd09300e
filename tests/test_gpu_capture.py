"""The step's calls in a caller's stream capture: what the captured graph's edges are, and that its replay
gives what the calls give one by one."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


class EdgeData(ctypes.Structure):
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte),
                ("reserved", ctypes.c_ubyte * 5)]


def edges(graph):
    """(from, to, programmatic) of a captured graph's edges."""
    cu = ctypes.CDLL("libcuda.so.1")
    f = cu.cuGraphGetEdges_v2
    f.argtypes = [ctypes.c_void_p] + [ctypes.c_void_p] * 3 + [ctypes.POINTER(ctypes.c_size_t)]
    n = ctypes.c_size_t(0)
    h = graph.raw_cuda_graph()
    assert f(h, None, None, None, ctypes.byref(n)) == 0
    a, b, d = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (EdgeData * n.value)()
    assert f(h, a, b, d, ctypes.byref(n)) == 0
    return [(a[k], b[k], d[k].type == 1 or d[k].from_port != 0) for k in range(n.value)]


# A general-path tree (above 16,384 particles) forks the work items to a stream of its own and joins them;
# then a download, an evaluation or a summarize.  A kernel that waits for two nodes waits for both completely:
# no programmatic edge leads into it.  Then the replay's results are those of the calls one by one.
@pytest.mark.parametrize("mode", ["stream", "walk", "fp64"])
@pytest.mark.parametrize("tail", ["store", "evaluate", "summarize"])
def test_calls_after_create_tree_in_a_capture(mode, tail):
    from barneshut.gb300 import native

    n, grid = 40000, 32
    rng = np.random.default_rng(n)
    kw = dict(stream=dict(), walk=dict(flags=native.BH_FLAG_WALK), fp64=dict(precision=native.BH_PREC_FP64))[mode]
    plan = native.Plan([n], [grid], native.make_params(1.0, 1e-5, 1e-3, 0.0, 0.5, 2, **kw))
    sets = [[torch.from_numpy(rng.random(n)).cuda() for _ in range(3)] for _ in range(2)]
    z = torch.zeros(n, dtype=torch.float64, device="cuda")

    def calls(cols):
        plan.load(*cols, z, z)
        plan.create_tree()
        if tail == "evaluate":  # (with the last summarize's cells)
            plan.evaluate()
        elif tail == "summarize":
            plan.summarize()
            plan.evaluate()
        out = plan.store()
        return torch.stack([out[k] for k in ("x", "y", "ax", "ay")])

    def cells():  # an evaluation without a summarize takes the cells that are there
        plan.load(*sets[0], z, z)
        plan.create_tree()
        plan.summarize()

    want = []
    for s in sets:
        cells()
        want.append(calls(s))
    cols = [c.clone() for c in sets[0]]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        out = calls(cols)
    into = {}
    for _, b, programmatic in edges(g):
        into.setdefault(b, []).append(programmatic)
    assert any(len(e) > 1 for e in into.values())  # (the join)
    assert any(any(e) for e in into.values())
    assert all(len(e) == 1 or not any(e) for e in into.values())
    g.instantiate()
    for k in range(4):
        cells()
        for c, src in zip(cols, sets[k & 1]):
            c.copy_(src)
        g.replay()
        assert torch.equal(out, want[k & 1])
    assert plan.error_flags() == 0
