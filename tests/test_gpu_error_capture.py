"""fc3dgpu_compute_error_device under stream capture: a captured call clears its
completion slot before every replay, and its replays and calls between them
give the same bits."""
import ctypes as C
import re

import numpy as np
import pytest

from test_zz_no_alloc import _call, _reaction

pytestmark = pytest.mark.gpu


@pytest.fixture
def case(built_lib):
    torch = pytest.importorskip("torch")
    from siconos_gb300.scene import lattice
    sc = lattice(6, 5, 4, seed=2)
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in
           dict(rowptr=sc.rowptr, colidx=sc.colidx, blocks=sc.blocks.reshape(-1), q=sc.q, mu=sc.mu,
                r=_reaction(sc.nc, 3)).items()}
    err = torch.zeros(1, dtype=torch.float64, device="cuda")

    def call(stream):
        assert _call(built_lib, sc.nc, sc.nnzb, dev, 1.0, None, err, stream.cuda_stream) == 0

    call(torch.cuda.current_stream())  # looks the scratch up before any capture
    torch.cuda.synchronize()
    return torch, call, err


def test_nodes_of_a_captured_call(case):
    """The clear and the kernel."""
    torch, call, _ = case
    path = next(m.group() for m in (re.search(r"/\S*libcudart\.so\S*", x) for x in open("/proc/self/maps")) if m)
    rt = C.CDLL(path)
    s = torch.cuda.Stream()
    graph, n = C.c_void_p(), C.c_size_t()
    assert rt.cudaStreamBeginCapture(C.c_void_p(s.cuda_stream), 2) == 0  # relaxed
    call(s)
    assert rt.cudaStreamEndCapture(C.c_void_p(s.cuda_stream), C.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, C.byref(n)) == 0
    rt.cudaGraphDestroy(graph)
    assert n.value == 2


def test_replays_among_calls(case):
    torch, call, err = case
    call(torch.cuda.current_stream())
    want = float(err)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(torch.cuda.current_stream())
    for k in range(40):  # more than the slots
        err.fill_(float("nan"))
        g.replay() if k % 3 else call(torch.cuda.current_stream())
        assert float(err) == want
