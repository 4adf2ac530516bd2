"""The launches a program is told of, against the kernel nodes of a capture."""
import ctypes

import pytest
import torch

from cpp_projects_b200 import CFdmtGpu
from cpp_projects_b200.pipeline import BatchedSearch, BeamShape, SearchPipeline, fdmt_launches

pytestmark = pytest.mark.gpu
P = ctypes.c_void_p


def captured_nodes(f):
    rt = ctypes.CDLL("libcudart.so.12")
    s, graph, n = torch.cuda.Stream(), P(), ctypes.c_size_t(0)
    f(s)   # (first launches set the kernels' shared memory)
    s.synchronize()
    assert rt.cudaStreamBeginCapture(P(s.cuda_stream), 2) == 0
    f(s)
    assert rt.cudaStreamEndCapture(P(s.cuda_stream), ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    rt.cudaGraphDestroy(graph)
    return n.value


@pytest.mark.parametrize("nchan,fuse,prec,levels", [(16, -1, 0, 0), (256, -1, 0, 0), (1024, 0, 0, 1), (256, 4, 0, 0),
                                                    (256, -1, 1, 0), (256, 0, 2, 0), (1024, -2, 1, 0)])
def test_fdmt_launches(cuda, nchan, fuse, prec, levels):
    f = CFdmtGpu(1200.0, 1600.0, nchan, 2000, nchan, fuse_depth=fuse, precision=prec, seg_levels=levels)
    x, y = torch.randn((nchan, 2000), device=cuda), torch.empty((nchan, 2000), device=cuda)
    assert captured_nodes(lambda s: f.process_image(x, y, False, s)) == fdmt_launches(f)


def test_batch_counts_the_same_schedules(cuda):
    shapes = [BeamShape(n, 3000, 1200.0, 1600.0, n) for n in (64, 256)]
    fdmt = [fdmt_launches(CFdmtGpu(1200.0, 1600.0, s.nchan, s.nsamp, s.max_dt, fuse_depth=-2)) for s in shapes]
    batch = BatchedSearch(shapes, capacity=1 << 16)
    assert batch.launches_per_run(0) == sum(fdmt) + 3 * len(shapes)
    pipe = SearchPipeline(shapes, capacity=1 << 16, device=cuda)
    for s in shapes:   # nothing to find: the FDMT, the statistics, the filter and the search
        pipe.run_beam(shapes.index(s), torch.zeros((s.nchan, s.nsamp), device=cuda))
    assert pipe.launches == sum(fdmt_launches(p) for p in pipe.plans) + 3 * len(shapes)
