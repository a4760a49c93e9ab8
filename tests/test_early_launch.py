"""Small queries' kernels start while the kernel before them ends.  Lookups of two images in turn, queued
on one stream without a wait between them (and the same replayed from a captured graph), reuse every
array of choices, states and table entries while the lookup before may still be running: each gives the
field that its image has when its kernels are launched strictly in order (a profiled lookup)."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu

ROUTES = {"default": ("-limit 1", (0, 0, 0)), "one candidate": ("-limit 1", (2, 2, 1, -1)),
          "one pass": ("-limit 1", (1, 2, 1, -1)), "window": ("-limit 1 -speed 1", (0, 0, 0)),
          "descriptors": ("-is_descriptor 1 -limit 0.05 -grid_ndims 3", (0, 0, 0)),
          "descriptors, capped": ("-is_descriptor 1 -limit 0.05 -grid_ndims 3", (0, 0, 5))}


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("size", [(48, 64), (100, 150), (9, 300)])
@pytest.mark.parametrize("route", sorted(ROUTES))
def test_lookups_in_turn_equal_ordered_ones(gpu, libc, route, size, captured):
    import torch
    sw, sched = ROUTES[route]
    p = ptb.PatchTableParams("-coherence_spatial 4 " + sw)
    p.set_schedule(sched)
    if p.is_descriptor:
        imgs, b = zip(*[synth.descriptor_pair(120, 310, 8, 60 + i) for i in range(2)])
        out_shape = (size[0], size[1], 3)
    else:
        imgs, b = zip(*[synth.pair(120, 310, 60 + i) for i in range(2)])
        out_shape = (size[0] - 7, size[1] - 7, 3)
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b[0])
    dev = [torch.from_numpy(np.ascontiguousarray(x[:size[0], :size[1]])).cuda() for x in imgs]
    want = []
    for d in dev:
        ann = torch.empty(out_shape, dtype=torch.float64, device="cuda")
        t.lookup_profile(d.data_ptr(), size[0], size[1], ann.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        want.append(ann)
    assert not torch.equal(want[0], want[1])
    got = [torch.full(out_shape, -1.0, dtype=torch.float64, device="cuda") for _ in range(12)]

    def enqueue():
        st = torch.cuda.current_stream().cuda_stream
        for i, ann in enumerate(got):
            t.lookup_device(dev[i & 1].data_ptr(), size[0], size[1], ann.data_ptr(), st)
    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            enqueue()
        for _ in range(3):
            for ann in got:
                ann.fill_(-1.0)
            g.replay()
    else:
        enqueue()
    torch.cuda.synchronize()
    for i, ann in enumerate(got):
        assert torch.equal(ann, want[i & 1]), i
    t.close()
