"""Descriptor-mode pulls that score every neighbour's candidate keep no sorted list and make the next
pass's choices themselves; a cap of 23 candidates (more than a patch can have here) runs the sorted walk
and separate chooses.  Both give the same field bit for bit, with exact ties in distance and key, masks,
one- and two-row images, radius 1 and 2, and every store width."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,sw", [((40, 53), ""), ((1, 70), ""), ((33, 1), ""), ((40, 53), " -speed 1"), ((2, 90), " -speed 6"),
                                     ((64, 128), " -gpu_prop_passes 1")])
@pytest.mark.parametrize("c", [3, 8, 13])
@pytest.mark.parametrize("ties,masked", [(False, False), (True, False), (True, True)])
def test_unsorted_pull_equals_sorted_walk(gpu, libc, size, sw, c, ties, masked):
    import torch
    a, b = synth.descriptor_pair(64, 128, c, 70 + c)
    a = np.ascontiguousarray(a[:size[0], :size[1]])
    if ties:
        rng = np.random.default_rng(71)
        a, b = (rng.integers(0, 2, x.shape).astype(np.float32) for x in (a, b))
    allowed = (np.random.default_rng(72).random((64, 128)) < 0.7).astype(np.int32) if masked else None
    p = ptb.PatchTableParams("-is_descriptor 1 -limit 0.02 -grid_ndims 3 -coherence_spatial 4" + sw)
    p.kcoherence = 0 if ties else p.kcoherence
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b, allowed_patches=allowed)
    da = torch.from_numpy(a).cuda()
    out = []
    for cap in (0, 23):
        p.gpu_pull_max = cap
        ann = torch.full((size[0], size[1], 3), float("nan"), dtype=torch.float64, device="cuda")
        t.lookup_device(da.data_ptr(), size[0], size[1], ann.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        out.append(ann.cpu().numpy())
    assert np.array_equal(out[0], out[1])
    t.close()
