"""What a profiled lookup reports: every stage by itself -- a choose and a pull launch per pass, also where
an ordinary lookup makes the next pass's choices inside the pull -- the field of an ordinary lookup, and
the rows that were scored."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu


def _profiled(t, a):
    import torch
    h, w = a.shape[:2]
    d = torch.from_numpy(a).cuda()
    shape = (h, w, 3) if t.params.is_descriptor else (h - 7, w - 7, 3)
    ann = torch.empty(shape, dtype=torch.float64, device="cuda")
    t.lookup(a)
    n0 = ptb.launch_count()
    ms, ctr = t.lookup_profile(d.data_ptr(), h, w, ann.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return ann.cpu().numpy(), ctr, ptb.launch_count() - n0


@pytest.mark.parametrize("sw,passes", [("", 4), (" -gpu_prop_passes 1", 1), (" -speed 1", 4),
                                       (" -is_descriptor 1 -grid_ndims 3", 4)])
def test_stages_are_apart(gpu, libc, sw, passes):
    p = ptb.PatchTableParams("-limit 0.5 -coherence_spatial 4" + sw)
    a, b = (synth.descriptor_pair(60, 90, 8, 44) if p.is_descriptor else synth.pair(60, 90, 44))
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)
    ann, ctr, launches = _profiled(t, a)
    first = 2 if p.is_descriptor else 1           # descriptors and table entries, or both in one
    assert launches == first + 2 * passes
    assert np.array_equal(ann, t.lookup(a))
    assert ctr["choose_cand"] > 0 and ctr["pull_cand"] > 0
    t.close()


def test_rows_of_few_candidates(gpu, libc):
    """A 2 x 2 patch image has at most four candidates at a time: they are scored in rounds of eight, which
    end after four rows when nothing can be accepted any more."""
    p = ptb.PatchTableParams("-limit 0.05 -coherence_spatial 4")
    rows = cand = 0
    for seed in range(12):
        a, b = synth.pair(40, 50, 100 + seed)
        srand_all(libc, 1)
        t = ptb.PatchTable(p, b)
        _, ctr, _ = _profiled(t, np.ascontiguousarray(a[:9, :9]))
        assert ctr["pull_rows"] % 4 == 0 and 4 * ctr["pull_cand"] <= ctr["pull_rows"] <= 8 * ctr["pull_cand"]
        rows += ctr["pull_rows"]
        cand += ctr["pull_cand"]
        t.close()
    assert rows < 8 * cand
