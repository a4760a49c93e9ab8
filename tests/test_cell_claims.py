"""The table's cell build keeps claim keys in the table's own words while they fit, with 4 or 5 edge
bits, and in an array of their own otherwise; its claims are unrolled over 6, 8 or 16 dimensions.  Each
combination gives the oracle's table bit for bit, at dimension counts on both sides of each line, with
single-slice dimensions, a mask, few patches and distance transforms cut short."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sw", ["", " -dt_iters 2", " -run_dt 0"])
@pytest.mark.parametrize("nslices", [(7, 1, 5), (3, 4, 5, 2, 6, 3), (2, 3, 4, 2, 3, 2, 5), (3, 2, 2, 3, 2, 1, 4, 3),
                                     (2, 2, 2, 2, 3, 2, 2, 2, 2), (2,) * 12, (130, 9, 40, 11, 4)])
@pytest.mark.parametrize("masked", [False, True])
def test_cells_equal_oracle(gpu, oracle, libc, sw, nslices, masked):
    c = max(3, len(nslices))
    b = synth.descriptor_pair(29, 37, c, 90 + c)[1]
    allowed = None
    if masked:
        allowed = (np.random.default_rng(5).random((29, 37)) < 0.3).astype(np.int32)
    p = ptb.PatchTableParams("-is_descriptor 1 -kcoherence 0 -grid_ndims %d%s" % (len(nslices), sw))
    p.nslices = nslices
    p.limit = float(np.prod(nslices))
    srand_all(libc, 1)
    ot = oracle.build(p.as_dict(), b, allowed=allowed) if masked else oracle.build(p.as_dict(), b)
    srand_all(libc, 1)
    gt = ptb.PatchTable(p, b, allowed_patches=allowed)
    assert gt.shape()[0] == list(nslices) == ot.shape()[0]
    assert gt.add_count() == ot.add_count()
    assert np.array_equal(gt.table(), ot.table())
    gt.close()


def test_claims_in_an_array_of_their_own(gpu, oracle, libc):
    """One cell more than the keys of 5 edge bits can number."""
    nslices = (8, 8, 8, 8, 8, 8, 8, 8, 6)
    b = synth.descriptor_pair(40, 50, 9, 99)[1]
    p = ptb.PatchTableParams("-is_descriptor 1 -kcoherence 0")
    p.nslices = nslices
    p.limit = float(np.prod(nslices))
    srand_all(libc, 1)
    ot = oracle.build(p.as_dict(), b)
    srand_all(libc, 1)
    gt = ptb.PatchTable(p, b)
    assert gt.shape() == (list(nslices), 100663296)
    assert np.array_equal(gt.table(), ot.table())
    gt.close()
