"""The k-nearest-neighbour search of the k-coherence step screens 32 x 32 pairs at a time with rounded
products and evaluates exactly what the rounding cannot rule out.  The k-coherence set must stay the
oracle's bit for bit where the screening's arithmetic could go wrong: every number of dimensions a
step of the products holds (3 .. 16, the last step full or not), point counts off the buckets of 32,
exact ties, isolated points (wide query groups), ranges from where a squared difference underflows
up to large ones, and the list widths from 12 to 64."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu


def _values(kind, h, w, c, seed):
    rng = np.random.default_rng(seed)
    b = synth.descriptor_pair(h, w, c, seed)[1].astype(np.float64)
    if kind == "ties":
        b = rng.integers(0, 3, (h, w, c)).astype(np.float64)
    elif kind == "isolated":
        far = rng.random((h, w)) < 0.02
        b[far] += rng.standard_normal((int(far.sum()), c)) * 1e3
    elif kind != "plain":
        b *= float(kind)
    return np.ascontiguousarray(b, np.float32)


@pytest.mark.parametrize("c", [3, 6, 7, 8, 13, 14, 15, 16])
@pytest.mark.parametrize("kind,kc", [("plain", 2), ("plain", 10), ("ties", 6), ("isolated", 2), ("1e-12", 2), ("1e-5", 20),
                                     ("1e6", 3)])
def test_kcoherence_equals_oracle(gpu, oracle, libc, c, kind, kc):
    b = _values(kind, 41, 53, c, 60 + c)
    p = ptb.PatchTableParams("-limit 0.02 -grid_ndims 3 -kcoherence %d -is_descriptor 1" % kc)
    srand_all(libc, 1)
    ot = oracle.build(p.as_dict(), b)
    srand_all(libc, 1)
    gt = ptb.PatchTable(p, b)
    kg, ko = gt.kcoherence(), ot.kcoherence()
    assert np.array_equal(kg[0], ko[0])
    assert np.array_equal(kg[1], ko[1])
    gt.close()
