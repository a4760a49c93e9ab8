"""The query's distance kernels score a candidate with four lanes that read one line of the table
image's row store.  Checked at the sizes where their indices can go wrong -- images of one patch, of
one row or column of patches, widths and heights around the tiles of 8 x 4 patches and the
two-pixel lines -- for every number of patches per CTA: the same field whatever the tile, and every
distance bit-exact with the reference's patch distance of its match."""
import ctypes as C

import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all
from tests.test_gpu_parity import check_nnf

pytestmark = pytest.mark.gpu


def _lookup(t, a):
    import torch
    h, w = a.shape[:2]
    da = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ann = torch.full((h - 7, w - 7, 3), float("nan"), dtype=torch.float64, device="cuda")
    t.lookup_device(da.data_ptr(), h, w, ann.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return ann.cpu().numpy()


@pytest.mark.parametrize("size", [(8, 8), (8, 40), (33, 8), (11, 15), (12, 16), (18, 23), (23, 39), (40, 64)])
@pytest.mark.parametrize("bsize", [(24, 30), (25, 31)])
@pytest.mark.parametrize("sched", ["", " -speed 1", " -gpu_prop_passes 1 -gpu_jump 2 -gpu_pull_max 1 -gpu_kc_max -1"])
def test_edges_of_tiles_and_lines(gpu, oracle, libc, size, bsize, sched):
    a = synth.image_a(size[0] + 4, size[1] + 4, 7)[2:-2, 2:-2]
    b = synth.pair(bsize[0], bsize[1], 8)[1]
    srand_all(libc, 1)
    p = ptb.PatchTableParams("-coherence_spatial 4 -limit 1" + sched)
    t = ptb.PatchTable(p, b)
    ref = None
    for tile in (0, 32, 64, 128, 256):        # 0: four warps share a tile of so small an image
        p.gpu_tile = tile
        ann = _lookup(t, a)
        if ref is None:
            ref = ann
            check_nnf(oracle, np.ascontiguousarray(a), b, ann, sample=ann.shape[0] * ann.shape[1])
        assert np.array_equal(ann, ref), tile
    t.close()


@pytest.mark.parametrize("sw", ["", " -speed 1", " -speed 6"])
def test_ties_keep_the_list_order(gpu, libc, sw):
    """Flat images: many candidates tie exactly in distance and key.  Four warps sharing a tile's list
    (tile 0), one warp per tile, and the zero-allocation lookup's separate chooses pick the same one."""
    import torch
    rng = np.random.default_rng(3)
    a, b = (np.repeat(np.repeat(rng.integers(0, 2, (h // 12 + 1, w // 12 + 1, 3)), 12, 0), 12, 1)[:h, :w].astype(np.float32)
            for h, w in ((60, 75), (50, 90)))
    srand_all(libc, 1)
    p = ptb.PatchTableParams("-coherence_spatial 4 -limit 0.1 -kcoherence 0" + sw)
    p.kcoherence = 0
    t = ptb.PatchTable(p, np.ascontiguousarray(b))
    a = np.ascontiguousarray(a)
    want = _lookup(t, a)
    for tile in (32, 64, 128, 256):
        p.gpu_tile = tile
        assert np.array_equal(_lookup(t, a), want), tile
    f = ptb.lib().pt_table_lookup_device_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    da = torch.from_numpy(a).cuda()
    ann = torch.empty(want.shape, dtype=torch.float64, device="cuda")
    assert f(t._h, da.data_ptr(), a.shape[0], a.shape[1], ann.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert np.array_equal(ann.cpu().numpy(), want)
    t.close()


def test_query_image_inside_the_field_buffer(gpu, libc):
    """A caller may hand over a query image that lies in the buffer the field is written to."""
    import torch
    a, b = synth.pair(60, 90, 11)
    srand_all(libc, 1)
    t = ptb.PatchTable(ptb.PatchTableParams("-limit 1"), b)
    want = _lookup(t, a)
    st = torch.cuda.current_stream().cuda_stream
    buf = torch.empty(want.size, dtype=torch.float64, device="cuda")
    f = ptb.lib().pt_table_lookup_device_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    qb = t.batch([a.shape[:2]])
    for call in (lambda: t.lookup_device(buf.data_ptr(), 60, 90, buf.data_ptr(), st),
                 lambda: f(t._h, buf.data_ptr(), 60, 90, buf.data_ptr(), st),
                 lambda: qb.lookup(buf.data_ptr(), buf.data_ptr(), st)):
        buf.view(torch.float32)[:a.size].copy_(torch.from_numpy(a.ravel()))
        call()
        torch.cuda.synchronize()
        assert np.array_equal(buf.cpu().numpy().reshape(want.shape), want)
    qb.close()
    t.close()
