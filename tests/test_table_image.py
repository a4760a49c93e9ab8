"""A finished table holds its image once, as the row store of the query: 64 bytes per pixel.  A saved file's
b0 is read back from it, at every width of a row's last line."""
import numpy as np
import pytest

import patchtable_b200 as ptb
from patchtable_b200 import synth
from tests.conftest import srand_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [8, 9, 10, 11, 46, 47])
@pytest.mark.parametrize("h", [8, 63, 65])
def test_saved_image_is_the_image(gpu, libc, tmp_path, h, w):
    _, b = synth.pair(h, w, 12)
    b[0, 0, 0] = -0.0
    p = ptb.PatchTableParams("-limit 0.01")
    p.kcoherence = 0
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)
    t.save(tmp_path / "t.bin")
    assert np.ascontiguousarray(b).tobytes() in (tmp_path / "t.bin").read_bytes()
    t.close()
    t = ptb.PatchTable.load(p, tmp_path / "t.bin")
    t.save(tmp_path / "u.bin")
    assert (tmp_path / "t.bin").read_bytes() == (tmp_path / "u.bin").read_bytes()
    t.close()


@pytest.mark.parametrize("loaded", [False, True])
@pytest.mark.parametrize("kcoherence", [0, 4])
def test_bytes_of_a_table(gpu, libc, tmp_path, loaded, kcoherence):
    h, w = 400, 500
    _, b = synth.pair(h, w, 13)
    p = ptb.PatchTableParams("-limit 0.05")
    p.kcoherence = kcoherence
    before = ptb.device_bytes_in_use()
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)
    if loaded:
        t.save(tmp_path / "t.bin")
        t.close()
        t = ptb.PatchTable.load(p, tmp_path / "t.bin")
    cells, patches = t.table().size, (h - 7) * (w - 7)
    image, descriptors, bins = 64 * h * w, 32 * patches, p.ndims * 16384 * 4
    assert ptb.device_bytes_in_use() - before <= image + descriptors + 4 * cells + 8 * kcoherence * patches + bins + 65536
    t.close()


def test_a_load_waits_for_no_other_stream(gpu, libc, tmp_path):
    """A load beside a kernel of about a second on another stream ends before that kernel: the image's
    copy goes back in the load's own order.  (A build's cooperative launch waits for a free GPU.)"""
    import torch
    _, b = synth.pair(60, 80, 14)
    p = ptb.PatchTableParams("-limit 0.05")
    path = tmp_path / "t.bin"
    srand_all(libc, 1)
    tables = [ptb.PatchTable(p, b)]
    tables[0].save(path)
    for _ in range(2):                            # kernels loaded, memory in the pool
        tables.append(ptb.PatchTable.load(p, path))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(2_000_000_000)
    tables.append(ptb.PatchTable.load(p, path))
    assert not side.query()
    side.synchronize()
    for t in tables:
        t.close()


def test_a_build_fits_without_room_for_the_row_store(gpu, libc):
    """The most that a build of many cells holds is those, their breadth-first lists and the image's
    16-byte copy, not the row store of 64 nor the partition's scratch."""
    h, w = 400, 500
    _, b = synth.pair(h, w, 15)
    p = ptb.PatchTableParams("-limit 5")
    srand_all(libc, 1)
    t = ptb.PatchTable(p, b)
    cells, patches = t.table().size, (h - 7) * (w - 7)
    t.close()
    # cells and lists, the populate order, descriptors and k-coherence sets, bins, the copy, small buffers
    bound = 22 * cells + (4 + 32 + 8 * p.kcoherence) * patches + p.ndims * 16384 * 4 + 16 * h * w + (1 << 20)
    old = ptb.set_device_alloc_limit(ptb.device_bytes_in_use() + bound)
    try:
        srand_all(libc, 1)
        ptb.PatchTable(p, b).close()
    finally:
        ptb.set_device_alloc_limit(old)


def test_bytes_of_a_lookup(gpu, libc):
    """12 bytes per pixel and 40 per patch: a lookup with the fused table step stores no descriptors, one
    with learned proposals (tests/test_proposal.py) or several tables does."""
    import torch
    h, w = 300, 400
    a, b = synth.pair(h, w, 16)
    patches = (h - 7) * (w - 7)
    d = torch.from_numpy(a).cuda()
    ann = torch.empty((h - 7, w - 7, 3), dtype=torch.float64, device="cuda")
    for ntables, each in ((1, 40), (2, 40 + 32 + 4)):
        p = ptb.PatchTableParams("-limit 0.05 -coherence_spatial 4")
        p.ntables = ntables
        srand_all(libc, 1)
        t = ptb.PatchTable(p, b)
        before = ptb.device_bytes_in_use()
        t.lookup_device(d.data_ptr(), h, w, ann.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert ptb.device_bytes_in_use() - before <= 12 * h * w + each * patches + 4096
        t.close()
