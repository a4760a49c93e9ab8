"""The library's device and page-locked memory pools, on the CPU over a stand-in for the CUDA runtime
(tests/cpp/fake_cuda): what is kept for reuse and its bound, failed allocations, devices and refused
waits."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

CPP = os.path.join(ROOT, "tests", "cpp")
CHECKS = ["reuse_beside_live", "bound", "retry", "pinned", "other_device", "refused_wait", "worker_device", "cap"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("memory") / "memory_pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-D__CUDACC__", "-I", os.path.join(CPP, "fake_cuda"),
                    "-I", os.path.join(ROOT, "patchtable_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(CPP, "memory_pool.cpp"), "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("check", CHECKS)
def test_pool(program, check):
    r = subprocess.run([program, check], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_threads_build_and_query_while_memory_is_given_back(gpu):
    """Two threads build, query and close tables while a third keeps giving the pools' memory back: every
    table and field equals the one built alone."""
    import threading

    import numpy as np

    import patchtable_b200 as ptb
    from patchtable_b200 import synth
    pairs = [synth.pair(90 + 20 * i, 140, 80 + i) for i in range(2)]
    p = [ptb.PatchTableParams("-limit 1 -populate_random 0") for _ in pairs]   # rand() is the process's

    def once(i):
        t = ptb.PatchTable(p[i], pairs[i][1])
        got = t.table(), t.lookup(pairs[i][0])
        t.close()
        return got
    want = [once(i) for i in range(2)]
    wrong, done = [], threading.Event()

    def work(i):
        try:
            for _ in range(6):
                for g, w in zip(once(i), want[i]):
                    if not np.array_equal(g, w):
                        wrong.append(i)
        except Exception as e:                    # noqa: BLE001 - reported by the assertion below
            wrong.append(e)

    def release():
        while not done.wait(0.002):
            ptb.release_memory()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    giver = threading.Thread(target=release)
    for th in threads + [giver]:
        th.start()
    for th in threads:
        th.join()
    done.set()
    giver.join()
    assert not wrong, wrong


@pytest.mark.gpu
def test_memory_kept_after_closing_stays_within_the_bound(gpu):
    import torch

    import patchtable_b200 as ptb
    from patchtable_b200 import synth
    t = ptb.PatchTable(ptb.PatchTableParams("-limit 1"), synth.pair(60, 80, 82)[1])
    ptb.release_memory()
    used = ptb.device_bytes_in_use()
    free = torch.cuda.mem_get_info()[0]
    batches = [t.batch([(4000, 4000)] * 4) for _ in range(3)]
    live = ptb.device_bytes_in_use() - used
    assert live > 6 << 30
    for b in batches:
        b.close()
    held = free - torch.cuda.mem_get_info()[0]
    slack = 64 << 20                              # the pool reserves whole granules
    assert held <= (4 << 30) + slack, held
    assert ptb.device_bytes_in_use() == used
    ptb.release_memory()
    assert free - torch.cuda.mem_get_info()[0] <= slack
    t.close()


@pytest.mark.gpu
def test_a_table_on_another_device(gpu, libc):
    """Build and query with device 1 current: the build's worker threads work there too."""
    import numpy as np
    import torch

    import patchtable_b200 as ptb
    from patchtable_b200 import synth
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    a, b = synth.pair(300, 200, 83)
    got = []
    for dev in range(2):
        with torch.cuda.device(dev):
            libc.srand(1)
            t = ptb.PatchTable(ptb.PatchTableParams("-limit 1"), b)
            got.append((t.table(), t.lookup(a)))
            t.close()
    assert all(np.array_equal(x, y) for x, y in zip(*got))


@pytest.mark.gpu
def test_memory_kept_stays_within_the_cap(gpu):
    import torch

    import patchtable_b200 as ptb
    from patchtable_b200 import synth
    a, b = synth.pair(60, 80, 84)
    t = ptb.PatchTable(ptb.PatchTableParams("-limit 1"), b)
    want = t.lookup(a)
    ptb.release_memory()
    used = ptb.device_bytes_in_use()
    free = torch.cuda.mem_get_info()[0]
    slack = 64 << 20                              # the pool reserves whole granules
    t.batch([(4000, 4000)] * 4).close()
    old = ptb.set_device_alloc_limit(used + (1 << 30))
    try:
        assert free - torch.cuda.mem_get_info()[0] <= (1 << 30) + slack
        with pytest.raises(ptb.PatchTableError):
            t.batch([(4000, 4000)] * 4)
        t.batch([(1000, 4000)]).close()
        assert (t.lookup(a) == want).all()
        assert free - torch.cuda.mem_get_info()[0] <= (1 << 30) + slack
    finally:
        ptb.set_device_alloc_limit(old)
    t.close()
