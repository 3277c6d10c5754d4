"""Several handles in one process: what they share (kernel attributes, the pool of workspaces) does not let one disturb another."""
import threading

import numpy as np
import pytest

from tests.util import anisotropic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import turbovec_b200
    return turbovec_b200


def test_handles_of_different_sizes_searched_from_two_threads(T):
    """The tables of the two handles need 2 KB and 96 KB of shared memory in the same kernels: neither's limit is the other's.
    A launch above a limit is refused by the runtime before anything runs."""
    shapes = [(64, 2, 4), (3072, 2, 4), (64, 3, 1), (3072, 3, 1)]
    work = []
    for dim, bits, nq in shapes:
        idx = T.TurboQuantIndex(dim, bits)
        idx.add(anisotropic(700, dim, seed=5))
        q = anisotropic(nq, dim, seed=5, offset=9)
        work.append((idx, q, idx.search(q, 5)))
    errors = []
    start = threading.Barrier(len(work))

    def search(idx, q, want):
        start.wait()
        for _ in range(800):
            try:
                s, i = idx.search(q, 5)
                assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])
            except Exception as e:  # noqa: BLE001
                errors.append(repr(e))
                return

    threads = [threading.Thread(target=search, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_idle_workspaces_are_bounded_and_given_back(T):
    import torch
    T.release_workspaces()
    x = anisotropic(9000, 512, seed=7)
    for _ in range(2):
        handles = [T.TurboQuantIndex(512, 4) for _ in range(4)]
        want = None
        for idx in handles:
            idx.add(x)
            got = idx.search(x[:40], 7)
            want = got if want is None else want
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        del handles, idx
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    assert T.release_workspaces() == 2
    assert torch.cuda.mem_get_info()[0] > before + (8 << 20)
    assert T.release_workspaces() == 0
    idx = T.TurboQuantIndex(512, 4)
    idx.add(x)
    got = idx.search(x[:40], 7)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("before", [0, 5, 32])
def test_host_add_in_chunks_of_whole_code_blocks(T, before):
    """16 MB of rows at a time: one launch per chunk, and one more only for rows that complete a block begun earlier."""
    n, dim = 12_001, 1536
    x = anisotropic(n + before, dim, seed=91)
    idx = T.TurboQuantIndex(dim, 4)
    if before:
        idx.add(x[:before])
    at = idx.launch_count
    idx.add(x[before:])
    chunks = -(-(n + before % 32) // (2730 // 32 * 32))
    assert idx.launch_count - at == chunks + (before % 32 != 0)
    whole = T.TurboQuantIndex(dim, 4)
    whole.set_option(T.OPT_INGEST_PIPELINE, 0)
    whole.add(x)
    assert np.array_equal(idx.codes_blocked_seq(), whole.codes_blocked_seq()) and np.array_equal(idx.scales(), whole.scales())
