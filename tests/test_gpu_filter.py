"""Batches over 2- and 3-bit codes that go through the filtering scan: identical to the oracle at ragged dimensions, partial
query groups and chunk ends, under masks, past 256 byte-groups of the flush family, and where the filter lets too much through."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.util import anisotropic
from turbovec_b200 import OPT_FILTER_REDONE

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import turbovec_b200
    return turbovec_b200


def built(T, x, bits):
    enc = O.encode(x, bits)
    idx = T.TurboQuantIndex(x.shape[1], bits)
    idx.add(x)
    idx.set_option(T.OPT_FILTER, 2)                         # whatever its expected time
    return idx, (O.packed_to_blocked(enc["packed"], bits, x.shape[1]), enc["scales"])


def check(idx, pre, q, k, mask=None, redone=0):
    n, bits = len(idx), idx.bit_width
    words = None if mask is None else O.pack_mask(mask)
    want = O.search(q, pre[0], pre[1], n, q.shape[1], bits, k, mask_words=words)
    s, i = idx.search(q, k, mask=mask)
    assert np.array_equal(s, want[0]) and np.array_equal(i, want[1]), (n, q.shape, bits, k)
    if redone is not None:
        assert idx.get_option(OPT_FILTER_REDONE) == redone, "the filter did not take this batch, or not to its end"


# dim 2072 at 2 bits has 518 byte-groups, not a multiple of four
@pytest.mark.parametrize("dim,bits,n,nq", [(64, 2, 270_001, 8), (200, 2, 90_017, 70), (200, 3, 45_003, 9), (1536, 2, 11_001, 65),
                                           (1000, 3, 9_000, 300), (2072, 2, 8_200, 8), (3072, 2, 6_007, 17), (64, 3, 33, 3)])
def test_filtering_scan_matches_oracle(T, dim, bits, n, nq):
    x = anisotropic(n, dim, seed=23)
    idx, pre = built(T, x, bits)
    q = anisotropic(nq, dim, seed=23, offset=n + 1)
    for k in (1, 10, 200):
        check(idx, pre, q, k)
    rng = np.random.default_rng(n)
    for share in (0.6, 0.02):
        mask = rng.random(n) < share
        check(idx, pre, q[:12], 10, mask)
    mask = np.zeros(n, bool)
    mask[rng.choice(n, min(7, n), replace=False)] = True            # fewer allowed than k
    check(idx, pre, q[:9], 10, mask)


@pytest.mark.parametrize("bits", [2, 3])
def test_filtering_scan_overflows_and_recovers(T, bits):
    """Every row the same but for a few, and a query that all of them score below zero: nothing can be dismissed."""
    n, dim = 300_000, 64
    x = np.repeat(anisotropic(1, dim, seed=2), n, axis=0)
    x[3::1117] = anisotropic(len(x[3::1117]), dim, seed=6)
    idx, pre = built(T, x, bits)
    q = np.concatenate([-x[:1], x[:1], anisotropic(6, dim, seed=7)])
    for batch, k in ((q, 10), (np.concatenate([q, np.zeros((1, dim), np.float32)]), 20)):
        check(idx, pre, batch, k, redone=None)
        assert idx.get_option(OPT_FILTER_REDONE) > 0


@pytest.mark.parametrize("bits", [2, 3])
def test_queries_that_the_filter_cannot_finish_are_redone_alone(T, bits):
    """Half of the rows are copies of one row: more ties at the k-th place than a list holds for the queries near it, none that
    matter for the others.  A zero query ties with every row, and the slots alone decide."""
    n, dim = 300_000, 64
    x = anisotropic(n, dim, seed=81)
    x[::2] = x[0]
    idx, pre = built(T, x, bits)
    q = anisotropic(16, dim, seed=81, offset=5)
    q[3] = 0.0
    check(idx, pre, q, 10)
    q[[0, 9]] = x[0]
    q[9] *= np.float32(3.0)
    mask = np.random.default_rng(1).random(n) < 0.97
    for m, redone in ((None, 2), (mask, 3)):                        # under a mask the slots come in any order
        check(idx, pre, q, 10, m, redone=redone)
    q[:12] = x[0]                                                   # most of the batch: all of it
    check(idx, pre, q, 10, redone=16)


def test_redone_queries_reach_every_kind_of_output(T):
    import torch
    n, dim, k = 300_000, 64, 10
    x = anisotropic(n, dim, seed=82)
    x[::2] = x[0]
    idx, pre = built(T, x, 2)
    q = anisotropic(16, dim, seed=82, offset=5)
    q[[2, 7]] = x[0]
    want = O.search(q, pre[0], pre[1], n, dim, 2, k)
    dq = torch.from_numpy(q).cuda()
    s = torch.empty((16, k), device="cuda")
    i = torch.empty((16, k), dtype=torch.int64, device="cuda")
    assert idx.search_device(dq.data_ptr(), 16, k, s.data_ptr(), i.data_ptr()) == k
    assert idx.get_option(OPT_FILTER_REDONE) == 2
    assert np.array_equal(s.cpu().numpy(), want[0]) and np.array_equal(i.cpu().numpy(), want[1])
    keys = torch.empty((16, k), dtype=torch.int64, device="cuda")
    idx.search_device_keys(dq.data_ptr(), 16, k, keys.data_ptr(), 1000)
    assert idx.get_option(OPT_FILTER_REDONE) == 2
    assert np.array_equal((keys.cpu().numpy() & 0xffffffff) - 1000, want[1])
    idx.search(q[:1], k)                                            # a search after one that was redone
    check(idx, pre, q[3:7], k)


@pytest.mark.parametrize("bits,n", [(2, 33_001), (3, 17_003)])
def test_filtering_scan_of_a_calibrated_index(T, bits, n):
    """The TQ+ pair moves the queries' coordinates and their bias; the bound has to follow."""
    dim = 512
    x = anisotropic(n, dim, seed=51) * np.float32(3.0)
    x[:, ::7] *= np.float32(2.5)
    sh, sc = O.fit_calibration(x[:4000], bits)
    idx = T.TurboQuantIndex(dim, bits)
    idx.calibrate(x[:4000])
    idx.add(x)
    idx.set_option(T.OPT_FILTER, 2)
    enc = O.encode(x, bits, sh, sc)
    q = anisotropic(20, dim, seed=51, offset=n + 3)
    want = O.search(q, O.packed_to_blocked(enc["packed"], bits, dim), enc["scales"], n, dim, bits, 10, shift=sh, scale=sc)
    s, i = idx.search(q, 10)
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])
    assert idx.get_option(T.OPT_FILTER_REDONE) == 0


def test_filtering_scan_of_rows_with_unused_bits_set(T):
    """set_row takes any bytes; bit 3 of a 3-bit nibble does not count in the exact score and must not in the filter."""
    n, dim = 20_011, 256
    x = anisotropic(n, dim, seed=61)
    idx, pre = built(T, x, 3)
    q = anisotropic(12, dim, seed=61, offset=4)
    want = O.search(q, pre[0], pre[1], n, dim, 3, 10)
    for slot in np.unique(np.concatenate([want[1].ravel(), np.arange(5, n, 997)])):
        groups, scale = idx.get_row(int(slot))
        idx.set_row(int(slot), groups | np.random.default_rng(slot).choice(np.array([0x08, 0x80, 0x88], np.uint8), groups.size), scale)
    for batch in (q, q[:1]):
        s, i = idx.search(batch, 10)
        assert np.array_equal(i, want[1][:len(batch)]) and np.array_equal(s, want[0][:len(batch)])


@pytest.mark.parametrize("n,k", [(20_011, 10), (300, 300)])
def test_filtering_scan_of_scores_that_overflow(T, n, k):
    """Scales and queries are bounded each on its own; their product can be infinite, of either sign, for the k-th result too."""
    dim = 64
    x = anisotropic(n, dim, seed=71)
    idx, pre = built(T, x, 2)
    scales = pre[1].copy()
    for slot in range(0, n, max(1, n // 300)):
        groups, _ = idx.get_row(slot)
        scales[slot] = 3e38
        idx.set_row(slot, groups, 3e38)
    q = anisotropic(9, dim, seed=71, offset=4) * np.float32(1000.0)
    with np.errstate(over="ignore"):
        want = O.search(q, pre[0], scales, n, dim, 2, k)
    assert np.isinf(want[0]).any()
    s, i = idx.search(q, k)
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])


@pytest.mark.parametrize("dim,bits,n,nq", [(1536, 2, 3000, 9), (1024, 3, 1500, 70), (64, 2, 40_000, 513), (3072, 2, 1500, 300)])
def test_one_hot_form_of_wide_batches_is_still_reached(T, dim, bits, n, nq):
    """A batch size that the caller sets selects the one-hot contraction, above 256 queries two query groups to a work item."""
    x = anisotropic(n, dim, seed=43)
    idx, pre = built(T, x, bits)
    idx.set_option(T.OPT_SCORE_MODE, T.SCORE_LUT_MULADD)
    idx.set_option(T.OPT_FILTER, 1)
    idx.set_option(T.OPT_MMA_MIN_BATCH, 1)
    q = anisotropic(nq, dim, seed=43, offset=7)
    want = O.search(q, pre[0], pre[1], n, dim, bits, 10, mode=O.MODE_LUT_MULADD)
    s, i = idx.search(q, 10)
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])
    assert idx.get_option(T.OPT_FILTER_REDONE) == -1
    idx.set_option(T.OPT_MMA_MIN_BATCH, -1)
    idx.set_option(T.OPT_FILTER, 0)
    s, i = idx.search(q, 10)
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])
    assert idx.get_option(T.OPT_FILTER_REDONE) == -1


@pytest.mark.parametrize("n,dim,bits,nq,k,chosen", [(500_000, 200, 2, 64, 10, True), (200_000, 1536, 2, 64, 10, True), (3_000, 3072, 2, 300, 10, False),
                                                    (100_000, 768, 3, 512, 200, False), (60_000, 2072, 2, 64, 10, True)])
def test_default_choice_on_both_sides_of_the_switch(T, n, dim, bits, nq, k, chosen):
    """Clearly inside and outside of the region where the filter pays; the results do not depend on it."""
    idx = T.TurboQuantIndex(dim, bits)
    for lo in range(0, n, 20_000):
        idx.add(anisotropic(min(20_000, n - lo), dim, seed=95, offset=lo))
    q = anisotropic(nq, dim, seed=95, offset=n + 1)
    s, i = idx.search(q, k)
    assert (idx.get_option(T.OPT_FILTER_REDONE) >= 0) == chosen
    idx.set_option(T.OPT_FILTER, 0)
    s0, i0 = idx.search(q, k)
    assert idx.get_option(T.OPT_FILTER_REDONE) == -1
    assert np.array_equal(i, i0) and np.array_equal(s, s0)


@pytest.mark.parametrize("api", ["host", "device"])
@pytest.mark.parametrize("n,dim,nq,share,masked", [(300_000, 200, 600, 0.01, False), (100_000, 1024, 40, 0.3, False), (300_000, 200, 600, 0.01, True)])
def test_filter_that_does_not_pay_is_given_up(T, n, dim, nq, share, masked, api):
    """Where all queries lie near a tight cluster, every vector of it survives the filter: the default decides that on what the
    scans counted, keeps the results of the chunks before (some, or none in the second case) and goes on without the filter."""
    import torch
    k = 10
    rng = np.random.default_rng(3)
    x = anisotropic(n, dim, seed=97)
    near = rng.random(n) < share
    x[near] = x[0] + np.float32(1e-3) * x[near]
    idx, pre = built(T, x, 2)
    idx.set_option(T.OPT_FILTER, 1)
    q = x[:1] + np.float32(0.01) * anisotropic(nq, dim, seed=97, offset=5)
    q[1] = 0.0
    mask = rng.random(n) < 0.9 if masked else None
    want = O.search(q, pre[0], pre[1], n, dim, 2, k, mask_words=None if mask is None else O.pack_mask(mask))
    if api == "host":
        s, i = idx.search(q, k, mask=mask)
    else:
        words = 0 if mask is None else torch.from_numpy(O.pack_mask(mask).view(np.int64)).cuda()
        dq, ds = torch.from_numpy(q).cuda(), torch.empty((nq, k), device="cuda")
        di = torch.empty((nq, k), dtype=torch.int64, device="cuda")
        assert idx.search_device(dq.data_ptr(), nq, k, ds.data_ptr(), di.data_ptr(), 0 if mask is None else words.data_ptr()) == k
        s, i = ds.cpu().numpy(), di.cpu().numpy()
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])
    if not masked:
        assert idx.get_option(T.OPT_FILTER_REDONE) > 0
    s, i = idx.search(anisotropic(9, dim, seed=97, offset=11), k)
    want = O.search(anisotropic(9, dim, seed=97, offset=11), pre[0], pre[1], n, dim, 2, k)
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0])
