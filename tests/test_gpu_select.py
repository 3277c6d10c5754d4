"""Top-k selection at the sizes where it can go wrong: one key, edges of a 4,096-key segment and of the longest list,
k at the limits of the merge and of the counting form, score ties, filters that leave fewer blocks than the first chunk."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.util import anisotropic

pytestmark = pytest.mark.gpu
DIM = 64


@pytest.fixture(scope="module")
def T():
    import turbovec_b200
    return turbovec_b200


def oracle_of(x, bits):
    enc = O.encode(x, bits)
    return O.packed_to_blocked(enc["packed"], bits, x.shape[1]), enc["scales"]


def check(idx, pre, q, k, n, bits, mask=None):
    words = None if mask is None else O.pack_mask(mask)
    want = O.search(q, pre[0], pre[1], n, q.shape[1], bits, k, mask_words=words)
    s, i = idx.search(q, k, mask=mask)
    assert np.array_equal(i, want[1]) and np.array_equal(s, want[0]), (n, k, q.shape[0])


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("n", [1, 33, 4095, 4097, 131_072, 131_105, 150_001])
def test_selection_edges(T, n, bits):
    x = anisotropic(n, DIM, seed=17)
    pre = oracle_of(x, bits)
    idx = T.TurboQuantIndex(DIM, bits)
    idx.add(x)
    rng = np.random.default_rng(n)
    for nq, k in ((1, 1), (1, 128), (2, 129), (3, 10), (1, 512), (1, 513), (40, 10)):
        check(idx, pre, anisotropic(nq, DIM, seed=17, offset=n + k), k, n, bits)
    for share in (0.9, 0.001):
        mask = rng.random(n) < share
        mask[rng.integers(n)] = True
        check(idx, pre, anisotropic(2, DIM, seed=17, offset=5), 100, n, bits, mask)


def test_selection_of_equal_scores(T):
    """Every key of a list shares its score: the cut falls back to the slots, which decide the order."""
    n = 70_000
    x = np.repeat(anisotropic(1, DIM, seed=3), n, axis=0)
    x[5::9973] = anisotropic(len(x[5::9973]), DIM, seed=4)
    pre = oracle_of(x, 4)
    idx = T.TurboQuantIndex(DIM, 4)
    idx.add(x)
    for k in (1, 10, 500, 600):
        check(idx, pre, np.concatenate([x[:1], -x[:1], anisotropic(1, DIM, seed=9)]), k, n, 4)


@pytest.mark.parametrize("bits,expanded", [(4, 1), (4, 0), (2, 1), (3, 1)])
@pytest.mark.parametrize("nq", [70, 300])
def test_batches_next_to_copies_of_a_row(T, bits, expanded, nq):
    """Half of the rows are copies of one row, and every query lies next to it: each copy ties with the k-th result of all columns
    of the tensor-memory scans, and the slots decide.  Some queries elsewhere, and copies with a smaller slot than a result's."""
    n, dim = 50_003, 200
    x = anisotropic(n, dim, seed=29)
    x[20_000::2] = x[0]
    x[7::5000] = x[0]
    pre = oracle_of(x, bits)
    idx = T.TurboQuantIndex(dim, bits)
    idx.add(x)
    idx.set_option(T.OPT_TC_EXPANDED, expanded)
    idx.set_option(T.OPT_MMA_MIN_BATCH, 8)                   # (2 and 3 bits: the one-hot form)
    q = x[:1] + np.float32(0.01) * anisotropic(nq, dim, seed=29, offset=3)
    q[::9] = anisotropic(len(q[::9]), dim, seed=29, offset=8)
    for k in (1, 10, 100):
        check(idx, pre, q, k, n, bits)
    check(idx, pre, q, 30, n, bits, np.random.default_rng(1).random(n) < 0.5)
