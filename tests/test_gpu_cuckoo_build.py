"""GPU cuckoo builds where the insert can go wrong: every bucket width (whole
words and unpacked slots), a table that already holds keys, batches of one key
and of ragged length, and more copies of a key than its two buckets hold."""
import numpy as np
import pytest

import dtlg as F
import oracle as O
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CONFIGS = [(t, b) for t in (4, 8, 12, 16, 32) for b in (1, 2, 4)]


def _dev(k):
    return torch.from_numpy(np.ascontiguousarray(k, dtype=np.uint32).view(np.int32)).cuda()


def _members(f, words, keys):
    out = torch.empty(len(keys), dtype=torch.int32, device="cuda")
    return f.batch_contains(words, keys, len(keys), out)


@pytest.mark.parametrize("t,b", CONFIGS)
def test_insert_in_two_batches(t, b):
    """All keys found and counted after a second, misaligned batch, and the
    oracle finds the same members in the GPU-built table.  Where the oracle's
    own insert cannot place the keys either (12-bit tags, one per bucket: an
    even MAGIC bucket count), every key is placed or reported lost."""
    m = (1 << 15) * t * b
    f, oc = F.cf(m, t, b), O.Cuckoo(t, b, m)
    n = int(f.block_cnt() * b * {1: 0.1, 2: 0.5, 4: 0.75}[b] * (0.5 if t == 4 else 1))
    keys = keygen.build_keys(n, 17 + t)
    dk, words = _dev(keys), f.alloc_filter_data()
    ok, lost = True, 0
    for part in (dk[:n // 3 + 1], dk[n // 3 + 1:n - 1], dk[n - 1:]):
        ok = f.batch_insert(words, part) and ok
        lost += f.last_failed
    assert f.count_occupied_slots(words) + lost == n and ok == (lost == 0)
    if oc.insert(np.zeros(f.alloc_words(), dtype=np.uint64), keys, seed=1):
        assert ok
        assert _members(f, words, dk) == n
        assert len(oc.batch_contains(words.cpu().numpy().view(np.uint64), keys)) == n


@pytest.mark.parametrize("t,b", [(16, 4), (8, 4), (12, 4), (8, 2)])
def test_copies_of_one_key(t, b):
    """20 000 copies of one key: its buckets (or both halves of one) and the
    victim record fill up, the rest is counted as lost, and it is found."""
    f = F.cf((1 << 12) * t * b, t, b)
    words = f.alloc_filter_data()
    n = 20000
    assert not f.batch_insert(words, _dev(np.full(n, 4242)))
    kept = f.count_occupied_slots(words)
    assert kept in (b + 1, 2 * b + 1) and f.last_failed == n - kept
    assert f.contains(words, 4242)
