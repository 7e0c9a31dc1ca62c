"""Cuckoo builds with more keys than the table holds, and with many copies of
few keys: every key is in the table or counted as lost, the table is nearly
full, and a table near its highest load still takes all keys."""
import numpy as np
import pytest

import dtlg as F
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KINDS = [(16, 4), (8, 4), (32, 2), (16, 2), (16, 1), (12, 4), (32, 4), (8, 2)]


def _table(t, b, buckets):
    f = F.cf(buckets * t * b, t, b)
    return f, f.alloc_filter_data(), int(f.block_cnt()) * b


@pytest.mark.parametrize("t,b", KINDS)
def test_more_keys_than_slots(t, b):
    f, words, slots = _table(t, b, 20001)
    for n in (slots + slots // 50, 2 * slots):
        words.zero_()
        assert not f.batch_insert(words, keygen.build_keys_torch(n, 71))
        kept = f.count_occupied_slots(words)
        assert kept + f.last_failed == n
        assert kept >= {1: 0.6, 2: 0.9, 4: 0.97}[b] * slots


@pytest.mark.parametrize("t,b", [k for k in KINDS if k[1] == 4 and k[0] > 8])
def test_high_load_places_every_key(t, b):
    f, words, slots = _table(t, b, 25001)
    n = int(slots * 0.965)
    keys = keygen.build_keys_torch(n, 72)
    assert f.batch_insert(words, keys) and f.last_failed == 0
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    assert f.batch_contains(words, keys, n, out) == n


@pytest.mark.parametrize("t,b", KINDS)
def test_many_copies_of_few_keys(t, b):
    f, words, slots = _table(t, b, 20001)
    few = keygen.build_keys_torch(200, 73)
    keys = few.repeat(100)
    assert not f.batch_insert(words, keys)
    kept = f.count_occupied_slots(words)
    assert kept + f.last_failed == keys.numel() and kept <= 200 * 2 * b + 1
    found = [f.contains(words, int(k)) for k in few[:20].cpu().numpy().view(np.uint32)]
    assert all(found)
