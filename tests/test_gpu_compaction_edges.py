"""The compaction (plan 2) where its tiles grow from two rows of mask words to
four and eight, and where the tiles' offsets change from a look-back to sums
and back, with sparse and dense matches: match lists equal the oracle's."""
import numpy as np
import pytest

import dtlg as F
import oracle as O
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGES = [5000, 1 << 21, 1 << 24, 1 << 25, 1 << 26]  # one tile, 4 rows, sums, 8 rows, look-back
N_BUILD = 40000


@pytest.mark.parametrize("hit", [0.0, 0.02, 0.9])
def test_compaction_at_tile_edges(hit):
    m = N_BUILD * 24
    ob, f = O.Bloom(4, 1, 1, 1, 4, m), F.bbf_32(m, 4, 1, 1)
    ref = ob.alloc()
    ob.insert(ref, keygen.build_keys(N_BUILD, 19))
    words = torch.zeros(f.alloc_words(), dtype=torch.int64)
    words[:len(ref)] = torch.from_numpy(ref.view(np.int64))
    words = words.cuda()
    pk, _ = keygen.probe_keys(N_BUILD, max(EDGES) + 32, hit, 19)
    keys, exp = torch.from_numpy(pk.view(np.int32)).cuda(), ob.batch_contains(ref, pk, 0)
    f.set_probe_options(2, -1)
    for edge in EDGES:
        for n in (edge - 31, edge, edge + 1):
            want = torch.from_numpy(exp[:np.searchsorted(exp, n)].view(np.int32)).cuda()
            out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
            got = f.batch_contains(words, keys, n, out, 0)
            assert got == len(want) and torch.equal(out[:got], want), n
            assert bool((out[got:] == -1).all()), n
