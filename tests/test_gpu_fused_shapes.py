"""The fused probe (plan 1) at the edges of its tile shapes: match lists equal
the oracle's where a batch goes from one tile to several, from one key per
thread to four, and from tiles of one round to tiles of four."""
import numpy as np
import pytest

import dtlg as F
import oracle as O
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGES = [1024, 256 * 5, 148 << 10, 2 << 20]  # one tile, ragged, four keys per thread, four rounds
N_BUILD = 40000


@pytest.fixture(scope="module", params=[(8, 8, 8, 1, 8), (4, 1, 1, 1, 4)], ids=["sectorized", "register"])
def case(request):
    wb, w, s, z, k = request.param
    m = N_BUILD * 12
    ob, f = O.Bloom(wb, w, s, z, k, m), F.construct(F.blocked_bloomfilter_config(k, wb, w, s, 0, z), m)
    ref = ob.alloc()
    ob.insert(ref, keygen.build_keys(N_BUILD, 8))
    words = torch.zeros(f.alloc_words(), dtype=torch.int64)
    words[:len(ref)] = torch.from_numpy(ref.view(np.int64))
    pk, _ = keygen.probe_keys(N_BUILD, max(EDGES) + 4, 0.3, 8)
    f.set_probe_options(1, -1)
    return f, words.cuda(), torch.from_numpy(pk.view(np.int32)).cuda(), ob.batch_contains(ref, pk, 0)


def test_slots_are_clean_between_calls_streams_and_threads(case):
    """Blocking calls share a bounded set of scratch slots: calls of different
    sizes, from more threads than slots, each on a stream of its own."""
    import threading
    f, words, keys, exp = case
    bad = []

    def work(t):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(12):
                n = (1 + 1031 * t + 70001 * i) % (1 << 20) + 1
                out = torch.empty(n, dtype=torch.int32, device="cuda")
                want = int(np.searchsorted(exp, n))
                got = f.batch_contains(words, keys, n, out, 0)
                if got != want or not np.array_equal(out[:got].cpu().numpy().view(np.uint32), exp[:got]):
                    bad.append((t, i, n, got, want))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(t,)) for t in range(20)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


@pytest.mark.parametrize("edge", EDGES)
def test_fused_probe_at_shape_edges(case, edge):
    f, words, keys, exp = case
    for n in (edge - 1, edge, edge + 1):
        for pad in (0, 3):
            want = exp[(exp >= pad) & (exp < pad + n)] - np.uint32(pad) + np.uint32(7)
            out = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda")
            got = f.batch_contains(words, keys[pad:pad + n], n, out, 7)
            assert got == len(want), (n, pad)
            assert np.array_equal(out[:got].cpu().numpy().view(np.uint32), want), (n, pad)
            assert bool((out[got:] == -1).all()), (n, pad)


def test_compaction_at_shape_edges():
    """The bitmask plan where the compaction's tiles grow from one row of mask
    words to two, four and eight."""
    edges = [1 << 23, 1 << 24, 1 << 25]
    m = N_BUILD * 12
    ob, f = O.Bloom(4, 1, 1, 1, 4, m), F.bbf_32(m, 4, 1, 1)
    ref = ob.alloc()
    ob.insert(ref, keygen.build_keys(N_BUILD, 9))
    words = torch.zeros(f.alloc_words(), dtype=torch.int64)
    words[:len(ref)] = torch.from_numpy(ref.view(np.int64))
    words = words.cuda()
    pk, _ = keygen.probe_keys(N_BUILD, max(edges) + 32, 0.2, 9)
    keys, exp = torch.from_numpy(pk.view(np.int32)).cuda(), ob.batch_contains(ref, pk, 0)
    f.set_probe_options(2, -1)
    for edge in edges:
        for n in (edge - 31, edge, edge + 1):
            want = torch.from_numpy(exp[:np.searchsorted(exp, n)].view(np.int32)).cuda()
            out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
            got = f.batch_contains(words, keys, n, out, 0)
            assert got == len(want) and torch.equal(out[:got], want), n
            assert bool((out[got:] == -1).all()), n
