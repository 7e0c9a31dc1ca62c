"""Bloom inserts that run at the same time: batches inserted into the same
words from several streams (and single keys beside them) leave the words that
one insert after the other leaves, whatever plan each batch takes."""
import pytest

import dtlg as F
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PART = 1 << 22  # from here on a build may be range by range


@pytest.mark.parametrize("m", [1 << 26, 3 * (1 << 25) + 4321, 1 << 30], ids=["pow2", "magic", "128MiB"])
@pytest.mark.parametrize("layout", [(8, 8, 8, 1, 8), (4, 16, 16, 2, 8), (8, 8, 2, 1, 8)])
def test_inserts_from_several_streams(layout, m):
    wb, w, s, z, k = layout
    f = F.construct(F.blocked_bloomfilter_config(k, wb, w, s, 0, z), m)
    keys = keygen.build_keys_torch(5 * PART, 51)
    parts = [keys[i * PART:(i + 1) * PART] for i in range(4)] + [keys[4 * PART:4 * PART + 1000]]
    f.set_build_options(1)
    want = f.alloc_filter_data()
    for p in parts:
        assert f.batch_insert(want, p)
    f.set_build_options(0)
    streams = [torch.cuda.Stream() for _ in parts]
    for _ in range(4):
        got = f.alloc_filter_data()
        torch.cuda.synchronize()
        for p, st in zip(parts, streams):
            with torch.cuda.stream(st):
                assert f.batch_insert(got, p)
        torch.cuda.synchronize()
        assert torch.equal(got, want)


def test_builds_of_different_sizes_from_several_threads():
    """Builds with different numbers and sizes of ranges (and so of shared
    memory) at the same time, each thread with filters and a stream of its own:
    every one succeeds and leaves the words of the one-kernel build."""
    import threading
    keys = keygen.build_keys_torch(1 << 23, 52)
    sizes = [5 << 23, 1 << 25, 1 << 27, 200 << 23, 300 << 20, 130 << 23]
    bad = []
    torch.cuda.synchronize()

    def work(t):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(6):
                f = F.construct(F.blocked_bloomfilter_config(8, 8, 8, 8, 0, 1), sizes[(t + i) % len(sizes)])
                got, want = f.alloc_filter_data(), f.alloc_filter_data()
                try:
                    assert f.batch_insert(got, keys)
                    f.set_build_options(1)
                    assert f.batch_insert(want, keys)
                    if not torch.equal(got, want):
                        bad.append((t, i, "words differ"))
                except Exception as e:  # noqa: BLE001
                    bad.append((t, i, repr(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]
