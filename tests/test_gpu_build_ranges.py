"""The range-by-range Bloom build: the same words as the one-kernel build (and
the oracle's) over layouts, addressing, ragged tiles and last ranges, words
that already hold keys, and key sets that overfill one range's bucket."""
import numpy as np
import pytest

import dtlg as F
import oracle as O
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N = 1 << 22        # from here on a build may be range by range
BIG = 48 << 20     # from here on every layout is, in a filter that fits L2


def _filter(layout, m):
    wb, w, s, z, k = layout
    return F.construct(F.blocked_bloomfilter_config(k, wb, w, s, 0, z), m)


def _both(f, keys, words=None):
    auto = f.alloc_filter_data() if words is None else words.clone()
    direct = auto.clone()
    assert f.batch_insert(auto, keys)
    f.set_build_options(1)
    assert f.batch_insert(direct, keys)
    f.set_build_options(0)
    return auto, direct


@pytest.mark.parametrize("m", [1 << 24, 5 * (1 << 22) + 777, 3 * (1 << 27) + 12345], ids=["pow2", "magic", "magic48M"])
@pytest.mark.parametrize("layout", [(8, 8, 8, 1, 8), (8, 16, 16, 1, 16), (4, 16, 16, 4, 8), (4, 16, 1, 1, 4),
                                    (8, 8, 2, 1, 8), (4, 16, 8, 1, 16)])
def test_words_equal_one_kernel_build(layout, m):
    f = _filter(layout, m)
    keys = keygen.build_keys_torch(N + (1 << 14) + 5, 31)
    for first, n in ((0, N), (1, N + (1 << 14) - 1), (3, N + (1 << 14) + 2)):
        auto, direct = _both(f, keys[first:first + n])
        assert torch.equal(auto, direct), (first, n)


@pytest.mark.parametrize("layout", [(4, 1, 1, 1, 4), (8, 1, 1, 1, 8), (4, 2, 1, 1, 6), (8, 4, 4, 1, 8), (8, 8, 8, 2, 8)])
def test_words_equal_many_keys(layout):
    f = _filter(layout, 3 * (1 << 24) + 999)
    auto, direct = _both(f, keygen.build_keys_torch(BIG + 321, 32)[1:])
    assert torch.equal(auto, direct)


def test_large_filter_and_words_in_place():
    f = _filter((8, 8, 8, 1, 8), 1 << 30)                       # 128 MiB
    first = f.alloc_filter_data()
    f.set_build_options(1)
    assert f.batch_insert(first, keygen.build_keys_torch(1 << 20, 33))
    f.set_build_options(0)
    auto, direct = _both(f, keygen.build_keys_torch(N, 34), first)
    assert torch.equal(auto, direct)
    assert bool(((auto & first) == first).all())


def test_overfull_range_and_oracle():
    """Most keys hash into the first of the ranges: its bucket overflows, and
    the rest goes straight into the words."""
    m = 1 << 25
    keys = keygen.build_keys(4 * N, 35)
    skew = keys[(keys.astype(np.uint64) * np.uint64(596572387) & np.uint64(0xFFFFFFFF)) < np.uint64(1 << 28)]
    ks = np.concatenate([np.tile(skew, 1 + 3 * N // len(skew)), keys[:N // 4]])
    f, ob = _filter((8, 8, 8, 1, 8), m), O.Bloom(8, 8, 8, 1, 8, m)
    auto, direct = _both(f, torch.from_numpy(ks.view(np.int32)).cuda())
    assert torch.equal(auto, direct)
    ref = ob.alloc()
    ob.insert(ref, np.unique(ks))
    assert np.array_equal(auto.cpu().numpy().view(np.uint64)[:len(ref)], ref)
