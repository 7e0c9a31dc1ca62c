"""Every build plan by name: the range-by-range build of filters beyond a few
MiB under MAGIC addressing and the build through the partition, against the
one-kernel build's words, with the plan each batch takes checked."""
import pytest

import dtlg as F
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _filter(layout, m):
    wb, w, s, z, k = layout
    return F.construct(F.blocked_bloomfilter_config(k, wb, w, s, 0, z), m)


def _equal_plans(f, keys, mode, plan):
    f.set_build_options(mode)
    assert f.build_plan(keys.numel()) == plan
    got, want = f.alloc_filter_data(), f.alloc_filter_data()
    assert f.batch_insert(got, keys)
    f.set_build_options(1)
    assert f.batch_insert(want, keys)
    f.set_build_options(0)
    assert torch.equal(got, want)


@pytest.mark.parametrize("layout", [(8, 8, 8, 1, 8), (8, 16, 16, 1, 16), (4, 16, 16, 4, 8), (4, 16, 1, 1, 4),
                                    (8, 8, 2, 1, 8), (4, 16, 8, 1, 16)])
def test_range_build_of_48_mib_magic(layout):
    f = _filter(layout, 3 * (1 << 27) + 12345)
    keys = keygen.build_keys_torch((1 << 23) + 4097, 41)
    for first, n in ((0, 1 << 23), (3, (1 << 23) + 4094)):
        _equal_plans(f, keys[first:first + n], 0, 3)


@pytest.mark.parametrize("layout,m", [((8, 8, 8, 1, 8), 1 << 31), ((8, 8, 8, 2, 8), (3 << 29) + 4096)])
def test_partitioned_build_of_large_filters(layout, m):
    """Many ranges, none overflowing; automatically such batches are built
    range by range."""
    f, keys = _filter(layout, m), keygen.build_keys_torch(1 << 25, 91)
    _equal_plans(f, keys, 2, 2)
    _equal_plans(f, keys, 0, 3)


@pytest.mark.parametrize("layout", [(8, 8, 8, 1, 8), (4, 1, 1, 1, 4)])
def test_automatic_partitioned_build(layout):
    """Few keys for the filter's size: the partition is the automatic plan."""
    f = _filter(layout, 3 << 30)
    _equal_plans(f, keygen.build_keys_torch(1 << 22, 92)[1:], 0, 2)
