"""Range builds whose keys repeat: buckets overflow, the scatter inserts what
does not fit, and the range build tests bits first.  The words equal those of
the one-kernel build for every shape of a layout's draws (one to sixteen word
groups, one and several bits per group, fixed and drawn words)."""
import pytest

import dtlg as F
from dtlg import keygen

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

N = (1 << 22) + 777
LAYOUTS = [(8, 8, 8, 1, 8), (4, 1, 1, 1, 8), (8, 1, 1, 1, 16), (4, 2, 1, 1, 6), (4, 16, 16, 4, 8), (8, 8, 8, 4, 8),
           (8, 4, 4, 1, 12), (4, 16, 8, 1, 16), (8, 16, 16, 1, 16), (4, 16, 1, 1, 3)]


def _check(f, keys):
    assert f.build_plan(keys.numel()) == 3
    auto, direct = f.alloc_filter_data(), f.alloc_filter_data()
    assert f.batch_insert(auto, keys)
    f.set_build_options(1)
    assert f.batch_insert(direct, keys)
    f.set_build_options(0)
    assert torch.equal(auto, direct)


def _copies(distinct, n, ordered):
    g = torch.Generator(device="cuda")
    g.manual_seed(distinct)
    i = torch.randint(0, distinct, (n,), device="cuda", generator=g)
    return keygen.build_keys_torch(max(distinct, 4), 61)[i.sort().values if ordered else i].contiguous()


@pytest.mark.parametrize("m", [1 << 30, 100 << 23], ids=["pow2", "magic"])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_repeated_keys(layout, m):
    wb, w, s, z, k = layout
    f = F.construct(F.blocked_bloomfilter_config(k, wb, w, s, 0, z), m + (12345 if m != 1 << 30 else 0))
    for distinct, ordered in ((1, False), (300, False), (20000, False), (50000, True)):
        _check(f, _copies(distinct, N, ordered)[1:])


@pytest.mark.parametrize("m", [1 << 24, 3 * (1 << 23) + 999], ids=["pow2", "magic"])
def test_one_hot_key_among_many(m):
    """Half the batch one key, the rest distinct, in a small filter."""
    f = F.construct(F.blocked_bloomfilter_config(8, 8, 8, 8, 0, 1), m)
    keys = keygen.build_keys_torch(N, 62)
    keys[torch.randint(0, 2, (N,), device="cuda").bool()] = 4242
    _check(f, keys)
