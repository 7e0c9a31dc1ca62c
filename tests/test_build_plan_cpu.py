"""The automatic build plan (host logic only): range by range in shared memory
for large batches into filters of enough ranges to fill the GPU, else the
plans of global atomics."""
import pytest

import dtlg as F


def _filter(layout, kib):
    wb, w, s, z, k = layout
    return F.construct(F.blocked_bloomfilter_config(k, wb, w, s, 0, z), kib << 13)


@pytest.mark.parametrize("layout", [(8, 8, 8, 1, 8), (4, 16, 16, 2, 8), (8, 8, 2, 1, 8), (4, 1, 1, 1, 4),
                                    (8, 4, 4, 1, 8), (8, 8, 8, 4, 8)])
def test_few_ranges_keep_the_one_kernel_build(layout):
    for kib in (8, 16, 64, 100, 256, 500):
        for ln in (22, 24, 26, 30):
            assert _filter(layout, kib).build_plan(1 << ln) == 1, (kib, ln)
    assert _filter(layout, 2048).build_plan(1 << 26) == 3


@pytest.mark.parametrize("layout,kib,n,plan", [
    ((8, 8, 8, 1, 8), 512, 1 << 22, 3), ((8, 8, 8, 1, 8), 8192, 1 << 22, 3),
    ((8, 8, 8, 1, 8), 8192, (1 << 22) - 1, 1), ((8, 8, 8, 1, 8), 64 << 10, 1 << 22, 1),
    ((8, 8, 8, 1, 8), 64 << 10, 1 << 23, 3), ((8, 8, 8, 1, 8), 128 << 10, 1 << 22, 3),
    ((8, 8, 8, 1, 8), 256 << 10, 1 << 22, 2), ((8, 8, 8, 1, 8), 512 << 10, 1 << 28, 3),
    ((4, 1, 1, 1, 4), 8192, 1 << 25, 1), ((4, 1, 1, 1, 4), 8192, 48 << 20, 3),
    ((8, 4, 4, 1, 8), 1024, 1 << 26, 1),
])
def test_plan_by_batch_and_filter_size(layout, kib, n, plan):
    f = _filter(layout, kib)
    assert f.build_plan(n) == plan
    for mode in (1, 2):
        f.set_build_options(mode)
        assert f.build_plan(n) == mode
    f.set_build_options(0)
    assert f.build_plan(0) == 0


def test_other_kinds():
    assert F.cf(1 << 20, 16, 4).build_plan(1 << 24) == 1
    assert F.bcf(1 << 26, 64, 16, 4).build_plan(1 << 24) == 1
    assert F.bloomfilter_logic(1 << 20, 4, F.POWER_OF_TWO).build_plan(1 << 24) == 1
