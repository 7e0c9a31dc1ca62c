"""The work that programs have this framework do, as cases that can be timed.

A case is one call, or a few calls that go together, through the public entry
points (`dtlg.filter_base`, `dtlg.batch.Batch`), with the inputs that such a
program has in hand:

  probe   batch_contains of device keys: ascending match positions and their count
  build   zeroed words and one batch_insert (Bloom filters: equal words)
  join    build, then probe, the build side of a semi-join (cuckoo kinds, whose
          words may legally differ from build to build: their match list may not)
  gather  batch_contains fused with the gather of two payload columns
  batch   many filters built and probed in one persistent launch
  host    batch_contains over pinned host buffers

A match list comes back in the caller's buffer, which is as long as the keys,
and its length as a number; what lies past it keeps the zeros of `prepare`.

Sizes run from the 1024-key batches of the reference's own benchmark to the
2^28 keys of bench.py's headline workload, filters from what fits in L1 to 512
MiB, hit ratios from 1 % to 50 %.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bloomfilter-bsd_b200"))

import dtlg  # noqa: E402
from dtlg import keygen  # noqa: E402
from dtlg.batch import Batch, BatchItem  # noqa: E402

# Layouts of blocked Bloom filters: word bytes, words per block, sectors, zones, bits per key.
SECTORIZED = dict(kind="bloom", word=8, w=8, s=8, z=1, k=8)    # bench.py's headline layout
REGISTER = dict(kind="bloom", word=4, w=1, s=1, z=1, k=4)      # one word per key
LAYOUTS = [
    SECTORIZED,
    REGISTER,
    dict(kind="bloom", word=4, w=1, s=1, z=1, k=8),            # blocked_bloomfilter_config()'s defaults
    dict(kind="bloom", word=8, w=8, s=8, z=2, k=8),            # zoned, as in the batched workload
    dict(kind="bloom", word=8, w=8, s=8, z=4, k=8),
    dict(kind="bloom", word=4, w=16, s=16, z=2, k=8),
    dict(kind="bloom", word=4, w=16, s=16, z=4, k=8),
    dict(kind="bloom", word=8, w=4, s=4, z=1, k=8),            # 32-byte blocks
    dict(kind="bloom", word=4, w=8, s=8, z=1, k=8),
    dict(kind="bloom", word=4, w=16, s=1, z=1, k=4),           # sectors wider than a word
    dict(kind="bloom", word=4, w=16, s=8, z=1, k=8),
    dict(kind="bloom", word=8, w=8, s=2, z=1, k=8),
]
CUCKOO = [dict(kind="cuckoo", tag=16, assoc=4), dict(kind="cuckoo", tag=12, assoc=4), dict(kind="cuckoo", tag=8, assoc=4)]
BCF = dict(kind="bcf", block=64, tag=16, assoc=4)              # dtl::bcf's defaults
CLASSIC = dict(kind="classic", k=4)
BATCH_LAYOUTS = [LAYOUTS[i] for i in (0, 3, 4, 5, 6)]


def listed():
    return [
        # a vectorised engine's smallest batch (the reference benchmarks 1024
        # keys at a time) against a small filter: latency and launches
        dict(name="probe_1k", op="probe", **LAYOUTS[2], n_build=20000, bits=16, n_probe=1024, hit=0.1),
        # one morsel of an operator, half of it passing, odd in length
        dict(name="probe_60k", op="probe", **LAYOUTS[6], n_build=150000, bits=12, n_probe=60001, hit=0.5),
        # a column chunk just under a million rows, L2-resident filter
        dict(name="probe_900k", op="probe", **SECTORIZED, n_build=1 << 22, bits=16, n_probe=900001, hit=0.1),
        # bench.py's register_blocked workload: few cache lines, many keys
        dict(name="probe_16m_register", op="probe", **REGISTER, n_build=1 << 20, bits=16, n_probe=1 << 24, hit=0.1),
        # a selective probe of a large L2-resident filter
        dict(name="probe_128m_l2", op="probe", **SECTORIZED, n_build=1 << 26, bits=8, n_probe=1 << 27, hit=0.01),
        # bench.py's headline workload: 512 MiB of words, 2^28 keys
        dict(name="probe_256m_dram", op="probe", **SECTORIZED, n_build=1 << 28, bits=16, n_probe=1 << 28, hit=0.1),
        # bench.py's cuckoo workload at half its probe keys
        dict(name="probe_128m_cuckoo", op="probe", **CUCKOO[0], n_build=1 << 26, load=0.95, n_probe=1 << 27, hit=0.1),
        # the build side of a join: a dimension table, and a large fact table
        dict(name="build_4m", op="build", **SECTORIZED, n_build=1 << 22, bits=16),
        dict(name="build_128m", op="build", **SECTORIZED, n_build=1 << 27, bits=16),
        # semi-join over a cuckoo filter, built for this query
        dict(name="join_3m_cuckoo", op="join", **CUCKOO[0], n_build=3000001, load=0.9, n_probe=5000003, hit=0.2),
        # a plan with one filter per partition: uneven sizes, one launch
        dict(name="batch_64", op="batch", filters=64, max_log2=21, hit=0.05),
        # keys that live on the host, positions wanted on the host
        dict(name="host_24m", op="host", **SECTORIZED, n_build=1 << 22, bits=16, n_probe=24000001, hit=0.1),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [2^lo, 2^hi]."""
    return int(2 ** rng.uniform(lo, hi))


def draw(rng):
    op = rng.choices(["probe", "build", "join", "gather", "batch", "host"], [9, 5, 2, 2, 1, 1])[0]
    hit = rng.choice([0.01, 0.05, 0.1, 0.2, 0.5])
    if op == "batch":
        return dict(op=op, filters=rng.randint(8, 96), max_log2=rng.randint(14, 21), hit=hit)
    kinds = LAYOUTS + [SECTORIZED] * 3
    if op == "join":
        kinds = CUCKOO + [BCF]
    elif op != "build":
        kinds = kinds + CUCKOO[:2] + [BCF, CLASSIC]
    kind = rng.choice(kinds)
    case = dict(op=op, **kind)
    # a classic filter's k words lie anywhere in it, so it is used while it
    # stays in L2; a join builds its filter anew for each query
    case["n_build"] = _log(rng, 10, 23 if kind in (CLASSIC, BCF) else 24 if op == "join" else 26.5)
    if kind["kind"] == "cuckoo":
        case["load"] = rng.choice([0.8, 0.9])
    elif kind["kind"] != "bcf":
        case["bits"] = rng.choice([8, 12, 16])
    if op != "build":
        case["n_probe"] = _log(rng, 10, 25 if op in ("host", "gather") else 27)
        case["hit"] = hit
    return case


def _cuckoo_bits(n, t, b, load):
    """Bits for n keys at `load` with an odd MAGIC bucket count (an even one
    stalls near 75 % occupancy, in the reference as here)."""
    buckets = int(-(-n // (b * load)))
    while True:
        f = dtlg.cf(buckets * t * b, t, b)
        if f.is_magic() and f.block_cnt() % 2 == 1 and f.block_cnt() * b * load >= n:
            return buckets * t * b
        buckets += 1


def _construct(c):
    if c["kind"] == "bloom":
        cfg = dtlg.blocked_bloomfilter_config(k=c["k"], word_size=c["word"], word_cnt_per_block=c["w"],
                                              sector_cnt=c["s"], zone_cnt=c["z"])
        return dtlg.construct(cfg, c["n_build"] * c["bits"])
    if c["kind"] == "cuckoo":
        return dtlg.cf(_cuckoo_bits(c["n_build"], c["tag"], c["assoc"], c["load"]), c["tag"], c["assoc"])
    if c["kind"] == "bcf":
        # a sixteenth of the slots: no bucket overflows, so the match list
        # does not depend on the order in which the keys were placed
        return dtlg.bcf(c["n_build"] * 16 * c["tag"] + 4096, c["block"], c["tag"], c["assoc"])
    # POW2: under MAGIC addressing every key of a classic filter sets bit 0 of
    # its words (as the reference does), which fills it up
    return dtlg.bloomfilter_logic(1 << (c["n_build"] * c["bits"] - 1).bit_length(), c["k"], dtlg.POWER_OF_TWO)


def _probe_side(c, seed):
    keys, _ = keygen.probe_keys_torch(c["n_build"], c["n_probe"], c["hit"], seed)
    return keys, torch.zeros(c["n_probe"], dtype=torch.int32, device="cuda")


def _prepare_batch(c, seed):
    rng = np.random.default_rng(seed)
    plan = []
    # the sizes belong to the case, the keys to the seed
    sizes = np.random.default_rng(c["filters"] * 100 + c["max_log2"])
    for _ in range(c["filters"]):
        lay = BATCH_LAYOUTS[int(sizes.integers(0, len(BATCH_LAYOUTS)))]
        n, p = int(2 ** sizes.uniform(10, c["max_log2"])), int(2 ** sizes.uniform(12, c["max_log2"]))
        bits = int(sizes.choice([8, 12, 16]))
        plan.append((_construct(dict(lay, n_build=n, bits=bits)), n, p))
    pad = lambda v, a: -(-v // a) * a  # noqa: E731
    words = torch.zeros(sum(pad(f.alloc_words(), 4) for f, _, _ in plan), dtype=torch.int64, device="cuda")
    pos = torch.zeros(sum(pad(p, 4) for _, _, p in plan), dtype=torch.int32, device="cuda")
    cnt = torch.zeros(len(plan), dtype=torch.int64, device="cuda")
    items, wo, po = [], 0, 0
    for i, (f, n, p) in enumerate(plan):
        ks = int(rng.integers(1, 1 << 30))
        bk = keygen.build_keys_torch(n, ks)
        pk, _ = keygen.probe_keys_torch(n, p, c["hit"], ks)
        items.append(BatchItem(f, words[wo:wo + f.alloc_words()], bk, pk, pos[po:po + p], cnt[i:i + 1], 0))
        wo += pad(f.alloc_words(), 4)
        po += pad(p, 4)
    return dict(op="batch", words=words, pos=pos, cnt=cnt, items=items, batch=Batch(items))


def prepare(case, seed):
    c = case
    if c["op"] == "batch":
        return _prepare_batch(c, seed)
    f = _construct(c)
    st = dict(op=c["op"], f=f, words=f.alloc_filter_data())
    build = keygen.build_keys_torch(c["n_build"], seed)
    if c["op"] == "build":
        st["build"] = build
        return st
    if c["op"] == "join":
        st["build"] = build
        st["keys"], st["pos"] = _probe_side(c, seed)
        return st
    f.batch_insert(st["words"], build)
    st["keys"], st["pos"] = _probe_side(c, seed)
    if c["op"] == "gather":
        n = c["n_probe"]
        st["cols"] = [torch.arange(n, dtype=torch.int32, device="cuda") * 3 + seed % 1000,
                      torch.arange(n, dtype=torch.int64, device="cuda") * 5 + seed % 1000]
        st["out"] = [torch.zeros_like(x) for x in st["cols"]]
    if c["op"] == "host":
        pinned = st["keys"].cpu().pin_memory()
        out = torch.zeros(c["n_probe"], dtype=torch.int32).pin_memory()
        st.update(pinned=(pinned, out), keys=pinned.numpy().view(np.uint32), pos=out.numpy().view(np.uint32))
    return st


def run(state):
    st, op = state, state["op"]
    if op == "batch":
        st["words"].zero_()
        st["batch"].run()
        return {"words": st["words"], "pos": st["pos"], "cnt": st["cnt"]}
    f, words = st["f"], st["words"]
    if op == "build":
        words.zero_()
        f.batch_insert(words, st["build"])
        return words
    if op == "host":
        n = f.batch_contains_host(words, st["keys"], st["pos"])
        return {"n": n, "pos": st["pos"]}
    if op == "gather":
        n = f.batch_contains_gather(words, st["keys"], st["cols"], st["out"], match_positions=st["pos"])
        return {"n": n, "pos": st["pos"], "cols": st["out"]}
    ok = True
    if op == "join":
        words.zero_()
        ok = f.batch_insert(words, st["build"])
    n = f.batch_contains(words, st["keys"], st["keys"].numel(), st["pos"])
    return {"ok": ok, "n": n, "pos": st["pos"]}


def _filter_bytes(c):
    if c["kind"] == "cuckoo":
        return c["n_build"] / c["load"] * c["tag"] / 8
    if c["kind"] == "bcf":
        return c["n_build"] * 16 * c["tag"] / 8
    if c["kind"] == "classic":
        return (1 << (c["n_build"] * c["bits"] - 1).bit_length()) / 8
    return c["n_build"] * c["bits"] / 8


def work(case):
    c = case
    if c["op"] == "batch":
        sizes = np.random.default_rng(c["filters"] * 100 + c["max_log2"])
        total = 0.0
        for _ in range(c["filters"]):
            sizes.integers(0, len(BATCH_LAYOUTS))
            n, p = int(2 ** sizes.uniform(10, c["max_log2"])), int(2 ** sizes.uniform(12, c["max_log2"]))
            bits = int(sizes.choice([8, 12, 16]))
            total += 4 * n + 2 * n * bits / 8 + 4 * p * (1 + c["hit"])
        return {"bytes": total, "flops": 0}
    fb = _filter_bytes(c)
    if c["op"] == "build":
        return {"bytes": 4 * c["n_build"] + fb, "flops": 0}
    n = c["n_probe"]
    # the keys, the match list, and the filter's words once (at most one
    # 32-byte sector of them per key)
    total = 4 * n + 4 * c["hit"] * n + min(fb, 32.0 * n)
    if c["op"] == "join":
        total += 4 * c["n_build"] + fb
    if c["op"] == "gather":
        total += 24 * c["hit"] * n
    return {"bytes": total, "flops": 0}
