"""Workloads that stand for how this framework is used: joins through its public entry points, from a dimension-table
lookup of a few thousand rows to the 2^26 x 2^28 joins that fill the card, one at a time and in batches.

A join's pairs come in no particular order, so every workload goes on as a query would and puts them where they
belong: the build row of each probe row (-1 without a match) in a column of the probe side, or, for repeated build
keys, each side's payload summed over its partners.  Large joins are selective ones (few probe rows have a match): with
many matches torch's own random scatter of them would take longer than the join.

kind
  one_shot   api.partitioned_join: plans, allocates and joins in one call
  reuse      api.Joiner: plan, workspace and output columns kept, new launch each pass
  payload    api.partitioned_join_payload with repeated build keys (sized by a counting join)
  count      api.join_count: how many pairs a join has, for sizing and for cost estimates
  batch      api.BatchJoiner replayed as a CUDA graph, all joins writing into one flat pair of columns
"""
import math

import torch

from partitioned_join_b200 import api

DEV = "cuda"
# pairs that one pass may scatter over a column larger than L2
MAX_SCATTER = 1 << 25


def listed():
    def join(name, kind, nb, np_, kb, match, zipf=0.0, plan="default"):
        return {"name": name, "kind": kind, "build": nb, "probe": np_, "key_bytes": kb, "match": match, "zipf": zipf,
                "plan": plan}

    return [
        # a lookup in a small dimension table, planned and allocated on the spot: launches and host work
        join("oneshot_1k_4k", "one_shot", 1 << 10, 1 << 12, 4, 0.7),
        # a mid-size dimension with 64-bit ids, sizes as they come
        join("reuse_20k_300k_i64", "reuse", 20011, 300007, 8, 0.8),
        # the plain uniform join of the benchmark's first configuration: a foreign key, every row matches
        join("reuse_1m_4m", "reuse", 1 << 20, 1 << 22, 4, 1.0),
        # 64-bit keys, odd sizes, a filter on the build side
        join("reuse_3m_10m_i64", "reuse", 3000017, 10000019, 8, 0.3),
        # repeated build keys (three rows a key), both payloads materialised and summed
        {"name": "payload_dup_1m_4m", "kind": "payload", "build": 1500007, "probe": 4000037, "key_bytes": 4,
         "match": 0.8, "per_key": 3},
        # equal sides, most rows match
        join("reuse_16m_16m", "reuse", 1 << 24, 1 << 24, 4, 0.9),
        # Zipf-skewed foreign keys (the skew sweep's top exponent), planned from the data's histograms
        join("zipf_16m_64m_i64", "reuse", 1 << 24, 1 << 26, 8, 1.0, 1.5, "exact"),
        # the headline sizes, every probe row with its build row: a selective join
        join("reuse_128m_128m", "reuse", 1 << 27, 1 << 27, 4, 0.125),
        # the headline join's cardinality
        join("count_128m_128m", "count", 1 << 27, 1 << 27, 4, 0.9),
        # the largest: a fact table of 2^28 rows with 64-bit keys
        join("reuse_64m_256m_i64", "reuse", 1 << 26, 1 << 28, 8, 0.125),
        # many joins of uneven sizes (2^10 .. 2^20 build rows, four probe rows each, a quarter of them Zipf-skewed)
        {"name": "batch_128_uneven", "kind": "batch", "joins": 128, "lo": 1 << 10, "hi": 1 << 20, "ratio": 4,
         "key_bytes": 4},
        # many small lookups with 64-bit ids
        {"name": "batch_64_small_i64", "kind": "batch", "joins": 64, "lo": 1 << 8, "hi": 1 << 13, "ratio": 7,
         "key_bytes": 8},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(2 ** rng.uniform(math.log2(lo), math.log2(hi))))

    kind = rng.choice(("one_shot", "reuse", "reuse", "reuse", "payload", "count", "batch"))
    kb = rng.choice((4, 8))
    if kind == "batch":
        hi = size(1 << 11, 1 << 20)
        return {"kind": kind, "joins": min(rng.randint(16, 160), (1 << 27) // hi), "lo": max(1 << 8, hi >> rng.randint(2, 10)),
                "hi": hi, "ratio": rng.choice((1, 3, 4, 7)), "key_bytes": kb}
    if kind == "payload":
        nb = size(1 << 12, 1 << 22)
        return {"kind": kind, "build": nb, "probe": min(1 << 23, size(nb, 8 * nb)), "key_bytes": kb,
                "match": round(rng.uniform(0.1, 1.0), 2), "per_key": rng.randint(2, 4)}
    nb = size(1 << 10, (1 << 21) if kind == "one_shot" else (1 << 26) if kb == 8 else (1 << 27))
    np_ = min(size(nb, 16 * nb), (1 << 23) if kind == "one_shot" else (1 << 27) if kb == 4 else (1 << 28))
    match = rng.uniform(0.1, 1.0)
    if kind != "count" and np_ > (1 << 24):
        match = min(match, MAX_SCATTER / np_)
    zipf = rng.choice((0.0, 0.0, 0.5, 1.0, 1.25, 1.5))
    return {"kind": kind, "build": nb, "probe": np_, "key_bytes": kb, "match": round(match, 4), "zipf": zipf,
            "plan": "exact" if zipf > 0 or rng.random() < 0.3 else "default"}


# ---- inputs ---------------------------------------------------------------

def _signed(x):
    return x - (1 << 64) if x >= 1 << 63 else x


def _mix(i):
    """A bijection of 64-bit integers (the SplitMix64 finaliser, shifts made logical): distinct in, distinct out."""
    def shr(v, s):
        return (v >> s) & ((1 << (64 - s)) - 1)

    i = i * _signed(0x9E3779B97F4A7C15)
    i = (i ^ shr(i, 30)) * _signed(0xBF58476D1CE4E5B9)
    i = (i ^ shr(i, 27)) * _signed(0x94D049BB133111EB)
    return i ^ shr(i, 31)


def _ranks(n, alphabet, theta, g):
    """n ranks in [0, alphabet), by a Zipf(theta) law (the inverse of its continuous distribution function)."""
    if theta == 0.0:
        return torch.randint(0, alphabet, (n,), generator=g, device=DEV)
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    if theta == 1.0:
        u.mul_(math.log(alphabet + 1.0)).exp_()
    else:
        u.mul_((alphabet + 1.0) ** (1.0 - theta) - 1.0).add_(1.0).pow_(1.0 / (1.0 - theta))
    return u.sub_(1.0).long().clamp_(0, alphabet - 1)


def _tables(nb, np_, kb, match, theta, g, seed):
    """Build keys (distinct: 1..nb shuffled, or random 64-bit values) and probe keys: one of them with probability
    match, else a key that no build row holds."""
    if kb == 4:
        build = torch.randperm(nb, generator=g, device=DEV, dtype=torch.int32) + 1
        pick = build[_ranks(np_, nb, theta, g)]
        if match < 1.0:
            miss = torch.rand(np_, generator=g, device=DEV) >= match
            other = torch.randint(nb + 1, (1 << 31) - 1, (np_,), generator=g, device=DEV, dtype=torch.int32)
            pick = torch.where(miss, other, pick)
        return build, pick
    # row r holds _mix(base + r); numbers from base + nb on belong to no row
    base = (seed * 0x9E3779B97F4A7C15 + 1) % (1 << 61)
    build = _mix(torch.arange(base, base + nb, device=DEV))
    at = _ranks(np_, nb, theta, g)
    if match < 1.0:
        miss = torch.rand(np_, generator=g, device=DEV) >= match
        at = torch.where(miss, at + nb, at)
    return build, _mix(at.add_(base))


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    kb, kind = case["key_bytes"], case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        n = case["joins"]
        span = math.log2(case["hi"] / case["lo"])
        # sizes spread evenly over their logarithm, the same for every seed
        nbs = [int(case["lo"] * 2 ** (span * i / max(n - 1, 1))) for i in range(n)]
        pairs = [_tables(nb, nb * case["ratio"], kb, 1.0, 1.0 if i % 4 == 3 else 0.0, g, seed * 512 + i)
                 for i, nb in enumerate(nbs)]
        s["joiner"] = j = api.BatchJoiner(pairs)
        total = sum(p.numel() for _, p in pairs)
        s["build_row"] = torch.empty(total, dtype=torch.int32, device=DEV)
        s["probe_row"] = torch.empty(total, dtype=torch.int32, device=DEV)
        starts, at = [], 0
        for i, (_, p) in enumerate(pairs):
            j.outs[i].build_row = s["build_row"].data_ptr() + 4 * at
            j.outs[i].probe_row = s["probe_row"].data_ptr() + 4 * at
            starts.append(at)
            at += p.numel()
        j.prepare()
        s["first"] = torch.repeat_interleave(torch.tensor(starts, dtype=torch.int32, device=DEV),
                                             torch.tensor([p.numel() for _, p in pairs], device=DEV))
        s["match"] = torch.empty(total, dtype=torch.int32, device=DEV)
        s["graph"] = j.graph()
        return s
    nb, np_ = case["build"], case["probe"]
    if kind == "payload":
        dt = torch.int32 if kb == 4 else torch.int64
        distinct = max(1, nb // case["per_key"])
        s["build"] = torch.randint(0, distinct, (nb,), generator=g, device=DEV, dtype=dt)
        s["probe"] = torch.randint(0, max(1, int(distinct / case["match"])), (np_,), generator=g, device=DEV, dtype=dt)
        s["build_val"] = torch.randint(0, 1000, (nb,), generator=g, device=DEV, dtype=torch.int32)
        s["probe_val"] = torch.randint(0, 1000, (np_,), generator=g, device=DEV, dtype=torch.int32)
        s["by_build"] = torch.empty(nb, dtype=torch.int32, device=DEV)
        s["by_probe"] = torch.empty(np_, dtype=torch.int32, device=DEV)
        return s
    s["build"], s["probe"] = _tables(nb, np_, kb, case["match"], case["zipf"], g, seed)
    s["plan"] = api.plan_exact(s["build"], s["probe"]) if case["plan"] == "exact" else None
    if kind != "count":
        s["match"] = torch.empty(np_, dtype=torch.int32, device=DEV)
    if kind == "reuse":
        s["joiner"] = api.Joiner(s["build"], s["probe"], plan=s["plan"])
    return s


# ---- one pass -------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "count":
        return api.join_count(s["build"], s["probe"], plan=s["plan"])
    if kind == "batch":
        s["graph"].replay()
        # foreign keys: every probe row of every join has its pair
        s["match"].scatter_(0, s["first"] + s["probe_row"], s["build_row"])
        return s["match"], s["joiner"].count
    if kind == "payload":
        br, pr, bv, pv = api.partitioned_join_payload(s["build"], s["probe"], s["build_val"], s["probe_val"],
                                                      unique_build_keys=False)
        s["by_build"].zero_().index_add_(0, br, pv)
        s["by_probe"].zero_().index_add_(0, pr, bv)
        return s["by_build"], s["by_probe"], br.numel()
    if kind == "one_shot":
        br, pr = api.partitioned_join(s["build"], s["probe"], plan=s["plan"])
    else:
        s["joiner"].launch()
        br, pr = s["joiner"].result()
    s["match"].fill_(-1).scatter_(0, pr, br)
    return s["match"], br.numel()


def work(case):
    kb = case["key_bytes"]
    if case["kind"] == "batch":
        n, span = case["joins"], math.log2(case["hi"] / case["lo"])
        nb = sum(int(case["lo"] * 2 ** (span * i / max(n - 1, 1))) for i in range(n))
        return {"bytes": nb * kb + nb * case["ratio"] * (kb + 4) + 8 * n, "flops": 0}
    nb, np_ = case["build"], case["probe"]
    if case["kind"] == "payload":
        return {"bytes": (nb + np_) * (kb + 4 + 4), "flops": 0}
    return {"bytes": (nb + np_) * kb + (8 if case["kind"] == "count" else 4 * np_), "flops": 0}
