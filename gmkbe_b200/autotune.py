"""Autotuner for the warp engine: occupancy, edge-hash capacity, intersection
strategy and per-degree-bucket chunking, per graph.

For one (graph, k, result limit) it times short enumerations and keeps the
fastest setting, by coordinate descent from the defaults (each knob in turn
over its values, the others fixed; `passes` rounds):
  * warps        resident search warps as a fraction of the occupancy limit
                 (the block-size / occupancy choice: one-warp blocks, fewer of
                 them per SM);
  * hash_load    the edge hash's maximum load in percent (its capacity:
                 gmk_graph_set_hash_load);
  * bits_min     k >= 2: the intersection strategy by list length -- candidate
                 lists of at least this many entries are filtered by bitmaps,
                 shorter ones by edge-hash probes (0xFFFFFFFF: probes only);
  * bucket_scale per root-degree bucket b = floor(log32 deg) (the reference's
                 32^b groups, include/partition.cuh:1136-1190): a factor on the
                 roots' costs, so that bucket's roots are cut into more (or
                 fewer) tasks by the planner -- the chunk size per bucket;
  * tasks_per_worker, donate_min_nodes, pair_limit: the planner's task count,
                 the in-launch sharing threshold (0: the kernel's own), the
                 node-rule threshold.
The defaults are what a run without any of these options uses.  A graph of at
most 128 vertices a side goes to its own kernel with them; other values of
bits_min and pair_limit are rules of the list-based one and take it there.
None of them changes the result set.  Winners are cached in a JSON file keyed
by graph fingerprint, k and limit, so a graph is tuned once.
"""
from __future__ import annotations

import json
import os
import time

import numpy as np

from .api import Graph

NONE = 0xFFFFFFFF
DEFAULTS = dict(warps=1.0, hash_load=25, bits_min=64, bucket_scale=(1.0, 1.0, 1.0),
                tasks_per_worker=8, donate_min_nodes=0, pair_limit=4096)
CHOICES = {
    "warps": [0.5, 0.75, 1.0],
    "hash_load": [25, 50, 90],
    "bits_min": [32, 64, 256, NONE],
    "bucket_scale": [(1.0, 1.0, 1.0), (1.0, 2.0, 4.0), (1.0, 4.0, 16.0), (2.0, 1.0, 1.0),
                     (0.5, 1.0, 2.0)],
    "tasks_per_worker": [2, 8, 32],
    "donate_min_nodes": [0, 4, 64],
    "pair_limit": [1024, 4096, 16384],
}


def degree_buckets(g_host, n_left: int) -> np.ndarray:
    """floor(log32 deg) of every root, capped at 2 (the root's degree bucket)."""
    deg = np.diff(np.asarray(g_host.offsets[: n_left + 1], dtype=np.int64))
    b = np.zeros(n_left, np.int64)
    b[deg > 32] = 1
    b[deg > 1024] = 2
    return b


def scaled_costs(base: np.ndarray, buckets: np.ndarray, scale) -> np.ndarray:
    return (base * np.asarray(scale, np.float64)[buckets]).astype(np.float32)


def _key(g: Graph, k: int, limit: int) -> str:
    return f"{g.fingerprint():016x}:k{k}:r{limit}"


def apply(g: Graph, settings: dict, base_cost: np.ndarray, buckets: np.ndarray,
          max_threads: int) -> dict:
    """enumerate() keyword arguments for `settings` (and the hash load, set on g)."""
    g.set_hash_load(int(settings["hash_load"]))
    warps = max(1, int(max_threads // 32 * settings["warps"]))
    return dict(schedule="ordered", task_cost=scaled_costs(base_cost, buckets,
                                                            settings["bucket_scale"]),
                threads=warps * 32, bits_min_list=int(settings["bits_min"]),
                tasks_per_worker=int(settings["tasks_per_worker"]),
                donate_min_nodes=int(settings["donate_min_nodes"]),
                pair_limit=int(settings["pair_limit"]))


def tune(g: Graph, g_host, k: int, base_cost: np.ndarray, result_limit: int = 0,
         repeats: int = 2, passes: int = 1, cache_path: str | None = None,
         knobs=None) -> dict:
    """Best settings for enumerating g at k (device time per result, lower is
    better), starting from DEFAULTS.  g_host: the graphgen.Graph of g (for the
    degree buckets); base_cost: per-root costs (the model's prediction or
    gmk_root_costs).  Returns {"settings", "ms", "default_ms", "gain",
    "results", "cached", "trials"}."""
    cache_path = cache_path or os.environ.get("GMK_AUTOTUNE_CACHE")
    key = _key(g, k, result_limit)
    cache = {}
    if cache_path and os.path.exists(cache_path):
        with open(cache_path) as f:
            cache = json.load(f)
        if key in cache:
            out = dict(cache[key], cached=True)
            out["settings"]["bucket_scale"] = tuple(out["settings"]["bucket_scale"])
            return out
    buckets = degree_buckets(g_host, g.n_left)
    max_threads = g.enumerate(k=k, result_limit=max(1, min(result_limit or 1000, 1000))).threads
    trials = []

    def run(settings):
        kw = apply(g, settings, base_cost, buckets, max_threads)
        ms, count = [], 0
        for _ in range(repeats + 1):
            st = g.enumerate(k=k, result_limit=result_limit, **kw)
            ms.append(st.kernel_ms)
            count = st.count
        best = min(ms[1:])
        trials.append({"settings": dict(settings), "ms": best, "results": count})
        return best / max(1, count), best, count

    best_s = dict(DEFAULTS)
    best_v, default_ms, results = run(best_s)
    for _ in range(passes):
        for knob in knobs or CHOICES:
            if knob == "bits_min" and k < 2:
                continue
            for val in CHOICES[knob]:
                if val == best_s[knob]:
                    continue
                s = dict(best_s, **{knob: val})
                v, _, _ = run(s)
                if v < best_v * 0.98:          # 2 %: below the run-to-run noise
                    best_v, best_s = v, s
    g.set_hash_load(int(best_s["hash_load"]))
    best_ms = best_v * max(1, results)
    out = {"settings": best_s, "ms": best_ms, "default_ms": default_ms,
           "gain": default_ms / best_ms if best_ms else None, "results": results,
           "trials": trials, "tuned_at": time.time()}
    if cache_path:
        cache[key] = out
        tmp = cache_path + f".tmp{os.getpid()}"
        with open(tmp, "w") as f:
            json.dump(cache, f, indent=1)
        os.replace(tmp, cache_path)
    return dict(out, cached=False)


# configurations the gain is reported on: (workload, k, result limit, induced prefix or None)
GAIN_CASES = [("cl20k", 1, 1_000_000, None), ("cl20k_sub", 1, 0, None),
              ("cl100k", 2, 10_000_000, None), ("cl100k", 1, 0, (20_000, 60_000)),
              ("cl500k", 1, 10_000_000, None), ("cl500k", 2, 0, (20_000, 40_000))]


def main(argv=None) -> int:
    """python -m gmkbe_b200.autotune [--passes 1]: tunes each GAIN_CASES workload
    (costs: the shipped model's predictions) and prints one JSON line per case
    with the default and the tuned device time."""
    import argparse
    import sys
    from . import graphgen as gg
    from . import learned as L
    ap = argparse.ArgumentParser(description="tuned vs default settings on cl20k, cl100k and cl500k")
    ap.add_argument("--passes", type=int, default=1)
    ap.add_argument("--repeats", type=int, default=2)
    a = ap.parse_args(argv)
    model = L.load_default()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for name, k, limit, sub in GAIN_CASES:
        if name == "cl20k_sub":
            h = gg.read_graph_bin(os.path.join(root, "tests", "golden", "cl20k_sub.graph.bin"))
        else:
            h = gg.read_graph_bin(gg.cached_workload(name))
            if sub:
                h = gg.induced_prefix(h, *sub)
        with Graph.from_graph(h) as g:
            cost = L.predicted_costs(model, g, k)
            r = tune(g, h, k, cost, result_limit=limit, repeats=a.repeats, passes=a.passes)
            print(json.dumps({"workload": name if not sub else f"{name} induced {sub[0]}x{sub[1]}",
                              "k": k, "result_limit": limit, "default_ms": r["default_ms"],
                              "tuned_ms": r["ms"], "gain": r["gain"], "settings": r["settings"],
                              "trials": len(r["trials"])}), flush=True)
            sys.stdout.flush()
    return 0


if __name__ == "__main__":
    raise SystemExit(main())
