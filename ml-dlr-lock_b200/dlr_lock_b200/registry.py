"""(model, batch size) -> implementation table, in the format of the reference's
``kernels/registry.py:17-135``: a list of entries per model with ``B_lo``,
``B_hi``, ``kernel``, ``callable`` (importable dotted path), ``config`` and
``note``.  This build has one backend behind one callable; it covers every batch
size of all four model shapes.  The library picks among its device paths per
call (``dlrb200_query`` reports the choice for a shape on the current device);
the ranges below name the path that serves most of each range on a B200, and
``describe`` fills an entry from the library's own answer.
"""

MODEL_CONFIGS = {  # kernels/reference.py:18-23
    "Qwen3-0.6B": {"d": 1024, "d_ff": 3072, "r": 32},
    "Qwen3-1.7B": {"d": 2048, "d_ff": 6144, "r": 64},
    "Qwen3-8B": {"d": 4096, "d_ff": 12288, "r": 128},
    "Qwen3-32B": {"d": 5120, "d_ff": 25600, "r": 256},
}

_CALLABLE = "dlr_lock_b200.ops.forward_xvu"

PATH_NAMES = {1: "b200_striped", 2: "b200_cluster", 3: "b200_cluster_small", 4: "b200_streamed",
              5: "b200_streamed_pairs", 6: "b200_striped_clusters", 7: "b200_resident"}
PATH_CONFIGS = {
    1: "width-striped cooperative grid, TMA weight ring, one exchange per layer through L2",
    2: "128-row tiles on clusters of d/512 CTAs, activations resident in tensor memory, tcgen05",
    3: "one cluster of d/256 CTAs per two rows, exchange in distributed shared memory",
    4: "128-row tiles, one cluster of 1/2/4 CTAs each, activations streamed through shared and tensor memory, tcgen05",
    5: "256-row tiles on CTA pairs (tcgen05 cta_group::2), activations streamed, exchange in distributed shared memory",
    6: "width-striped cooperative grid in clusters of 8: reduction inside a cluster in distributed shared memory, "
       "cluster sums through counted words in L2",
    7: "clusters of 4/8/16 CTAs that keep a few rows each in registers, exchange in distributed shared memory",
}


def _entry(lo, hi, path, note):
    return {"B_lo": lo, "B_hi": hi, "kernel": PATH_NAMES[path], "callable": _CALLABLE,
            "config": PATH_CONFIGS[path] + "; picked per call by dlrb200_query", "note": note}


# (first batch size, path) per width, at the depth of the SwiGLU budget.  Bounds between two paths move by some rows with the
# number of clusters that fit the GPU at once; from 4096 rows on, the large-batch kernels change places where a last wave of
# tiles would be nearly empty.
_RANGES = {1024: [(1, 7), (1057, 2)], 2048: [(1, 7), (481, 2), (5889, 5)], 4096: [(1, 7), (225, 2), (1921, 5), (3841, 4), (4225, 2), (5889, 5)],
           5120: [(1, 1), (12, 7), (449, 4)]}
_LAST = 131072
_NOTES = {1: "A few rows of the widest model: all SMs pull the weights.",
          2: "Row tiles on tensor cores, activations in tensor memory, one launch for all layers.",
          4: "Row tiles on tensor cores, activations streamed, one launch for all layers.",
          5: "256-row tiles on CTA pairs, activations streamed, one launch for all layers.",
          7: "Small and medium batches: a few rows per cluster in registers, one launch for all layers."}


def _entries(name):
    ranges = _RANGES[MODEL_CONFIGS[name]["d"]]
    ends = [lo - 1 for lo, _ in ranges[1:]] + [_LAST]
    return [_entry(lo, hi, path, _NOTES[path]) for (lo, path), hi in zip(ranges, ends)]


REGISTRY = {name: _entries(name) for name in MODEL_CONFIGS}


def resolve(model: str, batch_size: int):
    """Entry serving ``(model, batch_size)``, or None (kernels/registry.py:130-135)."""
    for entry in REGISTRY.get(model, []):
        if entry["B_lo"] <= batch_size <= entry["B_hi"]:
            return entry
    return None


def describe(model: str, batch_size: int, depth: int):
    """``resolve`` with ``kernel`` and ``config`` filled from what the library would run for this exact
    cell on the current CUDA device (needs the built library and a GPU)."""
    from . import ops
    entry = resolve(model, batch_size)
    if entry is None:
        return None
    cfg = MODEL_CONFIGS[model]
    plan = ops.query(batch_size, cfg["d"], cfg["r"], depth)
    out = dict(entry)
    out["kernel"] = PATH_NAMES.get(plan.path, f"path{plan.path}")
    out["config"] = (f"{PATH_CONFIGS.get(plan.path, '')}; grid {plan.grid}, cluster {plan.cluster}, "
                     f"{plan.passes} pass(es), {plan.smem_bytes} B shared memory")
    return out
