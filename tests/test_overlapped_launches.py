"""Kernels that are launched while the one before them still runs: what that one writes must not be read as memory that stays the same for
as long as the kernel is there (__ldg, const __restrict__).  Read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vq_b200", "csrc")
INVARIANT = re.compile(r"\b(__ldg|load_piece(?:<\w+>)?|load_slice(?:<\w+>)?)\(")

# What such a kernel, or a function that it reads memory with, may take for invariant.  Rows, the codebooks of an encode and the tree's
# `perm` of the spreads and splits were written two launches ago or earlier.
ALLOWED = {
    "walk_rows": set(), "dense_codebook_kernel": set(), "dense_shortlist_kernel": set(), "update_centroids_kernel": set(), "pq_update_centroids_kernel": set(),
    "rvq_stages_kernel": set(),  # (rows and codebooks by load4: written before the kernel in front of it)
    "pq_operand_b_kernel": set(), "pq_tc_kernel": {"P.x"}, "pq_queue_drain": {"P.x"}, "pq_expand_kernel": {"c16", "centroids"},
    "queue_sums_kernel": {"xp", "i"},  # (its load_piece takes a number)
    "resolve_kernel": {"x", "book", "c", "xr"}, "ordered_hist_kernel": set(), "ordered_lists_kernel": set(), "ordered_lists_cluster_kernel": set(),
    "ordered_sums_kernel": {"x"}, "ordered_sums_long_kernel": {"x"}, "init_tree_kernel": set(), "chunk_sums_kernel": {"x"}, "node_mean_kernel": set(), "node_stats_kernel": {"x"}, "node_stats_stream_kernel": {"x"},
    "node_spread_stream_kernel": {"x", "perm", "xcol", "p"}, "split_kernel": {"x", "perm"}, "next_level_kernel": set(), "no_children_kernel": set(),
}


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced")


def _functions():
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
        for m in re.finditer(r"\b(?:__global__|__device__)[^;{}()]*?\b(\w+)\s*\(", text):
            close = _closing(text, m.end() - 1, "()")
            body = re.match(r"\s*\{", text[close + 1:])
            if body:
                start = close + body.end()
                yield m.group(1), text[m.end():close], text[start:_closing(text, start, "{}")]


def _taken_for_invariant(params, body):
    names = set(re.findall(r"\bconst\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params))
    for m in INVARIANT.finditer(body):
        args = body[m.end():_closing(body, m.end() - 1, "()")]
        args = re.sub(r"^\w+,\s*", "", args) if m.group(1) != "__ldg" and "," in args else args  # (the first argument is the destination)
        args = re.sub(r"reinterpret_cast<[^>]*>\(", "", args)
        name = re.match(r"[\s(]*([A-Za-z_][\w.]*)", args)
        names |= {name.group(1)} if name else set()
    return names - {"const"}


def test_what_the_kernel_before_writes_is_not_taken_for_invariant():
    seen = set()
    for name, params, body in _functions():
        if name in ("walk_rows", "pq_queue_drain") or "after_previous_kernel();" in body:
            seen.add(name)
            assert name in ALLOWED, f"{name} may start before its predecessor ends: say here what it may take for invariant"
            extra = _taken_for_invariant(params, body) - ALLOWED[name]
            assert not extra, f"{name} reads {sorted(extra)} as invariant"
    assert seen == set(ALLOWED), seen ^ set(ALLOWED)
