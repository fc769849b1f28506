"""Kernels of one cluster whose sums go into every CTA's shared memory
(tail_sum2, apbs_b200/csrc/mixed.cu): distributed shared memory may be stored to
only once all CTAs of the cluster are known to have started, so in each kernel a
cluster barrier comes before anything that makes such a sum.  Checked on the
source, since a CTA that starts late cannot be brought about."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "apbs_b200", "csrc", "mixed.cu")


def _functions():
    """name -> (is a kernel, body) of the functions of the file."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(SRC).read(), flags=re.S)
    text = re.sub(r"__launch_bounds__\([^)]*\)|__forceinline__", "", text)
    out = {}
    for m in re.finditer(r"^(__global__|__device__)[^;{]*?\b(\w+)\([^;{]*\)\s*\{", text, re.M):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out[m.group(2)] = (m.group(1) == "__global__", text[m.end():end])
    return out


def _first(body, names):
    at = [m.start() for n in names for m in [re.search(r"\b%s\s*(<|\()" % n, body)] if m]
    return min(at, default=len(body))


def test_a_cluster_barrier_precedes_the_first_sum():
    funcs = _functions()
    # functions by what comes first in them, itself or by what it calls
    pushers, barriers = {"tail_sum2"}, {"tail_sync"}
    for _ in range(5):  # as deep as the calls go
        for n, (_, body) in funcs.items():
            push, wait = _first(body, pushers), _first(body, barriers)
            if n not in ("tail_sum2", "tail_sync") and push != wait:
                (pushers if push < wait else barriers).add(n)
                (barriers if push < wait else pushers).discard(n)
    assert "tail_damp" in pushers and "tail_cycle" in barriers
    kernels = {n for n, (k, b) in funcs.items() if k and re.search(r"\btail_(sum2|damp|cycle)\b", b)}
    assert {"k_vcycle_tail", "k_coarse_exact", "k_batch_solve"} <= kernels
    assert not kernels & pushers
