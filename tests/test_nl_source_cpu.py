"""Orderings in the block search's source that no run shows reliably: a warp's
copy of the chunk prefixes is written by its lanes and read by others, so a
warp barrier must stand between (a shuffle orders no memory)."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "akitsushima_b200", "csrc")


def test_chunk_prefixes_are_ordered_before_the_ranks():
    with open(os.path.join(CSRC, "mbf_nl.cu")) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    store = src.index("ahead_w[wid][lane] =")
    read = src.index("ahead_w[wid][x >> 12]")
    assert store < read
    assert re.match(r"[^;]*;\s*__syncwarp\(\);", src[store:]) or "__syncthreads();" in src[store:read]
