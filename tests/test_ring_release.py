"""A consumer warp hands a ring slot back with one lane's arrive on the slot's `empty` barrier. The other lanes' reads of the slot
come before that arrive only if the warp synchronises (__syncwarp orders memory among its lanes; a vote does not), so in the source
every such arrive directly follows a __syncwarp."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bats_gb300", "csrc")


def test_every_release_follows_a_syncwarp():
    found, bare = 0, []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        lines = [l.split("//")[0].strip() for l in open(os.path.join(CSRC, name))]
        for i, line in enumerate(lines):
            if re.search(r"mbar_arrive\(&\w+\.empty\[", line):
                found += 1
                before = next(l for l in reversed(lines[:i]) if l)
                if before != "__syncwarp();":
                    bare.append(f"{name}:{i + 1}")
    assert found >= 4 and not bare, bare
