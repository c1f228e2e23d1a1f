"""The cluster kernel's barriers, checked on the host with the library's own
constants and rule (csrc/ne2b_layout.h): for every hop length, with hops cut
short as windows cut them, no delivery lands in a slot that its hop reads,
every delivery is read in a later hop, and between a slot's read and the next
add to it lies a barrier at which every warp releases."""
import ctypes as C
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "neuro_edit_v2_b200", "csrc")
SOURCE = """
#include <stdint.h>
#include "ne2b_layout.h"
extern "C" {
uint32_t spare() { return ne2b::kRingSpare; }
uint32_t max_hop() { return ne2b::kMaxHop; }
int due(uint32_t since, uint32_t hop) { return ne2b::release_due(since, hop); }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "rule.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "rule.cpp"), "-o",
                    str(d / "librule.so")], check=True)
    return C.CDLL(str(d / "librule.so"))


@pytest.mark.parametrize("cut", [0, 3, 7, 10])
def test_reads_and_adds_of_a_slot_are_ordered(rule, cut):
    rng = random.Random(cut)
    for hop in range(1, rule.max_hop() + 1):
        for longest in sorted({hop, hop + 1, 2 * hop, hop + 13, 40}):
            slots = longest + 1 + rule.spare()
            delays = sorted({hop, min(hop + 1, longest), (hop + longest) // 2, max(hop, longest - 1), longest})
            read_at, released = {}, 0  # last step that read each slot; steps done at the last full release
            start = since = 0
            while start < 4 * slots:
                nb = min(hop, rng.randint(1, cut)) if cut else hop
                steps = range(start, start + nb)
                reads = {t % slots: t for t in steps}
                for t in steps:
                    for d in delays:
                        s = (t + d) % slots
                        assert s not in reads
                        assert t + d >= start + nb
                        assert read_at.get(s, -1) < released, (hop, longest, t, d)
                read_at.update(reads)
                since += nb
                start += nb
                if rule.due(since, hop):
                    since, released = 0, start
