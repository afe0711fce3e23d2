"""The warp-collective (.sync.aligned) tensor-memory instructions are undefined in a warp whose lanes
have parted, and the epilogues part them around the stores of partial tiles.  So they stand in the
wrappers of umma.cuh alone, and each of those brings the warp together before its first one."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "binder_b200", "csrc")


def read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_wrappers_bring_the_warp_together():
    bodies = re.findall(r"void (\w+)\(.*?\) \{\n(.*?)\n\}", read("umma.cuh"), re.S)
    collective = {n: b for n, b in bodies if re.search(r'"tcgen05\.\S*aligned', b)}
    assert set(collective) == {"tmem_alloc", "tmem_dealloc", "tmem_ld32", "tmem_ld16"}
    for name, body in collective.items():
        head = body.split('"tcgen05')[0]
        assert "__syncwarp();" in head, name


def test_no_collective_outside_the_wrappers():
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")) and name != "umma.cuh":
            assert not re.search(r'"[^"\n]*tcgen05[^"\n]*aligned', read(name)), name
