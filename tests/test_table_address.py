"""The E-steps read theta in an asm that is neither volatile nor clobbers memory, so nothing but its
address keeps such a load behind the barrier that completes the table: every address must come from
table_address, whose value comes out of a volatile asm that clobbers memory."""
import os
import re

from conftest import ROOT


def test_addresses_come_out_of_the_barrier():
    with open(os.path.join(ROOT, "binder_b200", "csrc", "estep.cu")) as f:
        s = f.read()
    body = re.search(r"unsigned table_address\(.*?\n\}", s, re.S).group(0)
    assert re.search(r'asm volatile\(""\s*:\s*"\+r"\(a\)\s*::\s*"memory"\)', body)
    loads = re.findall(r'asm\("ld\.shared.*?;\n|asm\("ld\.shared[^;]*;', s, re.S)
    assert loads and all(re.search(r"__dp4a\([^;]*\btha\b", x) for x in loads)
    sources = re.findall(r"\btha(?:\[m\])? = (\w+)\(", s)
    assert sources and set(sources) == {"table_address"}
