"""Checks of the kernel sources that need no GPU: what the compiler has to be told and no run would show reliably."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "sla_b200", "csrc", "*.cu*")))


def _asm_statements(path):
    """The text between the parentheses of every asm statement, comments taken out."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"\basm\b\s*(?:volatile)?\s*\(", text):
        depth, quoted, i = 1, False, m.end()
        while depth:
            ch = text[i]
            if ch == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += {"(": 1, ")": -1}.get(ch, 0)
            i += 1
        yield text[m.end():i - 1]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_asynchronous_copies_clobber_memory(path):
    """Without the clobber the compiler may read a copied slot before the wait, or after the next copy into it."""
    for asm in _asm_statements(path):
        if "cp.async" in asm or "cp.reduce.async" in asm:
            assert '"memory"' in asm, " ".join(asm.split())


def test_the_asynchronous_copies_are_seen():
    found = [a for p in SOURCES for a in _asm_statements(p) if "cp.async" in a]
    assert any("commit_group" in a for a in found) and any("wait_group" in a for a in found) and len(found) >= 6
