"""Inline assembly that writes memory, waits or orders tells the compiler so: the
C++ code around it reads and writes the same arrays, and `volatile` alone only
keeps the statement itself."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sph-dem_gb300", "csrc")
TOUCHES_MEMORY = re.compile(r"\b(st|ld|red|atom|cp|mbarrier|fence|barrier|bar|membar)\.")


def asm_statements(text):
    """(line, statement) of every asm(...) of a source file."""
    for m in re.finditer(r"\basm\b\s*(volatile)?\s*\(", text):
        i, depth, quoted = m.end(), 1, False
        while depth:
            ch = text[i]
            if ch == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (ch == "(") - (ch == ")")
            i += 1
        yield text.count("\n", 0, m.start()) + 1, text[m.start():i]


def test_memory_clobbers():
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as fh:
            text = fh.read()
        for line, stmt in asm_statements(text):
            if not TOUCHES_MEMORY.search(stmt):
                continue
            seen += 1
            assert "volatile" in stmt and re.search(r':\s*"memory"\s*\)$', stmt), f"{name}:{line}"
    assert seen > 0
