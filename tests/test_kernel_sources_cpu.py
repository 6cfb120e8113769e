"""What can be checked in the kernels' source text."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "grouped-sparse-gemm_b200", "csrc")


def asm_statements():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            for m in re.finditer(r"\basm( volatile)?\s*\(", text):
                depth, i, quoted = 1, m.end(), False
                while depth:
                    c = text[i]
                    if c == '"' and text[i - 1] != "\\":
                        quoted = not quoted
                    elif not quoted:
                        depth += (c == "(") - (c == ")")
                    i += 1
                yield name, bool(m.group(1)), text[m.end():i - 1]


def test_inline_asm_on_global_memory_is_ordered():
    """A kernel may start before its predecessor has ended and waits (griddepcontrol.wait) before it touches what the
    predecessor wrote.  Only a volatile statement with a memory clobber is kept behind that wait by the compiler."""
    seen = 0
    for name, volatile, body in asm_statements():
        if re.search(r"\b(ld|st|red|atom)\.global|\.global\b", body):
            seen += 1
            assert volatile and '"memory"' in body, f"{name}: {body[:80]}"
    assert seen >= 3
