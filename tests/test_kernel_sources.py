"""Inline assembly of the kernels states what it touches: a statement that reads or writes memory, or
orders such accesses, is volatile and clobbers memory, so the compiler keeps it behind the wait for
the kernel before (griddepcontrol.wait) and in order with the thread's own accesses."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "openlb_b200" / "csrc"


def statements(text):
    """(head, body) of every asm statement: what stands before its parenthesis and inside it."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\basm\b([^(]*)\(", text):
        depth, i, quoted = 1, m.end(), False
        while depth:
            c = text[i]
            if c == '"' and text[i - 1] != "\\":
                quoted = not quoted
            elif not quoted:
                depth += (c == "(") - (c == ")")
            i += 1
        yield m.group(1), text[m.end():i - 1]


def test_inline_assembly_that_touches_memory_is_ordered():
    seen = 0
    for path in sorted(CSRC.glob("*.cu*")):
        for head, body in statements(path.read_text()):
            seen += 1
            code = " ".join(re.findall(r'"((?:[^"\\]|\\.)*)"', body.split('"memory"')[0]))
            touches = re.search(r"\[[^\]]*%|\b(wait|wait_all|wait_group|commit_group|fence|griddepcontrol)\b", code)
            if touches:
                assert "volatile" in head, f"{path.name}: {code}"
                assert '"memory"' in body, f"{path.name}: {code}"
    assert seen > 10
