"""Inline assembly that stores to memory tells the compiler so.

keep_candidate (csrc/cells.cuh) stores to shared memory from an asm statement without a "memory"
clobber, so that the candidates' loads around it can overlap.  The compiler does not know of such a
store; a statement with the clobber has to stand between the last of them and the first read of what
they stored.  This CPU test reads the CUDA sources.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "vt-physics_b200" / "csrc"
STORE = re.compile(r"@?p?\s*(st|red|atom)\.(shared|global)|cp\.async")


def _functions(text):
    """(name, body) of the functions defined at the start of a line."""
    for m in re.finditer(r"^(?:__device__|__global__|static|template)[^;{]*?\b(\w+)\([^;{]*\)\s*(?:const\s*)?\{", text, re.M):
        i, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


def test_asm_stores_are_followed_by_a_clobber_before_they_are_read():
    texts = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu*"))}
    bodies = {name: body for t in texts.values() for name, body in _functions(t)}
    stores = {n for n, b in bodies.items() if any(STORE.search(a) and '"memory"' not in a
                                                  for a in re.findall(r"asm[^;]*\((?:[^;]|;(?=[^\n]*\\n))*?\);", b, re.S))}
    assert stores == {"keep_candidate"}
    through = {n for n, b in bodies.items() if any(re.search(rf"\b{s}\(", b) for s in stores)}
    assert through == {"test4"}
    users = {n: b for n, b in bodies.items() if "test4(" in b}
    assert users
    fences = [n for n, b in bodies.items() if re.fullmatch(r'\s*asm volatile\(""\s*::: "memory"\);\s*\}', b)]
    for name, body in users.items():
        last, read = body.rindex("test4("), body.index(".kept[0][0]")
        between = body[last:read]
        assert any(f"{f}()" in between for f in fences), f"{name} reads kept candidates without a clobber"
