"""CPU test of how chained kernels read what the kernels before them write.

A kernel that launch_dep starts behind its predecessor lives while that one
still writes.  `__restrict__` on a pointer to const (and __ldg) lets the compiler
load through the read-only path, which holds only for data that nobody writes
during the kernel's whole life, and which griddepcontrol.wait does not order.
So neither stands in a chained kernel, nor in a device function that it calls.
"""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "vcp_gb300" / "csrc"
WORD = re.compile(r"\b[A-Za-z_]\w*\b")
HEAD = re.compile(r"\b([A-Za-z_]\w*)\s*\(([^;{}()]*(?:\([^;{}()]*\)[^;{}()]*)*)\)\s*(?:const\s*)?\{")


def functions():
    """name -> [(is a kernel, parameters, body)] of every function under csrc."""
    out = {}
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        text = re.sub(r"__launch_bounds__\([^\n]*?\)(?=\s)", "", text)
        for h in HEAD.finditer(text):
            name = h.group(1)
            if name in ("if", "for", "while", "switch"):
                continue
            depth, end = 1, h.end()
            while depth and end < len(text):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            before = text[:h.start()]
            start = max(before.rfind(";"), before.rfind("}"), before.rfind("{"))
            kernel = "__global__" in before[start + 1:]
            out.setdefault(name, []).append((kernel, h.group(2), text[h.end():end]))
    return out


def test_chained_kernels_load_coherently():
    fs = functions()
    kernels = {n for n, ds in fs.items() if any(d[0] for d in ds)}
    chained = set()
    for ds in fs.values():
        for _, _, body in ds:
            if "launch_dep(" in body:
                plain = set(re.findall(r"(\w+)\s*(?:<[^<>;]*>)?\s*<<<", body))
                chained |= {w for w in WORD.findall(body) if w in kernels} - plain
    assert {"oz_crt_split", "oz_slice_gemm_kernel", "oz_crt_assemble_kernel", "dd_split",
            "dd_crt_assemble_kernel"} <= chained
    seen, todo = set(), sorted(chained)
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for _, params, body in fs[n]:
            assert "__restrict__" not in params, f"{n}: __restrict__ parameter"
            assert "__restrict__" not in body and "__ldg" not in body, n
            todo += [w for w in WORD.findall(body) if w in fs and w not in seen]
