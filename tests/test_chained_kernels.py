"""Kernels that run while the one in front still writes (chain_begin, dg_common.cuh) read
nothing through the path for data that does not change: neither their own pointers nor
those of the functions they call are __restrict__. Read off the sources."""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "diorama_gb300" / "csrc"
DEFINITION = re.compile(r"(?:__global__|__device__)[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*(?:const\s*)?(?::[^;{}]*)?\{")


def definitions():
    """(name, text from the name's line to the closing brace) of every device function."""
    for path in sorted(CSRC.glob("*.cu*")):
        source = re.sub(r"//[^\n]*", "", path.read_text())
        for match in DEFINITION.finditer(source):
            name = match.group(1)
            if name in ("__launch_bounds__", "__align__"):  # the kernel's name follows
                name = re.findall(r"\b(\w+)\s*\(", match.group(0))[-1]
            depth, at = 1, match.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(source[at], 0)
                at += 1
            names = re.findall(r"\b(\w+)\s*\(", match.group(0).split("{")[0])
            yield [n for n in names if not n.startswith("__")][0], match.group(0), source[match.end():at]


def test_nothing_in_a_chained_kernel_is_restrict():
    functions = {}
    for name, head, body in definitions():
        functions.setdefault(name, []).append((head, body))
    chained = {n for n, defs in functions.items() for _, body in defs if re.search(r"\bchain_begin\(\)", body)}
    assert {"preprocess_kernel", "rasterize_backward_kernel", "sort_pass_kernel", "bin_scatter_kernel",
            "scan_tiles_kernel", "preprocess_backward_adam_kernel"} <= chained
    reached, todo = set(), list(chained)
    while todo:
        name = todo.pop()
        if name in reached:
            continue
        reached.add(name)
        for _, body in functions[name]:
            todo += [n for n in set(re.findall(r"\b(\w+)\s*(?:<[^<>;]*>)?\(", body)) if n in functions]
    assert {"load_gaussian", "preprocess_backward_one", "adam_param_slot"} <= reached
    bad = {n for n in reached for head, body in functions[n] if "__restrict__" in head + body}
    assert not bad, sorted(bad)
