"""Kernels that read before they wait for their predecessor (load_early) must not declare what a predecessor writes `const __restrict__`: the compiler
may then move those loads to the other side of the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "jasmine_b200" / "csrc"
# constants of a model, and what describes a pass (copied from the host before its first kernel)
OLDER = re.compile(r"(seg|tile|tok)_\w+|block_table|rows|rope|gain|bias|w|b")


def kernels():
    for f in sorted(CSRC.glob("*.cu")):
        text = f.read_text()
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^{;]*?\)\s*)?(\w+)\(([^{;]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield f.name, m[1], m[2], text[m.end():end]


def test_no_kernel_that_reads_early_promises_constant_inputs():
    seen = 0
    for file, name, params, body in kernels():
        if "chain_wait()" not in body or "load_early(" not in body.split("chain_wait()")[0]:
            continue
        seen += 1
        for p in params.split(","):
            if "const " in p and "__restrict__" in p:
                assert OLDER.fullmatch(p.split()[-1]), (file, name, p.strip())
    assert seen >= 7
