"""Precompiled kernels that may start before the previous grid has ended (they
wait for it themselves): nothing they read is declared invariant."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "skelcl_gb300" / "csrc"


def test_no_restrict_before_the_wait():
    kernels = 0
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for part in re.split(r"__global__", text)[1:]:
            head, body = part.split("{", 1)
            body = body.split("\n}\n", 1)[0]
            if "dependency_wait()" in body:
                kernels += 1
                assert "__restrict__" not in head, (f.name, head)
                # what the kernel hands on to device functions of its file
                for name in re.findall(r"\b([a-z_0-9]+)\(", body):
                    d = re.search(rf"__device__[^;{{}}]*\b{name}\(([^)]*)\)\s*\{{", text)
                    assert not d or "__restrict__" not in d.group(1), (f.name, name)
    assert kernels >= 8
