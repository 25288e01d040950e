"""A kernel's shared-memory limit (cudaFuncSetAttribute) belongs to the device, so contexts on several threads
share it: every call in the sources sets a constant.  One that sets the size of the moment can be lowered by
another thread between the call and the launch, which then fails."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "latticemodels.jl_gb300" / "csrc"
CONSTANT = re.compile(r"^(\(int\)\s*)?(k[A-Z]\w*|[A-Z][A-Z_0-9]+)(\s*-\s*[A-Z][A-Z_0-9]+)?$")


def test_limits_are_constants():
    seen = 0
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"\\\n", "\n", f.read_text())
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*?)\)[,;]", text):
            arg = " ".join(m.group(1).split())
            assert CONSTANT.match(arg), f"{f.name}: {arg}"
            seen += 1
    assert seen >= 7
