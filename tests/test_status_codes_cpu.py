"""The status word of a context tells which kernel's wait gave up: every code stands once, in one list."""
import re
from pathlib import Path

KERNELS = Path(__file__).resolve().parent.parent / "lithos_b200" / "csrc" / "kernels"
CODE = re.compile(r"^#define\s+(\w+)\s+(0x1[0-9a-f]{3})u\b", re.M)


def test_codes_are_listed_once():
    codes = {}
    for f in sorted(KERNELS.glob("*.cu*")):
        for name, value in CODE.findall(f.read_text()):
            assert f.name == "common.cuh", (f.name, name)
            assert value not in codes, (name, codes.get(value))
            codes[value] = name
    assert len(codes) >= 14
    text = "".join(f.read_text() for f in KERNELS.glob("*.cu*") if f.name != "common.cuh")
    assert {n for n in codes.values() if not re.search(rf"\b{n}\b", text)} <= {"LB_DEV_OK"}
