"""Tensor-memory loads in the kernels' sources: a loaded register is valid only
behind its wait, and the compiler knows of that only through the wait's operands.
So every wait names the values in flight, each of them, and the wait's definition
hands them back."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "spmv_b200" / "csrc"
FILES = sorted(p.name for p in CSRC.iterdir() if "tmem_ld(" in p.read_text())
TOKEN = re.compile(r"tmem_ld\(\s*[^;]*?,\s*(\w+)(?:\[\w+\])*\s*\);|tmem_wait_ld\(([^)]*)\);")


def code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_the_wait_hands_its_values_back():
    text = code("sell_ring.cuh")
    wait = text.index("tcgen05.wait::ld")
    body = text[wait:text.index("}", text.index("\n", wait))]
    assert "tmem_landed" in body
    for kind in ("Tmem64", "Tmem32"):
        landed = text[text.index("tmem_landed(%s&" % kind):]
        assert '"+r"' in landed[:landed.index("}")]


@pytest.mark.parametrize("name", [f for f in FILES if f.endswith(".cu")])
def test_every_wait_names_the_values_in_flight(name):
    flying, waits = set(), 0
    for m in TOKEN.finditer(code(name)):
        if m.group(1):
            flying.add(m.group(1))
        else:
            assert {a.strip() for a in m.group(2).split(",") if a.strip()} == flying
            flying, waits = set(), waits + 1
    assert waits > 0 and not flying
