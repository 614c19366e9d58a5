"""Per-thread species arrays have Spec<NS>::A elements: the species count of an instantiation for a fixed
count, the tables' capacity (kMS) only in the generic one.  A loop to a capacity constant therefore runs past
the end of the fixed instantiation's array, and no device test can show it (the stores land in the thread's
registers or stack).  Read from the sources: loops over such arrays take their bound from the array or the count.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "openstc-mixinglayer_b200" / "csrc"
SIZED = sorted(p.name for p in CSRC.glob("*.cuh") if "Spec<NS>::A" in p.read_text())


@pytest.mark.parametrize("name", SIZED)
def test_no_loop_to_a_table_capacity(name):
    text = (CSRC / name).read_text()
    loops = re.findall(r"for \([^;)]*;[^;]*<=?[^;]*\bkM[A-Z]+\b[^;]*;[^)]*\)", text)
    assert not loops, loops


def test_sources_are_found():
    assert {"mix_math.cuh", "ostc_mix.cuh", "ostc_adj.cuh", "pv_mix.cuh", "ostc_steady.cuh"} <= set(SIZED)
