"""Slot indexes of the split stepper's scratch stay in range for every pool the slot arrays can hold.

A pose array of four components per slot, indexed by 32-bit integers, limits a pool to 2^29 slots; an array
of `width` values a slot then needs an index of more than 31 bits from width 4 on."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pystarc_b200" / "csrc"
MAX_SLOTS = 2 ** 29


def test_products_of_a_slot_and_a_width_fit_their_type():
    src = (CSRC / "bd_split.cuh").read_text()
    for width in re.findall(r"\[(\d+) \* slot\b", src):  # 32-bit products
        assert int(width) * MAX_SLOTS <= 2 ** 31, f"{width} * slot overflows 32 bits"


def test_list_lengths_are_not_multiplied_past_32_bits():
    src = (CSRC / "bd_split.cuh").read_text()
    for name in ("fwd_warps", "rev_warps"):
        body = re.search(name + r"\(int n, int n_warps\) \{(.*?)\n\}", src, re.S).group(1)
        for factor in re.findall(r"\bn \* (\d+)", body):
            assert int(factor) * MAX_SLOTS <= 2 ** 31, f"{name}: n * {factor} overflows 32 bits"
