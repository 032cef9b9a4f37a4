"""The candidates' exchange between the warps of a panel CTA: every order that the column's
barrier and the wait for the owner's message leave open, on the sets that
panel_slots.h gives the columns.  No read of a column's candidates may meet another's."""
import itertools
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bem_gb300", "csrc")
COLUMNS = 4


def _first_clash(sets, warps, owners):
    """Depth-first over the interleavings.  A warp's step in column j: 0 write its slot, 1 pass the
    barrier (all warps have written column j), 2 read all slots, 3 pass the wait (the owner has read column j)."""
    start = ((0,) * warps, ((-1,) * warps,) * (max(sets) + 1))
    seen, stack = {start}, [start]
    while stack:
        at, slots = stack.pop()
        for w in range(warps):
            j, step = divmod(at[w], 4)
            if j == COLUMNS:
                continue
            new = slots
            if step == 0:
                row = list(slots[sets[j]])
                row[w] = j
                new = slots[:sets[j]] + (tuple(row),) + slots[sets[j] + 1:]
            elif step == 1 and any(a < 4 * j + 1 for a in at):
                continue
            elif step == 2 and any(v != j for v in slots[sets[j]]):
                return at, slots
            elif step == 3 and at[owners[j]] < 4 * j + 3:
                continue
            nxt = (at[:w] + (at[w] + 1,) + at[w + 1:], new)
            if nxt not in seen:
                seen.add(nxt)
                stack.append(nxt)
    return None


def _sets(tmp_path):
    src, exe = tmp_path / "slots.cpp", tmp_path / "slots"
    src.write_text('#include <cstdio>\n#include "panel_slots.h"\n'
                   'int main() { for (int j = 0; j < %d; j++) std::printf("%%d ", panel_slot_set(j)); }\n' % COLUMNS)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]


@pytest.mark.parametrize("warps", [2, 3])
def test_no_read_meets_another_column(tmp_path, warps):
    sets = _sets(tmp_path)
    for owners in itertools.product(range(warps), repeat=COLUMNS):
        assert _first_clash(sets, warps, owners) is None, owners


def test_one_set_would_clash():
    assert _first_clash([0] * COLUMNS, 2, (0,) * COLUMNS) is not None
