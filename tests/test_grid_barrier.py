"""The grid barrier's control word: 64 bits, and only ever accessed whole.

PTX orders nothing between racing accesses that overlap in part, so every
access to the word that arrivals and errors share has to be 64 bits wide; the
arithmetic on it is run here for many barriers in a row, past its wrap (the
reference launches a kernel per phase and has no such barrier).
"""
import glob
import os
import re

import pytest


def source(root, name):
    text = open(os.path.join(root, "thievory_b200", "csrc", name)).read()
    return re.sub(r"//.*", "", text)


def test_word_is_accessed_whole(root):
    dev = source(root, "thv_device.cuh")
    members = re.search(r"struct (?:alignas\(\d+\) )?GridBar \{(.*?)\n\};", dev, re.S).group(1)
    fields = [m for m in re.findall(r"^\s*([^()\n]+);", members, re.M)]
    assert [f.split() for f in fields] == [["unsigned", "long", "long", "word"]]
    sync = dev[dev.index("bool grid_sync(GridBar *bar"):dev.index("struct BlockCounts")]
    widths = re.findall(r'asm volatile\("((?:atom|ld|st|red)[^ ]*) ', sync)
    assert len(widths) == 2 and all(w.endswith(".u64") for w in widths)
    assert not re.findall(r"atomic\w+", sync)
    flag = re.search(r"void flag_error.*?\n\}", dev, re.S).group(0)
    assert "atomicOr(&bar->word, 1ull <<" in flag
    for path in glob.glob(os.path.join(root, "thievory_b200", "csrc", "*.cu")):
        text = source(root, os.path.basename(path))
        assert not re.findall(r"bar(?:\.|->)(?!error\(\))\w+", text), path


@pytest.mark.parametrize("blocks", [1, 2, 148, 296, 1184])
def test_top_bit_flips_with_the_last_arrival(blocks):
    word = 0
    for _ in range(9):  # the arrivals wrap every second barrier
        olds = []
        for b in range(blocks):
            add = 0x80000000 - (blocks - 1) if b == 0 else 1
            olds.append(word)
            passed = [(word ^ o) >> 63 for o in olds]
            assert not any(passed)
            word = (word + (add << 32)) & (2**64 - 1)
            word |= 1 << 2 if b == blocks // 2 else 0  # an error set on the way
            assert all((word ^ o) >> 63 for o in olds) == (b == blocks - 1)
            assert word & 0xFFFFFFFF == (4 if b >= blocks // 2 or _ else 0)
