"""What the library is compiled from: every line length with kernels of its own is a module
of its own (a program loads the kernels of its lengths, not those of a whole radix), and the
library stays as small as it was before there were such lengths (57 MB)."""
import os

from pyfwix_b200 import build


def test_a_module_per_length():
    units = build.units()
    names = [u[2] for u in units]
    assert len(set(names)) == len(names)
    own = {}
    for src, flags, name in units:
        base = os.path.basename(src)[:-3]
        if flags:
            rt = int(base.split("_")[1])
            ra, rb = (int(f.split("=")[1]) for f in flags[:2])
            assert name == f"{base}_{ra}_{rb}"
            own[rt * ra * rb] = "-DFWIX_FLEX_ROWS_ONLY" in flags
    # two-stage lengths from 48 to 300, ten three-stage ones; rows of the planned lengths
    assert sorted(n for n, rows in own.items() if rows) == [64, 96, 128, 160, 192, 320, 384, 512, 640]
    assert sum(not rows for rows in own.values()) == 50
    assert {48, 105, 135, 270, 300, 250, 504} <= set(own) and 147 not in own and 256 not in own


def test_library_size():
    assert os.path.getsize(build.build()) < 57e6
