"""What a tile of a 16-bit run segment reads from shared memory it has written:
k_fdmt_run16 decides by all the columns it forms, written ones or not, whether
its sums left the type's range, and values left by an earlier kernel sent whole
warps through the element-by-element form (256 x 65536, depth 0: 176 us against
111)."""
import re
from pathlib import Path

import pytest

from test_run16 import MID, TT, plan16

SRC = (Path(__file__).resolve().parent.parent / "cpp_projects_b200" / "csrc" / "internal.h").read_text()
OVER = int(re.search(r"constexpr int kRun16Over = (\d+);", SRC).group(1))


@pytest.mark.parametrize("nchan,ncols,max_dt,fuse", [(64, 1300, 64, -1), (256, 65536, 256, -1), (256, 40000, 384, 2),
                                                     (512, 32768, 512, 2), (1024, 8000, 512, -1), (4096, 2050, 4096, 2)])
def test_tiles_read_what_they_wrote(nchan, ncols, max_dt, fuse):
    assert OVER % 8 == 0
    seen = 0
    for _, _, pr, tiles, rows, ent in plan16(nchan, ncols, max_dt, fuse):
        s1, s2, _, pitch, zx, y0, zy, ent0 = (int(v) for v in pr[:8])
        for _, e0, n_in, n1, n2, _, _, _ in tiles:
            seen += 1
            x_end = zx if n_in * pitch == zx else n_in * pitch + OVER   # written: its rows, then cleared or the -0.0 row
            for first, n, stage, cols, base, end, zero in ((e0, n1, s1, MID, 0, x_end, zx), (e0 + n1, n2, s2, TT, y0, y0 + n1 * MID, zy)):
                q = ent[first:first + n][:, :2 * stage] // 2   # value offsets (bit 0: the moved flag)
                odd = q % 2
                last = q - odd + cols + 2 * odd                # an odd offset reads one word more
                ok = (q == zero) | ((q >= base) & (last <= (end if end != zx else zx + MID)))
                assert ok.all()
    assert seen
