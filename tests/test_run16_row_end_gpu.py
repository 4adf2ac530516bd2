"""Run segments over 16-bit planes read nothing past a row's end: columns there
are never written by the pass before, and a NaN or an infinity left in them sent
the row's warps through the element-by-element form."""
import pytest
import torch

from cpp_projects_b200 import CFdmtGpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("ncols", [1, 511, 1025, 1027, 1029, 1031])   # every odd rest of 8
def test_columns_past_the_end_are_not_read(cuda, prec, ncols):
    nchan, max_dt = 256, 256
    f = CFdmtGpu(1200.0, 1600.0, nchan, ncols, max_dt, fuse_depth=2, precision=prec, external_ws=True)
    p = f.passes()
    assert f.info.fuse_depth == 2 and [q[:2] for q in p] == [[2, 5], [5, 8]]
    x = torch.randn((nchan, ncols), generator=torch.Generator(device=cuda).manual_seed(ncols), device=cuda)
    out = torch.empty((2, max_dt, ncols), device=cuda)
    ends = []
    for k, fill in enumerate((0x00, 0xff)):   # 0xffff is a NaN in both types
        ws = torch.full((f.workspace_size(),), fill, dtype=torch.uint8, device=cuda)
        f.process_image_ws(x, out[k], False, ws)
        # the second pass's input plane follows the first's; an odd row's last
        # stored word holds one column past its end
        rows, pitch = f.rows_per_level(), (ncols + 63) // 64 * 64
        at = (int(rows[2]) * pitch * 2 + 255) // 256 * 256
        plane = ws[at:at + int(rows[5]) * pitch * 2].view(torch.float16 if prec == 1 else torch.bfloat16)
        ends.append(plane.view(int(rows[5]), pitch)[:, ncols].float().clone())
    assert torch.equal(out[0], out[1])
    assert bool(torch.isfinite(ends[1]).all()) and torch.equal(ends[0], ends[1])
