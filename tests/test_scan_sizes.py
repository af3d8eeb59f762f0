"""Prefix sums at the sizes where their form changes: one block, one cluster, and the
two-launch form with full and ragged rows.  The cell starts of a frame are the scan of
its cell counts, so grids of chosen sizes exercise each; integers, compared exactly.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# cells per axis spanned by the particles (the grid adds its margin around them)
@pytest.mark.parametrize("cells", [(1, 1, 1), (9, 8, 10), (11, 11, 9), (45, 44, 44), (45, 46, 45), (77, 61, 52), (300, 90, 41)])
def test_cell_starts_are_the_scan_of_the_counts(pms_lib, tmp_config, cells):
    from postmps_gb300 import synth
    cs, n = 0.015, 3001
    pos = np.stack([synth.uniform(5, k, n) * cells[k] * cs for k in range(3)], 1).astype(np.float32)
    pos[0], pos[1] = 0.0, np.asarray(cells, np.float32) * np.float32(cs)
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        size = ctx.grid().sp_size
        keys, start, end = (ctx.debug(k) for k in ("keys_sorted", "cell_start", "cell_end"))
    count = np.bincount(keys, minlength=size)
    first = np.concatenate([[0], np.cumsum(count)[:-1]])
    np.testing.assert_array_equal(start, np.where(count > 0, first, 0))
    np.testing.assert_array_equal(end, np.where(count > 0, first + count, 0))
    np.testing.assert_array_equal(keys, np.sort(keys))


@pytest.mark.parametrize("elem", [4, 8])
@pytest.mark.parametrize("n", [1, 31, 4096, 4097, 131072, 131073, 3000001])
def test_scan_forms(pms_lib, tmp_config, elem, n):
    """Both element types at the lines between the forms, outputs on and off a 16-byte boundary, and
    device counts from none to all: the sums before the count, the total, and nothing written past it."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    from postmps_gb300 import synth
    f = pms_lib.lib().pms_debug_scan
    f.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_uint64, C.c_void_p, C.POINTER(C.c_uint64)]
    f.restype = C.c_int
    dtype, top = (np.int32, 1 << 9) if elem == 4 else (np.int64, 1 << 40)
    values = np.random.default_rng(n).integers(0, top, n).astype(dtype)
    sums = np.concatenate([[0], np.cumsum(values, dtype=np.int64)])
    mark = -77
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        for count in (None, 0, 1, n // 100, n - 1, n):
            m = n if count is None else count
            d_n = None if count is None else torch.tensor([count], dtype=torch.int32, device="cuda")
            for off_in, off_out in ((0, 0), (0, 1), (3, 0)):
                src = torch.full((n + 4,), mark, dtype=torch.from_numpy(values).dtype, device="cuda")
                src[off_in:off_in + n] = torch.from_numpy(values).cuda()
                dst = torch.full_like(src, mark)
                torch.cuda.synchronize()
                total = C.c_uint64()
                st = f(ctx.handle, elem, src.data_ptr() + elem * off_in, dst.data_ptr() + elem * off_out, n,
                       None if d_n is None else d_n.data_ptr(), C.byref(total))
                assert st == 0
                got = dst.cpu().numpy()
                assert total.value == sums[m]
                np.testing.assert_array_equal(got[off_out:off_out + m], sums[:m])
                assert np.all(got[:off_out] == mark) and np.all(got[off_out + m:] == mark)
