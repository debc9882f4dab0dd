"""Which step kernel runs: the launch's blocks tell k_resident (one per task, fewer than the SMs at
these sizes) from k_persist (one or two per SM), so a comparison of the two cannot pass by running one
kernel twice.  And the resident kernel's paths for tiles that do not fit whole, bitwise against
k_persist: the moments of a tile in chunks of 4 of 8 rows (1024 x 1024 with compiled transforms, 1040 x
1001 with a last tile of one row), 4 of 6, 2 of 8 (last tile of two rows), 2 of 6; the tallest tiles;
350 x 350 with its compiled transforms, every buffer resident."""
import numpy as np
import pytest

from test_gpu_resident import _run

pytestmark = pytest.mark.gpu
SMS = 148


@pytest.mark.parametrize("nx,ny,grid", [
    (4, 4, 2), (5, 7, 4), (33, 24, 12), (64, 64, 32), (130, 165, 83), (96, 96, 48), (128, 128, 64), (192, 192, 96),
    (256, 256, 128), (40, 297, 75), (64, 298, 75), (597, 40, 75), (512, 512, 129), (1100, 64, 138),
])
def test_kernel_of_each_size(monkeypatch, nx, ny, grid):
    _, a = _run(monkeypatch, True, nx, ny, 1.0, False)
    _, b = _run(monkeypatch, False, nx, ny, 1.0, False)
    assert a["grid"] == grid and b["grid"] in (SMS, 2 * SMS), (a["grid"], b["grid"])


@pytest.mark.parametrize("nx,ny,grid,mask", [
    (350, 350, 117, False), (1024, 1024, 129, False), (1040, 1001, 131, True), (1100, 594, 138, False),
    (1100, 890, 138, False), (1300, 600, 109, True), (300, 2001, 144, False),
])
def test_large_tiles_bitwise(monkeypatch, nx, ny, grid, mask):
    a, sa = _run(monkeypatch, True, nx, ny, 3.0, mask)
    b, sb = _run(monkeypatch, False, nx, ny, 3.0, mask)
    assert sa["grid"] == grid and sb["grid"] in (SMS, 2 * SMS), (sa["grid"], sb["grid"])
    assert sa["naccept"] > 2 and sa["nsparse"] >= 1
    for k in ("naccept", "nreject", "nf", "nsparse"):
        assert sa[k] == sb[k], (k, sa[k], sb[k])
    for f in a:
        assert np.all(np.isfinite(a[f])) and np.array_equal(a[f], b[f]), (f, np.abs(a[f] - b[f]).max())


@pytest.mark.parametrize("nx,ny,grid,mask", [
    (64, 299, 76, False), (64, 303, 77, True), (64, 351, 89, False), (512, 323, 129, False), (96, 645, 109, True),
    (300, 2003, 144, False), (1040, 1003, 131, True),
])
def test_odd_rows_take_their_even_neighbours_height(monkeypatch, nx, ny, grid, mask):
    """The last of an odd number of rows is a tile of its own; the others are as high as one row fewer
    asks for (4, 4, 4, 4, 6, 14 and 8 here; the tile before the last row 2, 2, 2, 2, 2, 14 and 2)."""
    a, sa = _run(monkeypatch, True, nx, ny, 3.0, mask)
    b, sb = _run(monkeypatch, False, nx, ny, 3.0, mask)
    assert sa["grid"] == grid and sb["grid"] in (SMS, 2 * SMS), (sa["grid"], sb["grid"])
    assert sa["naccept"] > 2 and sa["nsparse"] >= 1
    for k in ("naccept", "nreject", "nf", "nsparse"):
        assert sa[k] == sb[k], (k, sa[k], sb[k])
    for f in a:
        assert np.all(np.isfinite(a[f])) and np.array_equal(a[f], b[f]), (f, np.abs(a[f] - b[f]).max())
