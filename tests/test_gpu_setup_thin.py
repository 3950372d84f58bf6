"""The curvature d of thin volumes (a thread per voxel) and of sizes on both sides
of the line to the blocked form, against the FP64 oracle as in test_gpu_setup."""
import pytest

from test_gpu_setup import test_setup_against_oracle as check

pytestmark = pytest.mark.gpu

# (nx, ny, nz), (BINSx, BINSy): one row, one column, blocks of 128 left over, many
# planes; 32 x 6 and 32 x 7 (0.375 and 0.44 of a block)
SIZES = [((129, 1, 3), (70, 9)), ((1, 41, 4), (9, 50)), ((5, 3, 40), (14, 12)),
         ((32, 6, 3), (40, 12)), ((32, 7, 3), (40, 12))]


@pytest.mark.parametrize("size", SIZES, ids=["%dx%dx%d" % s[0] for s in SIZES])
def test_thin_volumes(size):
    check(size, "length")
