"""The C interface's version goes with the layout of its argument structs: a changed size has to come with another
number in the header, or a host built against the older header is read past its structs' ends."""
import ctypes
import re

from tests.test_capi import HEADER
from textured_gaussians_b200 import _backend as B

# bytes of (tg_raster_fwd_args, tg_raster_bwd_args) by version
SIZES = {1: (376, 544), 2: (400, 576)}


def test_version_goes_with_the_struct_sizes():
    declared = re.findall(r"^#define TG_ABI_VERSION (\d+)$", open(HEADER).read(), flags=re.M)
    assert declared == [str(B.lib().tg_version())]
    assert SIZES[int(declared[0])] == (ctypes.sizeof(B.RasterFwdArgs), ctypes.sizeof(B.RasterBwdArgs))
