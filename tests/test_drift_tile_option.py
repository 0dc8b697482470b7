"""The drift medium's passes come in tiles of 1, 2 and 4 rows.  The build option
that fixes the height (FOLD3D_DRIFT_TV; 0: by grid size) admits those and nothing
else: another height has no kernel, and no place in the context's occupancy table."""
import os
import subprocess

import pytest


@pytest.mark.parametrize("rows", [0, 1, 2, 3, 4, 5, 8, -1])
def test_drift_tile_option(rows):
    import build as pkg_build  # fgcs-openacc-advanced_b200/build.py

    cmd = [pkg_build.NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=compute_100a", "-x", "cu",
           "-DFOLD3D_DRIFT_TV=%d" % rows, "-I", pkg_build.INCLUDE, "-I", pkg_build.CSRC, "-cuda", "-", "-o", os.devnull]
    r = subprocess.run(cmd, capture_output=True, text=True, input='#include "fold3d_internal.h"\n')
    assert (r.returncode == 0) == (rows in (0, 1, 2, 4)), r.stderr
