"""Every tile height that the build options admit for the elliptical medium
(FOLD3D_WAVE_TV) compiles: the kernel sources through the device front end."""
import os
import subprocess

import pytest


@pytest.mark.parametrize("rows", [1, 2, 4, 8])
@pytest.mark.parametrize("source", ["fold3d_wavefront.cu", "fold3d_adjoint.cu"])
def test_elliptical_tile_heights_compile(tmp_path, source, rows):
    import build as pkg_build  # fgcs-openacc-advanced_b200/build.py

    cmd = [pkg_build.NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=compute_100a", "--fmad=false",
           "-DFOLD3D_WAVE_TV=%d" % rows, "-I", pkg_build.INCLUDE, "-I", pkg_build.CSRC, "-cuda",
           os.path.join(pkg_build.CSRC, source), "-o", str(tmp_path / "out.ii")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
