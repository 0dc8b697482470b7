"""bench.py reports the captured pipe shares only for grids that run the captured
form of the drift kernel, tiles of 4 rows, and names it; the limit is the
library's own."""
import os
import re

from conftest import PKG, ROOT


def test_capture_belongs_to_its_kernel(monkeypatch):
    monkeypatch.syspath_prepend(ROOT)
    import bench

    src = open(os.path.join(PKG, "csrc", "fold3d_api.cu")).read()
    limit = float(re.search(r"rows < 12000\.0 \? 1 : rows < ([0-9.]+) \? 2 : 4", src).group(1))
    for n in (128, 512, 1011, 1012, 1280):
        rows = 3.0 * n ** 3 / 32.0 / (3.0 * n)
        got = bench.fp64_capture(n)
        assert (got is not None) == (rows >= limit), n
        assert got is None or got["kernel"] == "drift_pass_kernel<4>"
