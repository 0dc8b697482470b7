"""The reference driver's argument lists are there without its sources: six
calls of six spacings, F and three drifts each (AN_ISO_1_OpenACC.c:1195-1236),
and a call into its own build says why it cannot be made."""
import math

import pytest

from oracle import _REF_CALLS, REF_A, REF_F, RefLib, build, ref_spacing


def test_argument_lists_need_no_reference(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "REF_DIR", str(tmp_path))
    monkeypatch.setattr(build, "REF_OUT", str(tmp_path / "out"))
    n = 16
    h, r = ref_spacing(n), RefLib(n)
    d = math.sqrt(h * h + h * h)
    assert [c[0] for c in _REF_CALLS] == ["function_x_down", "function_x_up", "function_k_up", "function_k_down",
                                          "function_y_up", "function_y_down"]
    for entry in _REF_CALLS:
        args = r._args(entry)
        assert args[:7] == [h, h, h, d, d, d, REF_F]
        assert sorted(map(abs, args[7:])) == sorted(map(abs, REF_A))
    with pytest.raises(build.ReferenceMissing):
        r.L
