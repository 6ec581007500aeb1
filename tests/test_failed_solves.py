"""A device solve that fails midway (an allocation, a launch) returns only when neither stream can
still read the caller's arrays: the targets are sorted on the second stream from early on."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CAPI = open(os.path.join(ROOT, "2d-treecodes_b200", "csrc", "capi.cu")).read()


def test_device_solves_drain_both_streams_before_an_error_return():
    drain = CAPI[CAPI.index("static int drain_and_fail("):]
    drain = drain[:drain.index("\n}")]
    assert "wait_stream(c, c.aux)" in drain and "wait_stream(c, c.stream)" in drain
    for fn in ("potential_device", "force_device"):
        body = CAPI[CAPI.index(f"static int {fn}("):]
        queued = body[body.index("phase_mark(c, 0)"):body.index("phase_mark(c, 5)")]
        assert re.findall(r"return [^;]*;", queued) == ["return drain_and_fail(c, rc);"], fn
