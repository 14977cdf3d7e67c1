"""The autotuner keeps the fastest schedule it has measured: each uniform one and the composed one (host code)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dnsbox_b200", "csrc")


@pytest.mark.parametrize("uniform,composed,want", [
    ([4.5, 3.3], 3.6, 1),      # a mix slower than a run its passes come from, and faster than the default
    ([4.5, 3.3], 3.2, -1),
    ([3.0, 3.3], 3.2, 0),      # the default
    ([3.3], 3.3, -1),
    ([5.0, 4.0, 2.0, 2.5], 3.0, 2),
])
def test_fastest_schedule(tmp_path, uniform, composed, want):
    src = tmp_path / "pick.cpp"
    src.write_text('#include "tune_pick.h"\n#include <cstdio>\nint main() { const double u[] = {%s}; std::printf("%%d", '
                   "fastest_schedule(u, %d, %r)); }\n" % (", ".join(map(repr, uniform)), len(uniform), composed))
    exe = tmp_path / "pick"
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)])
    assert int(subprocess.check_output([str(exe)])) == want
