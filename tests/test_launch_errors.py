"""Which launch errors let a one-launch search run level by level instead
(psb_launch.h); the others are reported."""
import os
import subprocess

from puzzlesearch_b200 import build

ROOM = ["InvalidClusterSize", "InvalidConfiguration", "LaunchOutOfResources", "MemoryAllocation", "NotSupported"]
REPORTED = ["InvalidValue", "InvalidDeviceFunction", "InvalidResourceHandle", "IllegalAddress", "IllegalInstruction",
            "MisalignedAddress", "LaunchFailure", "LaunchTimeout", "ContextIsDestroyed", "StreamCaptureUnsupported"]


def test_only_a_lack_of_room_is_no_error(tmp_path):
    lines = ['#include "psb_launch.h"', "static_assert(!psb::launch_has_no_room(cudaSuccess));"]
    lines += [f"static_assert(psb::launch_has_no_room(cudaError{e}));" for e in ROOM]
    lines += [f"static_assert(!psb::launch_has_no_room(cudaError{e}));" for e in REPORTED]
    src = tmp_path / "launch_errors.cpp"
    src.write_text("\n".join(lines) + "\n")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run([build.host_compiler(), "-std=c++17", "-fsyntax-only", "-I" + build.CSRC, "-I" + cuda, str(src)],
                   check=True)
    # and the one-launch search asks
    text = open(os.path.join(build.CSRC, "psb_host.cu")).read()
    body = text[text.index("int small_search("):text.index("int session_run(")]
    assert "psb::launch_has_no_room(" in body
