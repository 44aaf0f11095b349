"""What a kernel is granted (more shared memory) holds on one device: every device of a process asks for itself."""
import os
import re
import subprocess

from xyntetik_runner_b200.csrc import build

PROGRAM = r"""
#include "per_device.h"
#include <cstdio>
int main() {
    bool done[XR_DEVICES] = {};
    int asked = 0;
    bool grant = false;
    auto ask = [&] { asked++; return grant; };
    bool ok = !xr_once_on_device(done, 0, ask) && asked == 1;                 // refused: asked again later
    grant = true;
    ok = ok && xr_once_on_device(done, 0, ask) && asked == 2 && xr_once_on_device(done, 0, ask) && asked == 2;
    ok = ok && xr_once_on_device(done, 1, ask) && asked == 3;                 // another device asks for itself
    ok = ok && xr_once_on_device(done, XR_DEVICES - 1, ask) && asked == 4;
    ok = ok && xr_once_on_device(done, XR_DEVICES, ask) && xr_once_on_device(done, -1, ask) && asked == 6;
    return ok ? 0 : 1;
}
"""


def test_every_device_asks_once(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run([build.find_cxx(), "-std=c++17", "-I", build.HERE, "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_launcher_remembers_for_the_whole_process():
    """A launcher that opts a kernel into more shared memory does so through xr_once_per_device, or at every launch."""
    for name in sorted(os.listdir(build.HERE)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(build.HERE, name)) as f:
            text = f.read()
        assert not re.search(r"static\s+(const\s+)?bool\s+\w+\s*=", text), name
        for at in (m.start() for m in re.finditer(r"xr_allow_smem\(", text)):
            near = text[max(0, at - 600):at]
            assert "xr_once_per_device" in near or "known[dev]" in near or "inline bool" in near[-80:], (name, text[at:at + 80])
