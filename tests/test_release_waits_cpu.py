"""Memory of the host layer's arrays is handed out again only when nothing can use it: what a release waits for."""
import os
import subprocess

import fake_device

ROOT = fake_device.ROOT


def test_release_waits_for_every_stream_the_array_was_used_on(tmp_path):
    from thundersvm_b200 import build
    lib = os.path.dirname(build.build())
    runtime, exe = fake_device.compile_runtime(tmp_path), str(tmp_path / "release_waits")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-pthread", "-I/usr/local/cuda/include",
                           "-I" + os.path.join(ROOT, "thundersvm_b200", "csrc", "host", "include"),
                           os.path.join(ROOT, "tests", "release_waits.cpp"), "-o", exe, runtime, "-L" + lib,
                           "-lthundersvm_b200", "-Wl,-rpath," + lib, "-Wl,--allow-shlib-undefined"])
    fake_device.run_child(runtime, [exe])
