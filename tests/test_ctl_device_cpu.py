"""Reading a handle's state from a thread whose current device is another GPU (tests/host/ctl_device.cpp: a fake CUDA
runtime that refuses a launch on a stream of another device, as CUDA does). nsf_get_time, nsf_sync (and with it
nsf_ensemble_sync) and nsf_upload_conserved work from any thread, and leave the thread's device as it was."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "3d-ns-fsi_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_control_block_is_read_on_the_handles_device(tmp_path):
    exe = str(tmp_path / "ctl_device")
    subprocess.run(["g++", "-std=c++17", "-O1", "-no-pie", "-fno-pie", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
                    "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "host", "ctl_device.cpp"),
                    os.path.join(CSRC, "nsf_capi.cpp"), "-o", exe, "-Wl,--unresolved-symbols=ignore-all"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stderr)
    assert r.stdout.split("\n")[:3] == ["nsf_get_time 0 0", "nsf_sync 0 0", "nsf_upload_conserved 0 0"]
