"""Copies of pageable memory: whole, and on the stream they were asked for - which for a context on
cudaStreamPerThread only the calling thread can name. Runs against a stand-in for the CUDA runtime."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_copies_stay_on_their_stream(tmp_path):
    exe = str(tmp_path / "host_copy_check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(CUDA, "include"), "-o", exe,
                           os.path.join(HERE, "native", "host_copy_check.cpp"),
                           os.path.join(HERE, "..", "cortexsdr_b200", "csrc", "host", "host_copy.cpp")])
    done = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout + done.stderr
