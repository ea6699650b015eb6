"""The predictor's staging of small feeds, on the host alone: repeated feeds of one input without a forward, more inputs than
descriptors, more bytes than the buffer, drops in between, and batches still being read. (tests/feed_stage_check.cc, built
with AddressSanitizer.)"""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "x-deeplearning_b200")


def test_feeds_stay_inside_the_staging_buffer_and_the_last_one_arrives(tmp_path):
    exe = str(tmp_path / "feed_stage_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-fno-omit-frame-pointer",
                           "-I" + os.path.join(PKG, "host", "src"), "-I" + os.path.join(PKG, "host", "include"),
                           "-I" + os.path.join(os.path.dirname(PKG), "include"), "-I" + os.path.join(cuda, "include"),
                           os.path.join(HERE, "feed_stage_check.cc"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr[-2000:]
