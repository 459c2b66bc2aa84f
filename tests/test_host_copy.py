"""Uploads of images in ordinary memory (csrc/host_copy.cu) on the CPU, against a CUDA runtime made of host memory whose transfers
are as late as they may be (tests/host_copy_check.cc)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host_copy") / "host_copy_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", f"-I{cuda}/include", "-x", "c++", os.path.join(ROOT, "tests", "host_copy_check.cc"),
                    os.path.join(ROOT, "darknet_b200", "csrc", "host_copy.cu"), "-pthread", "-ldl", "-o", out], check=True)

    def run(*args):
        r = subprocess.run([out, *args], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout.strip().endswith("ok"), (r.returncode, r.stdout[-500:], r.stderr[-500:])
    return run


@pytest.mark.parametrize("how", ["in_turn", "threads"])
def test_ring_slots_are_rewritten_only_after_their_transfers(check, how):
    check(how)


@pytest.mark.parametrize("how", ["no_threads", "no_memory", "little_memory"])
def test_what_cannot_be_had_is_done_without(check, how):
    check(how)


def test_small_images_take_little(check):
    check("small")
