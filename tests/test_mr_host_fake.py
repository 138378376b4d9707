"""The Miller-Rabin engine's host code when device memory runs out.

tests/cpp/mr_host_fake.cpp runs csrc/mr.cu unchanged against a stand-in CUDA
runtime (host memory under a limit, kernels that only mark their candidates
finished), so that an allocation can fail at any point without a GPU.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("fake") / "mr_host_fake")
    subprocess.run(["g++", "-O1", "-std=c++20", "-w", "-x", "c++",
                    "-I", os.path.join(ROOT, "tests", "cpp", "emul"),
                    "-I", os.path.join(ROOT, "prime-finder_b200", "csrc"),
                    "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "mr_host_fake.cpp"), "-o", exe, "-lpthread"], check=True)

    def run(lines):
        out = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True,
                             timeout=300).stdout.strip().split("\n")
        assert out[-1] == "left 0"  # every block was freed
        return out[:-1]
    return run


@pytest.mark.parametrize("bits", [3_000, 123_100, 344_000])
def test_server_needs_no_memory_beyond_the_slot(host, bits):
    """A server whose device has room for the slot and nothing more runs the
    request; without room for the slot it reports the request, and stays up."""
    assert host(["server -1 %d" % bits, "server 1 %d" % bits, "server 0 %d" % bits]) == \
        ["verdict 0 fft", "verdict 0 fft", "verdict -1 none"]


def test_context_fits_where_the_integer_engine_does(host):
    """Moduli of 166 000 bits go to the integer engine where only its buffers,
    21 words a point, fit the device; at 20 000 bits the floating-point
    engine's buffers are no larger than those."""
    def integer_bytes(points, bits, n):  # with four 64-bit words per 16-bit limb, and tables
        return n * (21 * 4 * points + 4 * 8 * ((bits + 15) // 16)) + 8192

    rc, size, eng = host(["ctx -1 166000 4"])[0].split()[1:]
    assert (rc, eng) == ("0", "fft") and int(size) > integer_bytes(8192, 166000, 4)
    rc, small, eng = host(["ctx %d 166000 4" % (int(size) - 1)])[0].split()[1:]
    assert (rc, eng) == ("0", "int") and int(small) <= integer_bytes(8192, 166000, 4)
    assert host(["ctx %d 166000 4" % (int(small) - 1)])[0].split()[1:] == ["-3", "0", "none"]
    rc, size, eng = host(["ctx -1 20000 4"])[0].split()[1:]
    assert (rc, eng) == ("0", "fft") and int(size) <= integer_bytes(1024, 20000, 4)


@pytest.mark.parametrize("bits", [700, 20_000, 123_100, 344_000])
def test_batch_falls_back_to_the_integer_engine(host, bits):
    """Where the floating-point engine's buffers do not fit the device, the
    batch runs on the integer engine; below that it is refused."""
    rc, size, eng = host(["batch -1 %d 6" % bits])[0].split()[1:]
    assert (rc, eng) == ("0", "fft")
    rc, small, eng = host(["batch %d %d 6" % (int(size) - 1, bits)])[0].split()[1:]
    assert (rc, eng) == ("0", "int") and int(small) < int(size)
    assert host(["batch %d %d 6" % (int(small) - 1, bits)])[0].split()[1:] == ["-3", "0", "none"]


def test_autotune_times_what_a_quantum_changes(host):
    """With a block for each candidate the quantum has no part in the launch, so
    the shape of one candidate per SM is timed once per chunk: 1 + 3 launches,
    and 1 + 9 with two per SM; equal rates keep the defaults."""
    assert host(["tune 12", "tune 15"]) == ["rc 0 14 64 2048"] * 2


def test_server_runs_classes_in_turn_without_more_streams(host):
    """Two length classes run side by side on streams of their own, or one
    after the other where no further stream can be created."""
    assert host(["mixed 1", "mixed 0"]) == ["verdict 0 0 fft"] * 2
