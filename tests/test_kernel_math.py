"""The arithmetic that kernels and host share, compiled for the host and run on the CPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_hit_sums_and_reservations(tmp_path):
    # 32 query windows over one repeat of 140 M positions have 4.48 G raw hits: the
    # sum must not wrap to a number that fits the hit buffer.
    exe = str(tmp_path / "kernel_math")
    csrc = os.path.join(HERE, "..", "lastz-gxy_b200", "csrc")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-I", csrc,
                    os.path.join(HERE, "harness", "kernel_math.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.stdout.strip() == "ok", r.stdout + r.stderr
