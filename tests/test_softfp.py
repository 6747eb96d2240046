"""The integer-pipe FP64 product (csrc/dcpse_softfp.cuh) equals the IEEE
product bit for bit over its whole range: 2e7 pairs on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_integer_product_is_the_ieee_product(tmp_path):
    exe = str(tmp_path / "softfp")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++",
                    os.path.join(ROOT, "tests", "cpp", "test_softfp.cpp"), "-o", exe,
                    "-I" + os.path.join(ROOT, "openfpm_numerics_gb300", "csrc")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
