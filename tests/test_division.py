"""The quotient by one correction that the bit-exact row structure rests on."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_one_correction_gives_the_quotient(tmp_path):
    exe = str(tmp_path / "div")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "cpp", "div_one_correction.cpp"),
                    "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.strip() == "0"
