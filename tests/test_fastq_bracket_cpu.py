"""The float reconstruction and quantiser of the common path
(faz_gb300/csrc/fastq.cuh) on the CPU, against the double computation on random and
adversarial inputs over the whole ranges of values, bounds and radii."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bracket_matches_double(tmp_path):
    exe = str(tmp_path / "fastq_bracket_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(ROOT, "tests", "fastq_bracket_check.cpp")])
    for seed in (21, 22):
        r = subprocess.run([exe, "3000000", str(seed)], stdout=subprocess.PIPE, text=True)
        assert r.returncode == 0, r.stdout
