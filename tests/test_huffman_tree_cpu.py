"""The Huffman tree parser of the decoder, on the CPU: the second tables have a
slot for every prefix that needs one, also for damaged trees."""
import os
import subprocess

from faz_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_decoder_slots_cover_every_prefix(tmp_path):
    exe = str(tmp_path / "huffman_tree_check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-I" + B.cuda_include(), "-o", exe,
                           os.path.join(ROOT, "tests", "huffman_tree_check.cpp"),
                           os.path.join(ROOT, "faz_gb300", "csrc", "huffman_host.cpp")])
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
