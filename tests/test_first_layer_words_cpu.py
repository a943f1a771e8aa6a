"""Loads of the first layer's row kernel for rows that are not whole 16-byte pieces (conv_first_words.h): compiled for the
host, every start and length beside the end of a tensor.  Runs without a GPU."""
import os
import subprocess


def test_row_pieces_stay_inside_the_tensor(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "first_layer_words_test"
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(root, "tests", "first_layer_words_test.cpp"), "-o", str(exe),
                    "-I" + os.path.join(root, "ai-gamer_b200", "csrc")], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout[-2000:] + done.stderr
