"""The ring of bias half tiles that two streams of the D = 96 / 128 forward share, on a model without a GPU: no order in
which its loads land lets a stream read a half tile that is not there, or one that is being replaced."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bias_ring_model(tmp_path):
    exe = str(tmp_path / "ring")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "megakernel-exploration_b200", "csrc"),
                    "-x", "c++", os.path.join(ROOT, "tests", "bias_ring_model.cpp"), "-o", exe], check=True)
    said = dict(line.split(": ") for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines())
    assert said["kernel"] == "ok"
    assert said["by slot"] == "a stream reads a half tile that has not landed"      # what the model is there to find
