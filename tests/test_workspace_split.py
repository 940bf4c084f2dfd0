"""The stand-alone kernels use the workspace as one array of words: whatever call an entry point accepts, its words are
there (``split_model.cpp``, on the launchers' own arithmetic), and a launch that did not fit would be refused."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_every_accepted_call_fits_its_workspace(tmp_path):
    exe = tmp_path / "split_model"
    csrc = HERE.parent / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-I", str(csrc / "include"), "-I", str(csrc / "cuda"),
                    str(HERE / "split_model.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout


def test_launchers_check_the_words():
    for name, words in (("hc_encode.cu", "encode_words"), ("hc_decode.cu", "run_words")):
        src = (HERE.parent / "csrc" / "cuda" / name).read_text()
        assert words + "(split" in src and "> p.ws.words) return cudaErrorInvalidValue;" in src
