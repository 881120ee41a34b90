"""Row export in pieces (csrc/export.cuh) on the CPU, over a fake device: the
rows, and each call that can fail.  A copy or a mark that was not queued ends
the export with an error, with nothing left in flight; without pinned memory
nothing is written and the caller takes the keys in one copy."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_rows_and_failures(tmp_path):
    exe = str(tmp_path / "export_pieces")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-pthread", "-Wall", "-Wextra", "-Werror",
                    "-o", exe, os.path.join(HERE, "cpp", "export_pieces.cpp")], check=True)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=120)
    assert (out.returncode, out.stdout) == (0, "ok\n")
