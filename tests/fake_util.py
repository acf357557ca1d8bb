"""Host sources of the library built with tests/fake_cuda instead of the CUDA runtime."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "new_fgssjoin_b200", "csrc")


def run(tmp_path, program, sources=(), timeout=300):
    """Compiles `program` (C++ text) with the named files of csrc, runs it, returns its output."""
    src = tmp_path / "main.cpp"
    src.write_text(program)
    exe = str(tmp_path / "main")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(HERE, "fake_cuda"), "-I", CSRC, "-o",
                           exe, str(src)] + [os.path.join(CSRC, s) for s in sources] + ["-lpthread"])
    p = subprocess.run([exe], capture_output=True, text=True, timeout=timeout)
    assert p.returncode == 0, p.stdout + p.stderr
    return p.stdout
