"""Large results on their way to pageable host memory, without a GPU: the part
of the copy that runs on the host (csrc/hostmove.h)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def _program(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-rdynamic", "-pthread", os.path.join(HERE, "native", name + ".cpp"),
                    "-o", exe, "-ldl"], check=True)
    return exe


def test_pieces_through_the_ring(tmp_path):
    """Sizes around a piece and the ring's length; every allocation, every thread start and every call of the link
    failing in its turn: the bytes are right or the verdict says why not, and nothing reaches the C caller as an
    exception."""
    r = subprocess.run([_program(tmp_path, "host_move")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.splitlines()[-1] == "all right", r.stdout + r.stderr


def test_which_results_take_the_ring(tmp_path):
    """Results of 6 to 16 MiB take the ring only when memory for a MiB or more of them is not there yet: a result
    buffer that is used again goes by plain copies, which are faster at these sizes."""
    r = subprocess.run([_program(tmp_path, "ring_rule")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.splitlines()[-1] == "all right", r.stdout + r.stderr
