"""Inside the tracking run (csrc/tracking.cu, gn_track_kernel): what no call
of the library reaches, by a program that shares its arena."""
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def program(gbf, tmp_path_factory):
    from libfusion_gb300 import build as B
    exe = tmp_path_factory.mktemp("run") / "track_run"
    subprocess.run([B.nvcc(), *B.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", str(HERE / "track_run_main.cu"),
                    str(B.LIB), "-Xlinker", f"-rpath={B.LIB.parent}", "-lcuda", "-o", str(exe)], check=True,
                   capture_output=True)

    def run(*args):
        r = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout + r.stderr
    return run


def test_run_numbers_wrap(program):
    """The numbers of a run's words go on from frame to frame for the session's life:
    past 2^31 and past 2^32 the frames are those of a new session."""
    program("numbers")


def test_run_whose_wait_ran_out(program):
    """CTA 0 gives up waiting: the run ends at once, the frame is not tracked and carries a
    flag of its own, and the session's next run is as if that one had not been."""
    program("lost")


def test_frames_on_a_stream_with_few_sms(program):
    """A green context's stream has too few SMs for all CTAs of the run at once: those that
    are there make it, with the same result."""
    program("few_sms")
