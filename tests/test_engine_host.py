"""The engine's host path on a machine without a GPU: its objects linked with a
stand-in for the CUDA runtime (cpp/fake_cudart.cpp), in which device memory is
host memory and kernels do not run. Each program checks one property and prints
"ok"."""
import importlib.util
import shutil
import subprocess
from pathlib import Path

import pytest

from torpedo_gb300 import build as B

ROOT = Path(__file__).resolve().parent.parent
CPP = ROOT / "tests" / "cpp"


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    B.build()
    cuda = Path(B.nvcc()).resolve().parents[1] / "include"
    out = tmp_path_factory.mktemp("engine_host")

    def go(program):
        exe = out / program
        objects = [str(B.OUT / (src + ".o")) for src in B.SOURCES]
        cmd = [gxx, "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(cuda), str(CPP / f"{program}.cpp"),
               str(CPP / "fake_cudart.cpp"), *objects, "-lpthread", "-o", str(exe)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stdout + r.stderr
        return r.stdout.splitlines()[:-1]

    return go


def test_compile_beside_another_threads_capture(run):
    run("engine_compile_capture")


def test_failed_allocations_leave_nothing_stale(run):
    run("engine_alloc_failures")


def test_bench_counts_the_launches_of_a_frame(run):
    """The bench's launch count (frame_launches) against the launches that the engine makes."""
    spec = importlib.util.spec_from_file_location("bench_under_test", ROOT / "bench.py")
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    lines = run("engine_frame_launches")
    assert len(lines) >= 20
    for line in lines:
        views, n, w, h, lookback, ctas, launches = map(int, line.split())
        settings = {"key_sort_lookback": lookback, "sort_ctas_per_sm": ctas}
        assert bench.frame_launches(views, n, (w + 15) // 16, (h + 15) // 16, settings) == launches, line
