"""The runtime's host-side decisions, compiled as plain C++ from the library's
own headers and run without a GPU."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from cuminlp_gb300 import build

ROOT = Path(__file__).resolve().parents[1]


def run(tmp_path, header: str, body: str) -> None:
    """Compiles a program that includes a csrc header; every CHECK must hold."""
    cc = shutil.which("g++") or pytest.skip("g++ not found")
    src = tmp_path / "check.cpp"
    src.write_text(f'#include <cstdio>\n#include "{header}"\n'
                   "#define CHECK(x) if (!(x)) { std::printf(\"line %d: %s\\n\", __LINE__, #x); return 1; }\n"
                   "using namespace cmn;\nint main() {\n" + body + "\nreturn 0;\n}\n")
    cuda = Path(build._nvcc()).resolve().parents[1] / "include"
    exe = tmp_path / "check"
    subprocess.run([cc, "-std=c++17", "-w", f"-I{cuda}", f"-I{ROOT / 'cuminlp_gb300' / 'csrc'}", str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_planes_beyond_the_largest_pitch_go_one_by_one(tmp_path):
    run(tmp_path, "handles.hpp", """
    const uint64_t most = (1ull << 31) - 1;
    CHECK(plane_copy(4, 100, 100, most) == PlaneCopy::kPacked);
    CHECK(plane_copy(4, 100, 101, most) == PlaneCopy::kPitched);
    CHECK(plane_copy(4, 100, most / 8, most) == PlaneCopy::kPitched);
    CHECK(plane_copy(4, 100, most / 8 + 1, most) == PlaneCopy::kEach);
    CHECK(plane_copy(4, 1ull << 28, 1ull << 28, most) == PlaneCopy::kPacked);
    CHECK(plane_copy(4, 1ull << 28, (1ull << 28) + 1, most) == PlaneCopy::kEach);
    CHECK(plane_copy(1, 100, 1ull << 40, most) == PlaneCopy::kPacked);
    """)


def test_a_device_error_ends_the_search(tmp_path):
    # a barrier's wait that ran out in one iteration: the kernels behind it
    # stop, and the burst's other iterations begin nothing
    run(tmp_path, "search.hpp", """
    static SolverDev d;
    d.pool_size = 5;
    d.improved = 1;
    CHECK(begin_search(d) && !halted(d) && d.improved == 0);
    d.ticket = 3;
    d.error = 1;
    CHECK(halted(d));
    for (int i = 0; i < 63; ++i) {
      d.improved = 1;
      CHECK(!begin_search(d) && halted(d) && d.done == 1 && d.improved == 0);
    }
    CHECK(d.pool_size == 5 && d.error == 1);
    static SolverDev stopped;
    stopped.done = 1;
    CHECK(!begin_search(stopped) && halted(stopped) && stopped.error == 0);
    """)
