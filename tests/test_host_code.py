"""Host-only parts of the library, compiled by g++ with a small program of
the test's own: what no device is needed for is shown without one."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ablsteadyrans_b200", "csrc")

needs_gxx = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def _run(tmp_path, source, *include):
    """Compiles and runs a program; its output lines."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    cmd = ["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror"]
    for d in include:
        cmd += ["-I", str(d)]
    r = subprocess.run(cmd + [str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout.split("\n")[:-1]


@needs_gxx
@pytest.mark.parametrize("counts", [(4,), (16, 16, 4), (16, 2), ()])
def test_forgetting_chunks_keeps_the_neighbours(tmp_path, counts):
    """Vectors of other allocations right below and right above the chunks (a
    full one of 16 vectors and a short last one) stay in the list, in order;
    those in the chunks, the first and the last of each, leave it."""
    sizes = ", ".join(str(c) for c in counts)
    out = _run(tmp_path, f"""
#include "gb_krylov.h"
#include <cstdio>
int main()
{{
    constexpr int vol = 5;
    const std::vector<int> counts{{{sizes}}};
    std::vector<double> memory(1000);
    double* at = memory.data();
    std::vector<double*> list, kept;
    std::vector<gb::KrylovChunk> chunks;
    auto keep = [&](int n) {{
        for (int q = 0; q < n; ++q, at += vol) {{ list.push_back(at); kept.push_back(at); }}
    }};
    keep(3);
    for (int n : counts) {{
        chunks.push_back(gb::KrylovChunk{{at, vol * n}});
        for (int q = 0; q < n; ++q, at += vol) {{ list.push_back(at); }}
        keep(3);
    }}
    gb::forget_chunks(chunks, list);
    std::printf("%d\\n", list == kept ? 1 : 0);
}}
""", CSRC)
    assert out == ["1"]
