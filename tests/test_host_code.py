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


STUB = os.path.join(ROOT, "tests", "cuda_stub")

# A fork with two branches (one entered twice, one joined early), the main
# stream between and after them; every launch records the stream it went to.
BRANCHES = """
#include "gb_branches.h"
#include <cstdio>
int main()
{
    Handle home{"main"};
    cudaStream_t stream = &home;
    {
        gb::SideStreams sides;
        if (!sides.ready()) { return 1; }
        calls.clear();
        n_calls = 0;
        fail_at = FAIL;
        auto launch = [&](const char* what) { calls.push_back(std::string(what) + " on " + stream->name); };
        launch("before");
        {
            gb::SideBranches br(sides, stream, true);
            br.on(1);
            launch("a1");
            br.on(2);
            launch("b1");
            br.join(1);
            launch("after a1");
            br.on(1);
            launch("a2");
            gb::SideBranches inner(sides, stream, true);
            inner.on(3);
            launch("inner");
        }
        launch("after all");
        if (stream != &home || sides.forked) { return 1; }
        if (last_error != cudaSuccess) { calls.push_back("error left"); }
    }
    for (const std::string& c : calls) { std::printf("%s\\n", c.c_str()); }
    return n_made == n_destroyed ? 0 : 1;
}
"""


def _precedes(log, first, then):
    """Whether a log of streams, events and host waits orders launch `first` before launch `then`."""
    at = {}  # stream or event -> the launches it comes after
    for line in log:
        if line.endswith(" fails"):
            continue
        w = line.split()
        if w[0] == "record":
            at[w[1]] = set(at.get(w[3], ()))
        elif w[1:3] == ["waits", "for"] and w[0] != "host":
            at[w[0]] = at.get(w[0], set()) | at.get(w[3], set())
        elif w[0] == "host":
            # what any stream is sent after it comes after
            for s in ("main", "stream1", "stream3", "stream5", "stream7"):
                at[s] = at.get(s, set()) | at.get(w[3], set())
        elif " on " in line:
            what, stream = line.rsplit(" on ", 1)
            if what == then:
                return first in at.get(stream, set())
            at.setdefault(stream, set()).add(what)
    raise AssertionError((first, then, log))


@needs_gxx
@pytest.mark.parametrize("fail", range(-1, 10))
def test_branches_keep_their_order_when_a_call_fails(tmp_path, fail):
    """The fork, each wait and each record in turn fail: what follows a branch
    still comes after it (through the host where no event can say so), a
    branch that cannot wait for the fork stays on the main stream, and no
    error is left behind."""
    log = _run(tmp_path, BRANCHES.replace("FAIL", str(fail)), CSRC, STUB)
    for what in ("a1", "b1", "after a1", "a2", "inner"):
        assert _precedes(log, "before", what), (what, log)
    assert _precedes(log, "a1", "after a1")
    for what in ("a1", "b1", "after a1", "a2", "inner"):
        assert _precedes(log, what, "after all"), (what, log)
    assert "error left" not in log
    if fail < 0:
        # the branches run beside the main stream: b1 is not waited for before the join
        assert not _precedes(log, "b1", "after a1")
        assert sum("host" in ln for ln in log) == 0
    elif fail >= 9:
        assert not any("fails" in ln for ln in log)  # all calls have had their turn
