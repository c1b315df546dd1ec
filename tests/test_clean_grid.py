"""The state of the grid that the NUFFT adjoint accumulates into (csrc/clean_grid.cuh), with fakes of
the launches, so that calls can fail: no later call adds to a grid that is not zero."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cstdio>
#include <functional>
#include <vector>
#include "clean_grid.cuh"

struct Stream {  // a grid, work that runs at once or is recorded, and calls that fail on request
    int grid = 0, result = 0;
    bool dirty = false, capturing = false, fail_run = false, fail_clear = false;
    std::vector<std::function<void()>> graph;
    void enqueue(std::function<void()> f) { capturing ? graph.push_back(f) : f(); }
    int adjoint(int value)
    {
        return lentils::accumulate_clean(
            dirty,
            [&] {
                enqueue([this, value] { grid += value; });
                if (fail_run) return 1;  // between the gridding and the transform
                enqueue([this] { result = grid; grid = 0; });
                return 0;
            },
            [&] {
                if (fail_clear) return 2;
                enqueue([this] { grid = 0; });
                return 0;
            },
            [&] { return capturing; });
    }
    void replay() { for (auto &f : graph) f(); }
};

static int bad = 0;
#define EXPECT(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); ++bad; } } while (0)

int main()
{
    {   // plain calls, and a failed one between them
        Stream s;
        EXPECT(s.adjoint(3) == 0 && s.result == 3 && s.adjoint(4) == 0 && s.result == 4);
        s.fail_run = true;
        EXPECT(s.adjoint(100) == 1);
        s.fail_run = false;
        EXPECT(s.adjoint(5) == 0 && s.result == 5 && !s.dirty);
    }
    {   // a failed call whose clearing fails too; the next call clears
        Stream s;
        s.fail_run = s.fail_clear = true;
        EXPECT(s.adjoint(100) == 1 && s.dirty);
        EXPECT(s.adjoint(1) == 2 && s.dirty);
        s.fail_run = s.fail_clear = false;
        EXPECT(s.adjoint(5) == 0 && s.result == 5 && !s.dirty && s.adjoint(6) == 0 && s.result == 6);
    }
    for (int launched = 0; launched < 2; ++launched) {
        // a dirty grid, a call that is only captured, then calls before, between and after replays
        Stream s;
        s.fail_run = s.fail_clear = true;
        EXPECT(s.adjoint(100) == 1);
        s.fail_run = s.fail_clear = false;
        s.capturing = true;
        EXPECT(s.adjoint(7) == 0);
        s.capturing = false;
        if (launched) {
            s.replay();
            EXPECT(s.result == 7);
        }
        EXPECT(s.adjoint(5) == 0 && s.result == 5);
        s.replay();
        EXPECT(s.result == 7 && s.adjoint(6) == 0 && s.result == 6);
    }
    {   // a graph captured from a clean grid, and a failed call before its replay
        Stream s;
        s.capturing = true;
        EXPECT(s.adjoint(7) == 0 && s.graph.size() == 2);  // no memset
        s.capturing = false;
        s.fail_run = true;
        EXPECT(s.adjoint(100) == 1);
        s.fail_run = false;
        s.replay();
        EXPECT(s.result == 7);
    }
    {   // a call that fails while it is captured changes nothing
        Stream s;
        s.capturing = s.fail_run = true;
        EXPECT(s.adjoint(100) == 1 && !s.dirty);
        s.capturing = s.fail_run = false;
        EXPECT(s.adjoint(5) == 0 && s.result == 5);
    }
    return bad;
}
"""


def test_no_call_adds_to_a_dirty_grid(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "driver"
    out = subprocess.run([cxx, "-std=c++17", "-I", os.path.join(REPO, "lentils_gb300", "csrc"),
                          str(src), "-o", str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
