"""A staged run that fails part way (host side, compiled here): what it queued
is joined all the same, the first error is the run's, and a scope's clean-up
runs on every way out of it."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include <cstdio>
#include "staged_run.hpp"

// a run whose fork, chunk `bad` or join fails; prints the order of its steps, its status and its message
static void run(const char *name, bool fork_ok, int bad, bool join_ok) {
    std::string steps;
    mcg::clear_error();
    mcg_status st;
    {
        const mcg::AtExit plain([&] { steps += " plain"; });
        st = mcg::forked_run(
            [&] { steps += "fork"; return fork_ok ? MCG_OK : mcg::fail(MCG_ERR_CUDA, "fork"); },
            [&]() -> mcg_status {
                for (int c = 0; c < 3; ++c) {
                    steps += " chunk";
                    if (c == bad) return mcg::fail(MCG_ERR_OOM, "chunk " + std::to_string(c));
                }
                return MCG_OK;
            },
            [&] { steps += " join"; return join_ok ? MCG_OK : mcg::fail(MCG_ERR_CUDA, "join"); });
    }
    std::printf("%s: %s: %d %s\n", name, steps.c_str(), (int)st, mcg::last_error().c_str());
}

int main() {
    run("whole", true, -1, true);
    run("second chunk", true, 1, true);
    run("first chunk and join", true, 0, false);
    run("fork", false, -1, true);
    run("join", true, -1, false);
}
"""


def test_what_a_failed_run_queued_is_joined(tmp_path):
    src, exe = tmp_path / "run.cc", tmp_path / "run"
    src.write_text(SOURCE)
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'mcscram_b200/csrc'}", str(src), str(ROOT / "mcscram_b200/csrc/error.cpp"), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    cuda, oom = 2, 3  # MCG_ERR_CUDA, MCG_ERR_OOM
    assert out == [
        "whole: fork chunk chunk chunk join plain: 0 ",
        f"second chunk: fork chunk chunk join plain: {oom} chunk 1",
        f"first chunk and join: fork chunk join plain: {oom} chunk 0",
        f"fork: fork join plain: {cuda} fork",
        f"join: fork chunk chunk chunk join plain: {cuda} join",
    ]
