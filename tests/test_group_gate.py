"""Warps that take their steps together (csrc/group_gate.h), with threads for the warps: whichever of them gives up on whichever wait, every one of them ends."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "umbrella_b200", "csrc")

# A group as gemm_wide.cu's: units of its own to wait for, tiles to leave in between (a barrier each) and a last tile.  A barrier that a warp waits at while
# another has ended is one that nobody ever leaves.
HARNESS = r"""
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
#include "group_gate.h"

struct Barrier {
    std::mutex m;
    std::condition_variable cv;
    int here = 0, round = 0, ended = 0;
    bool all = true, result = true, stuck = false;
    bool operator()(bool ok) {
        std::unique_lock<std::mutex> lock(m);
        all = all && ok;
        const int mine = round;
        if (++here == 4) {
            result = all;
            all = true;
            here = 0;
            ++round;
            cv.notify_all();
            return result;
        }
        cv.wait(lock, [&] { return round != mine || ended > 0; });
        if (round != mine) return result;
        stuck = true;
        return false;
    }
    void end() {
        std::lock_guard<std::mutex> lock(m);
        ++ended;
        cv.notify_all();
    }
};

// waits of a warp in order: of units (even) and of the tiles left in between (odd)
static void warp(Barrier& bar, bool gated, unsigned fails, int steps) {
    umb::GroupGate gate;
    auto together = [&](bool ok) { return gated ? gate.pass(ok, bar) : bar(ok); };
    bool ok = true;
    for (int i = 0; ok && i < steps; ++i) {
        const bool passed = !(fails >> i & 1);
        ok = i & 1 ? together(passed) : passed;
    }
    together(ok);
    bar.end();
}

int main(int, char** argv) {
    const bool gated = atoi(argv[1]) != 0;
    int stuck = 0, runs = 0;
    for (int steps = 0; steps <= 5; ++steps)
        for (int who = 0; who < 16; ++who)
            for (int at = 0; at <= steps; ++at) {
                Barrier bar;
                std::vector<std::thread> t;
                for (int w = 0; w < 4; ++w) t.emplace_back([&, w] { warp(bar, gated, who >> w & 1 ? 1u << at : 0u, steps); });
                for (auto& x : t) x.join();
                stuck += bar.stuck;
                ++runs;
            }
    printf("%d %d\n", runs, stuck);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_every_warp_ends(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h")], check=True)
    stuck = [int(subprocess.run([str(tmp_path / "h"), gated], check=True, capture_output=True, text=True, timeout=120).stdout.split()[1]) for gated in "01"]
    assert stuck[0] > 0 and stuck[1] == 0                       # (without the gate some never do)


def test_the_kernels_barriers_pass_the_gate():
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "gemm_wide.cu")).read())
    uses = re.findall(r"[^\n]*\bgroup_all\([^\n]*", text)
    assert len(uses) == 2 and uses[0].startswith("__device__") and "gate.pass" in uses[1]


def test_what_is_handed_to_the_other_block_names_its_scope():
    """An arrival without a scope orders what its own block sees; the barriers of a pair are arrived at from the other block, by its threads or by the end of
    products of both.  So every remote arrival names the cluster, and so does every wait for a barrier that has one."""
    shared = {"gemm_wide.cu": {"full_a", "acc_empty", "done", "acc_full", "last_full"}, os.path.join("seq", "seq_gemm_pair.cu"): {"acc_empty", "empty"}}
    for name, bars in shared.items():
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        remote = [a for a in re.findall(r'"mbarrier\.arrive[^ ]*', text) if "shared::cluster" in a]
        assert remote and all(re.search(r"\.(release|relaxed)\.cluster\.", a) for a in remote), (name, remote)
        for bar in bars:
            waits = re.findall(r"(\w+)\(%s\b[^;{]*?, quit\)" % bar, text)
            assert waits and set(waits) <= {"spin_pair", "wait_pair"}, (name, bar, waits)
        assert re.search(r"test_wait\.parity\.(acquire|relaxed)\.cluster|UMB_TEST_WAIT\(\"\.relaxed\.cluster\"\)", text), name
