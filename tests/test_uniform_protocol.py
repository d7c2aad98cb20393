"""How PROPOSE's threads agree that the proposal of uniform tiles is in shared
memory (csrc/pearl_uniform.hpp), on the CPU under ThreadSanitizer.

A block is a handful of host threads that walk tiles with one barrier a tile, as
the kernel does, and ask the header's own class when to write and when to read
the shared proposal.  Nothing else orders them, so an access that the votes do
not order is reported as a race.  The same walk with a flag that is read after
the barrier, which does not order the leader's next tile, is reported: the check
sees what it is there for.
"""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fe-c_eutectoid_phase-field_simulation_b200" / "csrc"

SOURCE = r"""
#include <atomic>
#include <barrier>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "pearl_uniform.hpp"

constexpr int kThreads = 8, kTiles = 400;
struct Proposal { double q[8]; int flag; } U;  // plain shared words

#ifdef LATE_FLAG
struct Agreement {  // the flag is looked at after the vote
    bool filled = false;
    bool takes(bool same) const { return same && filled; }
    bool fills(bool same, bool leader) const { return same && leader && !filled; }
    void vote(bool) { if (!filled) filled = U.flag != 0; }
};
#else
using Agreement = pearl_gpu::FilledByVote;
#endif

int main(int, char** argv) {
    const unsigned seed = std::atoi(argv[1]);
    // a tile is uniform as a whole, at a few threads, or nowhere
    std::vector<std::vector<char>> same(kTiles, std::vector<char>(kThreads, 0));
    std::srand(seed);
    for (auto& tile : same) {
        const int kind = std::rand() % 8;
        for (auto& s : tile) s = kind == 0 ? 1 : kind < 5 ? std::rand() % 2 : 0;
    }
    std::vector<std::atomic<int>> votes(kTiles);
    std::barrier<> end(kThreads);
    std::atomic<int> taken{0}, wrong{0}, filled{0};
    std::vector<std::thread> block;
    for (int id = 0; id < kThreads; ++id)
        block.emplace_back([&, id] {
            Agreement a;
            for (int t = 0; t < kTiles; ++t) {
                const bool s = same[t][id];
                if (a.takes(s)) {
                    ++taken;
                    for (double q : U.q) wrong += q != 0.25;
                } else if (a.fills(s, id == 0)) {
                    ++filled;
                    for (double& q : U.q) q = 0.25;
                    U.flag = 1;
                }
                votes[t] += s;
                end.arrive_and_wait();
                a.vote(votes[t] == kThreads);
            }
        });
    for (auto& t : block) t.join();
    std::printf("%d %d %d\n", taken.load(), filled.load(), wrong.load());
    return 0;
}
"""


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    d = tmp_path_factory.mktemp("uniform")
    (d / "probe.cpp").write_text("int main() { return 0; }\n")
    (d / "walk.cpp").write_text(SOURCE)

    def compile_(source, name, *flags):
        subprocess.run(["g++", "-O1", "-g", "-std=c++20", "-fsanitize=thread", f"-I{CSRC}", *flags, str(d / source),
                        "-pthread", "-o", str(d / name)], check=True, capture_output=True)
        return d / name

    try:
        subprocess.run([str(compile_("probe.cpp", "probe"))], check=True, capture_output=True)
    except (subprocess.CalledProcessError, OSError):
        pytest.skip("ThreadSanitizer does not run here")
    return compile_


@pytest.mark.parametrize("seed", range(4))
def test_votes_order_every_access(build, seed):
    r = subprocess.run([str(build("walk.cpp", "walk")), str(seed)], capture_output=True, text=True)
    assert r.returncode == 0 and "data race" not in r.stderr, r.stderr[:3000]
    taken, filled, wrong = map(int, r.stdout.split())
    assert taken > 100 and filled >= 1 and wrong == 0


def test_a_flag_read_after_the_vote_is_a_race(build):
    r = subprocess.run([str(build("walk.cpp", "late", "-DLATE_FLAG")), "0"], capture_output=True, text=True)
    assert "data race" in r.stderr
