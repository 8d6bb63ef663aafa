"""The walk of an epilogue team over its tiles (csrc/team_walk.hpp, used by the
Adam kernel) with host threads in the place of a team's threads: a wait that
gives up in some of them and not in the others -- in any tile, whether or not
the team has a chunk of it -- ends the walk of all of them at the same tile,
and none is left behind at a barrier that the others never reach.
"""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "team_walk.hpp"

constexpr int kThreads = 4, kTiles = 5, kTeams = 3;

// all_good: every thread waits for all; a barrier that is not met in time
// ends the program.
struct Agreement {
    std::mutex m;
    std::condition_variable cv;
    int in = 0, round = 0;
    bool all = true, result = true;
    bool operator()(bool ok) {
        std::unique_lock<std::mutex> lock(m);
        all = all && ok;
        const int mine = round;
        if (++in == kThreads) {
            result = all;
            all = true;
            in = 0;
            ++round;
            cv.notify_all();
        } else if (!cv.wait_for(lock, std::chrono::seconds(5), [&] { return round != mine; })) {
            std::puts("left at a barrier");
            std::exit(1);
        }
        return result;
    }
};

int main() {
    int runs = 0;
    for (int chunks = 0; chunks <= 2; ++chunks)
        for (int team = 0; team < kTeams; ++team)
            for (int at = 0; at < kTiles; ++at)
                for (int on_chunk = 0; on_chunk < 2; ++on_chunk)
                    for (int failing = 0; failing < 1 << kThreads; ++failing) {
                        Agreement agreement;
                        std::vector<int> result(kThreads), left(kThreads), worked(kThreads);
                        std::vector<std::thread> threads;
                        for (int t = 0; t < kThreads; ++t)
                            threads.emplace_back([&, t] {
                                const bool fails = (failing >> t) & 1;
                                auto count = [&](int) { return chunks; };
                                auto wait_tile = [&](int k) { return on_chunk || k != at || !fails; };
                                auto wait_chunk = [&](int i) { return !on_chunk || i != at || !fails; };
                                auto agree = [&](bool ok) { return agreement(ok); };
                                auto work = [&](int, int) { ++worked[t]; };
                                auto leave = [&](int) { ++left[t]; };
                                result[t] = pdlpgpu_mlp_impl::team_walk(0, 1, kTiles, team, kTeams, count, wait_tile,
                                                                        wait_chunk, agree, work, leave);
                            });
                        for (std::thread& t : threads) t.join();
                        // Without a failure every tile and every third chunk; else all stop together.
                        int mine = 0;
                        for (int n = 0; n < kTiles * chunks; ++n) mine += n % kTeams == team;
                        const bool met = failing != 0 && (on_chunk ? at < mine : true);
                        for (int t = 0; t < kThreads; ++t) {
                            const bool ok = result[t] == !met && left[t] == left[0] && worked[t] == worked[0] &&
                                            (met ? left[t] <= kTiles : left[t] == kTiles && worked[t] == mine) &&
                                            (!met || on_chunk || left[t] == at + 1);
                            if (!ok) {
                                std::printf("chunks %d team %d at %d on_chunk %d failing %d\n", chunks, team, at,
                                            on_chunk, failing);
                                return 1;
                            }
                        }
                        ++runs;
                    }
    std::printf("%d walks\n", runs);
    return 0;
}
"""


def test_a_wait_that_gives_up_in_some_threads_ends_the_walk_of_all(tmp_path):
    source, program = tmp_path / "walk.cpp", tmp_path / "walk"
    source.write_text(SOURCE)
    include = os.path.join(ROOT, "optimisation_solver_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-Wall", "-Werror", "-I", include, str(source), "-o",
                    str(program)], check=True)
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
    assert run.stdout == f"{3 * 3 * 5 * 2 * 16} walks\n"
