"""The word of the grid barrier (rift_bar.cuh) on the CPU: CTAs arrive in any
order, some raise an event, and each polls as early or as late as it can.  None
may leave before the last has arrived, and all count the same events."""
import os
import subprocess

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "rift_bar.cuh"
using namespace rift;

// Two barriers a step: events are raised at the first only.  `start`: arrivals so far
// (the counter's wrap).
int play(int n, int raisers, unsigned start, unsigned seed) {
    std::mt19937 g(seed);
    unsigned word = start;
    std::vector<unsigned> target(n, start);
    std::vector<int> at(n, 0), in(n, 0);  // barriers passed; arrived at the next one
    std::vector<int> arrived(9, 0), raisedAt(9, 0);
    for (int b = 0; b < 8; b += 2) raisedAt[b] = (int)(g() % (raisers + 1));
    std::vector<int> raised(9, 0);
    for (int done = 0; done < n;) {
        const int c = (int)(g() % n);
        if (at[c] == 8) continue;
        const int b = at[c];
        if (!in[c]) {  // any CTA among the first raisedAt[b] arrivals raises
            const bool raise = raised[b] < raisedAt[b];
            raised[b] += raise;
            target[c] += n;
            word += barArrival(raise);
            arrived[b]++;
            in[c] = 1;
        } else if (barPassed(word, target[c])) {
            if (arrived[b] != n) return printf("left early: barrier %d, %d of %d\n", b, arrived[b], n), 1;
            if (b % 2 == 0) {
                const unsigned k = barEvents(word, target[c]);
                if ((int)k != raised[b]) return printf("events\n"), 1;
                target[c] = barSeen(target[c], k);
            }
            in[c] = 0;
            if (++at[c] == 8) done++;
        }
    }
    return 0;
}
int main() {
    for (unsigned seed = 0; seed < 300; seed++)
        for (int n : {1, 2, 7, 40})
            for (int r : {0, 1, n})
                for (unsigned start : {0u, 0xffffffffu - 3u * n, 0x7fffffffu - n, 0xffffu - 3u * n})
                    if (play(n, r, start, seed)) return 1;
    return 0;
}
"""


def test_no_one_leaves_early_and_all_count_the_same(tmp_path):
    (tmp_path / "bar.cpp").write_text(SRC)
    csrc = os.path.join(os.path.dirname(__file__), "..", "rift_gb300", "csrc")
    exe = str(tmp_path / "bar")
    subprocess.run(["g++", "-O1", "-x", "c++", "-I", csrc, str(tmp_path / "bar.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
