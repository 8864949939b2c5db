"""CPU check of the run kernel's buffer ring (csrc/ring.hpp): every wait is on the phase
of the use it means.  A model of the barriers (phases, a try_wait by parity) runs all
stages; copies of the stages from `lost` on never land by themselves.  The warp then
waits, per buffer, for the last stage copied into it, and may leave only when that
copy has landed: a wait on a fixed parity lets it leave early (the model shows that
too), with a copy still on its way into shared memory that is given back."""
import os
import subprocess

from conftest import REPO

SRC = r"""
#include "ring.hpp"
#include <cstdio>
#include <vector>
template <int N> int check()
{
    using R = raft::Ring<N>;
    int early_fixed = 0;
    for (int nst = 1; nst <= 6 * N + 1; nst++)
        for (int lost = 0; lost <= nst; lost++) {
            std::vector<unsigned> done(N, 0);            // completed phases per buffer
            std::vector<int> armed(N, -1);
            auto try_wait = [&](int b, unsigned parity) { return ((done[b] - 1) & 1u) == (parity & 1u); };
            for (int s = 0; s < nst; s++) {
                const int b = R::buffer(s);
                if (R::reused(s)) {                      // the stage before it in this buffer has landed and is summed
                    if (R::before(s) != armed[b]) return 1;
                    if (R::before(s) >= lost) break;     // its wait ran out: no further copies
                } else if (armed[b] != -1) return 2;
                if (try_wait(b, R::parity(s))) return 3; // the copy is only being issued
                armed[b] = s;
                if (s < lost) {
                    done[b]++;                           // it lands
                    if (!try_wait(b, R::parity(s))) return 4;
                }
            }
            for (int b = 0; b < N; b++) {                // the drain
                if (armed[b] < 0) continue;
                const bool flight = armed[b] >= lost;
                if (flight && try_wait(b, 1)) early_fixed++;
                if (try_wait(b, R::parity(armed[b])) == flight) return 5;
                if (flight) {
                    done[b]++;
                    if (!try_wait(b, R::parity(armed[b]))) return 6;
                }
            }
        }
    return early_fixed > 0 ? 0 : 7;
}
int main()
{
    const int r[] = {check<2>(), check<3>(), check<4>()};
    printf("%d %d %d\n", r[0], r[1], r[2]);
    return r[0] || r[1] || r[2];
}
"""


def test_waits_are_on_the_phase_they_mean(tmp_path):
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-I", os.path.join(REPO, "ssc-raft_b200", "csrc"), str(src), "-o",
                           str(exe)])
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.split() == ["0", "0", "0"]


def test_the_kernel_uses_the_ring():
    with open(os.path.join(REPO, "ssc-raft_b200", "csrc", "bp_run.cuh")) as f:
        kernel = f.read()
    # waits and the drain take their parity from the ring
    assert kernel.count("Stages::parity(") == 3 and "mbar_wait_bounded(&full[i], 1," not in kernel
