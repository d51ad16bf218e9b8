// The bounded drain of a ring of TMA loads after a wait ran out (spk_ring.cuh),
// on the host: a model of the stages' barriers for a walk of `ntiles` tiles
// whose wait for tile `fail` runs out.  Argument "line": the remaining tiles
// are walked without loading, and the loads that went out are counted (k_line);
// "axis": the walk ends at once (k_axis2).
// Prints the number of loads still in flight after the drain, and of waits
// for a load that never went out, summed over all cases: both must be 0.
#include <cstdio>
#include <cstring>
#include <vector>

#include "spk_ring.cuh"

struct Ring {
    int nst, issued = 0;
    std::vector<int> last;      // last load of each stage, -1: none
    std::vector<char> waited;   // by load
    Ring(int n, int ntiles) : nst(n), last(n, -1), waited(ntiles, 0) {}
    void issue(int j, int stage) { last[stage] = j; issued++; }
    // a wait that lasts until the stage's phase of this parity completes: it
    // covers the stage's last load only if the parity is that load's
    bool wait(int stage, unsigned parity) {
        const int j = last[stage];
        if (j < 0 || ((unsigned)(j / nst) & 1u) != parity) return false;
        waited[j] = 1;
        return true;
    }
    int in_flight() const {
        int n = 0;
        for (int j = 0; j < issued; j++) n += !waited[j];
        return n;
    }
};

int main(int argc, char** argv) {
    const bool line = argc > 1 && std::strcmp(argv[1], "line") == 0;
    int left = 0, idle = 0;
    for (int nst = line ? 2 : 1; nst <= 4; nst++)
        for (int ntiles = 1; ntiles <= 11; ntiles++)
            for (int fail = 0; fail < ntiles; fail++) {
                Ring r(nst, ntiles);
                for (int s = 0; s < nst && s < ntiles; s++) r.issue(s, s);
                for (int it = 0; it < fail; it++) {
                    r.waited[it] = 1;
                    // k_line refills the previous tile's stage, k_axis2 this one's
                    const int tn = line ? it + nst - 1 : it + nst;
                    if (tn < ntiles && (!line || it > 0)) r.issue(tn, tn % nst);
                }
                if (line) {
                    for (int j = spk::ring_first_pending(r.issued, nst); j < r.issued; j++)
                        idle += !r.wait(spk::ring_stage(j, nst), spk::ring_parity(j, nst));
                } else {
                    // the loads issued by tile `fail`: up to nst ahead, as far as there are tiles
                    for (int j = fail; j < fail + nst && j < ntiles; j++)
                        idle += !r.wait(spk::ring_stage(j, nst), spk::ring_parity(j, nst));
                }
                left += r.in_flight();
            }
    printf("in_flight %d\nidle_waits %d\n", left, idle);
    return 0;
}
