// Host-only replay of how a face tile's threads leave the TMA-staged kernels
// after a wait that ran out (no GPU needed): threads, mbarriers and bulk copies
// as a state machine in which copies land as late as they can, waits give up in
// any set of threads at any plane, and the next step is taken by a random
// thread.  No thread may be gone while a bulk copy that it issued is in
// flight.  Prints "OK <runs>", or the first violation.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>
#include "../multiphaselb_b200/csrc/tma_util.cuh"

using namespace mplb;

constexpr int NT = 4, NSTAGE = 2;

struct Bar {
    int count = NT, arrived = 0, tx = 0, phase = 0;
    void check() {
        if (arrived == count && tx == 0) { phase++; arrived = 0; }
    }
    bool done(uint32_t parity) const { return (uint32_t)(phase & 1) != parity; }
};

struct Op { bool arrive; int s; uint32_t parity; };

enum At { START, FACE, PSI, PSI_WAIT, LEAVE, GONE };

struct Thread {
    At at = START;
    int j = 0;
    uint32_t fparity = 0;
    bool landed = true;
    std::vector<Op> ops;  // of leave_face_tile, to be run
    size_t op = 0;
    std::vector<int> copies;  // stages of its bulk copies in flight
};

// One run: threads of `face_mask` (`psi_mask`) give up their wait for wrapped
// parts (psi) at plane `plane`; drain: as the kernels do, or not at all.
static bool run(int planes, int plane, int face_mask, int psi_mask, bool drain, uint32_t seed) {
    std::mt19937 rng(seed);
    Bar face[NSTAGE], psi;
    std::vector<Thread> th(NT);
    bool s_fail = false, ok = true;
    auto patch = [&](Thread& t, int s) {  // every thread issues a bulk copy and arrives
        face[s].tx++;
        t.copies.push_back(s);
        face[s].arrived++;
        face[s].check();
    };
    auto leave = [&](Thread& t) {
        s_fail = true;
        t.at = LEAVE;
        if (drain)
            leave_face_tile(t.j, NSTAGE, t.fparity, t.j + 1 < planes, [&](int s) { t.ops.push_back({true, s, 0}); },
                            [&](int s, uint32_t par) { t.ops.push_back({false, s, par}); });
    };
    // one step of thread i if it can take one; `out`: its wait's limit is reached
    auto step = [&](int i, bool out) -> bool {
        Thread& t = th[i];
        const int s = t.j % NSTAGE;
        switch (t.at) {
        case START:
            patch(t, 0);
            t.at = FACE;
            return true;
        case FACE: {
            const bool give_up = t.j == plane && ((face_mask >> i) & 1);
            if (!give_up && !out && !face[s].done((t.fparity >> s) & 1u)) return false;
            t.landed = !give_up && !out;
            t.fparity ^= 1u << s;
            t.at = PSI;
            return true;
        }
        case PSI:
            if (!t.landed) s_fail = true;
            psi.arrived++;
            psi.check();
            t.at = PSI_WAIT;
            return true;
        case PSI_WAIT: {
            const bool give_up = t.j == plane && ((psi_mask >> i) & 1);
            if (!give_up && !out && !psi.done((uint32_t)t.j & 1u)) return false;
            if (give_up || out || s_fail) {
                leave(t);
                return true;
            }
            if (t.j + 1 < planes) patch(t, (t.j + 1) % NSTAGE);
            t.j++;
            t.at = t.j < planes ? FACE : GONE;
            return true;
        }
        case LEAVE:
            if (t.op == t.ops.size()) {
                if (!t.copies.empty()) ok = false;
                t.at = GONE;
                return true;
            }
            if (t.ops[t.op].arrive) {
                face[t.ops[t.op].s].arrived++;
                face[t.ops[t.op].s].check();
            } else if (!out && !face[t.ops[t.op].s].done(t.ops[t.op].parity)) {
                return false;
            }
            t.op++;
            return true;
        default: return false;
        }
    };
    for (int guard = 0; guard < 100000; guard++) {
        std::vector<int> order = {0, 1, 2, 3};
        std::shuffle(order.begin(), order.end(), rng);
        bool moved = false, left = false;
        for (int i : order) {
            left |= th[i].at != GONE;
            if (!moved) moved = step(i, false);
        }
        if (!left) return ok;
        if (moved) continue;
        // nobody can move: the copies land; without copies, a limit is reached
        bool landed = false;
        for (Thread& t : th) {
            for (int s : t.copies) { face[s].tx--; face[s].check(); landed = true; }
            t.copies.clear();
        }
        for (size_t i = 0; !landed && i < order.size(); i++)
            if (th[order[i]].at != GONE) { step(order[i], true); break; }
    }
    return false;  // never ended
}

int main() {
    int runs = 0, bad = 0, control = 0;
    for (int planes : {2, 3, 6})
        for (int plane = 0; plane < planes; plane++)
            for (int fm = 0; fm < 1 << NT; fm++)
                for (int pm = 0; pm < 1 << NT; pm++)
                    for (uint32_t seed = 0; seed < 4; seed++, runs++) {
                        if (!run(planes, plane, fm, pm, true, seed) && bad++ < 5)
                            printf("FAIL planes %d plane %d masks %x %x seed %u\n", planes, plane, fm, pm, seed);
                        control += !run(planes, plane, fm, pm, false, seed);
                    }
    if (!control) { printf("FAILED: the replay sees no copy in flight without leave_face_tile\n"); return 1; }
    if (bad) { printf("FAILED %d runs\n", bad); return 1; }
    printf("OK %d\n", runs);
    return 0;
}
