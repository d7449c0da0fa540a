// comb_roles_host.cpp — host build of the asynchronous roles of k_comb256
// (comb_roles.cuh) over barriers that say a wait was for nothing, would not
// have waited, or ran out, for tests/test_comb_roles_host.py.  TEST HARNESS
// ONLY.
#include "../../libftcrypto_gb300/csrc/comb_roles.cuh"

// an mbarrier as its waiter sees it, phases completed only when waited for
struct Bar {
    unsigned phases = 0; // completed
    // waits for the phase after those completed; *wrong if the parity is that
    // of an earlier one (the wait would return at once)
    bool wait(unsigned parity, bool *wrong)
    {
        if (parity != (phases & 1)) *wrong = true;
        ++phases;
        return true;
    }
};

enum { OK = 1, WRONG = 2, IN_FLIGHT = 4 };

extern "C" {

// comb_load of `steps` rows, its fail-th wait running out (0: none).  Bits:
// OK as returned, WRONG a parity or a buffer that was not waited for,
// IN_FLIGHT a copy that may still land (or, with OK, a product that may still
// read or arrive) afterwards
int hr_load(unsigned steps, unsigned fail)
{
    Bar full[COMB_BUFS], empty[COMB_BUFS];
    unsigned loads[COMB_BUFS] = {}, waits = 0;
    bool wrong = false;
    const bool ok = comb_load(
        steps, [&](unsigned b, unsigned p) { return ++waits != fail && full[b].wait(p, &wrong); },
        [&](unsigned b, unsigned p) {
            if (++waits == fail) return false;
            empty[b].wait(p, &wrong);
            if (full[b].phases < empty[b].phases) full[b].phases = empty[b].phases; // what was read had landed
            return true;
        },
        [&](unsigned b) {
            if (loads[b] > empty[b].phases) wrong = true; // not free yet
            ++loads[b];
        });
    bool flying = false;
    unsigned total = 0;
    for (unsigned b = 0; b < COMB_BUFS; ++b) {
        total += loads[b];
        if (full[b].phases < loads[b] || (ok && empty[b].phases < loads[b])) flying = true;
    }
    if (ok && total != steps) wrong = true;
    return (ok ? OK : 0) | (wrong ? WRONG : 0) | (flying ? IN_FLIGHT : 0);
}

// comb_issue of `steps` products likewise (IN_FLIGHT: a product not waited for)
int hr_issue(unsigned steps, unsigned fail)
{
    Bar full[COMB_BUFS], ready;
    unsigned waits = 0, issued = 0, done = 0;
    bool wrong = false;
    const bool ok = comb_issue(
        steps, [&](unsigned b, unsigned p) { return ++waits != fail && full[b].wait(p, &wrong); },
        [&](unsigned p) { return ++waits != fail && ready.wait(p, &wrong); },
        [&](unsigned p) {
            if (++waits == fail) return false;
            if (p != ((issued - 1) & 1)) wrong = true; // not the last product's phase
            done = issued;
            return true;
        },
        [&](unsigned b) {
            if (full[b].phases != issued / COMB_BUFS + 1 || b != issued % COMB_BUFS) wrong = true;
            ++issued;
        });
    if (ok && issued != steps) wrong = true;
    return (ok ? OK : 0) | (wrong ? WRONG : 0) | (done != issued ? IN_FLIGHT : 0);
}

} // extern "C"
