// comb_roles.cuh — the two roles of a k_comb256 block (k_encrypt.cu) that only
// start asynchronous work: the thread that loads table rows into three buffers
// in turn, and the threads that issue a warpgroup's products.  What they wait
// for and start is the caller's, so that the host tests run them against waits
// that run out.
//
// The shared and the tensor memory of a block are another block's as soon as
// it ends.  So a role returns only when what it started is done: a copy into a
// buffer has landed, a product has read its buffer and written its columns,
// and the arrival that tells of it has been made.  That holds where a wait ran
// out, too (each of the last waits has the limit of any other).
#pragma once
#include "fe.cuh"

static constexpr unsigned COMB_BUFS = 3;

// Loads `steps` rows: load(b) starts the next row's copy into buffer b.
// wait_full(b, parity) waits for a copy into b to land, wait_empty(b, parity)
// for the products that read it.  False: a wait ran out.
template <class WaitFull, class WaitEmpty, class Load>
FT_DEV bool comb_load(unsigned steps, WaitFull wait_full, WaitEmpty wait_empty, Load load)
{
    bool ok = true;
    unsigned k = 0, buf = 0, use = 0; // step k is the use-th of buffer buf
#pragma unroll 1
    for (; k < steps; ++k) {
        if (use && !wait_empty(buf, (use - 1) & 1)) {
            ok = false;
            break;
        }
        load(buf);
        if (++buf == COMB_BUFS) {
            buf = 0;
            ++use;
        }
    }
#pragma unroll 1
    for (unsigned j = k < COMB_BUFS ? 0 : k - COMB_BUFS; j < k; ++j)
        if (!wait_full(j % COMB_BUFS, j / COMB_BUFS & 1)) ok = false;
    // (without a product that does not come there is nothing to wait for here)
#pragma unroll 1
    for (unsigned j = k < COMB_BUFS ? 0 : k - COMB_BUFS; ok && j < k; ++j)
        if (!wait_empty(j % COMB_BUFS, j / COMB_BUFS & 1)) ok = false;
    return ok;
}

// Issues `steps` products: issue(b) starts that of the row in buffer b, which
// completes a phase of `done`.  wait_ready(parity) waits for the warpgroup's
// one-hot rows.  False: a wait ran out.
template <class WaitFull, class WaitReady, class WaitDone, class Issue>
FT_DEV bool comb_issue(unsigned steps, WaitFull wait_full, WaitReady wait_ready, WaitDone wait_done, Issue issue)
{
    bool ok = true;
    unsigned q = 0, buf = 0, use = 0;
#pragma unroll 1
    for (; q < steps; ++q) {
        if (!wait_full(buf, use & 1) || !wait_ready(q & 1)) {
            ok = false;
            break;
        }
        issue(buf);
        if (++buf == COMB_BUFS) {
            buf = 0;
            ++use;
        }
    }
    if (q && !wait_done((q - 1) & 1)) ok = false;
    return ok;
}
