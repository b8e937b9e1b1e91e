// seq_exchange.h -- one thread's progress through the exchanges of a sequential
// pass on a cluster (seq_kernel.cuh).  Plain C++, so that the rules below can
// be run against a model of the barriers on the host
// (tests/seq_exchange_model.cpp).
//
// Each exchange is one phase of the receiver's mbarrier: armed once with the
// bytes it expects, completed when the senders' pushes have counted them off.
// A wait is bounded.  A thread whose wait gave up neither waits nor arms nor
// pushes again; it walks on through the rest of the pass, whose CTA and cluster
// barriers the others need it at (each thread gives up on its own clock, so
// none may leave the loops alone).  A row task's bytes are part of every CTA's
// column exchange and a column task's of one CTA's row exchange, so without them
// that exchange and, through the threads that then give up, all later ones
// stay incomplete: no barrier gets more than two exchanges' bytes beyond what it
// was armed for, at most 64 KB of the 2^20 - 1 its transaction count holds.  (Were
// pushes to go on, an unarmed barrier would pass that after 32 exchanges of 32 KB.)
#pragma once

#ifdef __CUDACC__
#define MSET_HD __host__ __device__ __forceinline__
#else
#define MSET_HD inline
#endif

namespace mset {

struct SeqProgress {
    unsigned ph[2] = {0, 0};  // exchanges waited for: rows, columns
    bool dead = false;        // a wait gave up

    MSET_HD bool waits() const { return !dead; }
    MSET_HD bool sends() const { return !dead; }
    MSET_HD bool arms() const { return !dead; }
    // parity of the phase the next wait on `which` is for
    MSET_HD unsigned parity(int which) const { return ph[which] & 1u; }
    MSET_HD void waited(int which, bool completed) {
        if (!completed) dead = true;
        ++ph[which];
    }
};

}  // namespace mset
