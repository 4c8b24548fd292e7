/*
 * run_ctl.h -- control state of a shared-step simulation's run kernels
 * (shared_run.cuh), and how a launch reports it.  Plain C++ without CUDA, for
 * the test.
 */
#ifndef ASSIST_GB300_RUN_CTL_H
#define ASSIST_GB300_RUN_CTL_H

#include "ieee_convert.cuh"

struct ShCtl {
    double t, tc, dt, dtls, dt_done;
    long long accepted, rejected, iterations;
    int status;
};

/* Device memory of a simulation's run kernel. */
struct ShRunMem {
    ShCtl ctl[2];                /* a launch reads one and writes the other */
    /* from here on zero at launch */
    unsigned long long red[9];   /* three rotating buffers of the maxima */
    unsigned bar[2];             /* grid barrier: arrivals, generation */
    unsigned gave_up;            /* a block stopped waiting at the barrier */
};

/* A block's last word: block 0 has the state that every block has, and a block
 * that stopped waiting says so in a word that nothing else writes (in the
 * state's own struct block 0's store could overwrite it). */
AG_HD void sh_run_report(const ShCtl& K, bool gave_up, int block, ShCtl* out, unsigned* word) {
    if (block == 0) *out = K;
    if (gave_up) *word = 1u;
}

#endif
