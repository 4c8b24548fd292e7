/*
 * batch_ws.h -- the global workspace of a batch that runs on two kernels at
 * once: the region of the groups with a deep pass behind the others', whatever
 * kernel builds take them (ag_k_coop's learned and variational builds keep the
 * groups' state there, the rest in shared memory).  Plain C++, for the test.
 */
#ifndef ASSIST_GB300_BATCH_WS_H
#define ASSIST_GB300_BATCH_WS_H

#include <cstddef>

struct AgBatchWs {
    size_t deep_at, total;       /* doubles */
};

/* per: doubles a slot (a particle's place in a resident block). */
inline AgBatchWs ag_batch_ws(size_t per, int slots, int deep_slots) {
    return {per * (size_t)slots, per * ((size_t)slots + (size_t)deep_slots)};
}

#endif
