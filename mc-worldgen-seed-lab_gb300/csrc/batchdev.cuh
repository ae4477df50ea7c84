/* batchdev.cuh -- device helpers shared by the persistent batch kernels (batch.cu, owtile.cu). */
#ifndef MG_BATCHDEV_CUH
#define MG_BATCHDEV_CUH
#include "batch.h"

namespace mg {

/* a biome id to the output: written once and never read back by the kernel, so stored with the streaming
 * (evict-first) policy, which keeps the streamed output from evicting the threads' local memory from L2 */
__device__ __forceinline__ void put_id(uint8_t *p, int v) { __stcs(p, (unsigned char)v); }

/* The request holding tile `tile`: the last r with reqs[r].tile0 <= tile (tile0 is non-decreasing and
 * reqs[0].tile0 == 0), found by the 32 lanes of a warp in rounds of 32 probes -- the probes that are <= tile
 * form a prefix, whose length narrows the range 32-fold -- so 3 rounds of loads for 10,000 requests where a
 * binary search by one thread made 14 dependent ones while the CTA waited. */
__device__ __forceinline__ int find_req(const MgBatchReq *__restrict__ reqs, int nreq, long long tile) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = nreq - 1;
    while (hi > lo) {
        const int step = (hi - lo + 31) / 32;
        const int p = lo + (lane + 1) * step;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, p <= hi && reqs[p].tile0 <= tile);
        lo += __popc(m) * step;
        hi = min(hi, lo + step - 1);
    }
    return lo;
}

}  // namespace mg
#endif
