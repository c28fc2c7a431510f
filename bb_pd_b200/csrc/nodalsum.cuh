// Per-node sums of bond forces in bond order, by warps.
//
// A node's list holds its bond ends in bond order: entry v = 2 k + side of bond
// k (side 0: +force, side 1: -force); with CHUNKS its top bit is set where a new
// OpenMP chunk begins after the first entry. A thread per node walked its list alone: 122
// dependent steps on a few warps, every load of its own sector. Here a warp
// takes 4 neighbouring nodes: a load instruction reads 8 consecutive entries of
// each list, so that it meets the bonds a node starts, which lie in a row, and
// the bonds of one other node to several of the four, which lie in a row too (32
// entries of one list at a time had every lane of the latter in a line of its
// own: 130 against 109 us). The forces go to shared memory, and 12 lanes, one per node
// and component, add 32 entries one after the other. What bounds it: the L1 lookups
// of the gathers at millions of bonds; the chain of additions and two round trips
// to L2 per 32 entries at thousands.
#pragma once

namespace bbpd {

constexpr int kNodes = 4;   // nodes of a warp (8 lanes load for each)

struct NodeSumShared {
    double f[kNodes][3][33];   // one column more than entries: no bank conflicts across rows
};

// t and a of lane l < 3 kNodes (node n0 + l / 3, component l % 3): on return the
// finished chunks have been added to t, and a holds the last chunk's sum. The
// caller sets t beforehand and adds a where the list is not empty. off[] has
// nN + 1 entries.
template <bool CHUNKS, class ENT>
__device__ __forceinline__ void warp_node_sums(const int64_t *__restrict__ off, const ENT *__restrict__ ent, int64_t n0,
                                               int64_t nN, const double *__restrict__ fX, const double *__restrict__ fY,
                                               const double *__restrict__ fZ, NodeSumShared &sm, double &t, double &a)
{
    constexpr ENT kFlag = CHUNKS ? (ENT)1 << (8 * sizeof(ENT) - 1) : (ENT)0;
    const int lane = threadIdx.x & 31;
    const int q = lane & (kNodes - 1), jq = lane / kNodes;   // this lane loads entries jq, jq + 8, ... of node q
    const int64_t p0 = n0 + q < nN ? off[n0 + q] : 0, p1 = n0 + q < nN ? off[n0 + q + 1] : 0;
    int64_t longest = p1 - p0;
    longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, 1));
    longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, 2));
    const int mq = min(lane / 3, kNodes - 1), mc = lane % 3;   // lanes below 12: the node and component they add
    a = 0.0;
    for (int64_t b = 0; b < longest; b += 32) {
        ENT v[4];
        double f[4][3];
        unsigned flags = 0;   // chunk starts of node mq
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const int64_t p = p0 + b + 8 * s + jq;
            v[s] = p < p1 ? ent[p] : (ENT)0;
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const bool in = p0 + b + 8 * s + jq < p1;
            const int64_t k = (int64_t)((v[s] & ~kFlag) >> 1);
            // an absent entry adds -0, which leaves every sum as it is
            f[s][0] = in ? fX[k] : -0.0;
            f[s][1] = in ? fY[k] : -0.0;
            f[s][2] = in ? fZ[k] : -0.0;
            if (CHUNKS) {
                const unsigned m = __ballot_sync(0xffffffffu, in && (v[s] & kFlag));
                if (m)
                    for (int j = 0; j < 8; j++) flags |= ((m >> (kNodes * j + mq)) & 1u) << (8 * s + j);
            }
        }
#pragma unroll
        for (int s = 0; s < 4; s++)
#pragma unroll
            for (int c = 0; c < 3; c++) sm.f[q][c][8 * s + jq] = (v[s] & 1) ? -f[s][c] : f[s][c];
        __syncwarp();
        if (lane < 3 * kNodes) {
            const double *row = sm.f[mq][mc];
            double x[8];
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
#pragma unroll
                for (int k = 0; k < 8; k++) x[k] = row[j + k];
                if (CHUNKS && ((flags >> j) & 0xFFu)) {
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        if (flags & (1u << (j + k))) {   // partial of the previous OpenMP thread is complete
                            t = t + a;
                            a = 0.0;
                        }
                        a = a + x[k];
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 8; k++) a = a + x[k];
                }
            }
        }
        __syncwarp();
    }
}

}  // namespace bbpd
