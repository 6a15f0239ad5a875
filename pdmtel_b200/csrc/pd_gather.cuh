// The MLS gather of the 2x2x2 rule with eight lanes per node, a lane per Gauss
// point, shared by the FP64 and the FP32 form.
//
// A node's contributors are taken in chunks of eight.  The coefficients of the
// chunks ahead are on their way to a shared-memory ring (cp.async, zero-filled
// past the list's end); each lane gathers the displacement of one contributor
// of the next chunk, with its id loaded a chunk earlier still, and leaves it in
// shared memory for the group.  A lane then adds its point's terms contributor
// by contributor, in the order of the list.  One thread per point (FP64) or per
// four points (FP32) gathered every contributor's displacement itself and
// waited on the id -> displacement chain of each batch of four.
//
// sum(c, v) is called for every contributor of the lane's node, in order, with
// its coefficient c at the lane's point and the triple v that fetch(id, v) gave.
#pragma once

#include "pd_internal.cuh"

namespace pd {

constexpr int kGatherChunk = 8;

// Coefficients and triples of a node's chunk with padding, so that the four
// nodes of a warp read different banks.
constexpr int kRingRow = kGatherChunk * 8 + 8, kTripRow = kGatherChunk * 3 + 4;
// shared bytes per warp: the ring of coefficients [stages][4 nodes] and two
// buffers of triples [4 nodes]
template <typename C>
__host__ __device__ constexpr int gather_warp_bytes(int stages) {
    return stages * 4 * kRingRow * (int)sizeof(C) + 2 * 4 * kTripRow * (int)sizeof(double);
}

template <typename C, int STAGES, typename Fetch, typename Sum>
__device__ __forceinline__ void gather_chunks(char* warp_sm, const C* __restrict__ coef, const int32_t* __restrict__ ids,
                                              int nc, const Fetch& fetch, const Sum& sum) {
    constexpr int kPieces = kGatherChunk * 8 * (int)sizeof(C) / 16 / 8;  // 16-byte copies per lane and chunk
    constexpr int kPer = 8 * (int)sizeof(C) / 16;                        // 16-byte pieces per contributor
    const int lane = threadIdx.x & 31, g = lane & 7, grp = lane >> 3;
    C* ring = reinterpret_cast<C*>(warp_sm);
    double* trip = reinterpret_cast<double*>(warp_sm + STAGES * 4 * kRingRow * sizeof(C)) + grp * kTripRow;
    const int most = __reduce_max_sync(0xffffffffu, nc);
    const int chunks = (most + kGatherChunk - 1) / kGatherChunk;
    auto copy = [&](int c) {  // the coefficients of chunk c
        if (c < chunks) {
            char* to = reinterpret_cast<char*>(ring + ((c % STAGES) * 4 + grp) * kRingRow);
            const char* from = reinterpret_cast<const char*>(coef) + (int64_t)c * kGatherChunk * 8 * sizeof(C);
#pragma unroll
            for (int p = 0; p < kPieces; ++p) {
                const int piece = 8 * p + g;
                const bool in = c * kGatherChunk + piece / kPer < nc;
                const unsigned sa = (unsigned)__cvta_generic_to_shared(to + 16 * piece);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa),
                             "l"(in ? from + 16 * piece : reinterpret_cast<const char*>(coef)), "r"(in ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto id = [&](int c) {
        const int k = c * kGatherChunk + g;
        return k < nc ? __ldg(ids + k) : -1;
    };
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) copy(c);
    double v[3] = {0.0, 0.0, 0.0};
    int m = id(0);
    if (m >= 0) fetch(m, v);
    m = id(1);
    for (int c = 0; c < chunks; ++c) {
        copy(c + STAGES - 1);
        double* t = trip + (c & 1) * 4 * kTripRow;
        t[3 * g] = v[0];
        t[3 * g + 1] = v[1];
        t[3 * g + 2] = v[2];
        const int next = id(c + 2);
        if (m >= 0) fetch(m, v);
        m = next;
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        __syncwarp();
        const C* r = ring + ((c % STAGES) * 4 + grp) * kRingRow + g;
        const int k0 = c * kGatherChunk;
        if (k0 + kGatherChunk <= nc) {
#pragma unroll
            for (int k = 0; k < kGatherChunk; ++k) sum(r[8 * k], t + 3 * k);
        } else {
#pragma unroll 1
            for (int k = 0; k < nc - k0; ++k) sum(r[8 * k], t + 3 * k);
        }
        __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace pd
