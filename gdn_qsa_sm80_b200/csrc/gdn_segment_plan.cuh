// How a long sequence is cut into segments that run as independent CTAs of one launch of the chain.
//
// The second level of the reference's scan has the same purpose (csrc/gdn_chunk/gdn_ops.cu:1002-1012,
// gdn_scan_stage1.cu:7-18); here it rests on an exact bound instead of a propagated transfer matrix.  A stretch of tokens
// maps its incoming state by S_out = A S_in + B with A = prod_t exp(g_t)(I - beta_t k_t k_t^T), and
// |I - beta k k^T|_2 <= 1 whenever 0 <= beta |k|^2 <= 2, so |A|_2 <= exp(sum of g).  Once that sum is below -115
// (exp(-115) < 2^-149) the incoming state no longer shows in fp32: the state after the stretch is the same from a zero
// state.  So a segment s >= 1 starts from a ZERO state p chunks before its first chunk, p the shortest stretch ending at
// the boundary whose sum of g is below -115 ("warm-up": its outputs are not formed), and from its first chunk on its state,
// its outputs and its final state are those of the serial run - bit for bit where the decay is strong (a sum of -10 a chunk);
// where the warm-up is a hundred chunks long the two states end a last bit apart and their bf16 copies round differently now and
// then (up to 5e-3 of a chunk's outputs, 120000 random calls, as far as either is from the exact result).
//
// The sums are prefix sums, and a difference of two prefixes has to be the sum of what lies between them whatever lies in front: in
// fp32 a gate of -1e9 (a reset, a mask's fill value) leaves prefixes with a spacing of 64 and more, and a rounding step behind it read
// as "-128, forgotten" where the decay was -2 (errors up to 100 % behind such a boundary).  So they are integers:
// -sum of g in units of 2^-10, rounded towards zero (a boundary counts as forgotten late, never early), and a chunk counts
// 128 at most - one below -115 forgets on its own.  kPlanChunks of them stay below 2^32, and integer sums are exact and monotone,
// which the binary search needs.  A sequence of more chunks is planned in units of several: the smallest number that leaves at most
// kPlanChunks units, each counting 128 at most.
//
// Every CTA of a head makes the same plan from the per-chunk scalars the prepare kernel left: for each number of segments
// g up to the launch's most (a warp each), equal segments first, then segment 0, which has no warm-up, longer by about the
// warm-up; the g with the fewest dependent chunk steps wins, the serial run (g = 1) included.  The prefix sums sit in
// shared memory, so a warm-up is a binary search there (a scan of the scalars in global memory per boundary took
// 3-5 microseconds of every launch, and the number of segments was the host's guess: sequences of fewer than 32 chunks were
// never split).  No host read, no data-dependent launch, no state passed between CTAs.
#pragma once

#include "gdn_common.cuh"

namespace gdn {

struct SegmentPlan {          // in chunks: segment 0 = chunks [0, L0), segment s >= 1 = L1 chunks from L0 + (s - 1) L1 on
    int g, L0, L1;
    int warm[kMaxSegments];    // chunks of warm-up before each segment s >= 1
};

constexpr float kForgetScale = 1024.f, kForgetCap = 128.f;
constexpr unsigned kForget = static_cast<unsigned>(-kForgetLn * kForgetScale);
static_assert(kForgetCap > -kForgetLn && kForgetCap * kForgetScale * kPlanChunks < 4294967296.0, "prefix sums of a whole sequence fit 32 bits");

// Smallest p <= t0 whose chunks [t0 - p, t0) forget (pre: prefix sums, non-decreasing); 0 = none.
__device__ __forceinline__ int forget_stretch(const unsigned* pre, int t0) {
    const unsigned at = pre[t0];
    if (at - pre[0] <= kForget) return 0;
    int lo = 1, hi = t0;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (at - pre[t0 - mid] > kForget) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// One warp: warm-ups of g segments, segment 0 = [0, L0), then L1 chunks each.  Lane s holds segment s's; returns the
// largest, or -1 when a segment has none.
__device__ __forceinline__ int warmups(const unsigned* pre, int NT, int g, int L0, int L1, int lane, int& mine) {
    int w = 0, bad = 0;
    if (lane >= 1 && lane < g) {
        const int t0 = L0 + (lane - 1) * L1;
        if (t0 < NT) {
            w = forget_stretch(pre, t0);
            bad = w == 0;
        }
    }
    mine = w;
    if (__any_sync(0xffffffffu, bad)) return -1;
    return __reduce_max_sync(0xffffffffu, w);
}

// All threads of the CTA: the split of this head (plan.g = 1: serial), `chunks` of them.  `pre`: kPlanChunks + 1 words of shared memory.
template <int THREADS>
__device__ __forceinline__ void plan_segments(const float* meta, int chunks, int G, unsigned* pre, SegmentPlan& plan, int* best) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int unit = 1, NT = chunks, bad = 0;   // chunks of a unit; units
    auto chunk = [&](int c) -> unsigned {
        const float2 m = *reinterpret_cast<const float2*>(meta + 2 * c);
        if (!(m.y <= 2.f) || !(m.x <= 0.f)) bad = 1;    // outside the premise (also NaN, and +inf for a gate out of range)
        return __float2uint_rd(fminf(-m.x, kForgetCap) * kForgetScale);
    };
    if (chunks <= kPlanChunks) {
        for (int t = tid; t < NT; t += THREADS) pre[t + 1] = chunk(t);
    } else {
        unit = (chunks + kPlanChunks - 1) / kPlanChunks;
        NT = (chunks + unit - 1) / unit;
        for (int t = tid; t < NT; t += THREADS) {
            unsigned sum = 0;
            for (int c = t * unit; c < min(chunks, (t + 1) * unit); ++c)
                sum = min(static_cast<unsigned>(kForgetCap * kForgetScale), sum + chunk(c));
            pre[t + 1] = sum;
        }
    }
    if (tid == 0) {
        pre[0] = 0;
        plan.g = 1;
        *best = NT * 64;                                // score of the serial run
    }
    bad = __syncthreads_or(bad);
    if (bad) return;
    if (warp == 0) {
        unsigned carry = 0;
        for (int base = 0; base < NT; base += 32) {
            unsigned x = base + lane < NT ? pre[base + lane + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            x += carry;
            if (base + lane < NT) pre[base + lane + 1] = x;
            carry = __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    const int g = warp + 2;
    int L0 = 0, L1 = 0, mine = 0, score = 1 << 30;
    if (g <= G) {
        L0 = L1 = (NT + g - 1) / g;
        int w0, p = warmups(pre, NT, g, L0, L1, lane, w0);
        mine = w0;
        if (p >= 0) {
            int steps = L1 + p;
            // equal work: segment 0, which has no warm-up, longer by about the warm-up
            const int M1 = max(1, (NT - p + g - 1) / g), M0 = NT - (g - 1) * M1;
            if (M0 >= M1) {
                int w1;
                const int p1 = warmups(pre, NT, g, M0, M1, lane, w1);
                if (p1 >= 0 && max(M0, M1 + p1) < steps) {
                    steps = max(M0, M1 + p1);
                    L0 = M0;
                    L1 = M1;
                    mine = w1;
                }
            }
            score = steps * 64 + g;
            if (lane == 0) atomicMin(best, score);
        }
    }
    __syncthreads();
    if (g <= G && score == *best) {
        if (lane == 0) {
            plan.g = g;
            plan.L0 = L0 * unit;
            plan.L1 = L1 * unit;
        }
        if (lane < g) plan.warm[lane] = mine * unit;
    }
    __syncthreads();
}

}  // namespace gdn
