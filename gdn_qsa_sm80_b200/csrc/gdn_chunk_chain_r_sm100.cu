// "chain", residual form: one CTA per (sequence, value head[, segment]) runs the serial state recurrence and the outputs
// of all 128 value columns.  Instead of W = T (beta e^gamma K), formed per chunk by the prepare step and read back here, it
// applies T'' = T diag(beta) to both parts of the chunk's residual V - e^gamma K S (notation of gdn_qsa_sm80/reference/gdn_chunk_ref.py:90-94;
// v_new = U - W S = T'' V - T'' diag(e^gamma) K S), all products transposed so that what the recurrence rewrites are A
// operands in tensor memory and every B operand is a tile as TMA loaded it:
//   E1   KS     = S^T K^T              (A = bf16 S^T)
//   E1'  O      = S^T Q^T              (same A)           O <- scale e^gamma_i O  (column factors, by the output warps)
//   E0   v_new  = V^T T''^T            (A = the raw V tile, MN-major)
//        X      = e^gamma_j KS         (column factors, bf16)
//   ER   v_new -= X^T T''^T            (A = bf16 X^T, negated)                                              (ref :91)
//   E2   ACC_S  = v~^T K               (A = bf16 v~^T, v~ = e^(gamma_C - gamma_i) v_new)
//        S^T   <- e^gamma_C S^T + ACC_S                                                                    (ref :94)
//   E3   O     += v_new^T P^T                                                                           (ref :92-93)
// Against the form with W (this library's chain before) a chunk has one hand-off more on its critical path, but reads 16 KB
// less and needs 256 tensor-memory columns, 110 KB of shared memory and 32 K registers, so TWO CTAs share an SM and
// each fills the other's waits: what counts here is the time of a chunk step per SM, not its latency.
//
// Tensor memory of a CTA (columns; each operand is written over an accumulator that is dead by then - UMMAs of one thread
// execute in order):
//   0..127    ACC_S; the state epilogue packs the bf16 state over columns it has read: the warps of half h own the blocks
//             32 h and 64 + 32 h of 32 columns and pack them into 32 h, so that A_S lies in 0..63, its k order permuted,
//             and 64..127 are free for v_new (E0, ER) while E1 and E1' read A_S
//   128..191  KS; X packed over it (128..143, 160..175); then v~ (128..159) and v_new (160..191) once ER has read X
//   192..255  O
// Order of issue: E1, E0, ER, E1', E2, E3 - E0 runs during the X epilogue and E1' during the v_new epilogue, so of the two
// products nothing on the critical path waits for, neither delays one that is on it.
// Shared memory: K, V and T'' in two slots, Q and P in one: every tile is used once (K twice, a few thousand cycles
// apart), and its slot is reloaded as soon as the UMMA that read it has completed.  V's slot is used again first: a chunk's outputs
// are staged where its V was and leave by TMA.  Two-byte stores by the lanes cost the output warps 190 instructions a chunk, two thirds
// of what they issue, and these share the issue slots of the critical warps (24.0 -> 20.0 million instructions on 4 x 2048 tokens, 32
// heads, with the paired arithmetic of the other epilogues).  us a call, before / after: 8192 tokens 97.2 / 91.8, 4 x 1999 101.7 / 95.0,
// 16 x 2048 322 / 310, 64 x 4096 2700 / 2580, 131072 tokens 1460 / 1380; the paired arithmetic alone is 0 to 1 % of it.  (Staged in Q's place, whose next tile is wanted a step earlier
// than V's, 8192 tokens took 104.)
//
// Roles (16 warps): 0-7 critical (warp w: TMEM lane quadrant w % 4, column half w / 4): X, v_new and state epilogues,
// fp32 state in registers; 8-11 output; 12 TMA producer; 13 issues every UMMA.  Registers are moved from the last two
// groups of four warps to the first two (64 each at launch -> 88, 88, 56, 24).
//
// Sequences are split into segments when there are too few of them (gdn_segment_plan.cuh).
// Stands in for the reference's gdn_recurrence_kernel (csrc/gdn_chunk/gdn_kernel.cu:1027-1271).
#include <cuda.h>

#include "../../include/gdn_chunk_sm100.h"
#include "gdn_common.cuh"
#include "gdn_launch.cuh"
#include "gdn_segment_plan.cuh"
#include "ptx_sm100.cuh"

namespace gdn {
namespace {

constexpr int kRThreads = 512;
constexpr uint32_t R_K = 0, R_V = 32768, R_Q = 65536, R_T2 = 81920, R_P = 98304, R_VEC = 106496, kRBytes = R_VEC + 2048;
constexpr uint32_t kRDynamic = kRBytes + 1024;
constexpr uint32_t C_S = 0, C_VN = 64, C_KS = 128, C_VS = 128, C_VP = 160, C_O = 192, kRTmemCols = 256;
constexpr int kRTimeout = 0x500;   // + the barrier's index

// barriers
enum : uint32_t { R_KFULL = 0, R_VFULL = 2, R_VEMPTY = 4, R_TFULL = 6, R_QFULL = 8, R_PFULL, R_KS, R_QS, R_X, R_VACC, R_VN, R_S, R_STATE = R_S + 2,
                  R_QSC, R_O, R_ODONE, R_OUT, R_STATE1 = R_OUT + 2, R_NEVER /* test hook */, kRBars };

// Byte offset, in a [64 tokens][128 dk] tile of two 64-column halves, of the 16 dk that k step `ks` of A_S holds (half ks / 4
// of the warps packed the column blocks 32 h .. and 64 + 32 h ..).
__device__ constexpr uint32_t dk_bytes(int ks) { return ((ks >> 1) & 1) * 8192 + (ks >> 2) * 64 + (ks & 1) * 32; }

// What a CTA runs, in shared memory (the roles re-read what they need instead of holding it in registers): `steps` chunks
// of the sequence from chunk t0 on, outputs stored from step `store_from` on.
struct RWork {
    int t0, steps, store_from, len;        // len: tokens of the sequence
    int b, s_first;                        // TMA coordinates of the sequence's first token
    int seg, segs;                         // which segment of the sequence this CTA runs, of how many at most
    size_t tok0, tile0;                    // first token and first workspace tile of the sequence and head
    const float* s_in;                     // state it starts from (null: zeros) and where the one it ends with goes
    float* s_out;
    int* status;
    int late;                              // code of the first wait that ran out
};

// Shared-memory descriptor of this file's operands: 1024 bytes between 8-row groups and the 128-byte swizzle throughout, so
// the upper word is a constant and only the lower one (address and, MN-major, the distance of 64-column groups) varies.
__device__ __forceinline__ uint64_t r_desc(uint32_t lo) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"((1024u >> 4) | (1u << 14) | (SWZ_128B << 29)));
    return d;
}
__device__ __forceinline__ uint64_t r_desc64(uint32_t lo) {   // triangular tiles: 64-byte rows and swizzle, 512 bytes per 8 rows
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"((512u >> 4) | (1u << 14) | (SWZ_64B << 29)));
    return d;
}
// Where k step `ks` (16 columns) of a triangular tile starts: steps 0, 1 are columns of all 64 rows, 2, 3 of rows 32-63 only -
// products with it are N = 64 and, for the later two, N = 32 into the second half of the accumulator.
__device__ constexpr uint32_t tri_bytes(int ks) { return (ks >> 1) * 4096 + (ks & 1) * 32; }
constexpr uint32_t kLoK = (16u >> 4) << 16, kLoMN = (8192u >> 4) << 16;

// Bounded wait; a role whose wait ran out leaves, the others' waits run out behind it, and the CTA reports the first at its end.  With the inline
// slow path of mbar_wait at 25 places (before / after, us a call): 2 x 1500 tokens, 8 / 8 heads 29.8 / 28.6, 333 tokens 21.5 / 20.9,
// 4 x 1999 104.0 / 102.2, 8192 100.1 / 98.7; nothing where HBM bounds it.
__device__ __forceinline__ bool r_wait(uint32_t bar, uint32_t parity, int code, RWork& work) {
    if (mbar_wait_compact(bar, parity)) return true;
    atomicCAS(&work.late, 0, code);
    return false;
}

__device__ __forceinline__ float2 as_float2(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ uint32_t mul_bf16x2(float2 a, float2 b) {
    const float2 x = mul2(a, b);
    return pack_bf16x2(x.x, x.y);
}

template <int N>
__device__ __forceinline__ void set_max_registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void set_max_registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

template <bool SPLIT, bool HOOKS>
__global__ void __launch_bounds__(kRThreads, 2)
gdn_chain_r_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_p,
                   const __grid_constant__ CUtensorMap tm_t2, const __grid_constant__ CUtensorMap tm_out, const __grid_constant__ Problem p,
                   const __grid_constant__ Workspace ws, const unsigned sms) {
    extern __shared__ uint8_t smem_raw[];
    // Rounded up as an offset: through an integer the pointer loses its address space, and every access by the roles becomes a generic one (us a call,
    // before / after: 333 tokens 19.9 / 19.1, 2 x 1500 with 8 / 8 heads 28.2 / 27.0, 4 x 1999 82.1 / 80.4, 8192 83.1 / 82.0, 64 x 4096 2179 / 2143).
    uint8_t* sm = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);
    const uint32_t sm_u32 = warp_uniform(smem_u32(sm));
    __shared__ __align__(8) uint64_t bars[kRBars];
    __shared__ uint32_t tmem_slot;
    __shared__ int plan_best;
    __shared__ SegmentPlan plan;
    __shared__ RWork work;

    const int tid = threadIdx.x, warp = static_cast<int>(warp_uniform(tid >> 5)), lane = tid & 31;
    const int hv = blockIdx.x, hq = hv / (p.Hv / p.Hq);
    const uint32_t bar0 = smem_u32(bars);
    auto cb = [&](uint32_t i) { return bar0 + 8u * i; };

    if (tid == 0) {
        for (uint32_t i = 0; i < kRBars; ++i) {
            const uint32_t count = i == R_VEMPTY || i == R_VEMPTY + 1 ? 12
                                   : i == R_X || i == R_VN || i == R_STATE || i == R_STATE1 ? 8 : i == R_QSC || i == R_ODONE ? 4 : 1;
            mbar_init(&bars[i], count);
        }
        work.late = 0;
        work.status = p.status;
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_slot, kRTmemCols);
        tmem_relinquish();
    }
    // Launched ahead of the end of the prepare kernel.  What that one makes is read behind this wait, where sequences are split by every thread (the plan), else
    // by the producer alone: the first tiles of K and V and the initial state are under way by then (whoever made them had ended when the prepare kernel's
    // CTAs let this one start).  us a call, before / after: 9 tokens 10.04 / 9.47, 200 15.27 / 14.70, 333 18.59 / 18.02, 4 x 200 17.76 / 17.23.
    const bool whole = SPLIT || p.pk_chunk || !p.behind_prepare;
    if (whole) grid_dependency_wait();

    if (tid == 0) {   // which sequence: its tokens, chunks and workspace tiles
        int seq;
        if (p.pk_chunk) {
            const int4 o = p.pk_order[blockIdx.y];
            seq = o.x;
            work.seg = o.z;
            work.segs = o.w;
            work.b = 0;
            work.s_first = p.pk_cu[seq];
            work.len = p.pk_cu[seq + 1] - work.s_first;
            work.tok0 = work.s_first;
            work.tile0 = static_cast<size_t>(o.y) * p.Hv + static_cast<size_t>(hv) * ((work.len + kChunk - 1) / kChunk);
        } else {
            seq = work.b = blockIdx.y;
            work.seg = blockIdx.z;
            work.segs = ws.n_seg;
            work.s_first = 0;
            work.len = p.S;
            work.tok0 = static_cast<size_t>(seq) * p.S;
            work.tile0 = (static_cast<size_t>(seq) * p.Hv + hv) * ((p.S + kChunk - 1) / kChunk);
        }
        const size_t state_off = (static_cast<size_t>(seq) * p.Hv + hv) * kD * kD;
        work.t0 = work.store_from = 0;
        work.steps = (work.len + kChunk - 1) / kChunk;
        work.s_in = p.h0 ? p.h0 + state_off : nullptr;
        work.s_out = p.hT ? p.hT + state_off : nullptr;
    }
    if (SPLIT) {
        __syncthreads();
        const int nt = work.steps;
        if (work.segs > 1) plan_segments<kRThreads>(ws.meta + 2 * work.tile0, nt, work.segs, reinterpret_cast<unsigned*>(sm), plan, &plan_best);
        else if (tid == 0) plan.g = 1;      // (of a packed batch whose longer sequences are cut)
        if (tid == 0) {
            const int seg = work.seg, g = plan.g;
            if (g > 1) {
                const int a = seg == 0 ? 0 : plan.L0 + (seg - 1) * plan.L1;
                const int e = min(nt, seg == 0 ? plan.L0 : a + plan.L1);
                if (seg >= g || a >= nt) {
                    work.steps = 0;
                } else {
                    work.store_from = seg == 0 ? 0 : plan.warm[seg];
                    work.t0 = a - work.store_from;
                    work.steps = e - work.t0;
                    if (seg > 0) work.s_in = nullptr;
                    if (e < nt) work.s_out = nullptr;
                }
            } else if (seg > 0) {
                work.steps = 0;
            }
        }
        fence_proxy_async_smem();   // the prefix sums lie where the ring's loads go
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = warp_uniform(tmem_slot);
#ifdef GDN_DIAGNOSTICS   // cycles of one thread of the critical warps (in shared memory: the roles have no registers to spare)
    __shared__ long long prof_acc[7];   // phases 0-5 and the last time stamp
    const bool prof_on = p.prof != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && tid == 0;
    if (prof_on)
        for (int n = 0; n < 7; ++n) prof_acc[n] = n == 6 ? clock64() : 0;
#define GDN_PHASE(n)                              \
    if (prof_on) {                                \
        const long long now_ = clock64();         \
        prof_acc[n] += now_ - prof_acc[6];        \
        prof_acc[6] = now_;                       \
    }
#else
#define GDN_PHASE(n)
#endif
    // Chunks before `from` are warm-up: their outputs are not formed (no Q, no P, no E1', no E3; the barriers of those count from `from` on).
    // One sequence of 8192 tokens, 5 of 20 steps: 98.6 -> 96.3 us a call; 4 x 1999 102.2 -> 101.2; 2 x 1500, 8 / 8 heads 28.4 -> 27.9.
    const int steps = work.steps, from = SPLIT ? work.store_from : 0;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        return r_wait(cb(bar), parity & 1, kRTimeout + static_cast<int>(bar), work);
    };

    if (steps == 0) {
    } else if (warp >= 12) {
        set_max_registers_down<24>();
        if (warp == 12) {
            // ------------------------------- TMA producer ----------------------------------------------------------
            auto load_k = [&](int n) {
                const uint32_t s = n & 1, fb = cb(R_KFULL + s), d = sm_u32 + R_K + s * 16384;
                const int s0 = work.s_first + (work.t0 + n) * kChunk;
                const int b = work.b;
                if (elect_one()) {
                    mbar_arrive_expect_tx_a(fb, 16384);
                    tma_load_4d_a(d, &tm_k, fb, 0, hq, s0, b);
                    tma_load_4d_a(d + 8192, &tm_k, fb, 64, hq, s0, b);
                }
            };
            auto load_v = [&](int n, bool tile, bool factors) {
                const uint32_t s = n & 1, fb = cb(R_VFULL + s);
                const int t = work.t0 + n, s0 = work.s_first + t * kChunk, b = work.b;
                const float* vec = ws.vec + (work.tile0 + t) * 256;
                if (elect_one()) {
                    if (tile) {
                        mbar_arrive_expect_tx_a(fb, 16384 + 1024);
                        tma_load_4d_a(sm_u32 + R_V + s * 16384, &tm_v, fb, 0, hv, s0, b);
                        tma_load_4d_a(sm_u32 + R_V + s * 16384 + 8192, &tm_v, fb, 64, hv, s0, b);
                    }
                    if (factors) bulk_load_1d_a(sm_u32 + R_VEC + s * 1024, vec, 1024, fb);
                }
            };
            auto load_tri = [](uint32_t dst, const void* map, uint32_t bar, int row0) {
                tma_load_2d_a(dst, map, bar, 0, row0);
                tma_load_2d_a(dst + 2048, map, bar, 0, row0 + 32);
                tma_load_2d_a(dst + 4096, map, bar, 32, row0 + 32);
            };
            auto prefetch_tri = [](const void* map, int row0) {
                tma_prefetch_2d(map, 0, row0);
                tma_prefetch_2d(map, 0, row0 + 32);
                tma_prefetch_2d(map, 32, row0 + 32);
            };
            // How many CTAs are at work: those of a head's segments that its plan does not use have left already, and so have
            // most of a packed batch's shorter sequences while its longest one runs.
            const unsigned g = SPLIT ? static_cast<unsigned>(plan.g) : 1u;
            const bool ahead = p.pk_chunk ? static_cast<unsigned long long>(p.Hv) * p.pk_chunks * g <= static_cast<unsigned long long>(sms) * p.pk_longest
                                          : gridDim.x * gridDim.y * g <= sms;
            auto load_t2 = [&](int n) {
                const uint32_t s = n & 1, fb = cb(R_TFULL + s);
                const int row0 = static_cast<int>((work.tile0 + work.t0 + n) * kChunk);
                if (elect_one()) {
                    mbar_arrive_expect_tx_a(fb, kTriBytes);
                    load_tri(sm_u32 + R_T2 + s * 8192, &tm_t2, fb, row0);
                }
            };
            auto dawdle = [&]() {                              // test hook: every barrier this role waits for is far ahead
                if (!HOOKS || p.dbg != kDbgLateProducer) return;
                const unsigned long long t0 = globaltimer_ns();
                while (globaltimer_ns() - t0 < 20000ull) {}
            };
            const bool tile = !HOOKS || p.dbg != kDbgNoTile;
            load_k(0);
            if (whole) {
                load_t2(0);
                if (tile) load_v(0, true, true);
            } else {
                if (tile) load_v(0, true, false);
                grid_dependency_wait();
                load_t2(0);
                if (tile) load_v(0, false, true);
            }
            // A slot's reload waits for the UMMA (or the epilogue) that read it, in the order in which those complete.  A wait names a parity,
            // so the next completion of its barrier has to need a tile that is loaded behind it.  In iteration n:
            //   R_S + slot of n - 1    next: E2 of n + 1, which needs K(n + 1), two lines below.  (One barrier for both slots would complete
            //                          next with E2 of n, and a warm-up chunk n needs nothing of this iteration: it has no Q.)
            //   R_O of n - 1           next: E3 of n, which needs P(n)
            //   R_VEMPTY, R_OUT + slot of n - 1    next: the epilogues and the outputs of n + 1, which need V(n + 1).  (All that chunk n's outputs
            //                          need has been loaded by then.)
            for (int n = 0; n < steps; ++n) {
                // Alone on its SM, a CTA waits for tiles whose load a slot holds up (Q and P have one; a step is shorter than
                // two HBM latencies under load), so what the next loads will read is brought into L2 first: 4 sequences of
                // 4096 tokens, 128 CTAs, 166 -> 141 us in this kernel.  With two CTAs per SM the other one fills those waits
                // and the extra requests cost more than they give (9 sequences, 288 CTAs: 221 -> 229 us).
                if (ahead && n + 1 < steps && elect_one()) {
                    const int s1 = work.s_first + (work.t0 + n + 1) * kChunk, b1 = work.b;
                    const int r1 = static_cast<int>((work.tile0 + work.t0 + n + 1) * kChunk);
                    if (n + 1 >= from) {
                        tma_prefetch_4d(&tm_q, 0, hq, s1, b1);
                        tma_prefetch_4d(&tm_q, 64, hq, s1, b1);
                        prefetch_tri(&tm_p, r1);
                    }
                    if (n + 2 < steps) {
                        tma_prefetch_4d(&tm_k, 0, hq, s1 + kChunk, b1);
                        tma_prefetch_4d(&tm_k, 64, hq, s1 + kChunk, b1);
                        tma_prefetch_4d(&tm_v, 0, hv, s1 + kChunk, b1);
                        tma_prefetch_4d(&tm_v, 64, hv, s1 + kChunk, b1);
                        prefetch_tri(&tm_t2, r1 + kChunk);
                    }
                }
                dawdle();
                if (n > 0 && !wait(R_S + ((n - 1) & 1), (n - 1) >> 1)) break;   // E2, hence also ER and E1', of chunk n - 1
                if (n + 1 < steps) {
                    load_k(n + 1);
                    load_t2(n + 1);
                }
                if (n >= from) {
                    const int s0 = work.s_first + (work.t0 + n) * kChunk, b = work.b;
                    const int row0 = static_cast<int>((work.tile0 + work.t0 + n) * kChunk);
                    if (elect_one()) {
                        mbar_arrive_expect_tx_a(cb(R_QFULL), 16384);
                        tma_load_4d_a(sm_u32 + R_Q, &tm_q, cb(R_QFULL), 0, hq, s0, b);
                        tma_load_4d_a(sm_u32 + R_Q + 8192, &tm_q, cb(R_QFULL), 64, hq, s0, b);
                    }
                    dawdle();
                    if (n > from && !wait(R_O, n - from - 1)) break;
                    if (elect_one()) {
                        mbar_arrive_expect_tx_a(cb(R_PFULL), kTriBytes);
                        load_tri(sm_u32 + R_P, &tm_p, cb(R_PFULL), row0);
                    }
                }
                if (n + 1 < steps) {
                    dawdle();
                    if (n > 0 && !wait(R_VEMPTY + ((n + 1) & 1), ((n + 1) >> 1) - 1)) break;
                    if (n > from && !wait(R_OUT + ((n - 1) & 1), (n - from - 1) >> 1)) break;   // the outputs of chunk n - 1, staged in its V's place, have left
                    load_v(n + 1, true, true);
                }
            }
        } else if (warp == 13) {
            // ------------------------------- UMMA issuer ------------------------------------------------------------
            constexpr uint32_t idesc_n64 = umma_idesc_bf16(128, 64, MAJOR_K, MAJOR_K);
            constexpr uint32_t idesc_n32 = umma_idesc_bf16(128, 32, MAJOR_K, MAJOR_K);
            constexpr uint32_t idesc_e0 = umma_idesc_bf16(128, 64, MAJOR_MN, MAJOR_K), idesc_e0_n32 = umma_idesc_bf16(128, 32, MAJOR_MN, MAJOR_K);
            constexpr uint32_t idesc_neg = umma_idesc_bf16(128, 64, MAJOR_K, MAJOR_K, 1);   // negated A
            constexpr uint32_t idesc_neg_n32 = umma_idesc_bf16(128, 32, MAJOR_K, MAJOR_K, 1);
            constexpr uint32_t idesc_e2 = umma_idesc_bf16(128, 128, MAJOR_K, MAJOR_MN);
            const uint32_t base = (sm_u32 & 0x3FFFFu) >> 4;   // (a cluster CTA's window address has bits above)
            for (int n = 0; n < steps; ++n) {
                const uint32_t s = n & 1;
                if (!wait(R_KFULL + s, n >> 1)) break;
                // E1.  Where sequences are split there are few of them and a step's length counts: the first four k steps begin when half of
                // the state's copy is there, while the epilogue works on the rest.  us a call, before / after: 700 tokens 27.0 / 26.4; 2 x 1500,
                // 8 / 8 heads 27.5 / 27.1; 2 x 2500, 8 / 16 heads 42.1 / 41.6; 4 x 1999 98.1 / 97.6, within the noise; with many sequences nothing.
                auto e1 = [&](int ks) {
                    umma_bf16_ts(tmem + C_KS, tmem + C_S + ks * 8, r_desc(base + s * (16384 >> 4) + kLoK + ((R_K + dk_bytes(ks)) >> 4)), idesc_n64, ks > 0);
                };
                if (SPLIT) {
                    if (!wait(R_STATE1, n)) break;
                    tc_fence_after_sync();
                    if (elect_one()) {
                        e1(0);
                        e1(1);
                        e1(4);
                        e1(5);
                    }
                    __syncwarp();
                }
                if (!wait(R_STATE, n)) break;
                tc_fence_after_sync();
                if (elect_one()) {
                    if (!SPLIT) {
                        e1(0);
                        e1(1);
                        e1(4);
                        e1(5);
                    }
                    e1(2);
                    e1(3);
                    e1(6);
                    e1(7);
                    umma_commit_a(cb(R_KS));
                }
                if (!wait(R_TFULL + s, n >> 1)) break;
                if (!wait(R_VFULL + s, n >> 1)) break;
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)               // E0
                        umma_bf16_ss(tmem + C_VN + (ks >> 1) * 32, r_desc(base + s * (16384 >> 4) + kLoMN + ((R_V + ks * 2048) >> 4)),
                                     r_desc64(base + s * (8192 >> 4) + kLoK + ((R_T2 + tri_bytes(ks)) >> 4)), ks < 2 ? idesc_e0 : idesc_e0_n32, ks > 0);
                }
                if (!wait(R_X, n)) break;
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)               // ER
                        umma_bf16_ts(tmem + C_VN + (ks >> 1) * 32, tmem + C_KS + (ks >> 1) * 32 + (ks & 1) * 8,
                                     r_desc64(base + s * (8192 >> 4) + kLoK + ((R_T2 + tri_bytes(ks)) >> 4)), ks < 2 ? idesc_neg : idesc_neg_n32, 1);
                    umma_commit_a(cb(R_VACC));
                }
                if (n >= from) {
                    if (!wait(R_QFULL, n - from)) break;
                    if (n > from && !wait(R_ODONE, n - from - 1)) break;   // chunk n - 1's outputs have been read
                    tc_fence_after_sync();
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)               // E1'
                            umma_bf16_ts(tmem + C_O, tmem + C_S + ks * 8, r_desc(base + kLoK + ((R_Q + dk_bytes(ks)) >> 4)), idesc_n64, ks > 0);
                        umma_commit_a(cb(R_QS));
                    }
                }
                if (!wait(R_VN, n)) break;
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)               // E2
                        umma_bf16_ts(tmem + C_S, tmem + C_VS + ks * 8, r_desc(base + s * (16384 >> 4) + kLoMN + ((R_K + ks * 2048) >> 4)), idesc_e2, ks > 0);
                    umma_commit_a(cb(R_S + s));
                }
                if (n < from) continue;
                if (!wait(R_PFULL, n - from)) break;
                if (!wait(R_QSC, n - from)) break;
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)               // E3
                        umma_bf16_ts(tmem + C_O + (ks >> 1) * 32, tmem + C_VP + ks * 8, r_desc64(base + kLoK + ((R_P + tri_bytes(ks)) >> 4)),
                                     ks < 2 ? idesc_n64 : idesc_n32, 1);
                    umma_commit_a(cb(R_O));
                }
            }
        }
    } else if (warp >= 8) {
        // ------------------------------- output warps ----------------------------------------------------------------
        set_max_registers_down<56>();
        const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
        const uint32_t o_addr = tmem_addr(tmem, lane_base, C_O);
        const bool leader = warp == 8;
        const uint32_t o_bar = HOOKS && p.dbg == kDbgWarpGivesUp && warp == 9 ? R_NEVER : R_O;
        // Row (token) whose address this lane gives to stmatrix, and its 16-byte chunk (8 value columns) before the swizzle; the warp's 32
        // value columns lie in one of the two halves of 64 columns.
        const uint32_t srow = 8 * (lane >> 4) + (lane & 7), sch = 4 * (warp & 1) + ((lane >> 3) & 1);
        const uint32_t stage = sm_u32 + R_V + ((warp >> 1) & 1) * 8192 + srow * 128;
        for (int n = 0; n < steps; ++n) {
            const uint32_t s = n & 1;
            if (!wait(R_VFULL + s, n >> 1)) break;            // the factors
            if (n < from) {                                   // (the slot's release counts these warps)
                __syncwarp();
                if (lane == 0) mbar_arrive_a(cb(R_VEMPTY + s));
                continue;
            }
            if (!wait(R_QS, n - from)) break;
            tc_fence_after_sync();
            const float* qf = reinterpret_cast<const float*>(sm + R_VEC + s * 1024) + kChunk + 2 * (lane & 3);   // scale e^gamma_j
#pragma unroll
            for (int u = 0; u < 4; ++u) {                     // tokens [16 u, +16) of 16 value columns at a time
                const float2 f[2] = {*reinterpret_cast<const float2*>(qf + 16 * u), *reinterpret_cast<const float2*>(qf + 16 * u + 8)};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t x[8];
                    const uint32_t at = o_addr + (static_cast<uint32_t>(16 * h) << 16) + 16 * u;
                    tmem_ld_16x256b_x2(at, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const float2 y = mul2(as_float2(x[e], x[e + 1]), f[e >> 2]);
                        x[e] = __float_as_uint(y.x);
                        x[e + 1] = __float_as_uint(y.y);
                    }
                    tmem_st_16x256b_x2(at, x);
                }
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_a(cb(R_QSC));
                mbar_arrive_a(cb(R_VEMPTY + s));
            }
            // The barrier below has no limit, so a warp whose tries run out here still takes part in it.  Whoever gets there has seen E3, hence
            // the arrivals of all four warps on R_QSC: none of them can have left earlier, and none gets to the next chunk's without the R_ODONE of
            // all.  (An mbarrier waited for with a limit: 700 tokens 26.3 -> 27.2 us a call.)
            if (!wait(o_bar, n - from)) {
                named_bar_arrive(1, 128);
                break;
            }
            tc_fence_after_sync();
            // O^T[dv][j] in fragments of 16 value columns by 32 tokens, transposed on their way into the place of V (E0 has read it)
#pragma unroll
            for (int u = 0; u < 4; ++u) {                     // value columns 16 (u & 1), tokens 32 (u >> 1)
                uint32_t x[16], pk[8];
                tmem_ld_16x256b_x4(o_addr + (static_cast<uint32_t>(16 * (u & 1)) << 16) + 32 * (u >> 1), x);
                tmem_ld_wait();
                if (u == 3) {                                 // the accumulator has been read
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_a(cb(R_ODONE));
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) pk[c] = pack_bf16x2(__uint_as_float(x[2 * c]), __uint_as_float(x[2 * c + 1]));
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    stmatrix_x4_trans(stage + s * 16384 + (32 * (u >> 1) + 16 * t) * 128 + (((sch + 2 * (u & 1)) ^ (srow & 7)) << 4), pk[4 * t], pk[4 * t + 1], pk[4 * t + 2], pk[4 * t + 3]);
            }
            const int t0 = (work.t0 + n) * kChunk, valid = work.len - t0;
            if (p.pk_chunk && valid < kChunk) {               // the rows below are the next sequence's: only this one's are copied
                named_bar_sync(1, 128);
                for (int e = tid & 127; e < valid * 16; e += 128) {
                    const int row = e >> 4, ch = e & 15;
                    const uint4 x = *reinterpret_cast<const uint4*>(sm + R_V + s * 16384 + (ch >> 3) * 8192 + row * 128 + (((ch & 7) ^ (row & 7)) << 4));
                    *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + ((work.tok0 + t0 + row) * p.Hv + hv) * (kD * 2) + ch * 16) = x;
                }
            } else {                                          // (rows behind a regular sequence's end are outside the map)
                fence_proxy_async_smem();
                named_bar_sync(1, 128);
                if (leader && elect_one()) {
                    tma_store_4d(&tm_out, sm + R_V + s * 16384, 0, hv, work.s_first + t0, work.b);
                    tma_store_4d(&tm_out, sm + R_V + s * 16384 + 8192, 64, hv, work.s_first + t0, work.b);
                    tma_store_commit();
                    tma_store_wait_read();
                    mbar_arrive_a(cb(R_OUT + s));
                }
                __syncwarp();
            }
        }
        if (leader && elect_one()) tma_store_wait_all();
    } else {
        // ------------------------------- critical warps ----------------------------------------------------------------
        set_max_registers_up<88>();
        const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
        const int dv = (warp & 3) * 32 + lane;
        const int hf = warp >> 2;                             // which half of the columns of each accumulator
        const uint32_t a_s = tmem_addr(tmem, lane_base, C_S + 32 * hf);
        const uint32_t a_ks = tmem_addr(tmem, lane_base, C_KS + 32 * hf);
        float st[64];                                         // S^T[dv][dk], dk = 32 hf + c (c < 32), 64 + 32 hf + c - 32
        const float* s_in = work.s_in ? work.s_in + 32 * hf * kD + dv : nullptr;
#pragma unroll
        for (int c = 0; c < 64; ++c) st[c] = s_in ? s_in[(c + (c & 32)) * kD] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            uint32_t pk[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) pk[c] = pack_bf16x2(st[16 * u + 2 * c], st[16 * u + 2 * c + 1]);
            tmem_st_x8(a_s + 8 * u, pk);
        }
        // The last tiles of a packed sequence hold the next sequence's first tokens below its own: beta and the gates are
        // zero there, but what the tiles hold (an infinity) must not reach this sequence, so those rows of K and V are
        // cleared before the step's first product.
        auto clear_tail = [&](int n) {
            const int valid = work.len - (work.t0 + n) * kChunk;
            if (!p.pk_chunk || valid >= kChunk) return;
            if (!wait(R_KFULL + (n & 1), n >> 1) || !wait(R_VFULL + (n & 1), n >> 1)) return;
            uint8_t* tile = sm + (n & 1) * 16384;
            for (int e = tid; e < (kChunk - valid) * 16; e += 256) {
                const uint32_t off = ((e >> 3) & 1) * 8192 + (valid + (e >> 4)) * 128 + (e & 7) * 16;
                *reinterpret_cast<uint4*>(tile + R_K + off) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(tile + R_V + off) = make_uint4(0, 0, 0, 0);
            }
            fence_proxy_async_smem();
        };
        if (steps == 1) clear_tail(0);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
            if (SPLIT) mbar_arrive_a(cb(R_STATE1));
            mbar_arrive_a(cb(R_STATE));
        }
        bool ok = true;
        for (int n = 0; n < steps; ++n) {
            const uint32_t s = n & 1;
            ok = wait(R_VFULL + s, n >> 1) && wait(R_KS, n);
            if (!ok) break;
            tc_fence_after_sync();
            GDN_PHASE(0)
            const float* vec = reinterpret_cast<const float*>(sm + R_VEC + s * 1024) + 32 * hf + 2 * (lane & 3);   // of this lane's columns
            const float dC = *reinterpret_cast<const float*>(sm + R_VEC + s * 1024 + 8 * kChunk);   // exp(gamma_C); read now, the slot is released below
#pragma unroll
            for (int u = 0; u < 2; ++u) {                     // X of tokens [32 hf + 16 u, +16), 16 value columns at a time
                const float2 f[2] = {*reinterpret_cast<const float2*>(vec + 3 * kChunk + 16 * u), *reinterpret_cast<const float2*>(vec + 3 * kChunk + 16 * u + 8)};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t x[8], pk[4];
                    const uint32_t at = a_ks + (static_cast<uint32_t>(16 * h) << 16);
                    tmem_ld_16x256b_x2(at + 16 * u, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 4; ++c) pk[c] = mul_bf16x2(as_float2(x[2 * c], x[2 * c + 1]), f[c >> 1]);
                    tmem_st_16x128b_x2(at + 8 * u, pk);
                }
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_a(cb(R_X));
            GDN_PHASE(1)
            ok = wait(R_VACC, n);
            if (!ok) break;
            tc_fence_after_sync();
            GDN_PHASE(2)
#pragma unroll SPLIT ? 2 : 1                          // (unsplit and unrolled, eight registers more are spilled: 64 x 4096 1 % slower)
            for (int u = 0; u < 2; ++u) {                     // v_new and v~ of tokens [32 hf + 16 u, +16)
                const float2 f[2] = {*reinterpret_cast<const float2*>(vec + 16 * u), *reinterpret_cast<const float2*>(vec + 16 * u + 8)};   // exp(gamma_C - gamma_j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t x[8], pk[4];
                    const uint32_t l16 = lane_base + 16 * h;
                    tmem_ld_16x256b_x2(tmem_addr(tmem, l16, C_VN + 32 * hf + 16 * u), x);
                    tmem_ld_wait();
                    if (n >= from) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) pk[c] = pack_bf16x2(__uint_as_float(x[2 * c]), __uint_as_float(x[2 * c + 1]));
                        tmem_st_16x128b_x2(tmem_addr(tmem, l16, C_VP + 16 * hf + 8 * u), pk);
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) pk[c] = mul_bf16x2(as_float2(x[2 * c], x[2 * c + 1]), f[c >> 1]);
                    tmem_st_16x128b_x2(tmem_addr(tmem, l16, C_VS + 16 * hf + 8 * u), pk);
                }
            }
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_a(cb(R_VN));
                mbar_arrive_a(cb(R_VEMPTY + s));
            }
            GDN_PHASE(3)
            ok = wait(R_S + s, n >> 1);
            if (!ok) break;
            tc_fence_after_sync();
            GDN_PHASE(4)
            const bool more = n + 1 < steps;
            if (SPLIT && n + 2 == steps) clear_tail(n + 1);   // (before E1 reads the tile)
#pragma unroll
            for (int u = 0; u < 4; ++u) {                     // S^T <- exp(gamma_C) S^T + v~^T K, 16 columns at a time
                uint32_t x[16];
                tmem_ld_x16(a_s + (u >> 1) * 64 + (u & 1) * 16, x);
                tmem_ld_wait();
                if (SPLIT && u == 2 && more) {                // the first two blocks' copies
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_a(cb(R_STATE1));
                }
#pragma unroll
                for (int c = 0; c < 16; c += 2) {
                    const float2 y = fma2(make_float2(dC, dC), make_float2(st[16 * u + c], st[16 * u + c + 1]), as_float2(x[c], x[c + 1]));
                    st[16 * u + c] = y.x;
                    st[16 * u + c + 1] = y.y;
                }
                if (more) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) x[c] = pack_bf16x2(st[16 * u + 2 * c], st[16 * u + 2 * c + 1]);
                    tmem_st_x8(a_s + 8 * u, reinterpret_cast<const uint32_t (&)[8]>(x));
                }
            }
            if (more) {
                if (!SPLIT && n + 2 == steps) clear_tail(n + 1);
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive_a(cb(R_STATE));
            }
            GDN_PHASE(5)
        }
#ifdef GDN_DIAGNOSTICS   // behind the prepare kernel's: waits for KS, v_new, the state's product and the epilogues behind them
        if (prof_on) {
            for (int n = 0; n < 6; ++n) p.prof[8 + n] = prof_acc[n];
            p.prof[14] = steps;
        }
#endif
        if (ok && work.s_out) {
            float* s_out = work.s_out + 32 * hf * kD + dv;
#pragma unroll
            for (int c = 0; c < 64; ++c) s_out[(c + (c & 32)) * kD] = st[c];
        }
    }

    if (!whole) grid_dependency_wait();   // (of a CTA without chunks: it does not end before the prepare kernel has)
    tc_fence_before_sync();
    __syncthreads();
    if (work.late) {   // let copies that may still be in flight land before the CTA's memory is released
        if (tid == 0) atomicCAS(work.status, 0, work.late);
        const unsigned long long w0 = globaltimer_ns();
        while (globaltimer_ns() - w0 < 100000ull) {}
        __syncthreads();
    }
    if (warp == 0) tmem_dealloc(tmem, kRTmemCols);
#undef GDN_PHASE
}

}  // namespace

int launch_chain_r(const Problem& p, const Workspace& ws, const TileMaps& maps, cudaStream_t stream) {
    auto map = [](const unsigned char* m) -> const CUtensorMap& { return *reinterpret_cast<const CUtensorMap*>(m); };
    auto go = [&](auto kernel, unsigned gz) -> int {
        if (allow_smem(reinterpret_cast<const void*>(kernel), kRDynamic)) return GDN_ERR_CUDA;
        // The value heads that share a qk head read the same K and Q tiles: as a cluster of two CTAs they start together
        // and run in step, so the second read of a tile finds it in L2 (nothing else of the cluster is used).
        // A grid's y ends at 65535: a packed batch of more entries takes several launches.
        Problem part = p;
        for (int done = 0, all = p.pk_chunk ? p.pk_n : 1; done < all; done += 65535) {
            unsigned gy = static_cast<unsigned>(p.B);
            if (p.pk_chunk) {
                part.pk_order = p.pk_order + done;
                gy = static_cast<unsigned>(all - done < 65535 ? all - done : 65535);
            }
            if (launch_dependent(kernel, dim3(p.Hv, gy, gz), dim3(kRThreads), kRDynamic, stream, (p.Hv / p.Hq) % 2 == 0, map(maps.q), map(maps.k),
                                 map(maps.v), map(maps.p), map(maps.t2), map(maps.out), part, ws, static_cast<unsigned>(sm_count())) != cudaSuccess)
                return GDN_ERR_CUDA;
        }
        return GDN_OK;
    };
    const int G = ws.n_seg;
    if (G <= 1 || G > kMaxSegments || !ws.meta) return p.dbg ? go(gdn_chain_r_kernel<false, true>, 1) : go(gdn_chain_r_kernel<false, false>, 1);
    const unsigned gz = p.pk_chunk ? 1u : static_cast<unsigned>(G);
    return p.dbg ? go(gdn_chain_r_kernel<true, true>, gz) : go(gdn_chain_r_kernel<true, false>, gz);
}

}  // namespace gdn
