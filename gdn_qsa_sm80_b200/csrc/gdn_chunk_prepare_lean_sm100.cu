// "prepare" for the residual-form chain (gdn_chunk_chain_r_sm100.cu): per chunk and value head only what that chain
// cannot form itself,
//   P [64][64] bf16 (masked, scaled Q K^T),  T'' = T diag(beta) [64][64] bf16,  the per-token factors  and the two
//   scalars of the decay bound (sum of g, max beta |k|^2)
// - no W, no U: the chain applies T'' to the residual V - exp(gamma) K S, so nothing of size [64][128] is formed, staged
// or written here, and P and T'' leave without the blocks above their diagonals (13 KB per chunk and head instead of 33 KB).
//
// HEADS = 2: one item = the chunk of the two value heads that share a qk head (the reference's head mapping,
// csrc/gdn_chunk/gdn_kernel.cu:385-387): one K / Q load and one [K;Q] K^T product, then one half of the CTA per head.
// HEADS = 1 (odd number of value heads per qk head): one head per CTA of 128 threads.
//
// The four warps of a head are roles that run several items apart, each with its own part of a chain of dependent phases (product, masks, triangular inverse,
// T''): a phase is some hundred instructions that wait for one another, and what an SM gets done is decided by how many of its 24 warps have one to issue.
//   role 0, 1   the two 32x32 diagonal blocks of T (lean_diagonal), item i; role 1 also the mask of A below them
//   role 2      tiles and product of item i + 1; P, rows 0-31, of item i; T'' below the diagonal blocks, left half, of item i - 1
//   role 3      gates and tables of item i + 1; P, rows 32-63, of item i; T'' below the diagonal blocks, right half, of item i - 1
// All four at the same item, with barriers of the head between the phases, left a quarter of the warps' time at them.
//
// What bounds it: the shared-memory pipe (16 sequences of 2048 tokens: 61 % of the cycles for loads and stores, about 25 % for operands and copies), then HBM (29 KB
// per chunk and head).  us alone, against the form that passed A and T through shared memory row by row and ran its phases in step: 16 x 2048 124 / 95.8, 8192 tokens
// 36.3 / 29.5, 4 x 1999 36.3 / 29.5 (with L2 normalisation 41.8 / 34.3), 64 x 4096 941 / 719; 16 x 2048 with 16 / 16 heads 81.5 / 66.0.
// Stands in for the reference's gdn_prepare_kernel (csrc/gdn_chunk/gdn_kernel.cu:343-710).
#include <cuda.h>

#include <type_traits>

#include "../../include/gdn_chunk_sm100.h"
#include "gdn_common.cuh"
#include "gdn_launch.cuh"
#include "gdn_prep_lean_device.cuh"
#include "ptx_sm100.cuh"

namespace gdn {
namespace {

template <int HEADS>
struct LeanSmem {
    static constexpr uint32_t KQ = 0;                    // [K;Q]: 2 k-halves x 128 rows x 128 B (K rows 0-63, Q rows 64-127);
                                                         //   P of head h on its way out in Q's rows of k-half h once the product is done
    static constexpr uint32_t T2 = 32768;                // T'' of head h on its way out at T2 + h * kTriBytes
    static constexpr uint32_t EX = T2 + HEADS * kTriBytes;
    static constexpr uint32_t kBytes = EX + HEADS * sizeof(LeanExchange);
    static constexpr uint32_t kDynamic = kBytes + 1024;
    static_assert(T2 % 512 == 0 && kTriBytes % 512 == 0, "the 64-byte swizzle repeats every 512 bytes");
};
constexpr uint32_t kLeanTmemCols = 128;                  // two accumulators of 64 columns
template <int HEADS>
constexpr int kLeanCtasPerSm = HEADS == 2 ? 3 : 4;

// Barriers; those with + head are one per head.  Each completes once an item.
enum : uint32_t {
    B_K = 0,         // K is there
    B_Q,             // Q is there
    B_MMA,           // the product is done
    B_ENT,           // every warp has seen the product (and the tables), and has read the accumulator of the item before
    B_SQ,            // with L2 normalisation: the rows' squares are there
    B_TAB,           // + head: the tables
    B_PAIR = B_TAB + 2,  // + head: both parts of P have left shared memory
    B_EXF = B_PAIR + 2,  // + head: the exchange is full
    B_EXE = B_EXF + 2,   // + head: and has been read
    B_LOW = B_EXE + 2,   // + head: role 3's half of T'' below the diagonal blocks is there
    B_BARS = B_LOW + 2,
    B_NEVER = B_BARS     // of a test hook: no arrival ever completes it
};

template <int HEADS, bool GATE_F32, bool HOOKS>
__global__ void __launch_bounds__(128 * HEADS, kLeanCtasPerSm<HEADS>)
gdn_prepare_lean_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_t2, Problem p,
                        Workspace ws, unsigned NT, unsigned num_items) {
    using L = LeanSmem<HEADS>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);   // (an offset, so that the compiler knows the address space)
    const uint32_t sm_u32 = warp_uniform(smem_u32(sm));
    __shared__ __align__(8) uint64_t bars[B_BARS + (HOOKS ? 1 : 0)];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) LeanScratch ps2[HEADS];
    __shared__ float squares[2][HEADS][128];      // with L2 normalisation: of the rows of [K;Q], per k-half

    const int tid = threadIdx.x, warp = static_cast<int>(warp_uniform(tid >> 5)), lane = tid & 31;
    const int h = HEADS == 2 ? warp >> 2 : 0;     // which head of the pair this half of the CTA prepares
    const int role = warp & 3;                    // and the warp's quadrant of the accumulator's lanes
    LeanScratch& ps = ps2[h];
    const float scale0 = rsqrtf(static_cast<float>(kD));
    const unsigned rep = p.Hv / p.Hq, groups = p.Hv / HEADS;
    uint8_t* t2tile = sm + L::T2 + h * kTriBytes;
    uint8_t* ptile = sm + L::KQ + 8192 + h * 16384;
    LeanExchange& ex = *reinterpret_cast<LeanExchange*>(sm + L::EX + h * sizeof(LeanExchange));
    uint8_t* kq = sm + L::KQ;
    const uint32_t bar0 = smem_u32(bars);
    auto cb = [&](uint32_t i) { return bar0 + 8u * i; };

    // Persistent CTA: items blockIdx.x, blockIdx.x + gridDim.x, ...; the head group index is the fastest, so the groups
    // that share a qk head are prepared at about the same time.
    int late = 0;                                 // code of this thread's first wait that ran out
    auto wait = [&](uint32_t bar, uint32_t item) {
        if (mbar_wait_compact(cb(HOOKS && p.dbg == kDbgLaneWaits && tid == 5 ? B_NEVER : bar), item & 1)) return true;
        if (late == 0) late = bar <= B_Q ? kDevTimeoutTma : kDevTimeoutMma;
        return false;
    };
    // Each lane counts its own tries.  The warp goes on, or leaves, as one: a lane that left by itself would be at the CTA's last barrier while the others
    // wait for it, without a limit, in the next instruction that needs the whole warp.
    auto agreed = [](bool ok) { return __all_sync(0xffffffffu, ok) != 0; };
    auto decode = [&](unsigned n) {
        LeanItem x{};
        const unsigned c = n / groups, grp = n - c * groups;
        unsigned seq, t, len, nt;
        size_t tile0;
        if (p.pk_chunk) {
            const int2 m = p.pk_chunk[c];
            seq = m.x;
            t = m.y;
            const int cu0 = p.pk_cu[seq];
            len = p.pk_cu[seq + 1] - cu0;
            nt = (len + kChunk - 1) / kChunk;
            x.b = 0;
            x.s0 = cu0 + t * kChunk;
            x.tok0 = x.s0;
            tile0 = static_cast<size_t>(c - t) * p.Hv;
        } else {
            seq = c / NT;
            t = c - seq * NT;
            len = p.S;
            nt = NT;
            x.b = seq;
            x.s0 = t * kChunk;
            x.tok0 = static_cast<size_t>(seq) * p.S + x.s0;
            tile0 = static_cast<size_t>(seq) * NT * p.Hv;
        }
        x.hv = HEADS * grp + h;
        x.hq = HEADS * grp / rep;
        x.valid = min(kChunk, static_cast<int>(len - t * kChunk));
        x.tile = tile0 + static_cast<size_t>(x.hv) * nt + t;
        return x;
    };
    auto load_k = [&](const LeanItem& x) {   // one thread; announces the bytes of Q as well
        mbar_arrive_expect_tx_a(cb(B_K), 2 * 8192);
        mbar_arrive_expect_tx_a(cb(B_Q), 2 * 8192);
        tma_load_4d_a(sm_u32 + L::KQ, &tm_k, cb(B_K), 0, x.hq, x.s0, x.b);
        tma_load_4d_a(sm_u32 + L::KQ + 16384, &tm_k, cb(B_K), 64, x.hq, x.s0, x.b);
    };
    auto load_q_half = [&](const LeanItem& x, int half) {
        tma_load_4d_a(sm_u32 + L::KQ + 8192 + half * 16384, &tm_q, cb(B_Q), 64 * half, x.hq, x.s0, x.b);
    };
    // Rows of padding tokens count as zeros.  In a packed batch they are the next sequence's (elsewhere the copies leave zeros): cleared by one warp before the product
    // (in the masks' registers instead, code that every role carried: 4 x 1999 tokens with L2 normalisation 35.6 us alone, now 34.3; 64 x 4096 726 / 719).
    auto clear_tail = [&](int valid) {
        uint32_t at = sm_u32 + L::KQ;
        asm volatile("" : "+r"(at));              // (its addresses are computed here, not kept in registers across the items' loop)
        at += ((lane >> 3) & 3) * 8192 + (lane & 7) * 16;
#pragma unroll 1
        for (int row = valid; row < kChunk; ++row) asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(at + row * 128), "r"(0) : "memory");
        fence_proxy_async_smem();
        __syncwarp();
    };
    auto issue_product = [&](uint32_t d) {   // raw K K^T (lanes 0-63) and Q K^T (lanes 64-127), shared by the heads
        tc_fence_after_sync();
        constexpr uint32_t idesc = umma_idesc_bf16(128, 64, MAJOR_K, MAJOR_K);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const uint64_t ad = umma_smem_desc(sm_u32 + L::KQ + (ks >> 2) * 16384 + (ks & 3) * 32, 16, 1024, SWZ_128B);
            umma_bf16_ss(d, ad, ad, idesc, ks > 0);
        }
        umma_commit_a(cb(B_MMA));
    };

    const bool prof_on = GDN_DIAG(p.prof != nullptr && tid == 0 && blockIdx.x == 0);
    long long prof_acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    long long prof_t = prof_on ? clock64() : 0, prof_n = 0;
#define GDN_PHASE(n)                                   \
    if (prof_on) {                                     \
        const long long now_ = clock64();              \
        prof_acc[n] += now_ - prof_t;                  \
        prof_t = now_;                                 \
    }

    if (warp == 2 && elect_one()) {
        for (uint32_t i = 0; i < B_BARS; ++i) {
            const uint32_t count = i == B_ENT ? 4 * HEADS : i == B_SQ ? 3 * HEADS : i == B_TAB || i == B_TAB + 1 ? (p.l2norm ? 2 : 1)
                                   : i >= B_PAIR && i < B_LOW ? 2 : 1;
            mbar_init(&bars[i], count);
        }
        if (HOOKS) mbar_init(&bars[B_NEVER], 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_slot, kLeanTmemCols);
        tmem_relinquish();
    }
    grid_dependency_wait();   // launched ahead of the end of the kernel before: no memory is touched above
    if (tid == 0 && p.clear_status && blockIdx.x == 0) *p.status = 0;
    // Role 2 looks ahead, two items.
    auto look = [&](unsigned item) {
        const LeanItem x = decode(blockIdx.x + item * gridDim.x);
        if (lane == 0) ps.item[item & 3] = x;
        __syncwarp();
    };
    const unsigned count = (num_items - 1 - blockIdx.x) / gridDim.x + 1;
    if (role == 3 || (role == 2 && count > 1)) look(3 - role);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = warp_uniform(tmem_slot);
    if (HOOKS && p.dbg == kDbgLaneGivesUp && tid == 5) late = kDevTimeoutTma;

    // Items of a CTA are counted from 0; `item & 1` names the buffer of its tables, its accumulator and the parity of its barriers.  A wait names a
    // parity, so the next completion of its barrier has to need something behind the wait: that of K, Q, MMA and TAB an arrival on ENT by each
    // warp that waits for them, the others an arrival by the one that waits.
    auto enter = [&](unsigned item) {
        const bool ok = wait(B_TAB + h, item) && wait(B_MMA, item);
        tc_fence_after_sync();
        if (ok && lane == 0) mbar_arrive_a(cb(B_ENT));
        return agreed(ok);
    };
    auto tables = [&](unsigned item) {
        const uint32_t buf = item & 1;
        return MaskTables{ps.gam[buf], p.l2norm ? ps.gcol[buf] : ps.gam[buf], p.l2norm ? ps.brow[buf] : ps.bet[item & 3], ps.t16[buf], ps.t32[buf]};
    };
    // L2 normalisation.  Squares of the next item's rows, of one k-half (of both where there is one head), by the warps of its head's diagonal blocks: role 0
    // K's, role 1 Q's.
    auto row_squares = [&](unsigned item) {
        if (!agreed(wait(role == 0 ? B_K : B_Q, item))) return false;
#pragma unroll 1
        for (int e = 0; e < 2; ++e) {
            const int row = 64 * role + 32 * e + lane;
            float ss = lean_row_squares(kq + h * 16384, row);
            if (HEADS == 1) ss += lean_row_squares(kq + 16384, row);
            squares[item & 1][h][row] = ss;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_a(cb(B_SQ));
        return true;
    };
    // What is made of them behind role 3's gates: role 3 the keys' share of the tables, role 2 the queries'.
    auto norms = [&](unsigned item) {
        const uint32_t buf = item & 1;
        if (!agreed(wait(B_SQ, item))) return false;
        const LeanItem& x = ps.item[item & 3];
        float* vec = ws.vec + x.tile * 256;
#pragma unroll 1
        for (int e = 0; e < 2; ++e) {
            const int tok = 32 * e + lane, row = 64 * (3 - role) + tok;
            lean_l2norm_fold(ps, item, role == 2, tok, HEADS == 1 ? squares[buf][0][row] : squares[buf][0][row] + squares[buf][HEADS - 1][row], scale0, vec, x.valid);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_a(cb(B_TAB + h));
        return true;
    };

    if (role < 2) {
        // ------------------------------- diagonal blocks of the inverse --------------------------------------------------
        bool go = !p.l2norm || row_squares(0);
#pragma unroll 1
        for (unsigned item = 0; go && item < count; ++item) {
            if (!enter(item)) break;
            GDN_PHASE(0)
            const uint32_t buf = item & 1;
            const LeanItem& x = ps.item[item & 3];
            auto ready = [&]() {                           // (the next item's squares while the exchange is still read)
                return (!p.l2norm || item + 1 == count || row_squares(item + 1)) && (item == 0 || agreed(wait(B_EXE + h, item - 1)));
            };
            go = lean_diagonal(tables(item), ps.bet[item & 3], p.l2norm != 0, ws.meta ? &ps.bound[buf][role] : nullptr, tmem + buf * 64, role, lane, ex,
                               t2tile + 4096 * role, &tm_t2, static_cast<int>(x.tile * kChunk), cb(B_EXF + h), ready);
            tc_fence_before_sync();
            GDN_PHASE(1)
            ++prof_n;
        }
    } else {
        // ------------------------------- role 2: tiles and product of `item`, role 3: its gates and tables; P of the one before, rows 0-31 and 32-63; T'' of
        //                                 the one before that, below the diagonal blocks, left and right half.  (One piece of code for both: what they share compiled
        //                                 twice is 9 KB more for the instruction cache, 64 x 4096 tokens 744 us alone, now 726, 4 x 1999 with L2 normalisation 38.6, now 35.6.)
        LaneGates gates{0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (unsigned item = 0; item < count + 2; ++item) {
            const bool more = item < count, one = item > 0 && item <= count;
            const LeanItem &next = ps.item[item & 3], &x = ps.item[(item - 1) & 3], &y = ps.item[(item - 2) & 3];
            if (one && !enter(item - 1)) break;
            if (more) {
                if (role == 3) gates = lean_load_gates<GATE_F32>(p, next.tok0, next.hv, next.valid, lane);
                else if (warp == 2 && elect_one()) load_k(next);
            }
            __syncwarp();
            if (one) {
                lean_mask_P(tables(item - 1), p.l2norm ? ps.prow[(item - 1) & 1] : nullptr, scale0, tmem + ((item - 1) & 1) * 64, role - 2, lane, ptile);
                tc_fence_before_sync();
                fence_proxy_async_smem();
                __syncwarp();
                if (elect_one()) {
                    const int row = static_cast<int>(x.tile * kChunk) + 32 * (role - 2);
                    tma_store_2d(&tm_p, ptile + 2048 * (role - 2), 0, row);
                    if (role == 3) tma_store_2d(&tm_p, ptile + 4096, 32, row);
                    tma_store_commit();
                }
                __syncwarp();
                if (role == 2 && item + 1 < count) look(item + 1);
            }
            if (item > 0) {
                if (elect_one()) {
                    tma_store_wait_read();           // (role 2: and T'' below the diagonal blocks of the item before that)
                    mbar_arrive_a(cb(B_PAIR + h));
                }
                __syncwarp();
            }
            if (role == 3 && more) {
                if (one && !agreed(wait(B_ENT, item - 1))) break;   // (nobody reads the tables any more)
                lean_gates(ps, item, gates, p.gate_act != 0, scale0, p.l2norm ? nullptr : ws.vec + next.tile * 256, lane);
                __syncwarp();
                if (lane == 0) mbar_arrive_a(cb(p.l2norm ? B_SQ : B_TAB + h));
            }
            if (item > 0 && !agreed(wait(B_PAIR + h, item - 1))) break;   // (T'' below the diagonal blocks has left its place; what role 2 looked up)
            if (role == 2 && more && elect_one()) {
                load_q_half(next, h);
                if (HEADS == 1) load_q_half(next, 1);
            }
            if (item > 1) {
                if (!agreed(wait(B_EXF + h, item - 2))) break;
                if (role == 2 && ws.meta && lane == 0) {
                    ws.meta[2 * y.tile] = y.decay;
                    ws.meta[2 * y.tile + 1] = y.gates_ok ? fmaxf(ps.bound[item & 1][0], ps.bound[item & 1][1]) : INFINITY;
                }
                lean_below(ps.bet[(item - 2) & 3], role - 2, lane, ex, t2tile + 2048, cb(B_EXE + h));
                if (role == 3) {
                    if (lane == 0) mbar_arrive_a(cb(B_LOW + h));
                } else {
                    if (!agreed(wait(B_LOW + h, item - 2))) break;
                    if (elect_one()) {
                        tma_store_2d(&tm_t2, t2tile + 2048, 0, static_cast<int>(y.tile * kChunk) + 32);
                        tma_store_commit();
                    }
                }
                __syncwarp();
            }
            if (more) {
                if (warp == 2) {
                    // (ENT: nobody reads the accumulator any more)
                    if (!agreed((!one || wait(B_ENT, item - 1)) && wait(B_K, item) && wait(B_Q, item))) break;
                    if (p.pk_chunk && next.valid < kChunk) clear_tail(next.valid);
                    tc_fence_after_sync();
                    if ((!HOOKS || one || p.dbg != kDbgNoProduct) && elect_one()) issue_product(tmem + (item & 1) * 64);
                    __syncwarp();
                }
                if (p.l2norm && !norms(item)) break;
            }
        }
    }
#undef GDN_PHASE
    if (prof_on) {
        for (int k = 0; k < 8; ++k) p.prof[k] = prof_acc[k];
        p.prof[15] = prof_n;
    }
    if (late) atomicCAS(p.status, 0, late);       // (each lane counts its own tries)
    // Only now may the chain kernel's CTAs start (and set up while the last CTAs of this grid finish): let in earlier, they
    // pile up two to an SM on the SMs that this grid leaves first while others stay empty.  (And never in front of this kernel's own wait: the chain
    // reads K, V and the initial state as soon as it starts.)
    grid_launch_dependents();
    if (elect_one()) tma_store_wait_all();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kLeanTmemCols);
}

}  // namespace

int launch_prepare_lean(const Problem& p, const Workspace& ws, const TileMaps& maps, cudaStream_t stream) {
    auto map = [](const unsigned char* m) -> const CUtensorMap& { return *reinterpret_cast<const CUtensorMap*>(m); };
    const int NT = (p.S + kChunk - 1) / kChunk;
    const long long chunks = p.pk_chunk ? p.pk_chunks : static_cast<long long>(p.B) * NT;
    auto go = [&](auto kernel, int heads, uint32_t smem, int per_sm) -> int {
        const long long items = chunks * (p.Hv / heads);
        if (items >= (1ll << 31)) return GDN_ERR_BAD_ARGUMENT;
        const long long max_ctas = static_cast<long long>(per_sm) * sm_count();
        const unsigned grid = static_cast<unsigned>(items < max_ctas ? items : max_ctas);
        if (allow_smem(reinterpret_cast<const void*>(kernel), smem)) return GDN_ERR_CUDA;
        const cudaError_t e = launch_dependent(kernel, dim3(grid), dim3(128 * heads), smem, stream, false, map(maps.q), map(maps.k), map(maps.p), map(maps.t2), p, ws,
                                               static_cast<unsigned>(NT), static_cast<unsigned>(items));
        return e == cudaSuccess ? GDN_OK : GDN_ERR_CUDA;
    };
    auto pick = [&](auto heads, auto hooks) -> int {
        constexpr int H = decltype(heads)::value;
        constexpr bool K = decltype(hooks)::value;
        return p.gate_f32 ? go(gdn_prepare_lean_kernel<H, true, K>, H, LeanSmem<H>::kDynamic, kLeanCtasPerSm<H>)
                          : go(gdn_prepare_lean_kernel<H, false, K>, H, LeanSmem<H>::kDynamic, kLeanCtasPerSm<H>);
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    if ((p.Hv / p.Hq) % 2 == 0) return p.dbg ? pick(Two{}, std::true_type{}) : pick(Two{}, std::false_type{});
    return p.dbg ? pick(One{}, std::true_type{}) : pick(One{}, std::false_type{});
}

}  // namespace gdn
