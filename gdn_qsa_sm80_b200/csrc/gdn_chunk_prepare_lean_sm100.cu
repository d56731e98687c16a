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
// What bounds it is latency: an item is a chain of dependent phases (product, mask, triangular inverse, T''), so what
// counts is how many items an SM has in flight.  A and T share one fp32 array (gdn_prep_lean_device.cuh) and K / Q are
// dead after the product, so a CTA needs 73 KB and 80 registers and three of them (24 warps) fit an SM; the next item's
// K is loaded as soon as this item's product is done, its Q as soon as P's staging tiles (in Q's place) have been read
// by their TMA store, and its product is issued, into a second accumulator, before this item's T'' is written.
// Stands in for the reference's gdn_prepare_kernel (csrc/gdn_chunk/gdn_kernel.cu:343-710).
#include <cuda.h>

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
                                                         //   P staging of head h in Q's rows of k-half h once the product is done
    static constexpr uint32_t AT = 32768;                // A, then T, fp32 64 x 68, of head h at AT + h * 17408; then its T'' staging
    static constexpr uint32_t kBytes = AT + HEADS * 17408;
    static constexpr uint32_t kDynamic = kBytes + 1024;
    static_assert(AT % 1024 == 0 && 17408 % 1024 == 0, "UMMA / TMA tiles must be 1024-byte aligned");
};
constexpr uint32_t kLeanTmemCols = 128;                  // two accumulators of 64 columns
template <int HEADS>
constexpr int kLeanCtasPerSm = HEADS == 2 ? 3 : 4;

template <int HEADS, bool GATE_F32>
__global__ void __launch_bounds__(128 * HEADS, kLeanCtasPerSm<HEADS>)
gdn_prepare_lean_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_t2, Problem p,
                        Workspace ws, unsigned NT, unsigned num_items) {
    using L = LeanSmem<HEADS>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sm_u32 = warp_uniform(smem_u32(sm));
    __shared__ __align__(8) uint64_t bar_tma;
    __shared__ __align__(8) uint64_t bar_mma;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) LeanScratch ps2[HEADS];
    __shared__ float squares[HEADS][128];         // with L2 normalisation: of the rows of [K;Q], per k-half

    const int tid = threadIdx.x, warp = static_cast<int>(warp_uniform(tid >> 5)), lane = tid & 31;
    const int h = HEADS == 2 ? tid >> 7 : 0;      // which head of the pair this half of the CTA prepares
    const int htid = tid & 127, hwarp = warp & 3, i = htid & 63;
    const PrepCtx ctx{htid, 1 + h};               // the half's own thread numbering and named barrier
    LeanScratch& ps = ps2[h];
    const float scale0 = rsqrtf(static_cast<float>(kD));
    const unsigned rep = p.Hv / p.Hq, groups = p.Hv / HEADS;
    float* At = reinterpret_cast<float*>(sm + L::AT + h * 17408);
    uint8_t* t2tile = sm + L::AT + h * 17408;
    uint8_t* ptile = sm + L::KQ + 8192 + h * 16384;
    uint8_t* kq = sm + L::KQ;

    // Persistent CTA: items blockIdx.x, blockIdx.x + gridDim.x, ...; the head group index is the fastest, so the groups
    // that share a qk head are prepared at about the same time.
    struct Item { int b, hv, hq, s0, valid; size_t tok0, tile; };
    int late = 0;                                 // code of this thread's first wait that ran out
    auto wait = [&](uint64_t* bar, uint32_t parity, int code) {   // (mbar_wait: 16 x 2048 tokens 125.8 us against 123.7, 8192 36.8 / 36.1)
        if (mbar_wait_compact(smem_u32(bar), parity)) return true;
        if (late == 0) late = code;
        return false;
    };
    auto decode = [&](unsigned n) {
        Item x;
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
    auto load_k = [&](const Item& x) {   // one thread; announces the bytes of Q as well
        mbar_arrive_expect_tx(&bar_tma, 4 * 8192);
        tma_load_4d(kq + 0, &tm_k, &bar_tma, 0, x.hq, x.s0, x.b);
        tma_load_4d(kq + 16384, &tm_k, &bar_tma, 64, x.hq, x.s0, x.b);
    };
    auto load_q_half = [&](const Item& x, int half) {
        tma_load_4d(kq + 8192 + half * 16384, &tm_q, &bar_tma, 64 * half, x.hq, x.s0, x.b);
    };
    auto issue_product = [&](uint32_t d) {   // raw K K^T (lanes 0-63) and Q K^T (lanes 64-127), shared by the heads
        tc_fence_after_sync();
        constexpr uint32_t idesc = umma_idesc_bf16(128, 64, MAJOR_K, MAJOR_K);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
            const uint64_t ad = umma_smem_desc(sm_u32 + L::KQ + (ks >> 2) * 16384 + (ks & 3) * 32, 16, 1024, SWZ_128B);
            umma_bf16_ss(d, ad, ad, idesc, ks > 0);
        }
        umma_commit(&bar_mma);
    };

    auto store_tri = [&](const void* map, const uint8_t* src, size_t tile) {   // the three blocks of a triangular tile
        const int row = static_cast<int>(tile * kChunk);
        tma_store_2d(map, src, 0, row);
        tma_store_2d(map, src + 2048, 0, row + 32);
        tma_store_2d(map, src + 4096, 32, row + 32);
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

    if (tid == 0) {
        mbar_init(&bar_tma, 1);
        mbar_init(&bar_mma, 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_slot, kLeanTmemCols);
        tmem_relinquish();
    }
    grid_dependency_wait();   // launched ahead of the end of the kernel before: no memory is touched above
    unsigned n = blockIdx.x;
    Item cur = decode(n);
    if (tid == 0) {
        if (p.clear_status && n == 0) *p.status = 0;
        load_k(cur);
        load_q_half(cur, 0);
        load_q_half(cur, 1);
    }
    LaneGates gates{0.f, 0.f, 0.f, 0.f};
    if (hwarp == 0) gates = lean_load_gates<GATE_F32>(p, cur.tok0, cur.hv, cur.valid, lane);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = warp_uniform(tmem_slot);
    const uint32_t lane_base = static_cast<uint32_t>(hwarp) * 32u;   // (warp % 4) * 32: the warp's TMEM lane quadrant
    uint32_t ph = 0;            // parity of both barriers: one load and one product per item
    bool ok = true;
    if (p.dbg == kDbgLaneGivesUp && tid == 5) late = kDevTimeoutTma;
    if (warp == 0) {
        ok = wait(&bar_tma, 0, kDevTimeoutTma);
        if (ok && p.dbg != kDbgNoProduct && elect_one()) issue_product(tmem);
    }

    for (; n < num_items; n += gridDim.x) {
        const size_t tile = cur.tile;
        float* vec = ws.vec + tile * 256;
        const uint32_t acc = tmem + ph * 64;
        const unsigned nn = n + gridDim.x;
        const bool more = nn < num_items;
        // the gate cumsum and the decay tables need nothing from the tiles: they run while the product does
        if (hwarp == 0) {
            if (elect_one()) tma_store_wait_read();   // (the lane that issued it) the previous item's T'' has left the array A goes into
            lean_gates(ps, gates, p.gate_act != 0, scale0, p.l2norm ? ps.vec : vec, lane);
        }
        ctx.sync();
        if (p.l2norm) {
            // The other half reads this half's sums of the item before in lean_l2norm_fold, and no barrier of the CTA lies behind that: this
            // wait does.  It needs the bytes of both halves of Q, which each half requests behind its own fold.
            ok = wait(&bar_tma, ph, kDevTimeoutTma);
            squares[h][htid] = lean_row_squares(kq + h * 16384, htid);
            if (HEADS == 1) squares[h][htid] += lean_row_squares(kq + 16384, htid);
        }
        GDN_PHASE(0)
        ok = wait(&bar_mma, ph, kDevTimeoutMma) && ok;
        ok = __syncthreads_and(ok);
        if (!ok) break;
        tc_fence_after_sync();
        if (p.l2norm) lean_l2norm_fold(ps, HEADS == 1 ? squares[0][htid] : squares[0][htid] + squares[HEADS - 1][htid], vec, cur.valid, ctx);
        GDN_PHASE(1)
        Item nxt = cur;
        if (more) {
            nxt = decode(nn);
            if (warp == 0 && elect_one()) load_k(nxt);
            if (hwarp == 0) gates = lean_load_gates<GATE_F32>(p, nxt.tok0, nxt.hv, nxt.valid, lane);
        }
        {   // mask epilogue: thread = row i = TMEM lane
            const bool low_rows = (hwarp & 1) == 0;          // rows 0-31: columns 32-63 lie above the diagonal
            if (hwarp < 2) {   // A = tril(beta_i * decay * K K^T, -1), fp32, and at once the inverse of the warp's 32x32 block
                const float ksq = lean_mask_row_A<HEADS == 2>(ps, p.l2norm != 0, tmem_addr(acc, lane_base, 0), i, low_rows, cur.valid, At);
                if (ws.meta) {
                    const float bound = lean_bound_of_rows(ps, p.l2norm != 0, i, ksq);
                    if (lane == 0) ps.bound[hwarp] = bound;
                }
                __syncwarp();
                lean_invert_diag32(At, hwarp, lane);
            } else {           // P = tril(scale * decay * Q K^T), bf16, into its staging tile in Q's place
                lean_mask_row_P(ps, p.l2norm != 0, scale0, tmem_addr(acc, lane_base, 0), i, low_rows, cur.valid, ptile);
                fence_proxy_async_smem();
                named_bar_sync(3 + h, 64);
                if (hwarp == 2 && elect_one()) {
                    store_tri(&tm_p, ptile, tile);
                    tma_store_commit();
                    if (more) {
                        tma_store_wait_read();
                        load_q_half(nxt, h);
                        if (HEADS == 1) load_q_half(nxt, 1);
                    }
                }
                __syncwarp();
            }
        }
        GDN_PHASE(2)
        tc_fence_before_sync();
        ctx.sync();
        GDN_PHASE(3)
        if (ws.meta && htid == 0) {
            ws.meta[2 * tile] = ps.gam[kChunk - 1] * (1.f / kLog2e);
            ws.meta[2 * tile + 1] = ps.gates_ok ? fmaxf(ps.bound[0], ps.bound[1]) : INFINITY;
        }
        lean_finish_T2(At, ps.bet, t2tile, ctx);
        GDN_PHASE(4)
        if (warp == 3 && more) {   // the next item's product, into the other accumulator (read last an item ago)
            ok = wait(&bar_tma, ph ^ 1, kDevTimeoutTma);
            if (ok && elect_one()) issue_product(tmem + (ph ^ 1) * 64);
            __syncwarp();
        }
        GDN_PHASE(5)
        fence_proxy_async_smem();
        ctx.sync();
        if (hwarp == 0 && elect_one()) {
            store_tri(&tm_t2, t2tile, tile);
            tma_store_commit();
        }
        GDN_PHASE(6)
        ++prof_n;
        cur = nxt;
        ph ^= 1;
    }
#undef GDN_PHASE
    if (prof_on) {
        for (int k = 0; k < 8; ++k) p.prof[k] = prof_acc[k];
        p.prof[15] = prof_n;
    }
    if (late) atomicCAS(p.status, 0, late);       // (each lane counts its own tries)
    // Only now may the chain kernel's CTAs start (and set up while the last CTAs of this grid finish): let in earlier, they
    // pile up two to an SM on the SMs that this grid leaves first while others stay empty.
    grid_launch_dependents();
    if ((hwarp & 1) == 0 && elect_one()) tma_store_wait_all();
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
    if ((p.Hv / p.Hq) % 2 == 0) {
        return p.gate_f32 ? go(gdn_prepare_lean_kernel<2, true>, 2, LeanSmem<2>::kDynamic, kLeanCtasPerSm<2>)
                          : go(gdn_prepare_lean_kernel<2, false>, 2, LeanSmem<2>::kDynamic, kLeanCtasPerSm<2>);
    }
    return p.gate_f32 ? go(gdn_prepare_lean_kernel<1, true>, 1, LeanSmem<1>::kDynamic, kLeanCtasPerSm<1>)
                      : go(gdn_prepare_lean_kernel<1, false>, 1, LeanSmem<1>::kDynamic, kLeanCtasPerSm<1>);
}

}  // namespace gdn
