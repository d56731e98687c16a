// Token-by-token gated delta rule for very short sequences (decode: one or a few new tokens per sequence on top
// of a stored state).  Same recurrence as the reference's recurrent torch definition
// (gdn_qsa_sm80/reference/gdn_chunk_ref.py:133-141), fp32 throughout:
//     S <- exp(g) S ;  delta = beta (v - S^T k) ;  S <- S + k delta^T ;  o = S^T q / sqrt(D)
// With one token the operator is nothing but a read and a write of the 64 KB state per (batch, value head), so the
// kernel is laid out for HBM.  The value columns of a state are independent, so the unit of work is a tile of
// [128 rows][32 columns] (16 KB): two warps own one, 64 values per thread, and a persistent CTA streams tiles through a
// ring of three TMA stages - the loads of the next tiles are in flight while this one is computed and the one before
// leaves by TMA store, which the load-compute-store phases of one CTA per state could not do (75 % of the copy bandwidth).  (A ring of two that
// writes states has no load in flight beside a computation: the next tile's place is the one whose store has to be read first.  The other CTAs of the SM fill that.)
// The tile is 128-byte swizzled; a lane owns eight pairs of rows and the four columns of a chunk, so that a 16-byte access of eight
// lanes covers all banks, a pair's two values of k arrive in one word, and the column sums a token needs (S^T k, S^T q) are three
// shuffles: no barrier.  With several tokens a tile what bounds it is the two warps' serial run through the tokens, not HBM (64 sequences
// of 4: DRAM 40 % busy, issue slots 37 % with six compute warps an SM): two multiply-adds in one instruction (f32x2).  32 heads, before
// and after: 8 sequences of 4 tokens 14.5 -> 12.7 us, 256 of 4 277 -> 241, 64 of 8 121 -> 111; 64 of one 47 us, 86 % of the copy bandwidth.
//   GROUPS = 1: a CTA of two compute warps and a producer warp, four per SM (from five tokens on, whose vectors take room in every stage,
//   three, or four with a ring of two: two_stages); 32 states give 128 CTAs.
//   PACKED: the sequences of a packed batch that have at most kDecodeMaxTokens tokens, of any lengths, found through a table.
//   GROUPS = 4: the four tiles of a state in one CTA, for the gated normalisation of the output rows (their sum of squares
//   needs all 128 columns: one barrier a token), which then costs no launch and no pass over the rows of its own.  One token: a ring of
//   three, one CTA per SM (HBM-bound).  Several: its barriers and instructions bound it, and two CTAs per SM with one stage each fill
//   each other's waits where there are states for both (8 sequences of 4 tokens 19.1 -> 15.7 us, 64 of 4 111 -> 94, 8 of 8 38.8 -> 26.9;
//   at 96 registers a thread, for which the compiler keeps 88 bytes of it in local memory).
#include <cuda.h>

#include "../../include/gdn_chunk_sm100.h"
#include "gdn_common.cuh"
#include "gdn_launch.cuh"
#include "ptx_sm100.cuh"

namespace gdn {
namespace {

constexpr int kDecTokens = 8;                      // tokens whose vectors travel through the ring (later ones: global loads)
constexpr int kDecTimeoutFull = 0x601, kDecTimeoutEmpty = 0x602;

struct DecodeGate {                                // gated normalisation of the output rows (z null: none)
    const __nv_bfloat16* z;
    const __nv_bfloat16* weight;
    float eps;
};

template <bool GATE_F32>
__device__ __forceinline__ float dec_gate(const void* p, size_t idx) {
    if (GATE_F32) return static_cast<const float*>(p)[idx];
    return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[idx]);
}
__device__ __forceinline__ float sum_rows(float x) {   // over the eight lanes that share a column
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    return x;
}

// bytes of the token area of one stage (a box's destination: a multiple of 128): k, q rows, 32 columns of v; g and beta there too, or, `apart`, behind all stages'
// areas (four tokens: 128 bytes a stage less, which fits a fourth CTA; the other forms are 1 to 3 % faster with them inside)
constexpr uint32_t kDecGateBytes = 2 * kDecTokens * 4;
__host__ __device__ constexpr uint32_t dec_token_bytes(int nt, bool apart) { return (nt * (256 + 256 + 64) + (apart ? 0 : kDecGateBytes) + 127) & ~127u; }

// Where the vectors of several tokens come from: a box of nt rows each, three copies a tile instead of three a token, where a CTA has
// more than one tile (32 heads, 18 sequences of 2 tokens 12.5 us, by rows 13.7; 32 of 2 22.0, 23.3; of 3 and more tokens the same within
// 2 %).  Smaller calls of up to four tokens are as long as the host takes to encode the maps and launch (one sequence of 2 to 4 tokens
// 5.7 us, by rows 5.1; of 6, whose kernel is as long as that, 5.8 and 6.5).  A packed batch's sequences have tokens of their own number
// each, and a box of the longest one's rows for all of them is slower (256 sequences of one token but one of 8: 174 us, by rows 164; of
// 1 to 8: 278, 271).
// ONE_ROW is ROWS for a single token: without the loop over tokens 8 sequences of one token take 7.0 us, with it 7.4.
enum class Fetch { ONE_ROW, ROWS, BOXES };
template <Fetch FETCH>
struct TokenMaps {};
template <>
struct TokenMaps<Fetch::BOXES> {
    CUtensorMap q, k, v;
};

__host__ __device__ constexpr bool gates_apart(int groups, int stages, Fetch fetch) { return fetch == Fetch::BOXES && (groups == 1 || stages == 1); }
__host__ __device__ constexpr int dec_ctas_per_sm(int groups, int stages) { return groups == 1 ? 4 : (stages == 3 ? 1 : 2); }

// Shared memory of a CTA, and the CTAs for which an SM's 228 KB suffice: each takes 1 KB more, and its own in steps of 128 bytes.
constexpr uint32_t dec_static_bytes(int groups, int stages, bool packed) {
    return (2 * 8 * groups * stages + (groups == 4 ? 64 : 0) + (packed ? 16 * stages : 0) + 4 + 15) & ~15;
}
constexpr uint32_t dec_dynamic_bytes(int groups, int stages, int nt, bool apart) {
    return groups * stages * (16384 + dec_token_bytes(nt, apart) + (apart ? kDecGateBytes : 0)) + 1024;
}
constexpr int dec_fit(uint32_t dynamic_bytes, uint32_t static_bytes) {
    return static_cast<int>(228 * 1024 / (((dynamic_bytes + static_bytes + 127) & ~127u) + 1024));
}
static_assert(dec_fit(dec_dynamic_bytes(1, 3, 4, true), dec_static_bytes(1, 3, false)) == 4, "four tokens: four CTAs of three stages an SM, to the byte");

template <int GROUPS, bool GATE_F32, bool PACKED, int STAGES, Fetch FETCH>
__global__ void __launch_bounds__(GROUPS * 64 + 32, dec_ctas_per_sm(GROUPS, STAGES))
gdn_decode_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out,
                  const __grid_constant__ TokenMaps<FETCH> maps, const __grid_constant__ Problem p, const __grid_constant__ DecodeGate gate, int items, int nt) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[GROUPS][STAGES], empty[GROUPS][STAGES];
    __shared__ float ssq[2][GROUPS * 2];
    __shared__ int4 seq_of[PACKED ? STAGES : 1];   // (sequence, first token, tokens) of the stage's tile
    __shared__ int failed;
    // (every variable above that the form uses counts: how many CTAs an SM holds goes by it)
    static_assert(sizeof(full) + sizeof(empty) + (GROUPS == 4 ? sizeof(ssq) : 0) + (PACKED ? sizeof(seq_of) : 0) + sizeof(failed) <= dec_static_bytes(GROUPS, STAGES, PACKED));

    const int tid = threadIdx.x, warp = static_cast<int>(warp_uniform(tid >> 5)), lane = tid & 31;
    constexpr bool APART = gates_apart(GROUPS, STAGES, FETCH);
    const uint32_t tok_bytes = dec_token_bytes(nt, APART);
    // stage s of group g: the tile at (g * STAGES + s) * 16 KB; the token areas behind all tiles
    auto tile_of = [&](int g, int s) { return sm + (g * STAGES + s) * 16384; };
    auto tok_of = [&](int g, int s) { return sm + GROUPS * STAGES * 16384 + (g * STAGES + s) * tok_bytes; };
    auto gates_of = [&](int g, int s) {
        return reinterpret_cast<float*>(APART ? sm + GROUPS * STAGES * (16384 + tok_bytes) + (g * STAGES + s) * kDecGateBytes : tok_of(g, s) + nt * (256 + 256 + 64));
    };
    const int rep = p.Hv / p.Hq;

    if (tid == 0) {
        for (int g = 0; g < GROUPS; ++g)
            for (int s = 0; s < STAGES; ++s) {
                mbar_init(&full[g][s], 2);       // the copies (bytes) and the gates (written by the producer warp)
                mbar_init(&empty[g][s], 1);
            }
        failed = 0;
        fence_mbar_init();
    }
    __syncthreads();
    grid_dependency_wait();
    grid_launch_dependents();
    if (p.clear_status && blockIdx.x == 0 && tid == 0) *p.status = 0;

    // work items: GROUPS = 1: a tile (state, quarter); GROUPS = 4: a state
    const int first = blockIdx.x, step = gridDim.x;
    if (warp == GROUPS * 2) {
        // ------------------------------- producer ---------------------------------------------------------------------
        int n = 0;
        for (int it = first; it < items; it += step, ++n) {
            const int s = n % STAGES;
            int state = GROUPS == 1 ? it >> 2 : it, tokens = nt;
            const int b = state / p.Hv, h = state - b * p.Hv, hq = h / rep;
            size_t tok0 = static_cast<size_t>(b) * p.S;
            int4 seq = {};
            if (PACKED) {
                seq = p.pk_short[b];
                state = seq.x * p.Hv + h;
                tok0 = seq.y;
                tokens = seq.z;
            }
            bool ok = true;
            for (int g = 0; g < GROUPS && ok; ++g) {
                if (n >= STAGES) ok = mbar_wait(&empty[g][s], ((n / STAGES) - 1) & 1, p.status, kDecTimeoutEmpty);
                const int quarter = GROUPS == 1 ? it & 3 : g;
                if (ok && elect_one()) {
                    uint8_t* tk = tok_of(g, s);
                    mbar_arrive_expect_tx(&full[g][s], (p.h0 ? 16384 : 0) + tokens * (256 + 256 + 64));
                    if (p.h0) tma_load_2d(tile_of(g, s), &tm_in, &full[g][s], quarter * 32, state * kD);
                    if constexpr (FETCH == Fetch::BOXES) {
                        tma_load_4d(tk, &maps.k, &full[g][s], 0, hq, 0, b);
                        tma_load_4d(tk + nt * 256, &maps.q, &full[g][s], 0, hq, 0, b);
                        tma_load_4d(tk + nt * 512, &maps.v, &full[g][s], quarter * 32, h, 0, b);
                    } else {
                        for (int t = 0; t < (FETCH == Fetch::ONE_ROW ? 1 : tokens); ++t) {
                            const size_t row = (tok0 + t) * p.Hq + hq;
                            bulk_load_1d(tk + t * 256, p.k + row * kD, 256, &full[g][s]);
                            bulk_load_1d(tk + (nt + t) * 256, p.q + row * kD, 256, &full[g][s]);
                            bulk_load_1d(tk + nt * 512 + t * 64, p.v + ((tok0 + t) * p.Hv + h) * kD + quarter * 32, 64, &full[g][s]);
                        }
                    }
                }
                __syncwarp();
            }
            if (!ok) {   // the compute warps then stop waiting as well
                *const_cast<volatile int*>(&failed) = 1;
                break;
            }
            float x = 0.f;
            if (lane < 2 * kDecTokens && (lane & 7) < tokens)
                x = dec_gate<GATE_F32>(lane < kDecTokens ? p.g : p.beta, (tok0 + (lane & 7)) * p.Hv + h);
            for (int g = 0; g < GROUPS; ++g) {
                if (PACKED && lane == 0) seq_of[s] = seq;
                if (lane < 2 * kDecTokens) gates_of(g, s)[lane] = x;
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[g][s]);
            }
        }
    } else {
        // ------------------------------- compute: two warps per tile ------------------------------------------------------
        const int g = warp >> 1, half = warp & 1;             // half: which 16 of the tile's 32 columns
        // Lane l owns the row pairs 16 m + 2 rg, + 1 (one word of k and one of q each) of 16-byte chunk ch of the 128-byte rows.  In the
        // swizzled tile rows eight apart share their banks, so lanes 4-7 of a column group take a pair's rows in the other order.
        const int rg = lane & 7, ch = half * 4 + (lane >> 3), odd = rg >> 2;
        const int row0 = 2 * rg + odd, row1 = 2 * rg + 1 - odd;
        const uint32_t off0 = row0 * 128 + ((ch ^ (row0 & 7)) << 4), off1 = row1 * 128 + ((ch ^ (row1 & 7)) << 4);
        const uint32_t first_half = odd ? 0x3244u : 0x1044u, second_half = odd ? 0x1044u : 0x3244u;   // byte selectors: a pair's rows as fp32
        const float scale = rsqrtf(static_cast<float>(kD));
        // Slot of ssq: changes with every row of the CTA, across work items too.  Between a warp's reads of a slot and its next
        // write to it lies the other slot's barrier, which every warp reaches only after those reads.
        int slot = 0;
        int n = 0;
        for (int it = first; it < items; it += step, ++n) {
            const int s = n % STAGES;
            int state = GROUPS == 1 ? it >> 2 : it, tokens = p.S;
            const int quarter = GROUPS == 1 ? it & 3 : g;
            const int b = state / p.Hv, h = state - b * p.Hv, hq = h / rep;
            size_t tok0 = static_cast<size_t>(b) * p.S;
            // after a wait that ran out nobody waits again, but every warp keeps to the loop: its barriers count all of them
            const bool ok = !*const_cast<volatile int*>(&failed) &&
                            mbar_wait(&full[g][s], (n / STAGES) & 1, p.status, kDecTimeoutFull);
            if (!ok) *const_cast<volatile int*>(&failed) = 1;
            if (PACKED) {
                const int4 seq = seq_of[s];
                state = seq.x * p.Hv + h;
                tok0 = seq.y;
                tokens = ok ? seq.z : 0;          // (nothing may have been written there)
            }
            uint8_t* tile = tile_of(g, s);
            const uint8_t* tk = tok_of(g, s);
            float2 st[16][2];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float4 x = p.h0 ? *reinterpret_cast<const float4*>(tile + (i >> 1) * 2048 + (i & 1 ? off1 : off0)) : make_float4(0.f, 0.f, 0.f, 0.f);
                st[i][0] = make_float2(x.x, x.y);
                st[i][1] = make_float2(x.z, x.w);
            }
            const float* gates = gates_of(g, s);
            for (int t = 0; t < tokens; ++t) {
                const size_t tok = tok0 + t;
                // this lane's rows of k and q, its four values, the gates
                const uint32_t *kr, *qr;
                uint2 vraw;
                float gt, bt;
                if (t < nt) {
                    kr = reinterpret_cast<const uint32_t*>(tk + t * 256);
                    qr = reinterpret_cast<const uint32_t*>(tk + (nt + t) * 256);
                    vraw = *reinterpret_cast<const uint2*>(tk + nt * 512 + t * 64 + ch * 8);
                    gt = gates[t];
                    bt = gates[kDecTokens + t];
                } else {
                    kr = reinterpret_cast<const uint32_t*>(p.k + (tok * p.Hq + hq) * kD);
                    qr = reinterpret_cast<const uint32_t*>(p.q + (tok * p.Hq + hq) * kD);
                    vraw = *reinterpret_cast<const uint2*>(p.v + (tok * p.Hv + h) * kD + quarter * 32 + ch * 4);
                    gt = dec_gate<GATE_F32>(p.g, tok * p.Hv + h);
                    bt = dec_gate<GATE_F32>(p.beta, tok * p.Hv + h);
                }
                if (p.gate_act) {   // raw gates: g = -softplus(.), beta = sigmoid(.)
                    gt = gt > 20.f ? -gt : -log1pf(__expf(gt));
                    bt = 1.f / (1.f + __expf(-bt));
                }
                const float dec = __expf(gt);
                uint32_t kw[8], qw[8];
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    kw[m] = kr[rg + 8 * m];
                    qw[m] = qr[rg + 8 * m];
                }
                auto both = [&](const uint32_t (&w)[8], int i) {   // row i of the lane's sixteen, twice
                    const float x = __uint_as_float(__byte_perm(w[i >> 1], 0, i & 1 ? second_half : first_half));
                    return make_float2(x, x);
                };
                float rk = 1.f, rq = 1.f;
                if (p.l2norm) {
                    float kk = 0.f, qq = 0.f;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float x = both(kw, i).x, y = both(qw, i).x;
                        kk = fmaf(x, x, kk);
                        qq = fmaf(y, y, qq);
                    }
                    rk = rsqrtf(sum_rows(kk) + 1e-6f);
                    rq = rsqrtf(sum_rows(qq) + 1e-6f);
                }
                float2 kv[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};   // S^T k
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 x = both(kw, i);
                    kv[0] = fma2(st[i][0], x, kv[0]);
                    kv[1] = fma2(st[i][1], x, kv[1]);
                }
                const float f = dec * rk, bk = bt * rk;
                float2 dl[2];   // delta = beta (v - (decayed S)^T k), with the key's norm folded in
                dl[0].x = (__uint_as_float(vraw.x << 16) - sum_rows(kv[0].x) * f) * bk;
                dl[0].y = (__uint_as_float(vraw.x & 0xffff0000u) - sum_rows(kv[0].y) * f) * bk;
                dl[1].x = (__uint_as_float(vraw.y << 16) - sum_rows(kv[1].x) * f) * bk;
                dl[1].y = (__uint_as_float(vraw.y & 0xffff0000u) - sum_rows(kv[1].y) * f) * bk;
                const float2 dec2 = make_float2(dec, dec);
                float2 oa[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 x = both(kw, i), y = both(qw, i);
                    st[i][0] = fma2(x, dl[0], mul2(dec2, st[i][0]));
                    st[i][1] = fma2(x, dl[1], mul2(dec2, st[i][1]));
                    oa[0] = fma2(st[i][0], y, oa[0]);
                    oa[1] = fma2(st[i][1], y, oa[1]);
                }
                rq *= scale;
                uint2 pk;
                pk.x = pack_bf16x2(sum_rows(oa[0].x) * rq, sum_rows(oa[0].y) * rq);
                pk.y = pack_bf16x2(sum_rows(oa[1].x) * rq, sum_rows(oa[1].y) * rq);
                const size_t o_at = (tok * p.Hv + h) * kD + quarter * 32 + ch * 4;
                if (GROUPS == 4 && gate.z) {
                    // the row as bf16, normalised and gated (the arithmetic of gdn_output_gate_sm100.cu on the rounded row)
                    const float a[4] = {__uint_as_float(pk.x << 16), __uint_as_float(pk.x & 0xffff0000u),
                                        __uint_as_float(pk.y << 16), __uint_as_float(pk.y & 0xffff0000u)};
                    const uint2 zr = *reinterpret_cast<const uint2*>(gate.z + o_at);
                    const uint2 wr = *reinterpret_cast<const uint2*>(gate.weight + quarter * 32 + ch * 4);
                    float ss = a[0] * a[0];
                    ss = fmaf(a[1], a[1], ss); ss = fmaf(a[2], a[2], ss); ss = fmaf(a[3], a[3], ss);
                    ss += __shfl_xor_sync(0xffffffffu, ss, 8);
                    ss += __shfl_xor_sync(0xffffffffu, ss, 16);
                    if (lane == 0) ssq[slot][warp] = ss;
                    named_bar_sync(1, GROUPS * 64);
                    float tot = 0.f;
#pragma unroll
                    for (int w = 0; w < GROUPS * 2; ++w) tot += ssq[slot][w];
                    slot ^= 1;
                    const float rstd = rsqrtf(tot * (1.f / 128.f) + gate.eps);
                    const float z4[4] = {__uint_as_float(zr.x << 16), __uint_as_float(zr.x & 0xffff0000u),
                                         __uint_as_float(zr.y << 16), __uint_as_float(zr.y & 0xffff0000u)};
                    const float w4[4] = {__uint_as_float(wr.x << 16), __uint_as_float(wr.x & 0xffff0000u),
                                         __uint_as_float(wr.y << 16), __uint_as_float(wr.y & 0xffff0000u)};
                    float o4[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) o4[e] = a[e] * (rstd * w4[e]) * __fdividef(z4[e], 1.f + __expf(-z4[e]));
                    pk.x = pack_bf16x2(o4[0], o4[1]);
                    pk.y = pack_bf16x2(o4[2], o4[3]);
                }
                if (rg == 0) *reinterpret_cast<uint2*>(p.out + o_at) = pk;
            }
            // the tile goes back into its stage and leaves by TMA; the stage before it is free once its store has been read
            if (p.hT) {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    *reinterpret_cast<float4*>(tile + (i >> 1) * 2048 + (i & 1 ? off1 : off0)) = make_float4(st[i][0].x, st[i][0].y, st[i][1].x, st[i][1].y);
                fence_proxy_async_smem();
            }
            named_bar_sync(2 + g, 64);
            if (half == 0 && elect_one()) {
                if (p.hT && STAGES > 1) {
                    tma_store_wait_read();                // tile n - 1's store has read its stage
                    if (n > 0) mbar_arrive(&empty[g][(n - 1) % STAGES]);
                    if (ok) tma_store_2d(&tm_out, tile_of(g, s), quarter * 32, state * kD);
                    tma_store_commit();
                } else if (p.hT) {                        // too few stages to wait a tile: the CTAs beside this one fill the time
                    if (ok) tma_store_2d(&tm_out, tile_of(g, s), quarter * 32, state * kD);
                    tma_store_commit();
                    tma_store_wait_read();
                    mbar_arrive(&empty[g][s]);
                } else {
                    mbar_arrive(&empty[g][s]);
                }
            }
            __syncwarp();
        }
        if (p.hT && half == 0 && elect_one()) tma_store_wait_all();
    }
}

// Gated rows: two CTAs per SM of one stage each, or one of three stages?  Two fill each other's barriers and instructions; one overlaps
// the next state's load and this one's store.  Of an odd number of states per SM the last runs alone, beside a CTA that has no more.
// 32 heads, fp32 states in and out, all a layer adds, us per call (two / one):
//   (states an SM) 1 (<= 1)     9 (2)         13 (3)        23 (5)        32 (7)        37 (8)        64 (14)
//   2 tokens       7.1 / 6.4    11.8 / 12.4   19.9 / 16.4   31.6 / 26.3   41.4 / 35.9   42.6 / 40.3   67.7 / 66.2
//   3 tokens       8.6 / 7.7    13.9 / 15.3   23.9 / 20.7   37.3 / 33.3   48.8 / 45.7   49.9 / 51.6   80.3 / 85.8
//   4 tokens       10.0 / 8.8   16.1 / 18.0   27.9 / 24.7   43.1 / 40.1   56.4 / 55.2   57.5 / 62.7   94.2 / 105
//   6 tokens       13.4 / 11.7  21.5 / 27.0   38.7 / 38.0   59.8 / 62.4   78.7 / 86.3   -             134 / 168
// A state that is not written weighs little beside the instructions: one CTA only at two and a half to three states per SM (13 sequences
// of 2 tokens, state in 15.5 / 14.2, none 12.2 / 10.7; 64 of 2, 46.8 / 52.4 and 38.9 / 43.0).  Out only, 2 tokens: 32 sequences
// 32.2 / 28.9, 37 33.8 / 34.0, 64 57.6 / 57.9.  Two tokens, in and out, on many states: 128 sequences (28) 125.9 / 125.8, 256 (56) 242 / 246.
bool two_gated_ctas(const Problem& p, long long states) {
    const long long sms = sm_count(), rounds = (states + sms - 1) / sms, pairs = (states + 2 * sms - 1) / (2 * sms);
    if (p.S == 1 || rounds == 1) return false;
    if (p.S > 4 || rounds == 2) return true;
    if (!p.hT) return rounds != 3 || 2 * states <= 5 * sms;
    if (p.S == 2 && p.h0) return rounds >= 40;
    return 10 * rounds >= (p.S == 2 ? 19 : p.S == 3 ? 18 : 17) * pairs;
}

// Five to eight tokens: four CTAs per SM with a ring of two, or three with a ring of three?  What bounds these tiles is their warps' run through the tokens, so
// four fill the SM's issue slots better, but a tile more at a time takes longer, and where the last round is not full three may have as many rounds.
// In hundredths of a round of three: a round of four 126 (five tokens: 130), a last round of one tile 50, of more 100.  32 heads, states in and out, us per
// call (three / two):
//   sequences (tiles an SM)  3 (3)      4 (4)      5 (5)        6 (6)        8 (7)        10 (9)       13 (12)      24 (21)      64 (56)
//   5 tokens                 6.3 / 7.0  8.2 / 6.9  10.1 / 8.6   10.2 / 10.4  14.5 / 11.9  14.9 / 15.8  18.7 / 17.1  30.9 / 31.8  76.3 / 76.9
//   6 tokens                 6.9 / 7.6  9.2 / 7.5  11.3 / 9.6   11.4 / 11.7  16.4 / 13.1  16.7 / 17.5  21.2 / 19.0  35.1 / 35.4  87.8 / 84.7
//   8 tokens                 8.2 / 8.8  11.1 / 8.8 13.8 / 11.5  13.8 / 13.8  20.2 / 15.6  20.5 / 21.2  26.3 / 22.7  44.1 / 43.2  112.0 / 100.2
// With states both in and out and many tiles an SM a round's three run into the next round, the tiles' traffic counts and a last round of one costs the form of four more. Above
// 20 tiles five tokens stay with three (21 to 84 tiles 0.6 to 5 % faster; two at 25, 28, 29 and 173 by 0.6 to 2 %); with six that last round counts 71 (21 tiles 35.3 / 35.8), and where two
// are taken they are up to 5 % ahead at 22 to 65 tiles but at 26, 27, 30, 31, 34, 43 and 46 (0.7 to 1.8 % behind).
// With one of them or neither two are ahead by 7 to 39 % wherever this rule takes them (64 sequences of 5 tokens: state in 71.2 / 55.2, out 73.4 / 66.6, neither 69.3 / 53.0).
// (Packed batches keep three: where most of their sequences are single tokens a ring of two is 8 % slower, 128 sequences with one of 8 86.7 / 94.3.)
bool two_stages(const Problem& p, long long tiles, long long sms) {
    if (p.S < 5) return false;
    const long long t = (tiles + sms - 1) / sms;
    const bool many = p.h0 && p.hT && t > 20;
    if (many && p.S == 5) return false;
    auto last = [](long long k, int one) { return k == 0 ? 0 : k == 1 ? one : 100; };
    return (p.S == 5 ? 130 : 126) * (t / 4) + last(t % 4, many && p.S == 6 ? 71 : 50) < 100 * (t / 3) + last(t % 3, 50);
}

}  // namespace

// `og`: gated normalisation applied to the output rows by the same kernel (null: none).
int launch_decode(const Problem& p, const OutputGate* og, cudaStream_t stream) {
    const long long states = static_cast<long long>(p.B) * p.Hv;   // (of a packed batch: all sequences', the map's extent)
    // a state's row is a map coordinate (2^31 rows of states: 1 TB); without states only the number of tiles is an int
    if (states * ((p.h0 || p.hT) ? kD : 4) >= (1ll << 31)) return GDN_ERR_BAD_ARGUMENT;
    alignas(64) CUtensorMap tin, tout;
    const unsigned long long d[2] = {kD, static_cast<unsigned long long>(states) * kD}, sb[1] = {kD * 4};
    const unsigned box[2] = {32, kD};
    const float* any = p.h0 ? p.h0 : p.hT;
    if (any) {   // a map nobody uses still has to be a valid one
        if (encode_tma(&tin, any, 4, 2, d, sb, box, 128)) return GDN_ERR_DRIVER;
        if (encode_tma(&tout, p.hT ? p.hT : any, 4, 2, d, sb, box, 128)) return GDN_ERR_DRIVER;
    } else {
        tin = tout = CUtensorMap{};
    }
    DecodeGate gate{};
    if (og) gate = DecodeGate{static_cast<const __nv_bfloat16*>(og->z), static_cast<const __nv_bfloat16*>(og->weight), og->eps};
    const bool gated = og && !p.pk_short;
    const long long sms = sm_count();
    const long long items = p.pk_short ? 4ll * p.pk_shorts * p.Hv : gated ? states : states * 4;
    const int groups = gated ? 4 : 1, stages = gated ? (two_gated_ctas(p, states) ? 1 : 3) : !p.pk_short && two_stages(p, items, sms) ? 2 : 3;
    const int most = gated ? 4 : kDecTokens;                       // tokens whose vectors fit three stages of four groups
    const int nt = p.S < most ? p.S : most;
    auto bytes = [&](bool apart) { return dec_dynamic_bytes(groups, stages, nt, apart); };
    auto resident = [&](uint32_t smem) {
        const int fit = dec_fit(smem, dec_static_bytes(groups, stages, p.pk_short != nullptr)), most_ctas = dec_ctas_per_sm(groups, stages);
        return sms * (fit > most_ctas ? most_ctas : fit);
    };
    // one tile a CTA: the host's time for three more maps is not hidden behind the kernel
    const bool by_rows = p.pk_short || p.S == 1 || (!gated && p.S <= 4 && items <= resident(bytes(false)));
    const uint32_t smem = bytes(!by_rows && gates_apart(groups, stages, Fetch::BOXES));
    const long long cap = resident(smem);
    auto go = [&](auto kernel, const auto& maps) -> int {
        if (allow_smem(reinterpret_cast<const void*>(kernel), smem)) return GDN_ERR_CUDA;
        const unsigned grid = static_cast<unsigned>(items < cap ? items : cap);
        const cudaError_t e = launch_dependent(kernel, dim3(grid), dim3(groups * 64 + 32), smem, stream, false, tin, tout, maps, p,
                                               gate, static_cast<int>(items), nt);
        return e == cudaSuccess ? GDN_OK : GDN_ERR_CUDA;
    };
    const TokenMaps<Fetch::ONE_ROW> one;
    const TokenMaps<Fetch::ROWS> rows;
    if (p.pk_short) return p.gate_f32 ? go(gdn_decode_kernel<1, true, true, 3, Fetch::ROWS>, rows) : go(gdn_decode_kernel<1, false, true, 3, Fetch::ROWS>, rows);
    if (p.S == 1 && gated) return p.gate_f32 ? go(gdn_decode_kernel<4, true, false, 3, Fetch::ONE_ROW>, one) : go(gdn_decode_kernel<4, false, false, 3, Fetch::ONE_ROW>, one);
    if (p.S == 1) return p.gate_f32 ? go(gdn_decode_kernel<1, true, false, 3, Fetch::ONE_ROW>, one) : go(gdn_decode_kernel<1, false, false, 3, Fetch::ONE_ROW>, one);
    if (by_rows)
        return p.gate_f32 ? go(gdn_decode_kernel<1, true, false, 3, Fetch::ROWS>, rows) : go(gdn_decode_kernel<1, false, false, 3, Fetch::ROWS>, rows);
    alignas(64) TokenMaps<Fetch::BOXES> maps;
    {
        const unsigned long long tokens = p.S, batch = p.B, Hq = p.Hq, Hv = p.Hv;
        const unsigned long long dq[4] = {kD, Hq, tokens, batch}, sq[3] = {kD * 2, Hq * kD * 2, tokens * Hq * kD * 2};
        const unsigned long long dv[4] = {kD, Hv, tokens, batch}, sv[3] = {kD * 2, Hv * kD * 2, tokens * Hv * kD * 2};
        const unsigned row[4] = {kD, 1, static_cast<unsigned>(nt), 1}, quarter[4] = {32, 1, static_cast<unsigned>(nt), 1};
        if (encode_tma(&maps.q, p.q, 2, 4, dq, sq, row, 0) || encode_tma(&maps.k, p.k, 2, 4, dq, sq, row, 0) || encode_tma(&maps.v, p.v, 2, 4, dv, sv, quarter, 0))
            return GDN_ERR_DRIVER;
    }
    if (gated && stages == 3) return p.gate_f32 ? go(gdn_decode_kernel<4, true, false, 3, Fetch::BOXES>, maps) : go(gdn_decode_kernel<4, false, false, 3, Fetch::BOXES>, maps);
    if (gated) return p.gate_f32 ? go(gdn_decode_kernel<4, true, false, 1, Fetch::BOXES>, maps) : go(gdn_decode_kernel<4, false, false, 1, Fetch::BOXES>, maps);
    if (stages == 2) return p.gate_f32 ? go(gdn_decode_kernel<1, true, false, 2, Fetch::BOXES>, maps) : go(gdn_decode_kernel<1, false, false, 2, Fetch::BOXES>, maps);
    return p.gate_f32 ? go(gdn_decode_kernel<1, true, false, 3, Fetch::BOXES>, maps) : go(gdn_decode_kernel<1, false, false, 3, Fetch::BOXES>, maps);
}

}  // namespace gdn
