// Device-side pieces of the "lean" prepare (gdn_chunk_prepare_lean_sm100.cu): the gate cumsum by one warp, the mask
// epilogues that write straight to their shared-memory destination, and the 64x64 unit-lower-triangular inverse IN
// PLACE.  Same mathematics as gdn_prep_device.cuh; what differs is what has to fit: three CTAs of two heads per SM
// leave 74 KB of shared memory and 80 registers to each, so A and T share one 64 x 68 fp32 array: T overwrites A block by
// block.
#pragma once

#include "gdn_common.cuh"
#include "gdn_prep_device.cuh"
#include "ptx_sm100.cuh"

namespace gdn {

struct alignas(16) LeanScratch {
    float gam[kChunk];      // gamma_j * log2(e): inclusive cumsum of the log gate inside the chunk
    float bet[kChunk];      // beta_j (0 for padding tokens)
    float gcol[kChunk];     // with L2 normalisation: gamma_j - log2(1/|k_j|), the mask epilogue's column table
    float rn[2 * kChunk];   // with L2 normalisation: 1/|k_j| (0..63) and 1/|q_i| (64..127)
    float vec[4 * kChunk];  // with L2 normalisation: the chain's factors before the norms are known
    float bound[2];         // per warp: max over its rows of beta_i |k_i|^2
    int gates_ok;           // every gate of the chunk is inside beta >= 0, g <= 0 (tested on the gates themselves: the
                            // cumsum's rounding can make two of its neighbours change places)
};

// Gates of a chunk held by ONE warp, two tokens per lane: (2 lane, 2 lane + 1).  A single warp needs no barrier inside
// the cumsum; the caller's next group barrier publishes the tables.
struct LaneGates {
    float g0, g1, b0, b1;
};

template <bool GATE_F32>
__device__ __forceinline__ LaneGates lean_load_gates(const Problem& p, size_t tok0, int hv, int valid, int lane) {
    const float pad = p.gate_act ? -INFINITY : 0.f;   // what the activations map to g = 0, beta = 0
    LaneGates x{pad, pad, pad, pad};
    const size_t idx = (tok0 + 2 * lane) * p.Hv + hv;
    if (2 * lane < valid) {
        x.g0 = prep_load_gate<GATE_F32>(p.g, idx);
        x.b0 = prep_load_gate<GATE_F32>(p.beta, idx);
    }
    if (2 * lane + 1 < valid) {
        x.g1 = prep_load_gate<GATE_F32>(p.g, idx + p.Hv);
        x.b1 = prep_load_gate<GATE_F32>(p.beta, idx + p.Hv);
    }
    return x;
}

// One warp.  Per-token factors of the chain kernel (fp32, vec_out[256]):
//   [0, 64) exp(gamma_C - gamma_i)   [64, 128) scale exp(gamma_i)   [128] exp(gamma_C)   [192, 256) exp(gamma_i)
__device__ __forceinline__ void lean_gates(LeanScratch& ps, LaneGates x, bool raw, float scale, float* vec_out, int lane) {
    if (raw) {
        prep_activate_gates(x.g0, x.b0);
        prep_activate_gates(x.g1, x.b1);
    }
    const bool in_range = __all_sync(0xffffffffu, x.g0 <= 0.f && x.g1 <= 0.f && x.b0 >= 0.f && x.b1 >= 0.f);
    if (lane == 0) ps.gates_ok = in_range;
    x.g0 = prep_floor_gate(x.g0);
    x.g1 = prep_floor_gate(x.g1);
    float s = x.g0 + x.g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    const float prev = __shfl_up_sync(0xffffffffu, s, 1);
    const float c0 = ((lane > 0 ? prev : 0.f) + x.g0) * kLog2e, c1 = s * kLog2e;
    const float cC = __shfl_sync(0xffffffffu, c1, 31);
    *reinterpret_cast<float2*>(ps.gam + 2 * lane) = make_float2(c0, c1);
    *reinterpret_cast<float2*>(ps.bet + 2 * lane) = make_float2(x.b0, x.b1);
    const float e0 = exp2f(c0), e1 = exp2f(c1);
    *reinterpret_cast<float2*>(vec_out + 2 * lane) = make_float2(exp2f(cC - c0), exp2f(cC - c1));
    *reinterpret_cast<float2*>(vec_out + kChunk + 2 * lane) = make_float2(scale * e0, scale * e1);
    *reinterpret_cast<float2*>(vec_out + 3 * kChunk + 2 * lane) = make_float2(e0, e1);
    if (lane == 0) vec_out[2 * kChunk] = exp2f(cC);
}

// L2 normalisation of q and k, folded into factors that exist anyway (see prep_l2norm_fold).  Sum of the squares of the 64 values that
// row `row` of the [K;Q] stack has in k-half `tile`; where two heads share the stack, each half of the CTA sums one k-half.
__device__ __forceinline__ float lean_row_squares(const uint8_t* tile, int row) {
    float2 ss = make_float2(0.f, 0.f);
#pragma unroll
    for (int ch = 0; ch < 8; ++ch) {
        const uint4 v = *reinterpret_cast<const uint4*>(tile + row * 128 + ((ch + row) & 7) * 16);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 x = make_float2(__uint_as_float(w[e] << 16), __uint_as_float(w[e] & 0xffff0000u));
            ss = fma2(x, x, ss);
        }
    }
    return ss.x + ss.y;
}
// 128 threads, thread r holds row r's sum (of two partial sums a k-half: against one running sum the norm's last bit differs here and
// there, and with it single bf16 roundings behind it; error against 64 bits the same).  Ends with a group barrier.  Rows of padding tokens
// count as zeros.  The chain's factors go from the tables (lean_gates wrote them to ps.vec) to vec_out: multiplied there in place, their
// way through L2 and back was most of what normalisation cost, and both heads summed all rows (four sequences of 1999 tokens with all
// a layer adds: 152.5 -> 146.6 us a call; prepare of 16 sequences of 2048 162.6 -> 143.4 us, 124.7 without normalisation).
__device__ __forceinline__ void lean_l2norm_fold(LeanScratch& ps, float ss, float* vec_out, int valid, PrepCtx ctx) {
    const int tid = ctx.tid;
    if ((tid & 63) >= valid) ss = 0.f;
    const float r = rsqrtf(ss + 1e-6f);
    ps.rn[tid] = r;
    vec_out[tid] = ps.vec[tid] * r;
    if (tid < kChunk) {
        ps.gcol[tid] = ps.gam[tid] - __log2f(r);
        vec_out[3 * kChunk + tid] = ps.vec[3 * kChunk + tid] * r;
    } else if (tid == kChunk) {
        vec_out[2 * kChunk] = ps.vec[2 * kChunk];
    }
    ctx.sync();
}

// The bits of the columns below `lim` (of 32).
__device__ __forceinline__ uint32_t columns_below(int lim) { return lim <= 0 ? 0u : lim >= 32 ? 0xffffffffu : (1u << lim) - 1u; }
// 2^(g - g_j) of two columns: the mask epilogues take two elements an instruction where they can, and their predicates from the bits of
// one word several at a time (prepare of 16 sequences of 2048 tokens, 32 heads: 128.3 -> 124.7 us; the same results).
__device__ __forceinline__ float2 decay2(float g, float gj0, float gj1) {
    const float2 d = fma2(make_float2(gj0, gj1), make_float2(-1.f, -1.f), make_float2(g, g));
    return make_float2(fast_exp2(d.x), fast_exp2(d.y));
}

// Row i of A = tril(beta_i * decay * K K^T, -1), fp32, into At (columns 32-63 of rows 0-31 are not written); rows of
// padding tokens (i >= valid) are zeros whatever the tile holds there.  Returns |k_i|^2.
// PAIRED: two elements an instruction.  With one head per CTA, 128 registers a thread, that gives nothing on many chunks (16 sequences of
// 2048 tokens, 16 / 16 heads: 217 us a call either way) and takes 0.2 us longer on a few (100 tokens, 16 / 16 heads: 13.58 -> 13.79).
template <bool PAIRED>
__device__ __forceinline__ float lean_mask_row_A(const LeanScratch& ps, bool l2norm, uint32_t trow, int i, bool low_rows,
                                                 int valid, float* At) {
    const float* gcol = l2norm ? ps.gcol : ps.gam;
    const float gi = ps.gam[i];
    const float bi = l2norm ? ps.bet[i] * ps.rn[i] : ps.bet[i];
    const int lim = i < valid ? i : 0;
    const float2 b2 = make_float2(bi, bi);
    float ksq = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        if (half == 1 && low_rows) break;
        const uint32_t keep = columns_below(lim - 32 * half);
        uint32_t r[32];
        tmem_ld_x32(trow + half * 32, r);
        tmem_ld_wait();
        if ((i >> 5) == half) {
#pragma unroll
            for (int c = 0; c < 32; ++c)
                if (c == (i & 31)) ksq = __uint_as_float(r[c]);
        }
#pragma unroll
        for (int c = 0; c < 32; c += 4) {
            const float4 gj = *reinterpret_cast<const float4*>(gcol + half * 32 + c);
            float4 o;
            if constexpr (PAIRED) {
                const float2 x = mul2(mul2(decay2(gi, gj.x, gj.y), b2), make_float2(__uint_as_float(r[c]), __uint_as_float(r[c + 1])));
                const float2 y = mul2(mul2(decay2(gi, gj.z, gj.w), b2), make_float2(__uint_as_float(r[c + 2]), __uint_as_float(r[c + 3])));
                o = make_float4(keep & (1u << c) ? x.x : 0.f, keep & (2u << c) ? x.y : 0.f, keep & (4u << c) ? y.x : 0.f, keep & (8u << c) ? y.y : 0.f);
            } else {
                const int col = half * 32 + c;
                o.x = col + 0 < lim ? bi * fast_exp2(gi - gj.x) * __uint_as_float(r[c + 0]) : 0.f;
                o.y = col + 1 < lim ? bi * fast_exp2(gi - gj.y) * __uint_as_float(r[c + 1]) : 0.f;
                o.z = col + 2 < lim ? bi * fast_exp2(gi - gj.z) * __uint_as_float(r[c + 2]) : 0.f;
                o.w = col + 3 < lim ? bi * fast_exp2(gi - gj.w) * __uint_as_float(r[c + 3]) : 0.f;
            }
            *reinterpret_cast<float4*>(At + i * kSolveStride + half * 32 + c) = o;
        }
    }
    return i < valid ? ksq : 0.f;
}

// Byte offset of the 16-byte chunk `ch` (8 columns) of row `row` in a lower-triangular 64x64 bf16 tile without its upper
// right block: 64-byte rows, 64-byte swizzle (see TileMaps).
__device__ __forceinline__ uint32_t tri_offset(uint32_t row, uint32_t ch) {
    return (ch < 4 ? 0u : 4096u - 2048u) + swz_chunk_offset<64>(row, ch & 3);
}

// Row i of P = tril(scale * decay * Q K^T) as bf16 into row i of a triangular tile.
__device__ __forceinline__ void lean_mask_row_P(const LeanScratch& ps, bool l2norm, float scale0, uint32_t trow, int i,
                                                bool low_rows, int valid, uint8_t* tile) {
    const float* gcol = l2norm ? ps.gcol : ps.gam;
    const float gis = ps.gam[i] + __log2f(l2norm ? scale0 * ps.rn[kChunk + i] : scale0);
    const int lim = i < valid ? i : -1;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        if (half == 1 && low_rows) break;          // above the diagonal
        const uint32_t keep = columns_below(lim + 1 - 32 * half);
        uint32_t r[32];
        tmem_ld_x32(trow + half * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
            float x[8];
#pragma unroll
            for (int c = 0; c < 8; c += 4) {
                const int col = half * 32 + 8 * ch + c;
                const float4 gj = *reinterpret_cast<const float4*>(gcol + col);
                const float2 y = mul2(decay2(gis, gj.x, gj.y), make_float2(__uint_as_float(r[8 * ch + c]), __uint_as_float(r[8 * ch + c + 1])));
                const float2 z = mul2(decay2(gis, gj.z, gj.w), make_float2(__uint_as_float(r[8 * ch + c + 2]), __uint_as_float(r[8 * ch + c + 3])));
                x[c + 0] = keep & (1u << (8 * ch + c)) ? y.x : 0.f;
                x[c + 1] = keep & (2u << (8 * ch + c)) ? y.y : 0.f;
                x[c + 2] = keep & (4u << (8 * ch + c)) ? z.x : 0.f;
                x[c + 3] = keep & (8u << (8 * ch + c)) ? z.y : 0.f;
            }
            uint4 pk;
            pk.x = pack_bf16x2(x[0], x[1]);
            pk.y = pack_bf16x2(x[2], x[3]);
            pk.z = pack_bf16x2(x[4], x[5]);
            pk.w = pack_bf16x2(x[6], x[7]);
            *reinterpret_cast<uint4*>(tile + tri_offset(i, 4 * half + ch)) = pk;
        }
    }
}

// max over the warp's rows of beta_i |k_i|^2; +inf when one of them is not a number (fmaxf would drop it): what such a key leaves in
// the state is bounded by nothing.
__device__ __forceinline__ float lean_bound_of_rows(const LeanScratch& ps, bool l2norm, int i, float ksq) {
    const float rk = l2norm ? ps.rn[i] : 1.f;
    float bound = ps.bet[i] * ksq * rk * rk;
    if (!(bound < INFINITY)) bound = INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bound = fmaxf(bound, __shfl_xor_sync(0xffffffffu, bound, o));
    return bound;
}

// In-place inverse of I + A (A strictly lower triangular, zeros on and above its diagonal inside the 32x32 diagonal
// blocks) in `At`, row stride kSolveStride.  The block above the two 32x32 diagonal blocks (rows 0-31, columns 32-63) is not used.
//
// What bounds the prepare kernel is the shared-memory pipe: it delivers one word to every lane per cycle, so a broadcast
// float4 costs as much as 512 bytes of data.  (With the 8 -> 16 level on CUDA cores, Y = A21 X11 passed through shared memory
// at every level and T read back for its conversion, that pipe was busy 72 % of the kernel's time.)  Products are therefore
// taken as (X22 A21) X11 with the accumulator of the first kept in registers as the A fragment of the second: an accumulator
// holds columns (2t, 2t + 1) where an A fragment wants k = (t, t + 4), so the second product runs over k in that order and
// its B fragments are rows 2t, 2t + 1 - which also lie in different banks.  Per call, before and after: 16 sequences of 2048
// tokens 418 -> 389 us, one of 8192 tokens 121.6 -> 117.0 us, 64 of 4096 tokens 3127 -> 2967 us.

__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    hi = f32_to_tf32(x) & 0xffffe000u;
    lo = f32_to_tf32(x - __uint_as_float(hi));
}
// Two 8x8x8 products at once with about fp32 precision (every factor as the sum of two TF32 numbers, the product of the low
// parts left out): d rows 0-7 = a rows 0-7 * B0, d rows 8-15 = a rows 8-15 * B1.  B fragments: words b[0] and b[step].
__device__ __forceinline__ void mma_split(float (&d)[4], const float (&av)[4], const float* b0, const float* b1, int step) {
    uint32_t ah[4], al[4], b0h[2], b0l[2], b1h[2], b1l[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) split_tf32(av[i], ah[i], al[i]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        split_tf32(b0[i * step], b0h[i], b0l[i]);
        split_tf32(b1[i * step], b1h[i], b1l[i]);
    }
    float c[4] = {0.f, 0.f, 0.f, 0.f}, e[4] = {0.f, 0.f, 0.f, 0.f};
    mma_tf32_16x8x8(c, ah, b0l);
    mma_tf32_16x8x8(e, ah, b1l);
    mma_tf32_16x8x8(c, al, b0h);
    mma_tf32_16x8x8(e, al, b1h);
    mma_tf32_16x8x8(c, ah, b0h);
    mma_tf32_16x8x8(e, ah, b1h);
    d[0] = c[0];
    d[1] = c[1];
    d[2] = e[2];
    d[3] = e[3];
}

// x = columns [8 N0, 8 N0 + 16) of z X: z (16 x 8 NT) in accumulator fragments, X lower triangular (8 NT x 8 NT).
template <int NT, int N0>
__device__ __forceinline__ void mma_times_lower(float (&x)[2][4], const float (&z)[NT][4], const float* X, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e >> 2][e & 3] = 0.f;
#pragma unroll
    for (int ks = N0; ks < NT; ++ks) {
        const uint32_t a[4] = {f32_to_tf32(z[ks][0]), f32_to_tf32(z[ks][2]), f32_to_tf32(z[ks][1]), f32_to_tf32(z[ks][3])};
#pragma unroll
        for (int nt = N0; nt < N0 + 2; ++nt) {
            if (nt > ks) continue;
            const float* b = X + (8 * ks + 2 * t) * kSolveStride + 8 * nt + g;
            const uint32_t bv[2] = {f32_to_tf32(b[0]), f32_to_tf32(b[kSolveStride])};
            mma_tf32_16x8x8(x[nt - N0], a, bv);
        }
    }
}

// One warp: the 32x32 diagonal block p.  8x8 blocks by forward substitution in fp32 registers, 8 -> 16 in split TF32,
// 16 -> 32 in TF32.  Needs the warp's own 32 rows only (a __syncwarp after they were written).
__device__ __forceinline__ void lean_invert_diag32(float* At, int p, int lane) {
    asm volatile("" : "+r"(lane));   // (its addresses are computed here, not kept in registers across the items' loop)
    {   // four 8x8 diagonal blocks: lane = (block, column)
        const int blk = 4 * p + (lane >> 3), c = lane & 7;
        float* a = At + (8 * blk) * kSolveStride + 8 * blk;
        float4 rowv[7][2];
#pragma unroll
        for (int i = 1; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (4 * q < i) rowv[i - 1][q] = *reinterpret_cast<const float4*>(a + i * kSolveStride + 4 * q);
        __syncwarp();                                  // all eight lanes of a block have read it
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = (i == c) ? 1.f : 0.f;
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            float acc0 = x[i], acc1 = 0.f;
#pragma unroll
            for (int j = 0; j < i; ++j) {
                const float4 v4 = rowv[i - 1][j >> 2];
                const float aij = (j & 3) == 0 ? v4.x : ((j & 3) == 1 ? v4.y : ((j & 3) == 2 ? v4.z : v4.w));
                if (j & 1) acc1 = fmaf(-aij, x[j], acc1);
                else acc0 = fmaf(-aij, x[j], acc0);
            }
            x[i] = acc0 + acc1;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i * kSolveStride + c] = x[i];
    }
    __syncwarp();
    const int g = lane >> 2, t = lane & 3;
    {   // 8 -> 16: X21 = -(X22 A21) X11 of the warp's two 16x16 blocks, rows 0-7 of the fragments block 0's, rows 8-15 block 1's
        float* b0 = At + (32 * p) * kSolveStride + 32 * p;
        float* b1 = b0 + 16 * kSolveStride + 16;
        const float* a0 = b0 + (8 + g) * kSolveStride + 8 + t;
        const float* a1 = b1 + (8 + g) * kSolveStride + 8 + t;
        const float av[4] = {a0[0], a1[0], a0[4], a1[4]};
        float z[4], x[4];
        mma_split(z, av, b0 + (8 + t) * kSolveStride + g, b1 + (8 + t) * kSolveStride + g, 4 * kSolveStride);
        const float zv[4] = {z[0], z[2], z[1], z[3]};   // the accumulator as an A fragment: its columns (2t, 2t + 1) are k
        mma_split(x, zv, b0 + 2 * t * kSolveStride + g, b1 + 2 * t * kSolveStride + g, kSolveStride);
        __syncwarp();
        *reinterpret_cast<float2*>(b0 + (8 + g) * kSolveStride + 2 * t) = make_float2(-x[0], -x[1]);
        *reinterpret_cast<float2*>(b1 + (8 + g) * kSolveStride + 2 * t) = make_float2(-x[2], -x[3]);
    }
    __syncwarp();
    {   // 16 -> 32 in TF32: X21 = -(X22 A21) X11 (16 x 16 each)
        float* x11 = At + (32 * p) * kSolveStride + 32 * p;
        float* a21 = x11 + 16 * kSolveStride;
        float z[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[4];
            load_a_frag(a, a21 + 16 + 8 * ks, kSolveStride, lane);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                uint32_t b[2];
                load_b_frag(b, a21 + (8 * ks) * kSolveStride + 8 * nt, kSolveStride, lane);
                mma_tf32_16x8x8(z[nt], a, b);
            }
        }
        float x[2][4];
        mma_times_lower<2, 0>(x, z, x11, lane);
        __syncwarp();
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) store_c_frag(a21 + 8 * nt, kSolveStride, lane, x[nt], -1.f);
    }
}

// The last level, X21 = -(X22 A21) X11 on 32x32 blocks, and T'' = T diag(beta) as bf16, 128 threads; both diagonal blocks
// are complete (one barrier before).  Warps 0 and 1 own 16 rows each of X21, which goes from the accumulators straight to
// its bf16 place; warps 2 and 3 convert the diagonal blocks meanwhile.  The tile overwrites the start of `At`,
// hence the barrier between reading and writing.
__device__ __forceinline__ void lean_finish_T2(const float* At, const float* bet, uint8_t* tile, PrepCtx ctx) {
    const int warp = ctx.tid >> 5;
    int lane = ctx.tid & 31;
    asm volatile("" : "+r"(lane));   // (see lean_invert_diag32)
    const int g = lane >> 2, t = lane & 3;
    if (warp < 2) {
        const int row0 = 32 + 16 * warp;
        float z[4][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            if (ks >= 2 * warp + 2) continue;              // X22 is lower triangular
            uint32_t a[4];
            load_a_frag(a, At + row0 * kSolveStride + 32 + 8 * ks, kSolveStride, lane);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                uint32_t b[2];
                load_b_frag(b, At + (32 + 8 * ks) * kSolveStride + 8 * nt, kSolveStride, lane);
                mma_tf32_16x8x8(z[nt], a, b);
            }
        }
        uint32_t pk[4][2];
        auto pack_half = [&](const float (&x)[2][4], int nt0) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const float2 b = *reinterpret_cast<const float2*>(bet + 8 * (nt0 + nt) + 2 * t);
                pk[nt0 + nt][0] = pack_bf16x2(-x[nt][0] * b.x, -x[nt][1] * b.y);
                pk[nt0 + nt][1] = pack_bf16x2(-x[nt][2] * b.x, -x[nt][3] * b.y);
            }
        };
        float x[2][4];
        mma_times_lower<4, 0>(x, z, At, lane);
        pack_half(x, 0);
        mma_times_lower<4, 2>(x, z, At, lane);
        pack_half(x, 2);
        ctx.sync();
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            *reinterpret_cast<uint32_t*>(tile + tri_offset(row0 + g, nt) + 4 * t) = pk[nt][0];
            *reinterpret_cast<uint32_t*>(tile + tri_offset(row0 + 8 + g, nt) + 4 * t) = pk[nt][1];
        }
    } else {
        const int blk = warp - 2, r = lane >> 3, c = lane & 7;   // four rows at a time, four columns a lane
        const float* src = At + (32 * blk + r) * kSolveStride + 32 * blk + 4 * c;
        const float4 b = *reinterpret_cast<const float4*>(bet + 32 * blk + 4 * c);
        uint2 pk[8];
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const float4 x = *reinterpret_cast<const float4*>(src + 4 * it * kSolveStride);
            pk[it] = make_uint2(pack_bf16x2(x.x * b.x, x.y * b.y), pack_bf16x2(x.z * b.z, x.w * b.w));
        }
        ctx.sync();
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            *reinterpret_cast<uint2*>(tile + tri_offset(32 * blk + 4 * it + r, 4 * blk + (c >> 1)) + (c & 1) * 8) = pk[it];
        }
    }
}

}  // namespace gdn
