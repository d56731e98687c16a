// Device-side pieces of the "lean" prepare (gdn_chunk_prepare_lean_sm100.cu): the gate cumsum by one warp, the mask
// epilogues that write straight to their shared-memory destination, and the 64x64 unit-lower-triangular inverse IN
// PLACE.  Same mathematics as gdn_prep_device.cuh; what differs is what has to fit: three CTAs of two heads per SM
// leave 73 KB of shared memory and 80 registers to each, so A, T and the merge temporaries share one 64 x 68 fp32 array:
// T overwrites A block by block, and the temporaries live in the block above the two 32x32 diagonal blocks (rows
// 0-31, columns 32-63), which neither matrix uses.
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

// L2 normalisation of q and k, folded into factors that exist anyway (see prep_l2norm_fold): 128 threads, thread r sums
// row r of the [K;Q] stack; ends with a group barrier.  Rows of padding tokens count as zeros.
__device__ __forceinline__ void lean_l2norm_fold(LeanScratch& ps, const uint8_t* kq, float* vec_out, int valid, PrepCtx ctx) {
    const int tid = ctx.tid;
    float ss = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
            const uint4 v = *reinterpret_cast<const uint4*>(kq + half * 16384 + tid * 128 + ((ch + tid) & 7) * 16);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float lo = __uint_as_float(w[e] << 16), hi = __uint_as_float(w[e] & 0xffff0000u);
                ss = fmaf(lo, lo, ss);
                ss = fmaf(hi, hi, ss);
            }
        }
    if ((tid & 63) >= valid) ss = 0.f;
    const float r = rsqrtf(ss + 1e-6f);
    ps.rn[tid] = r;
    if (tid < kChunk) {
        ps.gcol[tid] = ps.gam[tid] - __log2f(r);
        vec_out[tid] *= r;
        vec_out[3 * kChunk + tid] *= r;
    } else {
        vec_out[tid] *= r;           // scale exp(gamma_i) of token tid - 64
    }
    ctx.sync();
}

// Row i of A = tril(beta_i * decay * K K^T, -1), fp32, into At (columns 32-63 of rows 0-31 are not written); rows of
// padding tokens (i >= valid) are zeros whatever the tile holds there.  Returns |k_i|^2.
__device__ __forceinline__ float lean_mask_row_A(const LeanScratch& ps, bool l2norm, uint32_t trow, int i, bool low_rows,
                                                 int valid, float* At) {
    const float* gcol = l2norm ? ps.gcol : ps.gam;
    const float gi = ps.gam[i];
    const float bi = l2norm ? ps.bet[i] * ps.rn[i] : ps.bet[i];
    const int lim = i < valid ? i : 0;
    float ksq = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        if (half == 1 && low_rows) break;
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
            o.x = (half * 32 + c + 0 < lim) ? bi * fast_exp2(gi - gj.x) * __uint_as_float(r[c + 0]) : 0.f;
            o.y = (half * 32 + c + 1 < lim) ? bi * fast_exp2(gi - gj.y) * __uint_as_float(r[c + 1]) : 0.f;
            o.z = (half * 32 + c + 2 < lim) ? bi * fast_exp2(gi - gj.z) * __uint_as_float(r[c + 2]) : 0.f;
            o.w = (half * 32 + c + 3 < lim) ? bi * fast_exp2(gi - gj.w) * __uint_as_float(r[c + 3]) : 0.f;
            *reinterpret_cast<float4*>(At + i * kSolveStride + half * 32 + c) = o;
        }
    }
    return i < valid ? ksq : 0.f;
}

// Row i of P = tril(scale * decay * Q K^T) as bf16 into row i of a 128-byte-swizzled tile.
__device__ __forceinline__ void lean_mask_row_P(const LeanScratch& ps, bool l2norm, float scale0, uint32_t trow, int i,
                                                bool low_rows, int valid, uint8_t* tile) {
    const float* gcol = l2norm ? ps.gcol : ps.gam;
    const float gis = ps.gam[i] + __log2f(l2norm ? scale0 * ps.rn[kChunk + i] : scale0);
    const int lim = i < valid ? i : -1;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        if (half == 1 && low_rows) {               // above the diagonal: zeros
#pragma unroll
            for (int ch = 4; ch < 8; ++ch) *reinterpret_cast<uint4*>(tile + swz_chunk_offset<128>(i, ch)) = make_uint4(0, 0, 0, 0);
            break;
        }
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
                x[c + 0] = (col + 0 <= lim) ? fast_exp2(gis - gj.x) * __uint_as_float(r[8 * ch + c + 0]) : 0.f;
                x[c + 1] = (col + 1 <= lim) ? fast_exp2(gis - gj.y) * __uint_as_float(r[8 * ch + c + 1]) : 0.f;
                x[c + 2] = (col + 2 <= lim) ? fast_exp2(gis - gj.z) * __uint_as_float(r[8 * ch + c + 2]) : 0.f;
                x[c + 3] = (col + 3 <= lim) ? fast_exp2(gis - gj.w) * __uint_as_float(r[8 * ch + c + 3]) : 0.f;
            }
            uint4 pk;
            pk.x = pack_bf16x2(x[0], x[1]);
            pk.y = pack_bf16x2(x[2], x[3]);
            pk.z = pack_bf16x2(x[4], x[5]);
            pk.w = pack_bf16x2(x[6], x[7]);
            *reinterpret_cast<uint4*>(tile + swz_chunk_offset<128>(i, 4 * half + ch)) = pk;
        }
    }
}

// max over the warp's rows of beta_i |k_i|^2.
__device__ __forceinline__ float lean_bound_of_rows(const LeanScratch& ps, bool l2norm, int i, float ksq) {
    const float rk = l2norm ? ps.rn[i] : 1.f;
    float bound = ps.bet[i] * ksq * rk * rk;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bound = fmaxf(bound, __shfl_xor_sync(0xffffffffu, bound, o));
    return bound;
}

// In-place inverse of I + A (A strictly lower triangular, zeros on and above its diagonal inside the 32x32 diagonal
// blocks) in `At`, row stride kSolveStride.  The merge temporaries use the block above the diagonal (rows 0-31, columns
// 32-63), so neither function leaves anything defined there.

// One warp: the 32x32 diagonal block p.  8x8 blocks by forward substitution in fp32 registers, 8 -> 16 in fp32,
// 16 -> 32 with TF32 warp MMAs.  Needs the warp's own 32 rows only (a __syncwarp after they were written).
__device__ __forceinline__ void lean_invert_diag32(float* At, int p, int lane) {
    float* tmp = At + 16 * p * kSolveStride + 32;      // 16 rows of temporaries of this warp
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
    {   // 8 -> 16 in fp32: X21 = -X22 (A21 X11); lane = (16-block, row r, four columns c0 ..)
        const int b16 = 2 * p + (lane & 1), r = (lane >> 1) & 7, c0 = 4 * (lane >> 4);
        float* a21 = At + (16 * b16 + 8 + r) * kSolveStride + 16 * b16;
        const float* x11 = At + (16 * b16) * kSolveStride + 16 * b16 + c0;
        const float* x22 = a21 + 8;
        float* yb = tmp + 16 * (lane & 1);
        {
            const float4 a0 = *reinterpret_cast<const float4*>(a21), a1 = *reinterpret_cast<const float4*>(a21 + 4);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float4 xv = *reinterpret_cast<const float4*>(x11 + k * kSolveStride);
                acc.x = fmaf(av[k], xv.x, acc.x);
                acc.y = fmaf(av[k], xv.y, acc.y);
                acc.z = fmaf(av[k], xv.z, acc.z);
                acc.w = fmaf(av[k], xv.w, acc.w);
            }
            *reinterpret_cast<float4*>(yb + r * kSolveStride + c0) = acc;
        }
        __syncwarp();
        {
            const float4 b0 = *reinterpret_cast<const float4*>(x22), b1 = *reinterpret_cast<const float4*>(x22 + 4);
            const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float4 yv = *reinterpret_cast<const float4*>(yb + k * kSolveStride + c0);
                acc.x = fmaf(-bv[k], yv.x, acc.x);
                acc.y = fmaf(-bv[k], yv.y, acc.y);
                acc.z = fmaf(-bv[k], yv.z, acc.z);
                acc.w = fmaf(-bv[k], yv.w, acc.w);
            }
            *reinterpret_cast<float4*>(a21 + c0) = acc;
        }
    }
    __syncwarp();
    {   // 16 -> 32 with TF32 warp MMAs: Y = A21 X11, X21 = -X22 Y (16 x 16 each)
        float* a21 = At + (32 * p + 16) * kSolveStride + 32 * p;
        float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[4];
            load_a_frag(a, a21 + 8 * ks, kSolveStride, lane);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                uint32_t b[2];
                load_b_frag(b, At + (32 * p + 8 * ks) * kSolveStride + 32 * p + 8 * nt, kSolveStride, lane);
                mma_tf32_16x8x8(acc[nt], a, b);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) store_c_frag(tmp + 8 * nt, kSolveStride, lane, acc[nt], 1.f);
        __syncwarp();
        float acc2[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint32_t a[4];
            load_a_frag(a, a21 + 16 + 8 * ks, kSolveStride, lane);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                uint32_t b[2];
                load_b_frag(b, tmp + (8 * ks) * kSolveStride + 8 * nt, kSolveStride, lane);
                mma_tf32_16x8x8(acc2[nt], a, b);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) store_c_frag(a21 + 8 * nt, kSolveStride, lane, acc2[nt], -1.f);
    }
}

// 128 threads: the 32x32 lower-left block, X21 = -X22 (A21 X11); both diagonal blocks complete (one barrier before).
// Ends with a group barrier.
__device__ __forceinline__ void lean_invert_level2(float* At, PrepCtx ctx) {
    const int warp = ctx.tid >> 5, lane = ctx.tid & 31;
    const int rb = warp >> 1, cb = warp & 1;
    float* y = At + 32;                                // 32 x 32, row stride kSolveStride
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        uint32_t a[4];
        load_a_frag(a, At + (32 + 16 * rb) * kSolveStride + 8 * ks, kSolveStride, lane);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            if (ks < 2 * cb) continue;                 // X11 is lower triangular: rows above the column block are zero
            uint32_t b[2];
            load_b_frag(b, At + (8 * ks) * kSolveStride + 16 * cb + 8 * nt, kSolveStride, lane);
            mma_tf32_16x8x8(acc[nt], a, b);
        }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
        store_c_frag(y + (16 * rb) * kSolveStride + 16 * cb + 8 * nt, kSolveStride, lane, acc[nt], 1.f);
    ctx.sync();
    float acc2[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        if (ks >= 2 * rb + 2) continue;                // X22 is lower triangular
        uint32_t a[4];
        load_a_frag(a, At + (32 + 16 * rb) * kSolveStride + 32 + 8 * ks, kSolveStride, lane);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            uint32_t b[2];
            load_b_frag(b, y + (8 * ks) * kSolveStride + 16 * cb + 8 * nt, kSolveStride, lane);
            mma_tf32_16x8x8(acc2[nt], a, b);
        }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
        store_c_frag(At + (32 + 16 * rb) * kSolveStride + 16 * cb + 8 * nt, kSolveStride, lane, acc2[nt], -1.f);
    ctx.sync();
}

// T'' = T diag(beta) as bf16: 128 threads, thread = (row i, columns [32 hh, +32)); the tile (128-byte swizzle) overwrites
// the start of `At`, hence the barrier between reading and writing.  hh and i < 32 are uniform over a warp.
__device__ __forceinline__ void lean_store_T2(const float* At, const float* bet, int i, int hh, uint8_t* tile, PrepCtx ctx) {
    uint4 pk[4];
    if (hh == 1 && i < 32) {
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) pk[c4] = make_uint4(0, 0, 0, 0);
    } else {
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
            const int ch = 4 * hh + c4;
            const float4 t0 = *reinterpret_cast<const float4*>(At + i * kSolveStride + ch * 8);
            const float4 t1 = *reinterpret_cast<const float4*>(At + i * kSolveStride + ch * 8 + 4);
            const float4 b0 = *reinterpret_cast<const float4*>(bet + ch * 8), b1 = *reinterpret_cast<const float4*>(bet + ch * 8 + 4);
            pk[c4].x = pack_bf16x2(t0.x * b0.x, t0.y * b0.y);
            pk[c4].y = pack_bf16x2(t0.z * b0.z, t0.w * b0.w);
            pk[c4].z = pack_bf16x2(t1.x * b1.x, t1.y * b1.y);
            pk[c4].w = pack_bf16x2(t1.z * b1.z, t1.w * b1.w);
        }
    }
    ctx.sync();
#pragma unroll
    for (int c4 = 0; c4 < 4; ++c4) *reinterpret_cast<uint4*>(tile + swz_chunk_offset<128>(i, 4 * hh + c4)) = pk[c4];
}

}  // namespace gdn
