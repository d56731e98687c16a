// Device-side pieces of the "lean" prepare (gdn_chunk_prepare_lean_sm100.cu): the gate cumsum by one warp, the mask epilogues and the inverse of the
// 64x64 unit-lower-triangular matrix, on the accumulator fragments of 16x16 blocks that stay in registers from the raw product to T''.
#pragma once

#include "gdn_common.cuh"
#include "gdn_prep_device.cuh"
#include "ptx_sm100.cuh"

namespace gdn {

struct LeanItem {
    size_t tok0, tile;      // its first token and workspace tile
    int b, hv, hq, s0, valid;   // TMA coordinates, tokens of the sequence
    int gates_ok;           // every gate of the chunk is inside beta >= 0, g <= 0 (tested on the gates themselves: the
                            // cumsum's rounding can make two of its neighbours change places)
    float decay;            // sum of the log gates
};
// Items and tables of a head, by the items' numbers in the CTA: those of the next item are made while this one's are read, and the last part of T'' is
// formed an item later.
struct alignas(16) LeanScratch {
    float gam[2][kChunk];   // gamma_j * log2(e): inclusive cumsum of the log gate inside the chunk
    float bet[4][kChunk];   // beta_j (0 for padding tokens)
    float t16[2][kChunk];   // decay between a token and the last one of the first half of its 32 (t32: of the 64), times 1/|k_j| in the first half: the
    float t32[2][kChunk];   // decay of a pair across that line is the product of its two entries, both at most 1 (gates above zero: see lean_gates)
    float gcol[2][kChunk];  // with L2 normalisation: gamma_j - log2(1/|k_j|), the masks' column table
    float brow[2][kChunk];  // with L2 normalisation: beta_j / |k_j|, the row factors of A
    float prow[2][kChunk];  // with L2 normalisation: scale / |q_i|, the row factors of P
    LeanItem item[4];
    float bound[2][2];      // per warp of the inverse: max over its rows of beta_i |k_i|^2
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

// One warp.  Tables, and the per-token factors of the chain kernel (fp32, vec_out[256]; null: with L2 normalisation they are made when the norms are known):
//   [0, 64) exp(gamma_C - gamma_i)   [64, 128) scale exp(gamma_i)   [128] exp(gamma_C)   [192, 256) exp(gamma_i)
__device__ __forceinline__ void lean_gates(LeanScratch& ps, unsigned item, LaneGates x, bool raw, float scale, float* vec_out, int lane) {
    if (raw) {   // a token at a time, the lane's two in turn: compiled once (4 x 1999 tokens with all a layer adds but the output gate 83.1 us a call, now 82.5)
#pragma unroll 1
        for (int e = 0; e < 2; ++e) {
            float g = x.g1, b = x.b1;
            prep_activate_gates(g, b);
            x = LaneGates{g, x.g0, b, x.b0};
        }
    }
    const bool in_range = __all_sync(0xffffffffu, x.g0 <= 0.f && x.g1 <= 0.f && x.b0 >= 0.f && x.b1 >= 0.f);
    const uint32_t buf = item & 1;
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
    *reinterpret_cast<float2*>(ps.gam[buf] + 2 * lane) = make_float2(c0, c1);
    *reinterpret_cast<float2*>(ps.bet[item & 3] + 2 * lane) = make_float2(x.b0, x.b1);
    float c16 = __shfl_sync(0xffffffffu, c1, (lane & 16) + 7), c32 = __shfl_sync(0xffffffffu, c1, 15);
    const float s16 = lane & 8 ? 1.f : -1.f, s32 = lane & 16 ? 1.f : -1.f;
    if (!in_range) {
        // Gates above zero: gamma can fall by 90 in front of a line and rise by 85 behind it, and the decay between the tokens before and after both is exp(-5), but
        // exp(-90), what the line is from the first of them, is no fp32 number.  The tables then meet halfway between the smallest gamma before the line and the
        // largest behind it: no entry is above the root of the largest decay across the line, and what is lost is below 2^-126 times that root.
        auto halfway = [&](float s, int half, float line) {
            float u = fmaxf(s * c0, s * c1);
#pragma unroll 1
            for (int o = half >> 1; o > 0; o >>= 1) u = fmaxf(u, __shfl_xor_sync(0xffffffffu, u, o));
            const float v = __shfl_xor_sync(0xffffffffu, u, half);
            return u + v < 250.f ? 0.5f * s * (u - v) : line;   // (not of a gate of +inf)
        };
        c16 = halfway(s16, 8, c16);
        c32 = halfway(s32, 16, c32);
    }
    *reinterpret_cast<float2*>(ps.t16[buf] + 2 * lane) = make_float2(fast_exp2(s16 * (c0 - c16)), fast_exp2(s16 * (c1 - c16)));
    *reinterpret_cast<float2*>(ps.t32[buf] + 2 * lane) = make_float2(fast_exp2(s32 * (c0 - c32)), fast_exp2(s32 * (c1 - c32)));
    if (lane == 0) {
        ps.item[item & 3].gates_ok = in_range;
        ps.item[item & 3].decay = cC * (1.f / kLog2e);
    }
    if (!vec_out) return;
    const float e0 = exp2f(c0), e1 = exp2f(c1);
    *reinterpret_cast<float2*>(vec_out + 2 * lane) = make_float2(exp2f(cC - c0), exp2f(cC - c1));
    *reinterpret_cast<float2*>(vec_out + kChunk + 2 * lane) = make_float2(scale * e0, scale * e1);
    *reinterpret_cast<float2*>(vec_out + 3 * kChunk + 2 * lane) = make_float2(e0, e1);
    if (lane == 0) vec_out[2 * kChunk] = exp2f(cC);
}

// L2 normalisation of q and k, folded into factors that exist anyway (see prep_l2norm_fold).  Sum of the squares of the 64 values that
// row `row` of the [K;Q] stack has in k-half `tile`; where two heads share the stack, the warps of each sum one k-half.
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
// One token's share: its key's norm in the tables and the chain's factors (query = false), or its query's.  Padding tokens count as zeros.
__device__ __forceinline__ void lean_l2norm_fold(LeanScratch& ps, unsigned item, bool query, int tok, float ss, float scale, float* vec_out, int valid) {
    const uint32_t buf = item & 1;
    if (tok >= valid) ss = 0.f;
    const float r = rsqrtf(ss + 1e-6f), c = ps.gam[buf][tok], e = exp2f(c);
    if (query) {
        ps.prow[buf][tok] = scale * r;
        vec_out[kChunk + tok] = scale * e * r;
    } else {
        const float cC = ps.gam[buf][kChunk - 1];
        ps.gcol[buf][tok] = c - __log2f(r);
        ps.brow[buf][tok] = ps.bet[item & 3][tok] * r;
        if (!(tok & 16)) ps.t16[buf][tok] *= r;
        if (!(tok & 32)) ps.t32[buf][tok] *= r;
        vec_out[tok] = exp2f(cC - c) * r;
        vec_out[3 * kChunk + tok] = e * r;
        if (tok == 0) vec_out[2 * kChunk] = exp2f(cC);
    }
}

// 2^(g - g_j) of two elements, an instruction for both where the machine has it.
__device__ __forceinline__ float2 decay2(float2 g, float2 gj) {
    const float2 d = fma2(gj, make_float2(-1.f, -1.f), g);
    return make_float2(fast_exp2(d.x), fast_exp2(d.y));
}
__device__ __forceinline__ float2 twice(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 floats(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }

// Byte offset of the 16-byte chunk `ch` (8 columns) of row `row` in a lower-triangular 64x64 bf16 tile without its upper
// right block: 64-byte rows, 64-byte swizzle (see TileMaps).
__device__ __forceinline__ uint32_t tri_offset(uint32_t row, uint32_t ch) {
    return (ch < 4 ? 0u : 4096u - 2048u) + swz_chunk_offset<64>(row, ch & 3);
}
// The address a lane gives to stmatrix for a 16x16 block of such a tile, from the block's first row on; XOR 32 for the right one of 32 columns.
__device__ __forceinline__ uint32_t tri_lane_offset(int lane) { return tri_offset((lane & 7) + (lane & 8), lane >> 4); }

// A 16x16 block as two accumulator fragments of 8 columns, words rounded to TF32: lane (g, t) = (lane / 4, lane % 4) holds elements (g, 2t),
// (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1) of each.  The same registers are
//   an A fragment of the block (which wants k = (t, t + 4) where they hold columns 2t, 2t + 1: products run over k in that order), and
//   B fragments of the block's TRANSPOSE, in that same order of k: the first two n = g, the last two n = g + 8.
struct Block {
    uint32_t t[2][4];
};
__device__ __forceinline__ void mma_abt(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[4], int half) {   // d += a b^T, rows 8 half.. of b
    const uint32_t av[4] = {a[0], a[2], a[1], a[3]}, bv[2] = {b[2 * half], b[2 * half + 1]};
    mma_tf32_16x8x8(d, av, bv);
}
// d = a b^T: the first product of a sum, whose accumulator takes no registers.
__device__ __forceinline__ void mma_zero(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mma_abt_first(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[4], int half) {
    const uint32_t av[4] = {a[0], a[2], a[1], a[3]}, bv[2] = {b[2 * half], b[2 * half + 1]};
    mma_zero(d, av, bv);
}
__device__ __forceinline__ void to_tf32(uint32_t (&d)[4], const float (&x)[4], float sign = 1.f) {
#pragma unroll
    for (int e = 0; e < 4; ++e) d[e] = f32_to_tf32(sign * x[e]);
}

// Two 8x8x8 products at once with about fp32 precision (every factor as the sum of two TF32 numbers, the product of the low
// parts left out): d rows 0-7 = a rows 0-7 * B0, d rows 8-15 = a rows 8-15 * B1.
struct Split {
    uint32_t hi, lo;
};
__device__ __forceinline__ Split split_tf32(float x) {
    Split s;
    s.hi = f32_to_tf32(x) & 0xffffe000u;
    s.lo = f32_to_tf32(x - __uint_as_float(s.hi));
    return s;
}
__device__ __forceinline__ void mma_split(float (&d)[4], Split a0, Split a1, Split a2, Split a3, const Split (&b0)[2], const Split (&b1)[2]) {
    const uint32_t ah[4] = {a0.hi, a1.hi, a2.hi, a3.hi}, al[4] = {a0.lo, a1.lo, a2.lo, a3.lo};
    const uint32_t b0h[2] = {b0[0].hi, b0[1].hi}, b0l[2] = {b0[0].lo, b0[1].lo}, b1h[2] = {b1[0].hi, b1[1].hi}, b1l[2] = {b1[0].lo, b1[1].lo};
    float c[4], e[4];
    mma_zero(c, ah, b0l);
    mma_zero(e, ah, b1l);
    mma_tf32_16x8x8(c, al, b0h);
    mma_tf32_16x8x8(e, al, b1h);
    mma_tf32_16x8x8(c, ah, b0h);
    mma_tf32_16x8x8(e, ah, b1h);
    d[0] = c[0];
    d[1] = c[1];
    d[2] = e[2];
    d[3] = e[3];
}

// Inverses of four unit-lower-triangular 8x8 blocks by forward substitution in fp32, lane = (block, column).  `x`: the blocks' strictly lower
// parts, 64 floats apart, 8 a row; their inverses afterwards.  `xt`: the inverses' transposes.  Places of 16 bytes within a block are exchanged against
// bank conflicts (x8_at, xt8_at).  One warp, with a __syncwarp before and after.
__device__ __forceinline__ int x8_at(int blk, int row, int col) { return blk * 64 + ((2 * row + (col >> 2)) ^ (2 * blk)) * 4 + (col & 3); }
__device__ __forceinline__ int xt8_at(int blk, int row, int col) { return blk * 64 + row * 8 + (col ^ (row & 4)); }
__device__ __forceinline__ void lean_invert_8x8(float* x, float* xt, int lane) {
    const int blk = lane >> 3, c = lane & 7;
    float4 rowv[7][2];
#pragma unroll
    for (int i = 1; i < 8; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) {              // (no word more than the row has: what is read costs, not how often)
            const float* a = x + x8_at(blk, i, 4 * q);
            float4& v = rowv[i - 1][q];
            if (i - 4 * q >= 3) v = *reinterpret_cast<const float4*>(a);
            else if (i - 4 * q == 2) { const float2 u = *reinterpret_cast<const float2*>(a); v.x = u.x; v.y = u.y; }
            else if (i - 4 * q == 1) v.x = *a;
        }
    __syncwarp();                                  // all eight lanes of a block have read it
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (i == c) ? 1.f : 0.f;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        float acc0 = v[i], acc1 = 0.f;
#pragma unroll
        for (int j = 0; j < i; ++j) {
            const float4 v4 = rowv[i - 1][j >> 2];
            const float aij = (j & 3) == 0 ? v4.x : ((j & 3) == 1 ? v4.y : ((j & 3) == 2 ? v4.z : v4.w));
            if (j & 1) acc1 = fmaf(-aij, v[j], acc1);
            else acc0 = fmaf(-aij, v[j], acc0);
        }
        v[i] = acc0 + acc1;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) x[x8_at(blk, i, c)] = v[i];
    *reinterpret_cast<float4*>(xt + xt8_at(blk, c, 0)) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(xt + xt8_at(blk, c, 4)) = make_float4(v[4], v[5], v[6], v[7]);
}

// A fragment times a factor a row and one a column.
__device__ __forceinline__ void masked_tile(uint32_t (&d)[4], float2 f0, float2 f1, float2 col, const uint32_t* x) {
    const float2 v0 = mul2(mul2(f0, col), floats(x[0], x[1])), v1 = mul2(mul2(f1, col), floats(x[2], x[3]));
    d[0] = f32_to_tf32(v0.x);
    d[1] = f32_to_tf32(v0.y);
    d[2] = f32_to_tf32(v1.x);
    d[3] = f32_to_tf32(v1.y);
}

// What the warps of a head's diagonal blocks hand to those of the block below them, as fragments: 16 bytes a lane (8 for the two whose lower half is zero).
constexpr int kLeanTileWords = 128;
struct alignas(16) LeanExchange {
    uint32_t x11t[5 * kLeanTileWords];   // X11^T: its blocks (0, 0), (0, 1), (1, 1)
    uint32_t x22[6 * kLeanTileWords];    // X22: (0, 0), (1, 0), (1, 1)
    uint32_t a21[8 * kLeanTileWords];    // A21: rows 0-15, rows 16-31
};
__device__ __forceinline__ void put_tile(uint32_t* p, int n, const uint32_t (&t)[4], int lane) {
    *reinterpret_cast<uint4*>(p + n * kLeanTileWords + 4 * lane) = make_uint4(t[0], t[1], t[2], t[3]);
}
__device__ __forceinline__ void get_tile(uint32_t (&t)[4], const uint32_t* p, int n, int lane) {
    const uint4 v = *reinterpret_cast<const uint4*>(p + n * kLeanTileWords + 4 * lane);
    t[0] = v.x, t[1] = v.y, t[2] = v.z, t[3] = v.w;
}
// X11^T: rows 16 b, columns 8 k (k >= 2 b).
__device__ __forceinline__ void put_x11t(uint32_t* p, int b, int k, const uint32_t (&t)[4], int lane) {
    if (k == 2 * b) *reinterpret_cast<uint2*>(p + 4 * kLeanTileWords + 64 * b + 2 * lane) = make_uint2(t[0], t[1]);
    else put_tile(p, b ? 3 : k - 1, t, lane);
}
__device__ __forceinline__ void get_x11t(uint32_t (&t)[4], const uint32_t* p, int b, int k, int lane) {
    if (k == 2 * b) {
        const uint2 v = *reinterpret_cast<const uint2*>(p + 4 * kLeanTileWords + 64 * b + 2 * lane);
        t[0] = v.x, t[1] = v.y, t[2] = t[3] = 0;
    } else {
        get_tile(t, p, b ? 3 : k - 1, lane);
    }
}

// Two columns of T'' = T diag(beta).
__device__ __forceinline__ uint32_t pack_scaled(float x0, float x1, float2 b) {
    const float2 y = mul2(make_float2(x0, x1), b);
    return pack_bf16x2(y.x, y.y);
}

// Tables the masks read: gamma of rows and columns (with L2 normalisation less log2(1/|k_j|) in the latter), beta (times 1/|k_i|) of A's rows.  Across the
// lines between halves of 32 and 64 tokens the decay is a product of two table entries; exponentials are left for the diagonal 16x16 blocks.
struct MaskTables {
    const float *gam, *gcol, *brow, *t16, *t32;
};

// A = tril(beta_i * decay * K K^T, -1) from the raw product's accumulator, T = (I + A)^-1, T'' = T diag(beta).
//
// What bounded the prepare kernel was the shared-memory pipe: A written to and T built in a 64 x 64 array there, a row of the accumulator a
// thread, took it two thirds of the time (a broadcast float4 costs as much as 512 bytes of data, and the masks' column tables were read that way).
// Here everything but the 8x8 blocks stays in fragments.  A product M N takes N from fragments of N^T (see Block), so X21 = -X22 (A21 X11)
// = -X22 (X11^T A21^T)^T needs fragments of X22, A21 and X11^T:
//    8 -> 16   Z^T = X11^T A21^T, X21 = -X22 Z, X21^T = -Z^T X22^T, in split TF32
//   16 -> 32   the same in TF32, the transpose of the first 32 rows only
//   32 -> 64   in TF32, by two other warps (lean_below)
//
// lean_diagonal: one warp, the 32x32 diagonal block W from the accumulator's lanes 32 W .. + 31 (W = 1: also the mask of A21).  `stage`: its block of T'',
// 2 KB, where the 8x8 blocks lie before that.  `wait`: for the exchange's readers of the item before.
template <typename Wait>
__device__ __forceinline__ bool lean_diagonal(const MaskTables& tab, const float* bet, bool l2norm, float* bound, uint32_t acc, int W, int lane, LeanExchange& ex, uint8_t* stage, const void* map, int tile_row, uint32_t published, Wait&& wait) {
    asm volatile("" : "+r"(lane));   // (its addresses are computed here, not kept in registers across the items' loop)
    const int g = lane >> 2, t = lane & 3;
    const int R = 32 * W;            // first row, first column of the warp's diagonal block
    const uint32_t tmem = tmem_addr(acc, R, 0);
    float* x8 = reinterpret_cast<float*>(stage);
    float* xt8 = x8 + 4 * 64;
    float2 low0, low1;               // the 8x8 blocks below the diagonals of the two 16x16 blocks
    Block a10;                       // the 16x16 block below the diagonal
    {
        uint32_t x[8], y[16];        // rows 0-15 of columns 0-15, rows 16-31 of columns 0-31
        tmem_ld_16x256b_x2(tmem + R, x);
        tmem_ld_16x256b_x4(tmem + (16u << 16) + R, y);
        float gi[4], bi[4];
        float2 gj[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            gi[r] = tab.gam[R + 8 * r + g];
            bi[r] = tab.brow[R + 8 * r + g];
            gj[r] = *reinterpret_cast<const float2*>(tab.gcol + R + 8 * r + 2 * t);
        }
        tmem_ld_wait();
        if (bound) {                 // max beta_i |k_i|^2; a key that is not a number counts as infinity (fmaxf would drop it)
            float m = 0.f;
            if (t == (g >> 1)) {
                const uint32_t kk[4] = {g & 1 ? x[1] : x[0], g & 1 ? x[7] : x[6], g & 1 ? y[9] : y[8], g & 1 ? y[15] : y[14]};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    float b = bi[r] * __uint_as_float(kk[r]);
                    if (l2norm) b *= fast_exp2(gi[r] - (g & 1 ? gj[r].y : gj[r].x));   // 1/|k_i| once more
                    m = fmaxf(m, b < INFINITY ? b : INFINITY);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) *bound = m;
        }
        auto masked = [&](int r, int c, const uint32_t& v0, const uint32_t& v1) { return mul2(mul2(decay2(twice(gi[r]), gj[c]), twice(bi[r])), floats(v0, v1)); };
        const bool k0 = 2 * t < g, k1 = 2 * t + 1 < g;
        auto put8 = [&](int blk, float2 v) { *reinterpret_cast<float2*>(x8 + x8_at(blk, g, 2 * t)) = make_float2(k0 ? v.x : 0.f, k1 ? v.y : 0.f); };
        if (elect_one()) tma_store_wait_read();   // (the lane that issued it) the previous item's block has left its place
        __syncwarp();
        put8(0, masked(0, 0, x[0], x[1]));
        put8(1, masked(1, 1, x[6], x[7]));
        put8(2, masked(2, 2, y[8], y[9]));
        put8(3, masked(3, 3, y[14], y[15]));
        __syncwarp();
        low0 = masked(1, 0, x[2], x[3]);
        low1 = masked(3, 2, y[10], y[11]);
        const float f0 = bi[2] * tab.t16[R + 16 + g], f1 = bi[3] * tab.t16[R + 24 + g];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float2 col = *reinterpret_cast<const float2*>(tab.t16 + R + 8 * c + 2 * t);
            masked_tile(a10.t[c], twice(f0), twice(f1), col, y + 4 * c);
        }
    }
    lean_invert_8x8(x8, xt8, lane);
    __syncwarp();
    float2 xp[4], xq[4];             // the 8x8 inverses, their transposes
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        xp[b] = *reinterpret_cast<const float2*>(x8 + x8_at(b, g, 2 * t));
        xq[b] = *reinterpret_cast<const float2*>(xt8 + xt8_at(b, g, 2 * t));
    }
    float x21[4], x21t[4];           // of both 16x16 blocks: the first's in elements 0, 1, the second's in 2, 3
    {
        float z[4];
        const Split l0[2] = {split_tf32(low0.x), split_tf32(low0.y)}, l1[2] = {split_tf32(low1.x), split_tf32(low1.y)};
        mma_split(z, split_tf32(xq[0].x), split_tf32(xq[2].x), split_tf32(xq[0].y), split_tf32(xq[2].y), l0, l1);
        const Split z0[2] = {split_tf32(z[0]), split_tf32(z[1])}, z1[2] = {split_tf32(z[2]), split_tf32(z[3])};
        const Split p[2] = {split_tf32(xp[1].x), split_tf32(xp[1].y)}, q[2] = {split_tf32(xp[3].x), split_tf32(xp[3].y)};
        mma_split(x21, p[0], q[0], p[1], q[1], z0, z1);
        mma_split(x21t, z0[0], z1[0], z0[1], z1[1], p, q);
    }
    const float x0[2][4] = {{xp[0].x, xp[0].y, -x21[0], -x21[1]}, {0.f, 0.f, xp[1].x, xp[1].y}};
    const float x1[2][4] = {{xp[2].x, xp[2].y, -x21[2], -x21[3]}, {0.f, 0.f, xp[3].x, xp[3].y}};
    float x10[2][4];
    Block b, z;
    {
        const float x0t[2][4] = {{xq[0].x, xq[0].y, 0.f, 0.f}, {-x21t[0], -x21t[1], xq[1].x, xq[1].y}};
        Block a;
        float zt[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            to_tf32(a.t[n], x0t[n]);
            to_tf32(b.t[n], x1[n]);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int n = 0; n < 2; ++n) k == 0 ? mma_abt_first(zt[n], a.t[k], a10.t[k], n) : mma_abt(zt[n], a.t[k], a10.t[k], n);
#pragma unroll
        for (int n = 0; n < 2; ++n) to_tf32(z.t[n], zt[n]);
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int n = 0; n < 2; ++n) k == 0 ? mma_abt_first(x10[n], b.t[k], z.t[k], n) : mma_abt(x10[n], b.t[k], z.t[k], n);
        if (!wait()) return false;
        if (W == 0) {
            put_x11t(ex.x11t, 0, 0, a.t[0], lane);
            put_x11t(ex.x11t, 0, 1, a.t[1], lane);
        }
    }
    uint32_t w[4];
    if (W == 0) {
        float x10t[2][4];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int n = k; n < 2; ++n) k == 0 ? mma_abt_first(x10t[n], z.t[k], b.t[k], n) : mma_abt(x10t[n], z.t[k], b.t[k], n);
        const float x1t[2][4] = {{xq[2].x, xq[2].y, 0.f, 0.f}, {-x21t[2], -x21t[3], xq[3].x, xq[3].y}};
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            to_tf32(w, x10t[n], -1.f);
            put_x11t(ex.x11t, 0, 2 + n, w, lane);
            to_tf32(w, x1t[n]);
            put_x11t(ex.x11t, 1, 2 + n, w, lane);
        }
    } else {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            to_tf32(w, x0[n]);
            put_tile(ex.x22, n, w, lane);
            to_tf32(w, x10[n], -1.f);
            put_tile(ex.x22, 2 + n, w, lane);
            put_tile(ex.x22, 4 + n, b.t[n], lane);
        }
        const float f[4] = {tab.t32[32 + g] * tab.brow[32 + g], tab.t32[40 + g] * tab.brow[40 + g], tab.t32[48 + g] * tab.brow[48 + g], tab.t32[56 + g] * tab.brow[56 + g]};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            uint32_t y[16];
            tmem_ld_16x256b_x4(tmem + ((16u * r) << 16), y);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 col = *reinterpret_cast<const float2*>(tab.t32 + 8 * c + 2 * t);
                masked_tile(w, twice(f[2 * r]), twice(f[2 * r + 1]), col, y + 4 * c);
                put_tile(ex.a21, 4 * r + c, w, lane);
            }
        }
    }
    __syncwarp();                    // (and the 8x8 blocks have been read)
    if (lane == 0) mbar_arrive_a(published);
    __syncwarp();
    float2 be[4];
#pragma unroll
    for (int n = 0; n < 4; ++n) be[n] = *reinterpret_cast<const float2*>(bet + R + 8 * n + 2 * t);
    const uint32_t dst = smem_u32(stage) + tri_lane_offset(lane);
    stmatrix_x4(dst, pack_scaled(x0[0][0], x0[0][1], be[0]), pack_scaled(x0[0][2], x0[0][3], be[0]), 0, pack_scaled(x0[1][2], x0[1][3], be[1]));
    stmatrix_x4(dst ^ 32, 0, 0, 0, 0);
    stmatrix_x4(dst + 1024, pack_scaled(-x10[0][0], -x10[0][1], be[0]), pack_scaled(-x10[0][2], -x10[0][3], be[0]), pack_scaled(-x10[1][0], -x10[1][1], be[1]),
                pack_scaled(-x10[1][2], -x10[1][3], be[1]));
    stmatrix_x4((dst + 1024) ^ 32, pack_scaled(x1[0][0], x1[0][1], be[2]), pack_scaled(x1[0][2], x1[0][3], be[2]), 0, pack_scaled(x1[1][2], x1[1][3], be[3]));
    fence_proxy_async_smem();
    __syncwarp();
    if (elect_one()) {
        tma_store_2d(map, stage, R, tile_row + R);
        tma_store_commit();
    }
    __syncwarp();
    return true;
}

// Columns 16 b .. + 15 of X21 = -X22 (A21 X11), one warp, and of T'' into `stage` (its block below the diagonal).  `taken`: of the exchange, once it has been read.
__device__ __forceinline__ void lean_below(const float* bet, int b, int lane, const LeanExchange& ex, uint8_t* stage, uint32_t taken) {
    asm volatile("" : "+r"(lane));
    float zt[4][4] = {};             // Z^T: columns are rows of A21, 8 a fragment
#pragma unroll 1
    for (int k = 2 * b; k < 4; ++k) {
        uint32_t a[4], y0[4], y1[4];
        get_x11t(a, ex.x11t, b, k, lane);
        get_tile(y0, ex.a21, k, lane);
        get_tile(y1, ex.a21, 4 + k, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            mma_abt(zt[n], a, y0, n);
            mma_abt(zt[2 + n], a, y1, n);
        }
    }
    float x[2][2][4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        uint32_t z0[4], z1[4], a[4];
        to_tf32(z0, zt[k]);
        to_tf32(z1, zt[2 + k]);
#pragma unroll
        for (int r = 0; r < 3; ++r) {      // X22's blocks (0, 0), (1, 0), (1, 1)
            get_tile(a, ex.x22, 2 * r + k, lane);
#pragma unroll
            for (int n = 0; n < 2; ++n) k == 0 && r < 2 ? mma_abt_first(x[r > 0][n], a, z0, n) : mma_abt(x[r > 0][n], a, r == 2 ? z1 : z0, n);
        }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive_a(taken);
    __syncwarp();
    const uint32_t dst = (smem_u32(stage) + tri_lane_offset(lane)) ^ (32 * b);
    float2 be[2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        be[n] = *reinterpret_cast<const float2*>(bet + 16 * b + 8 * n + 2 * (lane & 3));
        be[n] = make_float2(-be[n].x, -be[n].y);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
        stmatrix_x4(dst + 1024 * r, pack_scaled(x[r][0][0], x[r][0][1], be[0]), pack_scaled(x[r][0][2], x[r][0][3], be[0]), pack_scaled(x[r][1][0], x[r][1][1], be[1]),
                    pack_scaled(x[r][1][2], x[r][1][3], be[1]));
    fence_proxy_async_smem();
    __syncwarp();
}

// P = tril(scale * decay * Q K^T) as bf16 into its triangular tile, rows 32 W .. + 31, one warp.
__device__ __forceinline__ void lean_mask_P(const MaskTables& tab, const float* prow, float scale0, uint32_t acc, int W, int lane, uint8_t* tile) {
    asm volatile("" : "+r"(lane));
    const int g = lane >> 2, t = lane & 3, R = 32 * W;
    const uint32_t tmem = tmem_addr(acc, 64 + R, 0), dst = smem_u32(tile) + 64 * R + tri_lane_offset(lane);   // (rows 32-63, columns 0-31 start at 2048)
    const bool k0 = 2 * t <= g, k1 = 2 * t + 1 <= g;
    float p[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) p[r] = prow ? prow[R + 8 * r + g] : scale0;
    auto pack2 = [](float2 f, float2 col, const uint32_t* v) {
        const float2 x = mul2(mul2(f, col), floats(v[0], v[1]));
        return pack_bf16x2(x.x, x.y);
    };
    auto block = [&](uint32_t at, float2 f0, float2 f1, float2 c0, float2 c1, const uint32_t* y) {
        stmatrix_x4(at, pack2(f0, c0, y), pack2(f1, c0, y + 2), pack2(f0, c1, y + 4), pack2(f1, c1, y + 6));
    };
    auto column = [&](const float* table, int c) { return *reinterpret_cast<const float2*>(table + 8 * c + 2 * t); };
    if (W == 1) {                    // columns 0-31
        const float2 c0 = column(tab.t32, 0), c1 = column(tab.t32, 1), c2 = column(tab.t32, 2), c3 = column(tab.t32, 3);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            uint32_t y[16];
            tmem_ld_16x256b_x4(tmem + ((16u * r) << 16), y);
            const float2 f0 = twice(p[2 * r] * tab.t32[32 + 16 * r + g]), f1 = twice(p[2 * r + 1] * tab.t32[40 + 16 * r + g]);
            tmem_ld_wait();
            block(dst + 1024 * r, f0, f1, c0, c1, y);
            block((dst + 1024 * r) ^ 32, f0, f1, c2, c3, y + 8);
        }
    }
    const uint32_t dg = dst + 64 * R;                      // the diagonal 32x32 block
    uint32_t x[8], y[16];
    tmem_ld_16x256b_x2(tmem + R, x);
    tmem_ld_16x256b_x4(tmem + (16u << 16) + R, y);
    float2 gj[4];
    float gi[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        gi[r] = tab.gam[R + 8 * r + g];
        gj[r] = column(tab.gcol + R, r);
    }
    tmem_ld_wait();
    auto diag = [&](uint32_t at, int r, const uint32_t* v) {   // the 16x16 block of rows and columns 8 r ..
        const float2 a = mul2(mul2(decay2(twice(gi[r]), gj[r]), twice(p[r])), floats(v[0], v[1]));
        const float2 b = mul2(mul2(decay2(twice(gi[r + 1]), gj[r]), twice(p[r + 1])), floats(v[2], v[3]));
        const float2 c = mul2(mul2(decay2(twice(gi[r + 1]), gj[r + 1]), twice(p[r + 1])), floats(v[6], v[7]));
        stmatrix_x4(at, pack_bf16x2(k0 ? a.x : 0.f, k1 ? a.y : 0.f), pack_bf16x2(b.x, b.y), 0, pack_bf16x2(k0 ? c.x : 0.f, k1 ? c.y : 0.f));
    };
    diag(dg, 0, x);
    stmatrix_x4(dg ^ 32, 0, 0, 0, 0);
    const float2 f0 = twice(p[2] * tab.t16[R + 16 + g]), f1 = twice(p[3] * tab.t16[R + 24 + g]);
    block(dg + 1024, f0, f1, column(tab.t16 + R, 0), column(tab.t16 + R, 1), y);
    diag((dg + 1024) ^ 32, 2, y + 8);
}

}  // namespace gdn
