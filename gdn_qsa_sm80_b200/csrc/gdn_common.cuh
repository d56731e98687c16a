// Declarations shared by the gdn_chunk translation units (internal; the public surface is
// include/gdn_chunk_sm100.h).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

// The kernels' cycle accounting is compiled in only with -DGDN_DIAGNOSTICS; otherwise every "is accounting on"
// test is the constant false and the accounting code disappears from the kernels.
#ifdef GDN_DIAGNOSTICS
#define GDN_DIAG(x) (x)
#else
#define GDN_DIAG(x) false
#endif

namespace gdn {

constexpr int kD = 128;      // head dimension (keys and values)
constexpr int kChunk = 64;   // tokens per chunk
constexpr float kLog2e = 1.4426950408889634f;

// Test hooks of Problem::dbg (7: gdn_chunk_coop_sm100.cu).  Those of the two-kernel path are compiled into instantiations of their own: a comparison
// in its loops made calls of a few tokens 0.3 to 1 % longer.
constexpr int kDbgLateProducer = 8;    // residual-form chain: the TMA producer sleeps 20 us before it looks at a barrier
constexpr int kDbgWarpGivesUp = 9;     // residual-form chain: one of the output warps waits for a barrier that nothing completes instead of the first outputs
constexpr int kDbgNoTile = 10;         // residual-form chain: the first tile of V is never announced
constexpr int kDbgNoProduct = 11;      // lean prepare: no CTA's first product is issued
constexpr int kDbgLaneGivesUp = 12;    // lean prepare: one lane of each CTA that is not its warp's first has given up
constexpr int kDbgLaneWaits = 13;      // lean prepare: the same lane waits for a barrier that nothing completes in place of its own

struct Problem {
    const __nv_bfloat16* q;
    const __nv_bfloat16* k;
    const __nv_bfloat16* v;
    const void* g;
    const void* beta;
    const float* h0;       // may be null
    __nv_bfloat16* out;
    float* hT;             // may be null
    int* status;           // device status word (never null)
    long long* prof;       // optional: 16 per-phase cycle counters written by CTA (0,0,0); null = off
    int B, S, Hq, Hv;
    int gate_f32;          // 0: g/beta are bf16, 1: fp32
    int gate_act;          // 1: g and beta hold raw values; the kernels apply g = -softplus(.), beta = sigmoid(.)
    int l2norm;            // 1: q and k are L2-normalised per head vector inside the kernels
    int clear_status;      // 1: the launch's first kernel clears the status word
    int behind_prepare;    // 1: the residual-form chain is launched right behind the prepare kernel of the same call
    int dbg;               // test hook (environment variable GDN_CHUNK_DBG); 0 in production
    // Packed batch (residual-form kernels only; null / 0 otherwise): B = 1, S = all tokens, sequences laid end to end
    const int* pk_cu;      // [pk_n + 1] first token of each sequence
    const int2* pk_chunk;  // [pk_chunks] (sequence, chunk within it), sequences in order
    const int4* pk_order;  // [pk_n] what a row of the chain's grid runs: (sequence, its first entry in pk_chunk, segment, segments
                           // it may be cut into)
    int pk_n, pk_chunks, pk_longest;   // entries of the two tables; chunks of the longest sequence
    const int4* pk_short;  // decode kernel: [pk_shorts] (sequence, first token, tokens); B = all sequences, S = the most tokens
    int pk_shorts;
};

// Workspace of the two-kernel path (device pointers into the caller's scratch buffer).
// One tile per (batch, value head, chunk): tile = (b * Hv + hv) * NT + t.
struct Workspace {
    __nv_bfloat16* W;   // [tiles][64][128]  W = T (beta e^gamma K)
    __nv_bfloat16* P;   // [tiles][64][64]   masked, scaled Q K^T
    __nv_bfloat16* U;   // [tiles][64][128]  U = T (beta V); the transposed chain's T'' = T diag(beta), [tiles][64][64], instead
    float* vec;         // [tiles][256]      exp(gamma_C-gamma_i) | scale exp(gamma_i) | exp(gamma_C), pad | exp(gamma_i)
    float* meta;        // [tiles][2]        sum of g over the chunk | max_j beta_j |k_j|^2 (+inf if a gate is out of range);
                        //                   null when sequences are not split
    int n_seg;          // segments a sequence is split into by the transposed chain (1 = not split)
};

// Byte offsets of the workspace arrays inside the scratch buffer (the status word sits at offset 0).
struct WorkspaceLayout {
    size_t W, P, U, vec, flags, flag_bytes, meta, total;
};
// with_meta: room for the two scalars per tile that the on-device decision to split sequences reads
inline WorkspaceLayout workspace_layout(size_t tiles, bool with_meta = false) {
    WorkspaceLayout l;
    l.W = 1024;
    l.P = l.W + tiles * 16384;
    l.U = l.P + tiles * 8192;
    l.vec = l.U + tiles * 16384;
    l.flags = l.vec + tiles * 1024;                      // one int per tile: "prepared" flags of the single-launch path
    l.flag_bytes = (tiles * 4 + 1023) / 1024 * 1024;
    l.meta = l.flags + l.flag_bytes;
    l.total = l.meta + (with_meta ? (tiles * 8 + 1023) / 1024 * 1024 : 0);
    return l;
}
// The most segments the chain may cut a sequence of NT chunks into (1 = not at all; how many a head uses is decided on
// the device, gdn_segment_plan.cuh): its share of the CTAs the GPU holds at once (`slots`) by its share of the launch's chunks
// (`chunks`: over all sequences and heads; equal sequences: slots / (sequences x heads) each), segments of at least four chunks on
// average.  A sequence of less than twice the average load of a slot is not cut: the CTAs beside it fill the time.
// A function of the lengths and of the SM count alone.  One of 30000 tokens with twenty of 50-100 beside it, 32 heads: 1.18 ms
// when the NUMBER of sequences decided, 0.36 now (the long one alone 0.31).
constexpr int kMaxSegments = 15;
constexpr int kPlanChunks = 24000;   // units of the plan: their prefix sums have to fit the ring's shared memory (longer sequences: several chunks a unit)
inline int chain_segments(long long chunks, int NT, int slots) {
    if (chunks <= 0) return 1;
    const long long share = static_cast<long long>(NT) * slots / chunks;
    int g = share > kMaxSegments ? kMaxSegments : static_cast<int>(share);
    if (g > NT / 4) g = NT / 4;
    return g < 2 ? 1 : g;
}
constexpr int kDecodeMaxTokens = 8;   // sequences this short take the decode kernel under GDN_PATH_AUTO
constexpr float kForgetLn = -115.f;   // exp(-115) < 2^-149: a transfer matrix bounded by it is zero in fp32

// Device status codes written by kernels (0 = fine).  The low byte says which wait gave up.
constexpr int kDevTimeoutTma = 0x101;
constexpr int kDevTimeoutMma = 0x102;

void count_launch();

// Token-by-token fp32 kernel on CUDA cores (one CTA per (batch, value head)).
cudaError_t launch_simt(const Problem& p, cudaStream_t stream);

// "prepare" (state-independent per-chunk quantities into the workspace) and "chain" (the serial
// state recurrence plus outputs, reading the workspace).  Both return a GDN_* status.
int launch_prepare(const Problem& p, const Workspace& ws, cudaStream_t stream);
int launch_chain(const Problem& p, const Workspace& ws, int nv, cudaStream_t stream);
// The two kernels of the automatic path: "lean" prepare (P, T'', factors; no W) and the transposed chain that applies T'' to
// the residual V - exp(gamma) K S, one CTA per (sequence, value head[, segment]); with ws.n_seg > 1 sequences may be cut
// into up to that many segments (gdn_segment_plan.cuh).
// TMA descriptors of both (128 bytes each, CUtensorMap): q, k, v and the outputs as 64 x 64 boxes, P and T'' (at the start of the
// U array) as 32 x 32 boxes (64-byte swizzle): both are lower triangular, so a tile travels as its three blocks on and below
// the diagonal and the fourth is neither written nor read (16 sequences of 2048 tokens: 391 -> 376 us per call, 64 of 4096
// 2958 -> 2870 us).  Encoded once per call: each encoding costs the host 0.1-0.2
// microseconds.
constexpr uint32_t kTriBytes = 6144;   // a triangular tile in shared memory: rows 0-63 of columns 0-31, then rows 32-63 of columns 32-63
struct alignas(64) TileMaps {
    unsigned char q[128], k[128], v[128], p[128], t2[128], out[128];
};
int encode_tile_maps(const Problem& p, const Workspace& ws, TileMaps& maps);
int launch_prepare_lean(const Problem& p, const Workspace& ws, const TileMaps& maps, cudaStream_t stream);
int launch_chain_r(const Problem& p, const Workspace& ws, const TileMaps& maps, cudaStream_t stream);
// Single-launch variant (prepare shared among the four column CTAs of a head, chain in the same kernel);
// only when all CTAs fit on the GPU at once.
bool coop_supported(const Problem& p);
// skip_prepare (measurement aid): run only the chain roles on a workspace an earlier call left behind.
int launch_coop(const Problem& p, const Workspace& ws, int* flags, size_t flag_bytes, cudaStream_t stream,
                bool skip_prepare = false);

// Host helper: encode a tiled TMA descriptor for a row-major tensor of `rank` dims
// (dims/strides innermost first; strides in bytes for dims 1..rank-1).  swizzle_bytes: 128 or 64.
// elem_bytes: 2 = bf16, 4 = fp32.  Returns 0 on success.
int encode_tma(void* tmap_out, const void* base, int elem_bytes, int rank, const unsigned long long* dims,
               const unsigned long long* strides_bytes, const unsigned* box, int swizzle_bytes);
inline int encode_tma_bf16(void* tmap_out, const void* base, int rank, const unsigned long long* dims,
                           const unsigned long long* strides_bytes, const unsigned* box, int swizzle_bytes) {
    return encode_tma(tmap_out, base, 2, rank, dims, strides_bytes, box, swizzle_bytes);
}
// TMA descriptors of the workspace arrays: W, P and U as 64x64 bf16 boxes (128-byte swizzle; what the prepare side
// stores and the chain side loads for W and P), and U as nv x 64 boxes (swizzle span 2*nv bytes) for the chain's
// column slice.  tu_load may be null.
int encode_workspace_maps(const Problem& p, const Workspace& ws, void* tw, void* tp, void* tu_store, void* tu_load, int nv);
// Number of SMs of the current device (cached per device).
int sm_count();
// z_ready: the kernel before it in the stream does not make z, and has waited for whatever did.
cudaError_t launch_rmsnorm_gated(const void* y, const void* z, const void* weight, void* out, long long n_rows,
                                 float eps, cudaStream_t stream, bool z_ready);
// The forward pass on device buffers (what gdn_chunk_fwd_sm100_ex does).  clear_status = false leaves the status
// word at the start of `scratch` as it is, so that several launches can share one sticky word.
// gate != nullptr: the output rows are replaced by rmsnorm_gated(row, z, weight), by the normalisation kernel
// launched right behind the forward pass.
struct OutputGate {
    const void* z;
    const void* weight;
    float eps;
};
// Token-by-token kernel for a few new tokens on stored states; og: gated normalisation of its rows in the same launch.
int launch_decode(const Problem& p, const OutputGate* og, cudaStream_t stream);
int forward_device(const void* q, const void* k, const void* v, const void* g, const void* beta, const float* h0,
                   void* out, float* hT, void* scratch, size_t scratch_bytes, int B, int S, int Hq, int Hv,
                   int gate_dtype, int path, unsigned flags, cudaStream_t stream, bool clear_status,
                   const OutputGate* gate = nullptr);
// TMA descriptors of q, k ([B,S,Hq,128], 64x64 boxes) and v ([B,S,Hv,128], v_box_cols x 64 boxes).
int encode_qkv_maps(const Problem& p, void* tq, void* tk, void* tv, int v_box_cols);

}  // namespace gdn
