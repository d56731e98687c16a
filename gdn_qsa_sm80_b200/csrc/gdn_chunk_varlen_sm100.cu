// Packed batch: sequences of different lengths laid end to end in [1, T, H, .] tensors, in one pass of the two-kernel path.
//
// The kernels find a chunk's sequence through three small tables (first token of each sequence; (sequence, chunk) per 64-token
// chunk; (sequence, first chunk, segment) in the order the chain's CTAs take them), written to the scratch buffer by a kernel whose parameters carry the lengths: no copy from the host, and a captured graph keeps them.
// The last tile of a sequence also holds the next one's first tokens; gates and beta count as zero there, and the kernels
// mask those rows (prepare) or clear them in the tile (chain), so no sequence ever sees another's values.
// Sequences of at most kDecodeMaxTokens tokens take the decode kernel, all of them in one launch through a table of their own (256
// sequences of 1 to 8 tokens, 32 heads: 1491 us with a launch per run of equal lengths, 271 now; before the packed route a padded
// batch, 957).
//
// Without this a packed batch was gathered into a padded one and scattered back (torch indexing: two passes over all
// tensors, and the padding's share of the work), or ran sequence by sequence.
#include <algorithm>
#include <vector>

#include "../../include/gdn_chunk_sm100.h"
#include "gdn_common.cuh"
#include "gdn_launch.cuh"
#include "ptx_sm100.cuh"

namespace gdn {
namespace {

constexpr int kPiece = 1024;          // sequences per launch of the table kernel (kernel parameters: 12 KB)
struct TablePiece {
    int first;                        // sequence of entry 0
    int start[kPiece + 1];
    int chunk0[kPiece];               // its first entry in the chunk table; -1: a short sequence, entry `rank` of their table
    unsigned rank[kPiece];            // 16 rank + segs: its entries in the chain's work list are layer[s] + rank for s < segs
    static_assert(kMaxSegments < 16, "segs in four bits");
    int layer[kMaxSegments];
};

__global__ void __launch_bounds__(64) gdn_pack_tables_kernel(const __grid_constant__ TablePiece piece, int* cu, int2* chunk, int4* order,
                                                             int4* shorts, int* status) {
    grid_dependency_wait();           // earlier kernels of the stream may still read the tables of their own call
    grid_launch_dependents();
    const int i = blockIdx.x, seq = piece.first + i, c0 = piece.chunk0[i], len = piece.start[i + 1] - piece.start[i];
    const int rank = static_cast<int>(piece.rank[i] >> 4), segs = piece.rank[i] & 15;
    if (threadIdx.x == 0) {
        cu[seq] = piece.start[i];
        cu[seq + 1] = piece.start[i + 1];   // (the next sequence's block writes the same value)
        if (c0 < 0) shorts[rank] = make_int4(seq, piece.start[i], len, 0);
        if (seq == 0 && status) *status = 0;
    }
    if (c0 < 0) return;
    const int nt = (len + kChunk - 1) / kChunk;
    if (threadIdx.x < segs) order[piece.layer[threadIdx.x] + rank] = make_int4(seq, c0, threadIdx.x, segs);
    for (int t = threadIdx.x; t < nt; t += blockDim.x) chunk[c0 + t] = make_int2(seq, t);
}

struct PackedLayout {
    WorkspaceLayout ws;
    size_t cu, chunk, order, shorts, total;
    size_t chunks;                    // 64-token chunks of the sequences that take the two-kernel path
    int longs;                        // how many those are
    int longest;                      // chunks of the longest
    int n_short, short_runs, most;    // the other sequences, their runs of equal lengths, the most tokens one has
};
PackedLayout packed_layout(const int* cu, int n_seq, int Hv) {
    PackedLayout l{};
    for (int i = 0; i < n_seq; ++i) {
        const int n = cu[i + 1] - cu[i], nt = (n + kChunk - 1) / kChunk;
        if (n <= kDecodeMaxTokens) {
            if (i == 0 || cu[i] - cu[i - 1] != n) ++l.short_runs;
            if (n > l.most) l.most = n;
            ++l.n_short;
            continue;
        }
        if (nt > l.longest) l.longest = nt;
        l.chunks += nt;
        ++l.longs;
    }
    l.ws = workspace_layout(l.chunks * Hv, true);
    auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
    l.cu = up(l.ws.total);
    l.chunk = up(l.cu + (static_cast<size_t>(n_seq) + 1) * 4);
    l.order = up(l.chunk + l.chunks * 8);
    l.shorts = up(l.order + static_cast<size_t>(l.longs) * kMaxSegments * sizeof(int4));
    l.total = up(l.shorts + static_cast<size_t>(l.n_short) * sizeof(int4));
    return l;
}
bool bounds_rise(const int* cu, int n_seq) {
    if (!cu || n_seq <= 0 || cu[0] != 0) return false;
    for (int i = 0; i < n_seq; ++i)
        if (cu[i + 1] <= cu[i]) return false;
    return true;
}

}  // namespace
}  // namespace gdn

using namespace gdn;

extern "C" {

size_t gdn_chunk_varlen_scratch_bytes(const int* cu_seqlens, int n_seq, int Hv) {
    return bounds_rise(cu_seqlens, n_seq) && Hv > 0 ? packed_layout(cu_seqlens, n_seq, Hv).total : 0;
}

int gdn_chunk_fwd_varlen_sm100(const void* q, const void* k, const void* v, const void* g, const void* beta, const float* h0,
                               void* out, float* hT, void* scratch, size_t scratch_bytes, const int* cu_seqlens, int n_seq,
                               int Hq, int Hv, int gate_dtype, unsigned flags, void* stream_) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (!bounds_rise(cu_seqlens, n_seq) || Hq <= 0 || Hv <= 0 || Hv % Hq != 0) return GDN_ERR_BAD_ARGUMENT;
    if (gate_dtype != GDN_GATE_BF16 && gate_dtype != GDN_GATE_F32) return GDN_ERR_BAD_ARGUMENT;
    if (flags & ~static_cast<unsigned>(GDN_FLAG_QK_L2NORM | GDN_FLAG_GATE_ACTIVATIONS)) return GDN_ERR_BAD_ARGUMENT;
    if (!q || !k || !v || !g || !beta || !out) return GDN_ERR_BAD_ARGUMENT;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                           reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(h0) | reinterpret_cast<uintptr_t>(hT);
    if (bits & 15u) return GDN_ERR_BAD_ARGUMENT;
    const PackedLayout l = packed_layout(cu_seqlens, n_seq, Hv);
    if (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 255u) || scratch_bytes < l.total) return GDN_ERR_SCRATCH;
    const EnqueueLock lock(scratch);
    uint8_t* base = static_cast<uint8_t*>(scratch);
    bool clear = true;                // whichever kernel comes first clears the status word

    Problem p = {};
    p.q = static_cast<const __nv_bfloat16*>(q);
    p.k = static_cast<const __nv_bfloat16*>(k);
    p.v = static_cast<const __nv_bfloat16*>(v);
    p.g = g;
    p.beta = beta;
    p.h0 = h0;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.hT = hT;
    p.status = static_cast<int*>(scratch);
    p.Hq = Hq;
    p.Hv = Hv;
    p.gate_f32 = gate_dtype == GDN_GATE_F32;
    p.l2norm = (flags & GDN_FLAG_QK_L2NORM) ? 1 : 0;
    p.gate_act = (flags & GDN_FLAG_GATE_ACTIVATIONS) ? 1 : 0;
    const bool listed = l.short_runs > 1;   // one run needs no table
    int most_segments = 1;
    if (l.longs > 0 || listed) {
        std::vector<int> rank, order, segs;
        try {
            rank.resize(n_seq);
            segs.resize(n_seq);
            order.reserve(l.longs);
        } catch (...) {               // nothing may be thrown through a C entry
            return GDN_ERR_SCRATCH;
        }
        int n_short = 0;
        auto chunks_of = [&](int s) { return (cu_seqlens[s + 1] - cu_seqlens[s] + kChunk - 1) / kChunk; };
        for (int i = 0; i < n_seq; ++i) {
            if (cu_seqlens[i + 1] - cu_seqlens[i] <= kDecodeMaxTokens) {
                rank[i] = n_short++;
                continue;
            }
            order.push_back(i);
            // two CTAs per SM; states in place: the CTA that reads a state must be the one that writes it
            segs[i] = h0 && h0 == hT ? 1 : chain_segments(static_cast<long long>(l.chunks) * Hv, chunks_of(i), 2 * sm_count());
        }
        // Order of the chain's work list.  First what takes long, segment by segment: the first segments of all sequences that may be
        // cut (and the long ones that may not), their second ones, ...: a head whose decay forbids the cut runs all of it in
        // its first segment's CTA, and those then find SMs of their own (4 sequences of 4096 tokens of slow decay, 32 heads: 220 us,
        // 278 us with the segments of a sequence side by side).  Last the short sequences, longest first: they fill what is left.
        int entries = 0, most = 1, longest_run = 0, layer[kMaxSegments] = {};
        auto run = [&](int s) { return chunks_of(s) / segs[s]; };
        for (int s : order) longest_run = std::max(longest_run, run(s));
        auto fills = [&](int s) { return segs[s] == 1 && 2 * run(s) < longest_run; };
        std::sort(order.begin(), order.end(), [&](int a, int b) {
            if (fills(a) != fills(b)) return fills(b);
            if (segs[a] != segs[b]) return segs[a] > segs[b];
            return run(a) != run(b) ? run(a) > run(b) : a < b;
        });
        int firsts = 0;
        for (int s : order) {
            if (fills(s)) break;
            rank[s] = firsts++;
            most = std::max(most, segs[s]);
        }
        for (int seg = 0; seg < most; ++seg) {
            layer[seg] = entries;
            for (int r = 0; r < firsts && segs[order[r]] > seg; ++r) ++entries;
        }
        for (int r = firsts; r < l.longs; ++r) rank[order[r]] = entries++;
        int* d_cu = reinterpret_cast<int*>(base + l.cu);
        int2* d_chunk = reinterpret_cast<int2*>(base + l.chunk);
        int4* d_order = reinterpret_cast<int4*>(base + l.order);
        int4* d_shorts = reinterpret_cast<int4*>(base + l.shorts);
        int c = 0;
        for (int i0 = 0; i0 < n_seq; i0 += kPiece) {
            TablePiece piece;
            piece.first = i0;
            std::copy(layer, layer + kMaxSegments, piece.layer);
            const int n = std::min(kPiece, n_seq - i0);
            for (int i = 0; i < n; ++i) {
                const int s = i0 + i, len = cu_seqlens[s + 1] - cu_seqlens[s];
                piece.start[i] = cu_seqlens[s];
                piece.rank[i] = 16u * static_cast<unsigned>(rank[s]) + static_cast<unsigned>(segs[s]);
                piece.chunk0[i] = len > kDecodeMaxTokens ? c : -1;
                if (len > kDecodeMaxTokens) c += (len + kChunk - 1) / kChunk;
            }
            piece.start[n] = cu_seqlens[i0 + n];
            const cudaError_t e = launch_dependent(gdn_pack_tables_kernel, dim3(n), dim3(64), 0, stream, false, piece, d_cu, d_chunk, d_order, d_shorts,
                                                   i0 == 0 ? static_cast<int*>(scratch) : static_cast<int*>(nullptr));
            if (e != cudaSuccess) return GDN_ERR_CUDA;
        }
        clear = false;
        p.pk_cu = d_cu;
        p.pk_chunk = d_chunk;
        p.pk_order = d_order;
        p.pk_n = entries;
        p.pk_chunks = static_cast<int>(l.chunks);
        p.pk_longest = l.longest;
        p.pk_short = d_shorts;
        p.pk_shorts = l.n_short;
        most_segments = most;
    }
    if (l.longs > 0) {
        p.B = 1;
        p.S = cu_seqlens[n_seq];
        Workspace ws = {};
        ws.P = reinterpret_cast<__nv_bfloat16*>(base + l.ws.P);
        ws.U = reinterpret_cast<__nv_bfloat16*>(base + l.ws.U);
        ws.vec = reinterpret_cast<float*>(base + l.ws.vec);
        ws.n_seg = most_segments;
        ws.meta = ws.n_seg > 1 ? reinterpret_cast<float*>(base + l.ws.meta) : nullptr;
        TileMaps maps;
        if (encode_tile_maps(p, ws, maps)) return GDN_ERR_DRIVER;
        int st = launch_prepare_lean(p, ws, maps, stream);
        if (st == GDN_OK) st = launch_chain_r(p, ws, maps, stream);
        if (st != GDN_OK) return st;
    }
    if (listed) {
        p.B = n_seq;
        p.S = l.most;
        return launch_decode(p, nullptr, stream);
    }
    // one run of short sequences (or none): a regular batch of the decode kernel
    const size_t gate_bytes = gate_dtype == GDN_GATE_F32 ? 4 : 2;
    for (int i = 0; i < n_seq;) {
        const int n = cu_seqlens[i + 1] - cu_seqlens[i];
        int j = i + 1;
        if (n <= kDecodeMaxTokens) {
            while (j < n_seq && cu_seqlens[j + 1] - cu_seqlens[j] == n) ++j;
            const size_t tok = cu_seqlens[i], state = static_cast<size_t>(i) * Hv * kD * kD;
            auto at = [](const void* x, size_t bytes) -> const void* { return static_cast<const char*>(x) + bytes; };
            const int st = forward_device(at(q, tok * Hq * kD * 2), at(k, tok * Hq * kD * 2), at(v, tok * Hv * kD * 2),
                                          at(g, tok * Hv * gate_bytes), at(beta, tok * Hv * gate_bytes), h0 ? h0 + state : nullptr,
                                          static_cast<char*>(out) + tok * Hv * kD * 2, hT ? hT + state : nullptr, scratch, scratch_bytes,
                                          j - i, n, Hq, Hv, gate_dtype, GDN_PATH_DECODE, flags, stream, clear);
            if (st != GDN_OK) return st;
            clear = false;
        }
        i = j;
    }
    return GDN_OK;
}

}  // extern "C"
