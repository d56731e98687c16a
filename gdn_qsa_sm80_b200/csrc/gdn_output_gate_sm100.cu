// Gated RMS normalisation of the operator's output rows, the step that follows gdn_chunk in the layer:
//     out[r, :] = y[r, :] * rsqrt(mean(y[r, :]^2) + eps) * weight[:] * silu(z[r, :])        (rows of 128)
// Same arithmetic as the reference's rmsnorm_gated kernel (csrc/output_gate/output_gate.cu:47-98: fp32 sums,
// rsqrtf(sum / 128 + 1e-6), silu as z / (1 + exp(-z))) and its test's torch expression
// (tests/test_output_gate.py:12-16).
//
// The work is pure streaming (three 256-byte rows per output row), so the kernel is laid out for HBM: 16 threads
// own one row (one 16-byte copy per thread and tensor), the grid is one resident wave and strides over the rows.  Behind the forward pass, in
// place (out == y), most of y comes from HBM again: the chain's inputs and workspace pass through the 126 MB L2 beside it (255,872 rows: 113 of 131 MB read).
// A thread fetches its next five rows into shared memory asynchronously while it works on one, and behind the forward pass z's first rows, which the
// forward pass does not make, before the kernel before has ended.  (Four rows at a time in registers, loaded, then worked on: a call of 333 tokens with all a
// layer adds 23.1 us, now 22.0; 100 tokens 16.2 / 14.4; 4 x 1999 121.6 / 117.9; 2 x 8192 230 / 224.  Alone, 255,872 rows 33.0 / 31.6, 2 M rows 297 / 298.
// Rows ahead: 4 with three blocks per SM 121.4 on 4 x 1999, 3 with four 125.7, 6 and 7 with two 118.9 and 119.6.)
#include "../../include/gdn_chunk_sm100.h"
#include "gdn_common.cuh"
#include "gdn_gate_device.cuh"
#include "gdn_launch.cuh"
#include "ptx_sm100.cuh"

namespace gdn {
namespace {

constexpr int kGateThreads = 512;
constexpr int kGateBlocksPerSm = 2;
constexpr int kGateAhead = 5;         // rows of a thread on their way
constexpr uint32_t kGateSmem = kGateThreads * kGateAhead * 32;

__device__ __forceinline__ void copy16_async(uint32_t smem, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(reinterpret_cast<uint64_t>(g)) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__global__ void __launch_bounds__(kGateThreads, kGateBlocksPerSm) gdn_rmsnorm_gated_kernel(const uint4* y,   // may alias out
                                                                         const uint4* __restrict__ z,
                                                                         const uint4* __restrict__ weight, uint4* out,
                                                                         long long n_rows, float eps, bool z_ready) {
    extern __shared__ uint4 slots[];                        // [row ahead][y, z][thread]: a thread reads what it fetched itself
    const int tid = threadIdx.x;
    const long long step = static_cast<long long>(gridDim.x) * (kGateThreads / 16);
    const long long first = static_cast<long long>(blockIdx.x) * (kGateThreads / 16) + (tid >> 4);
    const long long lane_at = first * 16 + (tid & 15);      // 16-byte chunk of this thread in its first row
    // the loop bound is taken on the warp's first row so that both rows of a warp run the same iterations
    const long long bound = first - ((tid >> 4) & 1);
    const uint32_t base = smem_u32(slots) + tid * 16;
    auto fetch = [&](const uint4* src, uint32_t slot, long long i) {
        if (first + i * step < n_rows) copy16_async(base + slot * (kGateThreads * 16), src + lane_at + i * step * 16);
    };
    if (z_ready) {
#pragma unroll
        for (int d = 0; d < kGateAhead; ++d) fetch(z, 2 * d + 1, d);
    }
    grid_dependency_wait();   // launched while the kernel before drains
#pragma unroll
    for (int d = 0; d < kGateAhead; ++d) {
        fetch(y, 2 * d, d);
        if (!z_ready) fetch(z, 2 * d + 1, d);
        copies_commit();
    }
    float w[8];
    gate_unpack8(weight[tid & 15], w);
    uint32_t d = 0;
    for (long long i = 0; bound + i * step < n_rows; ++i) {
        copies_wait<kGateAhead - 1>();
        // rows past the end are not stored: every lane takes part in the shuffles, because the two rows of a warp can fall on either side of the end
        const uint4 yv = slots[(2 * d) * kGateThreads + tid], zv = slots[(2 * d + 1) * kGateThreads + tid];
        const uint4 pk = gate_row_slice(yv, zv, w, eps);
        if (first + i * step < n_rows) out[lane_at + i * step * 16] = pk;
        fetch(y, 2 * d, i + kGateAhead);
        fetch(z, 2 * d + 1, i + kGateAhead);
        copies_commit();
        d = d + 1 == kGateAhead ? 0 : d + 1;
    }
}

}  // namespace

cudaError_t launch_rmsnorm_gated(const void* y, const void* z, const void* weight, void* out, long long n_rows,
                                 float eps, cudaStream_t stream, bool z_ready) {
    if (n_rows <= 0) return cudaSuccess;
    const long long rows_per_block = kGateThreads / 16;
    long long blocks = (n_rows + rows_per_block - 1) / rows_per_block;
    const long long cap = static_cast<long long>(sm_count()) * kGateBlocksPerSm;   // one wave; blocks stride over the rows
    if (allow_smem(reinterpret_cast<const void*>(gdn_rmsnorm_gated_kernel), kGateSmem)) return cudaErrorInvalidValue;
    if (blocks > cap) blocks = cap;
    return launch_dependent(gdn_rmsnorm_gated_kernel, dim3(static_cast<unsigned>(blocks)), dim3(kGateThreads), kGateSmem, stream, false,
                            static_cast<const uint4*>(y), static_cast<const uint4*>(z), static_cast<const uint4*>(weight),
                            static_cast<uint4*>(out), n_rows, eps, z_ready);
}

}  // namespace gdn

extern "C" int gdn_rmsnorm_gated_sm100(const void* y, const void* z, const void* weight, void* out, long long n_rows,
                                       float eps, void* stream) {
    if (n_rows < 0 || (n_rows > 0 && (!y || !z || !weight || !out))) return GDN_ERR_BAD_ARGUMENT;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z) |
                           reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(out);
    if (bits & 15u) return GDN_ERR_BAD_ARGUMENT;
    return gdn::launch_rmsnorm_gated(y, z, weight, out, n_rows, eps, static_cast<cudaStream_t>(stream), false) == cudaSuccess
               ? GDN_OK
               : GDN_ERR_CUDA;
}
