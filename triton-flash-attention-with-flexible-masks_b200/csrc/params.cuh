// Kernel parameter blocks, filled by api.cu.
#pragma once
#include <atomic>
#include "common.cuh"

namespace fa {

constexpr int kDkdvThreads = 608;  // dK / dV: sixteen compute warps and the producer, MMA and scheduler warps
// forward: 4 warpgroups, two softmax groups, an epilogue group, a producer / MMA group. Registers a thread after setmaxnreg
constexpr int kFwdThreads = 512, kFwdSoftmaxRegs = 192, kFwdEpilogueRegs = 80, kFwdServiceRegs = 48;
static_assert(256 * kFwdSoftmaxRegs + 128 * (kFwdEpilogueRegs + kFwdServiceRegs) <= kFwdThreads * 128, "registers at launch");

struct FwdParams {
    float* lse;  // [B, H, Mpad], log2 domain
    MaskArgs mask;
    int H, B, G;
    int gh;            // heads per scheduling group
    int by_length;     // take the blocks of a head in the plan's sorted order (few items per CTA)
    float scale_log2;  // sm_scale * log2(e)
    int* status;
    long long wait_limit;  // SM clocks a bounded wait may last
    // calls without ids that are short of items (fwd_kernel, SHORT)
    int pack;         // query heads of a group that share a tile; 1: none
    int rows;         // rows of a Q / O box
    int ns;           // runs an item's tiles are cut into; 1: none
    float* part_o;    // [ns, B, H, M, 64 or 128] normalised rows of each run (ns > 1)
    float* part_lse;  // [B, H, M, ns]
};

struct CombineParams {
    const float* part_o;
    const float* part_lse;
    OutTensor o;
    float* lse;  // [B, H, Mpad]
    int B, H, M, D, Dk, ns;  // Dk: columns of a row of part_o
    int64_t Mpad;
    const int* status;
};

struct DeltaParams {
    OutTensor o, d_o;
    float* delta;  // [B, H, Mpad]
    int B, H, M, D;
    int64_t Mpad;
    bool bf16;
};

struct DkdvParams {
    const float* lse;    // [B, H, Mpad]
    const float* delta;  // [B, H, Mpad]
    MaskArgs mask;
    int B, H, Hk, G;
    // Head dim / 16. The columns that 64-wide tiles have beyond it are zeros, and S and dP leave them out: 16 x 8 heads x 577 x 32, dK/dV
    // 46.5 -> 45.5 us, dQ 40.6 -> 39.8. (The forward's S, which nothing waits for, was no faster.)
    int ksteps;
    int gh;  // kv heads per scheduling group
    int by_length;  // take the blocks of a head in the plan's sorted order (few items per CTA)
    float scale_log2, sm_scale;
    int* status;
    long long wait_limit;  // SM clocks a bounded wait may last
};

struct DqParams {
    const float* lse;
    const float* delta;
    MaskArgs mask;
    int B, H, G;
    int ksteps;  // as in DkdvParams
    int gh;  // heads per scheduling group
    int by_length;  // take the blocks of a head in the plan's sorted order (few items per CTA)
    float scale_log2, sm_scale;
    int* status;
    long long wait_limit;  // SM clocks a bounded wait may last
};

// fp32 kernels (attn_f32.cu): plain pointers and element strides, no tensor maps
struct F32Tensor {
    float* ptr;
    int64_t sb, sh, sl;  // element strides; the D stride is 1
};

struct F32Params {
    F32Tensor q, k, v, o, d_o, dq, dk, dv;
    float* lse;    // [B, H, Mpad], natural log-sum-exp of the scaled scores; -inf for a row without keys
    float* delta;  // [B, H, Mpad]
    MaskArgs mask;
    int B, H, Hk, G;
    float scale;
};

// A number for the current CUDA context that no other context of the process ever has, or 0 (api.cu).
uint64_t context_number();

// The contexts in which a kernel may already use its dynamic shared memory. One per kernel.
struct SmemAllowed {
    std::atomic<uint64_t> context[16] = {};
};

// Lets `kern` use `bytes` of dynamic shared memory. The attribute belongs to the context (a process may have several on
// one device, and a device reset makes a new one), so it is set once per context, always to the same value.
template <class Kernel>
inline cudaError_t allow_smem(Kernel kern, int bytes, SmemAllowed& allowed) {
    const uint64_t number = context_number();
    std::atomic<uint64_t>& slot = allowed.context[number % 16];
    if (number && slot.load(std::memory_order_relaxed) == number) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) slot.store(number, std::memory_order_relaxed);
    return e;
}

// Launches `kern` so that it may start on SMs that the kernel before it in the stream has left, or leaves room on, once
// all of that one's blocks have called launch_dependents() or left. `kern` begins with follow_stream() (or with its two parts around
// the allocation of tensor memory), or, where it needs nothing of that kernel, ends with wait_prerequisites().
// Nearly all launches are of this kind: the gap from one kernel to the next, 2 to 3 us with a kernel's setup, shrinks to about 1.
template <class... Params, class... Args>
inline cudaError_t launch_overlapping(void (*kern)(Params...), dim3 grid, int threads, int smem, cudaStream_t stream, const Args&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

}  // namespace fa
