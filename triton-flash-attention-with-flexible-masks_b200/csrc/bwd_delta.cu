// delta[b,h,i] = sum_d O[b,h,i,d] * dO[b,h,i,d] in fp32. Replaces `_bwd_preprocess`
// (flash_triton.py:143-173). HBM-bound: reads O and dO once, writes one float per row.
// The output is padded to a multiple of 128 rows per (b,h); padding rows are written as 0 so
// that the backward kernels can bulk-copy whole 128-row slices.
#include <cuda_fp16.h>
#include "common.cuh"
#include "params.cuh"

namespace fa {

// D / 8 neighbouring threads read a row, 16 bytes of O and of dO each, so that a warp's load covers whole 128-byte lines, and each thread
// has the loads of its kRows rows in flight before it uses the first. Bound by HBM.
// us between events in a graph, eight threads a row with 2 x D / 8 elements and one row each | now: 16 x 8 x 577 x 32 6.1 | 2.8, 8 x 8 x 1024 x 64
// 5.2 | 3.3, 4 x 12 x 1000 x 64 4.1 | 3.0, 2 x 32 x 3001 x 128 16.2 | 14.2, 32 x 32768 x 128 96.7 | 83.1 (6.5 TB/s), 4 x 16 x 4096 x 128 21.1 | 21.2; one row
// a thread 18.3 and 103 in the fourth and fifth, four rows 21.7 in the last.
template <int D>
struct DeltaShape {
    static constexpr int kThreads = 256, kLanes = D / 8, kRows = 2;
    static constexpr int kStep = kThreads / kLanes;     // rows that the block's threads read together
    static constexpr int kBlockRows = kStep * kRows;
};

template <int D, bool BF16>
__global__ void __launch_bounds__(256) bwd_delta_kernel(const DeltaParams p) {
    using S = DeltaShape<D>;
    follow_stream();
    const int h = blockIdx.y, b = blockIdx.z;
    const int row0 = blockIdx.x * S::kBlockRows + int(threadIdx.x) / S::kLanes;
    const int part = int(threadIdx.x) % S::kLanes;
    const uint16_t* po = static_cast<const uint16_t*>(p.o.ptr) + int64_t(b) * p.o.sb + int64_t(h) * p.o.sh + part * 8;
    const uint16_t* pd = static_cast<const uint16_t*>(p.d_o.ptr) + int64_t(b) * p.d_o.sb + int64_t(h) * p.d_o.sh + part * 8;
    uint4 a[S::kRows], g[S::kRows];
#pragma unroll
    for (int r = 0; r < S::kRows; ++r) {
        const int row = row0 + r * S::kStep;
        a[r] = g[r] = make_uint4(0, 0, 0, 0);
        if (row < p.M) {
            a[r] = *reinterpret_cast<const uint4*>(po + int64_t(row) * p.o.sl);
            g[r] = *reinterpret_cast<const uint4*>(pd + int64_t(row) * p.d_o.sl);
        }
    }
#pragma unroll
    for (int r = 0; r < S::kRows; ++r) {
        const uint32_t aw[4] = {a[r].x, a[r].y, a[r].z, a[r].w};
        const uint32_t gw[4] = {g[r].x, g[r].y, g[r].z, g[r].w};
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float a0, a1, g0, g1;
            if constexpr (BF16) {
                a0 = __uint_as_float(aw[k] << 16); a1 = __uint_as_float(aw[k] & 0xffff0000u);
                g0 = __uint_as_float(gw[k] << 16); g1 = __uint_as_float(gw[k] & 0xffff0000u);
            } else {
                const __half2 ah = *reinterpret_cast<const __half2*>(&aw[k]);
                const __half2 gh = *reinterpret_cast<const __half2*>(&gw[k]);
                a0 = __low2float(ah); a1 = __high2float(ah);
                g0 = __low2float(gh); g1 = __high2float(gh);
            }
            acc = fmaf(a0, g0, acc);
            acc = fmaf(a1, g1, acc);
        }
#pragma unroll
        for (int o = 1; o < S::kLanes; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const int row = row0 + r * S::kStep;
        if (part == 0 && row < p.Mpad) p.delta[(int64_t(b) * p.H + h) * p.Mpad + row] = acc;
    }
}

template <int D>
static cudaError_t launch_delta_t(const DeltaParams& p, cudaStream_t stream) {
    const dim3 grid(unsigned((p.Mpad + DeltaShape<D>::kBlockRows - 1) / DeltaShape<D>::kBlockRows), p.H, p.B);
    return launch_overlapping(p.bf16 ? bwd_delta_kernel<D, true> : bwd_delta_kernel<D, false>, grid, DeltaShape<D>::kThreads, 0, stream, p);
}

cudaError_t launch_bwd_delta(const DeltaParams& p, cudaStream_t stream) {
    if (p.D == 128) return launch_delta_t<128>(p, stream);
    if (p.D == 64) return launch_delta_t<64>(p, stream);
    if (p.D == 32) return launch_delta_t<32>(p, stream);
    return launch_delta_t<16>(p, stream);
}

}  // namespace fa
