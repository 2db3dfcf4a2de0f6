// fp32 inputs (flash_triton.py:512 accepts any float dtype; testing.py:158 lists fp32). The tensor-core
// kernels of this library work on 16-bit operands; a 16-bit product cannot meet the 1e-4 tolerance
// asked of fp32 results, so fp32 tensors take the kernels below: the same flash-attention recurrence
// (flash_triton.py:94-133 forward, :250-311 dK/dV, :387-423 dQ), the same mask plan, tile
// classification and per-entry predicate as the 16-bit kernels, but all arithmetic in fp32 FMAs.
// They cover every head dim the reference accepts (16, 32, 64, 128).
//
// One CTA works on 32 or 16 "rows" (queries in the forward and dQ kernels, keys in the dK/dV kernel) against
// tiles of 64 "columns", which cp.async brings into the other of two shared-memory stages while a tile is worked
// on. A warp owns four rows from the scores to the result: lane x has columns x and x + 32 of the scores (4 x 2
// products in registers) and D / 32 columns of the result, so the softmax needs no barrier and P passes through the
// warp's own part of shared memory, where the four rows of a column lie side by side: two packed FMAs take them as they are. These calls are a few
// hundred rows of a few heads: what bounds them is the chain of tiles of the longest CTA, in it a warp's own steps and the shared-memory reads.
// A 16-byte read takes one pass per 8 lanes even where lanes repeat
// an address, so all lanes of a warp share the rows (one pass) and none shares a column: 12 passes per 32 FMAs of a
// warp, about half of what half-warps with two rows each took. (Eight rows a warp take 8 passes, but leave half as many warps: forward and
// backward of 8 heads x 512 x 64 127 us for 115, of 32 x 1024 714 for 729; two rows a warp 125 and 1012.) Packed FMAs for P V and its like and one
// reduction for the maximum: 118.5 -> 113 us for 8 heads x 512 x 64, 874 -> 851 for 32 x 1024.
#include "../../include/fa_b200.h"
#include "common.cuh"
#include "params.cuh"

namespace fa {

constexpr int kC = 64;          // columns per tile
constexpr int kRW = 4;          // rows per warp
__host__ __device__ constexpr int threads(int rows) { return rows / kRW * 32; }

template <int D, int R>
struct F32Smem {
    static constexpr int LD = D + 4;  // pitch: 8 lanes that read 16 bytes each of neighbouring rows hit all 32 banks
    static constexpr int rows = R * LD, cols = kC * LD, p = R * kC;  // floats
    static constexpr int vec = 3 * kC;                                   // per column: id code, lse, delta
    static constexpr int fwd_bytes = (rows + 4 * cols + p + 2 * kC) * 4, bwd_bytes = (2 * rows + 4 * cols + p + 2 * vec) * 4;
    static_assert(bwd_bytes + kListCap <= 232448, "shared memory budget");
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool real) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool real) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(real ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ bool rows_aligned(const float* base, int64_t sl) {
    return (reinterpret_cast<uintptr_t>(base) & 15u) == 0 && (sl & 3) == 0;
}

// starts the copy of rows [r0, r0 + NR) of a slice into a padded tile; rows outside [lo, hi) become zero: those outside
// the tensor, and those that the causal mask hides from the whole CTA, for their products with a P of 0 would be NaN
// where they hold a NaN or an infinity. Tensors are only promised to be 4-byte aligned: `vec` says that every row of
// this one starts on 16 bytes.
template <int D, int NR, int R>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int64_t sl, bool vec, int r0, int hi, int lo = 0) {
    constexpr int LD = F32Smem<D, R>::LD, kThreads = threads(R);
    if (vec) {
#pragma unroll 4
        for (int i = threadIdx.x; i < NR * (D / 4); i += kThreads) {
            const int r = i / (D / 4), c = i % (D / 4) * 4;
            const bool real = r0 + r >= lo && r0 + r < hi;
            cp_async16(smem_u32(dst + r * LD + c), real ? src + int64_t(r0 + r) * sl + c : src, real);
        }
    } else {
#pragma unroll 4
        for (int i = threadIdx.x; i < NR * D; i += kThreads) {
            const int r = i / D, c = i % D;
            const bool real = r0 + r >= lo && r0 + r < hi;
            cp_async4(smem_u32(dst + r * LD + c), real ? src + int64_t(r0 + r) * sl + c : src, real);
        }
    }
}

// s[r][c] = row (r0 + r) of A . row (x + 32 c) of B; even and odd elements are summed apart (packed FMAs)
template <int D>
__device__ __forceinline__ void rows_dot_cols(const float* A, const float* Bt, int r0, int x, float (&s)[kRW][2]) {
    constexpr int LD = D + 4;
    uint64_t t[kRW][2];
#pragma unroll
    for (int r = 0; r < kRW; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) t[r][c] = 0;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
        ulonglong2 b[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) b[c] = *reinterpret_cast<const ulonglong2*>(Bt + (x + 32 * c) * LD + d);
#pragma unroll
        for (int r = 0; r < kRW; ++r) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(A + (r0 + r) * LD + d);
#pragma unroll
            for (int c = 0; c < 2; ++c) t[r][c] = fma_f2(a.y, b[c].y, fma_f2(a.x, b[c].x, t[r][c]));
        }
    }
#pragma unroll
    for (int r = 0; r < kRW; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float lo, hi;
            unpack_f2(t[r][c], lo, hi);
            s[r][c] = lo + hi;
        }
}

// result columns of lane x, consecutive: 4x.. (D = 128), 2x.. (64), x (32), x of the lanes below 16 (16)
template <int D>
struct Own {
    static constexpr int N = D < 32 ? 1 : D / 32;
    static __device__ __forceinline__ bool has(int x) { return D >= 32 || x < D; }
    static __device__ __forceinline__ void load(const float* row, int x, float (&v)[N]) {
        if constexpr (N == 4) {
            const float4 t = *reinterpret_cast<const float4*>(row + 4 * x);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else if constexpr (N == 2) {
            const float2 t = *reinterpret_cast<const float2*>(row + 2 * x);
            v[0] = t.x; v[1] = t.y;
        } else {
            v[0] = row[D >= 32 ? x : x % D];
        }
    }
    static __device__ __forceinline__ void store(float* row, int x, bool vec, const float (&v)[N], float f) {
        if constexpr (N == 4) {
            if (vec) {
                *reinterpret_cast<float4*>(row + 4 * x) = make_float4(v[0] * f, v[1] * f, v[2] * f, v[3] * f);
                return;
            }
        } else if constexpr (N == 2) {
            if (vec) {
                *reinterpret_cast<float2*>(row + 2 * x) = make_float2(v[0] * f, v[1] * f);
                return;
            }
        }
        if (has(x)) {
#pragma unroll
            for (int k = 0; k < N; ++k) row[N * x + k] = v[k] * f;
        }
    }
};

// A warp's results: rows 2i and 2i + 1 of own column k in acc.v[i][k]
template <int D>
struct F32Acc {
    static constexpr int N = Own<D>::N;
    uint64_t v[kRW / 2][N];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < kRW / 2; ++i)
#pragma unroll
            for (int k = 0; k < N; ++k) v[i][k] = 0;
    }
    __device__ __forceinline__ void scale(const float (&f)[kRW]) {
#pragma unroll
        for (int i = 0; i < kRW / 2; ++i)
#pragma unroll
            for (int k = 0; k < N; ++k) v[i][k] = mul_f2(v[i][k], pack_f2(f[2 * i], f[2 * i + 1]));
    }
    // += sum_c P[c][row] * V[c][own column k], P being the warp's own (put_p). kHalves: over lo <= c < hi only
    template <bool kHalves>
    __device__ __forceinline__ void add(const float* P, const float* V, int x, int lo, int hi) {
        if (!kHalves || (lo <= 0 && hi >= kC)) {
#pragma unroll 8
            for (int c = 0; c < kC; ++c) add_column(P, V, x, c);
        } else {
            hi = min(hi, kC);
#pragma unroll 4
            for (int c = max(lo, 0); c < hi; ++c) add_column(P, V, x, c);
        }
    }
    __device__ __forceinline__ void add_column(const float* P, const float* V, int x, int c) {
        float own[N];
        Own<D>::load(V + c * (D + 4), x, own);
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(P + c * kRW);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint64_t o2 = pack_f2(own[k], own[k]);
            v[0][k] = fma_f2(w.x, o2, v[0][k]);
            v[1][k] = fma_f2(w.y, o2, v[1][k]);
        }
    }
    __device__ __forceinline__ void row(int r, float (&out)[N]) const {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            float lo, hi;
            unpack_f2(v[r / 2][k], lo, hi);
            out[k] = (r & 1) ? hi : lo;
        }
    }
};

// the lane's columns x and x + 32 of the warp's P, the rows of a column side by side
__device__ __forceinline__ void put_p(float* P, int x, const float (&w)[kRW][2]) {
#pragma unroll
    for (int c = 0; c < 2; ++c) *reinterpret_cast<float4*>(P + (x + 32 * c) * kRW) = make_float4(w[0][c], w[1][c], w[2][c], w[3][c]);
}

__device__ __forceinline__ float warp_max(float x) {
    float y;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// visited[o] for every 128-block o of the other side; the caller synchronises
template <int R>
__device__ __forceinline__ void find_visited(uint8_t* visited, const MaskArgs& mk, int b, int he, bool rows_are_queries, int own) {
    const int n = rows_are_queries ? mk.L.nK : mk.L.nQ;
    for (int o = threadIdx.x; o < n; o += threads(R))
        visited[o] = (classify_from_plan(mk, b, he, rows_are_queries ? own : o, rows_are_queries ? o : own) & TILE_VISIT) != 0;
}
// first column >= c (a multiple of kC) of a visited block, or end
__device__ __forceinline__ int next_tile(const uint8_t* visited, int c, int end) {
    while (c < end && !visited[c / kBlk]) c = c / kBlk * kBlk + kBlk;
    return c;
}

__device__ __forceinline__ int code_q(const MaskArgs& mk, int b, int he, int i) {
    return (mk.mode == 1 && i < mk.M) ? mk.plan[mk.L.off_qc + (int64_t(b) * mk.He + he) * mk.L.Mpad + i] : 0;
}
__device__ __forceinline__ int code_k(const MaskArgs& mk, int b, int he, int j) {
    return (mk.mode == 1 && j < mk.N) ? mk.plan[mk.L.off_kc + (int64_t(b) * mk.He + he) * mk.L.Npad + j] : 0;
}

// ---------------------------------------------------------------------------------------------
// forward: grid (H, B, ceil(M / R))
// ---------------------------------------------------------------------------------------------
template <int D, int R>
__global__ void __launch_bounds__(threads(R), R == 32 && D <= 32 ? 4 : 0) f32_fwd_kernel(const F32Params p) {
    using S = F32Smem<D, R>;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;
    float* KVs = Qs + S::rows;            // two stages of K, V
    float* Pall = KVs + 4 * S::cols;
    float* Ps = Pall + (threadIdx.x >> 5) * (kC * kRW);  // the warp's own
    int* codes = reinterpret_cast<int*>(Pall + S::p);  // two stages
    __shared__ uint8_t visited[kListCap];
    follow_stream();
    const MaskArgs& mk = p.mask;
    const int i0 = int(gridDim.z - 1 - blockIdx.z) * R, h = blockIdx.x, b = blockIdx.y, hk = h / p.G;  // long rows first
    const int he = (mk.He == 1) ? 0 : h;
    const int x = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * kRW;
    const float* qbase = p.q.ptr + int64_t(b) * p.q.sb + int64_t(h) * p.q.sh;
    const float* kbase = p.k.ptr + int64_t(b) * p.k.sb + int64_t(hk) * p.k.sh;
    const float* vbase = p.v.ptr + int64_t(b) * p.v.sb + int64_t(hk) * p.v.sh;
    const bool kvec = rows_aligned(kbase, p.k.sl), vvec = rows_aligned(vbase, p.v.sl);
    const int32_t* kcodes = mk.mode == 1 ? mk.plan + mk.L.off_kc + (int64_t(b) * mk.He + he) * mk.L.Npad : nullptr;
    const int end = mk.causal ? min(mk.N, i0 + R + mk.gap) : mk.N;  // keys beyond the last row's causal bound
    // In a block of 32 rows those beyond the first half's: the values there stay out of its P V, for a product with a P of 0 may be NaN.
    // What a NaN or an infinity reaches then does not go by the size of the blocks, which goes by what a sequence is batched with. us, forward and
    // forward with backward, products over the whole tile | over what the half sees: 4 x 8 heads x 1024 x 64 causal 179, 726 | 177, 712, not causal
    // 324, 1342 | 324, 1329; 4 x 8 x 1024 x 128 causal 363, 1462 | 359, 1466; 8 x 16 x 512 x 32 causal 121, 496 | 119, 488, not causal 205, 855 | 208, 859
    // (four blocks of head dims up to 32 share an SM only while a thread has 64 registers: 211 with three).
    const int end_half = mk.causal && r0 < 16 ? i0 + 16 + mk.gap : mk.N + kC;
    auto fetch = [&](int j0, int st) {
        load_tile<D, kC, R>(KVs + st * 2 * S::cols, kbase, p.k.sl, kvec, j0, end);
        load_tile<D, kC, R>(KVs + (st * 2 + 1) * S::cols, vbase, p.v.sl, vvec, j0, end);
        if (kcodes && threadIdx.x < kC) cp_async4(smem_u32(codes + st * kC + threadIdx.x), kcodes + j0 + threadIdx.x, true);
    };
    load_tile<D, R, R>(Qs, qbase, p.q.sl, rows_aligned(qbase, p.q.sl), i0, mk.M);
    find_visited<R>(visited, mk, b, he, true, i0 / kBlk);
    float m[kRW], l[kRW];
    F32Acc<D> acc;
    acc.clear();
    int qc[kRW];
#pragma unroll
    for (int r = 0; r < kRW; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
        qc[r] = code_q(mk, b, he, i0 + r0 + r);
    }
    __syncthreads();
    int j0 = next_tile(visited, 0, end);
    if (j0 < end) fetch(j0, 0);
    cp_async_commit();
    for (int st = 0; j0 < end; st ^= 1) {
        const int jn = next_tile(visited, j0 + kC, end);
        if (jn < end) fetch(jn, st ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const float* Ks = KVs + st * 2 * S::cols;
        float s[kRW][2], alpha[kRW];
        rows_dot_cols<D>(Qs, Ks, r0, x, s);
#pragma unroll
        for (int r = 0; r < kRW; ++r) {
            const int i = i0 + r0 + r;
            float mx = -INFINITY;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int j = j0 + x + 32 * c;
                const bool keep = keep_entry(i, j, qc[r], kcodes ? codes[st * kC + x + 32 * c] : 0, mk.N, mk.gap, mk.causal, mk.mode);
                s[r][c] = keep ? s[r][c] * p.scale : -INFINITY;
                mx = fmaxf(mx, s[r][c]);
            }
            const float mn = fmaxf(m[r], warp_max(mx));
            alpha[r] = (m[r] == -INFINITY) ? 0.f : expf(m[r] - mn);
            m[r] = mn;
            l[r] *= alpha[r];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                s[r][c] = (s[r][c] == -INFINITY) ? 0.f : expf(s[r][c] - mn);
                l[r] += s[r][c];
            }
        }
        acc.scale(alpha);
        put_p(Ps, x, s);
        __syncwarp();
        acc.template add<R == 32>(Ps, Ks + S::cols, x, 0, end_half - j0);
        __syncthreads();  // the stage may be refilled
        j0 = jn;
    }
    cp_async_wait<0>();  // a block without a visible tile has not waited for its Q
    float* obase = p.o.ptr + int64_t(b) * p.o.sb + int64_t(h) * p.o.sh;
    const bool ovec = rows_aligned(obase, p.o.sl);
#pragma unroll
    for (int r = 0; r < kRW; ++r) {
        const int i = i0 + r0 + r;
        const float lt = warp_sum(l[r]);
        if (i >= mk.M) continue;
        float own[Own<D>::N];
        acc.row(r, own);
        Own<D>::store(obase + int64_t(i) * p.o.sl, x, ovec, own, lt > 0.f ? 1.f / lt : 0.f);
        if (x == 0) p.lse[(int64_t(b) * p.H + h) * mk.L.Mpad + i] = lt > 0.f ? m[r] + logf(lt) : -INFINITY;
    }
}

// delta = rowsum(o * dO) (flash_triton.py:161-165): grid (ceil(M / 4), H, B), one warp per row
template <int D>
__global__ void __launch_bounds__(128) f32_delta_kernel(const F32Params p) {
    follow_stream();
    const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int h = blockIdx.y, b = blockIdx.z;
    if (i >= p.mask.L.Mpad) return;
    float a = 0.f;
    if (i < p.mask.M) {
        const float* po = p.o.ptr + int64_t(b) * p.o.sb + int64_t(h) * p.o.sh + int64_t(i) * p.o.sl;
        const float* pd = p.d_o.ptr + int64_t(b) * p.d_o.sb + int64_t(h) * p.d_o.sh + int64_t(i) * p.d_o.sl;
        for (int d = lane; d < D; d += 32) a = fmaf(po[d], pd[d], a);
    }
    a = warp_sum(a);
    if (lane == 0) p.delta[(int64_t(b) * p.H + h) * p.mask.L.Mpad + i] = a;
}

// ---------------------------------------------------------------------------------------------
// dQ: grid (H, B, ceil(M / R)). rows = queries, columns = keys
// ---------------------------------------------------------------------------------------------
template <int D, int R>
__global__ void __launch_bounds__(threads(R)) f32_bwd_dq_kernel(const F32Params p) {
    using S = F32Smem<D, R>;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;
    float* dOs = Qs + S::rows;
    float* KVs = dOs + S::rows;           // two stages of K, V
    float* Pall = KVs + 4 * S::cols;
    float* Ps = Pall + (threadIdx.x >> 5) * (kC * kRW);  // the warp's own
    int* codes = reinterpret_cast<int*>(Pall + S::p);
    __shared__ uint8_t visited[kListCap];
    const MaskArgs& mk = p.mask;
    const int i0 = int(gridDim.z - 1 - blockIdx.z) * R, h = blockIdx.x, b = blockIdx.y, hk = h / p.G;
    const int he = (mk.He == 1) ? 0 : h;
    const int x = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * kRW;
    const float* qbase = p.q.ptr + int64_t(b) * p.q.sb + int64_t(h) * p.q.sh;
    const float* dobase = p.d_o.ptr + int64_t(b) * p.d_o.sb + int64_t(h) * p.d_o.sh;
    const float* kbase = p.k.ptr + int64_t(b) * p.k.sb + int64_t(hk) * p.k.sh;
    const float* vbase = p.v.ptr + int64_t(b) * p.v.sb + int64_t(hk) * p.v.sh;
    const bool kvec = rows_aligned(kbase, p.k.sl), vvec = rows_aligned(vbase, p.v.sl);
    const int32_t* kcodes = mk.mode == 1 ? mk.plan + mk.L.off_kc + (int64_t(b) * mk.He + he) * mk.L.Npad : nullptr;
    const int end = mk.causal ? min(mk.N, i0 + R + mk.gap) : mk.N;  // keys beyond the last row's causal bound
    const int end_half = mk.causal && r0 < 16 ? i0 + 16 + mk.gap : mk.N + kC;  // (see the forward)
    auto fetch = [&](int j0, int st) {
        load_tile<D, kC, R>(KVs + st * 2 * S::cols, kbase, p.k.sl, kvec, j0, end);
        load_tile<D, kC, R>(KVs + (st * 2 + 1) * S::cols, vbase, p.v.sl, vvec, j0, end);
        if (kcodes && threadIdx.x < kC) cp_async4(smem_u32(codes + st * kC + threadIdx.x), kcodes + j0 + threadIdx.x, true);
    };
    load_tile<D, R, R>(Qs, qbase, p.q.sl, rows_aligned(qbase, p.q.sl), i0, mk.M);
    load_tile<D, R, R>(dOs, dobase, p.d_o.sl, rows_aligned(dobase, p.d_o.sl), i0, mk.M);
    find_visited<R>(visited, mk, b, he, true, i0 / kBlk);
    F32Acc<D> acc;
    acc.clear();
    float lse[kRW], dl[kRW];
    int qc[kRW];
#pragma unroll
    for (int r = 0; r < kRW; ++r) {
        const int i = i0 + r0 + r;
        const int64_t ro = (int64_t(b) * p.H + h) * mk.L.Mpad + i;
        lse[r] = (i < mk.M) ? p.lse[ro] : -INFINITY;
        dl[r] = (i < mk.M) ? p.delta[ro] : 0.f;
        qc[r] = code_q(mk, b, he, i);
    }
    __syncthreads();
    int j0 = next_tile(visited, 0, end);
    if (j0 < end) fetch(j0, 0);
    cp_async_commit();
    for (int st = 0; j0 < end; st ^= 1) {
        const int jn = next_tile(visited, j0 + kC, end);
        if (jn < end) fetch(jn, st ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const float* Ks = KVs + st * 2 * S::cols;
        float s[kRW][2], dp[kRW][2];
        rows_dot_cols<D>(Qs, Ks, r0, x, s);
        rows_dot_cols<D>(dOs, Ks + S::cols, r0, x, dp);
#pragma unroll
        for (int r = 0; r < kRW; ++r) {
            const int i = i0 + r0 + r;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int j = j0 + x + 32 * c;
                const bool keep = (i < mk.M) && keep_entry(i, j, qc[r], kcodes ? codes[st * kC + x + 32 * c] : 0, mk.N, mk.gap, mk.causal, mk.mode);
                const float pe = keep ? expf(s[r][c] * p.scale - lse[r]) : 0.f;  // a kept entry has a finite lse
                dp[r][c] = keep ? pe * (dp[r][c] - dl[r]) : 0.f;  // dS (flash_triton.py:301)
            }
        }
        put_p(Ps, x, dp);
        __syncwarp();
        acc.template add<R == 32>(Ps, Ks, x, 0, end_half - j0);  // dQ += dS K (flash_triton.py:420)
        __syncthreads();
        j0 = jn;
    }
    cp_async_wait<0>();
    float* dqbase = p.dq.ptr + int64_t(b) * p.dq.sb + int64_t(h) * p.dq.sh;
    const bool dqvec = rows_aligned(dqbase, p.dq.sl);
#pragma unroll
    for (int r = 0; r < kRW; ++r) {
        if (i0 + r0 + r >= mk.M) continue;
        float own[Own<D>::N];
        acc.row(r, own);
        Own<D>::store(dqbase + int64_t(i0 + r0 + r) * p.dq.sl, x, dqvec, own, p.scale);  // flash_triton.py:425
    }
    wait_prerequisites();  // what follows in the stream finds dK / dV complete too
}

// ---------------------------------------------------------------------------------------------
// dK, dV: grid (Hk, B, ceil(N / R)). rows = keys, columns = queries; the query heads of the group
// are walked one after the other, so the group sum (flash_triton.py:635-637) needs no second pass
// ---------------------------------------------------------------------------------------------
template <int D, int R>
__global__ void __launch_bounds__(threads(R)) f32_bwd_dkdv_kernel(const F32Params p) {
    using S = F32Smem<D, R>;
    extern __shared__ __align__(16) float sm[];
    follow_stream();  // (in this order: fa_bwd's dQ kernel reads nothing that this one writes, but delta, which is complete now)
    float* Ks = sm;
    float* Vs = Ks + S::rows;
    float* QDs = Vs + S::rows;            // two stages of Q, dO
    float* Pall = QDs + 4 * S::cols;
    float* Ps = Pall + (threadIdx.x >> 5) * (kC * kRW);  // the warp's own
    float* vecs = Pall + S::p;              // two stages of id code, lse, delta per query
    __shared__ uint8_t visited[kListCap];
    const MaskArgs& mk = p.mask;
    const int j0 = blockIdx.z * R, hk = blockIdx.x, b = blockIdx.y;
    const int x = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * kRW;
    const float* kbase = p.k.ptr + int64_t(b) * p.k.sb + int64_t(hk) * p.k.sh;
    const float* vbase = p.v.ptr + int64_t(b) * p.v.sb + int64_t(hk) * p.v.sh;
    load_tile<D, R, R>(Ks, kbase, p.k.sl, rows_aligned(kbase, p.k.sl), j0, mk.N);
    load_tile<D, R, R>(Vs, vbase, p.v.sl, rows_aligned(vbase, p.v.sl), j0, mk.N);
    F32Acc<D> dk, dv;
    dk.clear();
    dv.clear();
    // first query row that can see key j0 under the causal mask (flash_triton.py:214-218)
    const int first = mk.causal ? max(0, j0 - mk.gap) : 0;
    const int first_half = mk.causal && r0 >= 16 ? j0 + 16 - mk.gap : 0;  // the same for the second half of 32 keys (see the forward)
    for (int g = 0; g < p.G; ++g) {
        const int h = hk * p.G + g;
        const int he = (mk.He == 1) ? 0 : h;
        const float* qbase = p.q.ptr + int64_t(b) * p.q.sb + int64_t(h) * p.q.sh;
        const float* dobase = p.d_o.ptr + int64_t(b) * p.d_o.sb + int64_t(h) * p.d_o.sh;
        const bool qvec = rows_aligned(qbase, p.q.sl), dovec = rows_aligned(dobase, p.d_o.sl);
        const int64_t ro = (int64_t(b) * p.H + h) * mk.L.Mpad;
        const int32_t* qcodes = mk.mode == 1 ? mk.plan + mk.L.off_qc + (int64_t(b) * mk.He + he) * mk.L.Mpad : nullptr;
        auto fetch = [&](int i0, int st) {
            load_tile<D, kC, R>(QDs + st * 2 * S::cols, qbase, p.q.sl, qvec, i0, mk.M, first);
            load_tile<D, kC, R>(QDs + (st * 2 + 1) * S::cols, dobase, p.d_o.sl, dovec, i0, mk.M, first);
            for (int e = threadIdx.x; e < S::vec; e += threads(R)) {  // the per-row buffers are padded to 128 rows; what pads them is not used
                const int t = e % kC, what = e / kC;
                const void* src = what == 0 ? static_cast<const void*>(qcodes) : what == 1 ? p.lse + ro : p.delta + ro;
                if (src) cp_async4(smem_u32(vecs + st * S::vec + e), static_cast<const float*>(src) + i0 + t, true);
            }
        };
        if (g == 0 || mk.He != 1) {
            // A head without a visible tile has passed no barrier since its next_tile: without this one a fast warp
            // would rewrite the table while a slow one reads it, and the two would take different numbers of tiles.
            if (g > 0) __syncthreads();
            find_visited<R>(visited, mk, b, he, false, j0 / kBlk);
        }
        int kc[kRW];
#pragma unroll
        for (int r = 0; r < kRW; ++r) kc[r] = code_k(mk, b, he, j0 + r0 + r);
        __syncthreads();
        int i0 = next_tile(visited, first / kC * kC, mk.M);
        if (i0 < mk.M) fetch(i0, 0);
        cp_async_commit();
        for (int st = 0; i0 < mk.M; st ^= 1) {
            const int in = next_tile(visited, i0 + kC, mk.M);
            if (in < mk.M) fetch(in, st ^ 1);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            const float* Qs = QDs + st * 2 * S::cols;
            const float* dOs = Qs + S::cols;
            const float* vec = vecs + st * S::vec;
            float s[kRW][2], dp[kRW][2];
            rows_dot_cols<D>(Ks, Qs, r0, x, s);    // S^T
            rows_dot_cols<D>(Vs, dOs, r0, x, dp);  // dP^T
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = i0 + x + 32 * c;
                const int qc = qcodes ? __float_as_int(vec[x + 32 * c]) : 0;
                const float lse = vec[kC + x + 32 * c], dl = vec[2 * kC + x + 32 * c];
#pragma unroll
                for (int r = 0; r < kRW; ++r) {
                    const bool keep = (i < mk.M) && keep_entry(i, j0 + r0 + r, qc, kc[r], mk.N, mk.gap, mk.causal, mk.mode);
                    const float pe = keep ? expf(s[r][c] * p.scale - lse) : 0.f;
                    s[r][c] = pe;
                    dp[r][c] = keep ? pe * (dp[r][c] - dl) : 0.f;
                }
            }
            put_p(Ps, x, s);
            __syncwarp();
            dv.template add<R == 32>(Ps, dOs, x, first_half - i0, kC);  // dV += P^T dO (flash_triton.py:291)
            __syncwarp();
            put_p(Ps, x, dp);
            __syncwarp();
            dk.template add<R == 32>(Ps, Qs, x, first_half - i0, kC);   // dK += dS^T Q (flash_triton.py:308)
            __syncthreads();
            i0 = in;
        }
    }
    cp_async_wait<0>();
    float* dkbase = p.dk.ptr + int64_t(b) * p.dk.sb + int64_t(hk) * p.dk.sh;
    float* dvbase = p.dv.ptr + int64_t(b) * p.dv.sb + int64_t(hk) * p.dv.sh;
    const bool dkvec = rows_aligned(dkbase, p.dk.sl), dvvec = rows_aligned(dvbase, p.dv.sl);
#pragma unroll
    for (int r = 0; r < kRW; ++r) {
        const int j = j0 + r0 + r;
        if (j >= mk.N) continue;
        float own[Own<D>::N];
        dk.row(r, own);
        Own<D>::store(dkbase + int64_t(j) * p.dk.sl, x, dkvec, own, p.scale);  // flash_triton.py:313
        dv.row(r, own);
        Own<D>::store(dvbase + int64_t(j) * p.dv.sl, x, dvvec, own, 1.f);
    }
}

// ---------------------------------------------------------------------------------------------
template <int D, int R>
static cudaError_t launch_f32_t(int which, const F32Params& p, bool overlap, cudaStream_t stream) {
    using S = F32Smem<D, R>;
    const MaskArgs& mk = p.mask;
    static SmemAllowed allowed[4];
    auto run = [&](auto kern, int smem, int rows, int heads) {
        const cudaError_t e = allow_smem(kern, smem, allowed[which]);
        if (e != cudaSuccess) return e;
        // the blocks of all heads with many tiles first: with those of one head behind each other the last long ones started late (4 x 8
        // heads x 1024 x 64, forward and backward 851 -> 729 us)
        const dim3 grid(heads, p.B, cdiv(rows, R));
        if (which != 3 || overlap) return launch_overlapping(kern, grid, threads(R), smem, stream, p);
        kern<<<grid, threads(R), smem, stream>>>(p);
        return cudaGetLastError();
    };
    if (which == 0) return run(f32_fwd_kernel<D, R>, S::fwd_bytes, mk.M, p.H);
    if (which == 2) return run(f32_bwd_dkdv_kernel<D, R>, S::bwd_bytes, mk.N, p.Hk);
    return run(f32_bwd_dq_kernel<D, R>, S::bwd_bytes, mk.M, p.H);
}

// Blocks of 16 rows while those of 32 fit on the GPU all at once (`slots`): they have a chain of as many tiles but half the work, and the
// longest of them get an SM to themselves. For the backward both kernels' blocks count, and a third more is still worth it. us, 32 rows | 16, heads of
// 64 x 512: forward of 8 heads 31.7 | 32.2, 12 40.1 | 34.2, 16 45.8 | 37.6, 24 47.6 | 56.5; backward of 8 88.8 | 55.5, 12 82.9 | 77.5, 16
// 86.2 | 100. 32 x 512: forward of 24 44.7 | 38.7, 32 54.0 | 40.0, backward of 16 58.1 | 55.5, 24 80.3 | 81.2, 32 102 | 107. 128 x 512: forward of 4
// 48.8 | 36.0, 8 49.3 | 39.6, 16 52.4 | 77.3, backward of 4 86.2 | 62.7, 8 86.7 | 116. The same bits.
template <int D>
static cudaError_t launch_f32_rows(int which, const F32Params& p, bool overlap, int sms, cudaStream_t stream) {
    const MaskArgs& mk = p.mask;
    if (which == 1) return launch_overlapping(f32_delta_kernel<D>, dim3(unsigned(mk.L.Mpad / 4), p.H, p.B), 128, 0, stream, p);
    using S = F32Smem<D, 32>;
    constexpr int kStatic = kListCap + 1024;  // of a block: the table of visited tiles, and what the system takes
    constexpr int room = 232448 / ((S::fwd_bytes) + kStatic), per_sm = room < 4 ? room : 4;
    const int64_t rows = int64_t(cdiv(mk.M, 32)) * p.H * p.B, cols = int64_t(cdiv(mk.N, 32)) * p.Hk * p.B, slots = int64_t(per_sm) * sms;
    const bool small = which == 0 ? rows <= slots : 10 * (rows + cols) <= 13 * slots;
    return small ? launch_f32_t<D, 16>(which, p, overlap, stream) : launch_f32_t<D, 32>(which, p, overlap, stream);
}

// which: 0 forward, 1 delta, 2 dK / dV, 3 dQ. overlap: the launch directly before this one in the stream is the dK/dV
// kernel of the same backward, and the blocks of this one (dQ) may run beside its: two of 32 rows fit on an SM up to D = 64, and
// one alone leaves its FMA pipes idle most of the time. Whole backward, us, one behind the other and side by side (blocks of 32 rows): 8 heads x 512 x 64 causal 104,
// 82; 8 heads x 1024 283, 223; 32 heads x 1024 694, 634; 2 heads x 100 36, 22; D = 128, 8 heads x 512, 160, 136 (there dQ only
// starts on SMs that are free); 128 / 32 heads of 777 queries against 1024 keys, where dK/dV fills the GPU, 3291, 3222.
cudaError_t launch_f32(int which, int D, const F32Params& p, bool overlap, int sms, cudaStream_t stream) {
    switch (D) {
        case 16: return launch_f32_rows<16>(which, p, overlap, sms, stream);
        case 32: return launch_f32_rows<32>(which, p, overlap, sms, stream);
        case 64: return launch_f32_rows<64>(which, p, overlap, sms, stream);
        case 128: return launch_f32_rows<128>(which, p, overlap, sms, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace fa
