// fa_group_rows / fa_permute_rows: grouping of the queries by document id for calls without a
// causal mask.
//
// Without a causal mask the order of the query rows is free: row i of the output depends on query
// i, its id and all keys, not on its position. When the query ids are scattered (every block of 128
// queries holds every document) no tile can be skipped and every tile needs the entry-by-entry id
// check; after a stable sort of the rows by id the blocks are (nearly) uniform, the mask plan skips
// the tiles of other documents, and the few mixed blocks are the only ones that pay for the check.
// The reference has no counterpart: it evaluates every tile whatever the ids (flash_triton.py:94-129).
//
//  - fa_group_rows sorts each id row [M] of eq by the 32-bit code the mask plan uses for it
//    (ids >= 0, "attend to all", share one code that sorts last; flash_triton.py:114), keeping the
//    caller's order inside a document (stable; rows that are grouped already keep their places), and
//    writes the permutation, its inverse and the ids in the new order;
//  - fa_permute_rows moves the rows of a [B, H, M, D] tensor through such an index:
//    dst[b, h, i, :] = src[b, h, index[b, he, i], :]. With the permutation it gathers q (and dO) into
//    the grouped order; with the inverse it puts o (and dQ) back into the caller's order. It is plain
//    HBM traffic: every row is read once and written once, 16 bytes per thread.
//
// Short rows are sorted by counting: the place of a query is the number of codes before its own, and of equal ones at earlier places. Long
// rows are sorted by one CTA each in shared memory: a bitonic network over 64-bit keys (code, position), which
// are all distinct, so the order is the stable one whatever the network does with equal codes.
#include "../../include/fa_b200.h"
#include "common.cuh"
#include "params.cuh"

namespace {

struct IdRows {
    const void* ptr;
    int64_t sb, sh, sl;
    int is64;
};

constexpr int kSortThreads = 1024;

// The mask plan's code of an id, in an order in which ids >= 0 come last; same rule and status code as there.
__device__ __forceinline__ uint32_t sort_code(const IdRows& eq, int b, int he, int i, int* status) {
    const int64_t off = int64_t(b) * eq.sb + int64_t(he) * eq.sh + int64_t(i) * eq.sl;
    const long long id = eq.is64 ? static_cast<const long long*>(eq.ptr)[off] : static_cast<long long>(static_cast<const int*>(eq.ptr)[off]);
    int code = fa::kCodeAny;
    if (id < 0) {
        if (id >= -2147483648LL) {
            code = int(id);
        } else {
            code = int(-2147483647 - 1);
            atomicCAS(status, 0, fa::ST_ID_RANGE);
        }
    }
    return uint32_t(code) ^ 0x80000000u;
}

// grid (ceil(M / 64), He, B): the places of 64 queries, each counted by four threads over a quarter of the row's codes.
// Its work grows with the square of M, the network's time hardly faster than M while every row has an SM. us a launch, this | the network below: 8 rows
// of 300 3.0 | 8.6, of 1024 4.5 | 12.2, of 2048 8.9 | 21.0, of 4096 25.0 | 39.7; 64 rows of 1024 13.0 | 12.1, 16 of 4096 43.7 | 39.6, 128 of 512
// 8.1 | 8.5.
constexpr int kRankRows = 4096, kRankThreads = 256, kRankBlock = 64;
constexpr int64_t kRankCodes = 49152;  // id rows x M up to which counting is faster

// Does the range of bytes that holds the ids meet that of the int32 array `out` of n elements?
bool overlaps(const IdRows& eq, int B, int He, int M, const int32_t* out, int64_t n) {
    const int64_t item = eq.is64 ? 8 : 4, last[3] = {(B - 1) * eq.sb, (He - 1) * eq.sh, (M - 1) * eq.sl};
    int64_t lo = 0, hi = 0;  // of the offsets, in elements
    for (int64_t x : last) (x < 0 ? lo : hi) += x;
    const uintptr_t base = reinterpret_cast<uintptr_t>(eq.ptr), o = reinterpret_cast<uintptr_t>(out);
    return base + lo * item < o + n * 4 && o < base + (hi + 1) * item;
}
__global__ void __launch_bounds__(kRankThreads) group_rank_kernel(IdRows eq, int M, int He, int32_t* order, int32_t* inverse,
                                                                  int32_t* grouped, int* status) {
    __shared__ uint4 codes4[kRankRows / 4];
    __shared__ int part[4][kRankBlock];
    fa::follow_stream();
    uint32_t* codes = reinterpret_cast<uint32_t*>(codes4);
    const int he = blockIdx.y, b = blockIdx.z, first = blockIdx.x * kRankBlock;
    const int quarter = (M + 15) / 16 * 4;  // codes a thread counts
    for (int i = threadIdx.x; i < 4 * quarter; i += kRankThreads)
        codes[i] = i < M ? sort_code(eq, b, he, i, status) : ~0u;  // (what pads the row comes before nothing)
    __syncthreads();
    const int e = threadIdx.x % kRankBlock, q = threadIdx.x / kRankBlock, i = first + e;
    const uint32_t own = i < M ? codes[i] : 0u;
    const int lo = q * quarter, hi = lo + quarter;
    const int before = min(max(first, lo), hi), behind = min(max(first + kRankBlock, lo), hi);  // multiples of 4
    int n = 0;
#pragma unroll 4
    for (int j = lo; j < before; j += 4) {
        const uint4 c = codes4[j / 4];
        n += (c.x <= own) + (c.y <= own) + (c.z <= own) + (c.w <= own);
    }
    for (int j = before; j < behind; ++j) n += codes[j] < own || (codes[j] == own && j < i);
#pragma unroll 4
    for (int j = behind; j < hi; j += 4) {
        const uint4 c = codes4[j / 4];
        n += (c.x < own) + (c.y < own) + (c.z < own) + (c.w < own);
    }
    part[q][e] = n;
    __syncthreads();
    if (q == 0 && i < M) {
        const int64_t row = (int64_t(b) * He + he) * M;
        const int place = part[0][e] + part[1][e] + part[2][e] + part[3][e];
        order[row + place] = i;
        inverse[row + i] = place;
        grouped[row + place] = int(own ^ 0x80000000u);
    }
}

// grid (He, B). P = M rounded up to a power of two; dynamic shared memory = P * 8 bytes.
__global__ void __launch_bounds__(kSortThreads) group_rows_kernel(IdRows eq, int M, int P, int He, int32_t* order,
                                                                  int32_t* inverse, int32_t* grouped, int* status) {
    extern __shared__ __align__(16) unsigned long long keys[];
    fa::follow_stream();
    const int he = blockIdx.x, b = blockIdx.y;
    const int64_t row = (int64_t(b) * He + he) * M;
    for (int i = threadIdx.x; i < P; i += kSortThreads) {
        unsigned long long key = ~0ull;  // padding sorts behind every row
        if (i < M) key = (static_cast<unsigned long long>(sort_code(eq, b, he, i, status)) << 32) | uint32_t(i);
        keys[i] = key;
    }
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int t = threadIdx.x; t < (P >> 1); t += kSortThreads) {
                const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
                const int l = i | j;
                const bool up = (i & k) == 0;
                const unsigned long long a = keys[i], c = keys[l];
                if ((a > c) == up) {
                    keys[i] = c;
                    keys[l] = a;
                }
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < M; i += kSortThreads) {
        const unsigned long long key = keys[i];
        const int src = int(uint32_t(key));
        order[row + i] = src;
        inverse[row + src] = i;
        grouped[row + i] = int(uint32_t(key >> 32) ^ 0x80000000u);
    }
}

struct RowTensor {
    const uint4* src;
    uint4* dst;
    int64_t s_sb, s_sh, s_sl;  // strides in 16-byte units
    int64_t d_sb, d_sh, d_sl;
};

// grid (blocks of rows, H, B): `vec` neighbouring threads move a row, 16 bytes each, so that a warp reads and writes whole 128-byte (or longer)
// stretches, and each thread has kPermuteRows rows in flight. us, one row a thread, its place by
// divisions | now (four rows a thread in brackets): 8 x 8 x 1024 x 64 in 16 bits 5.0 | 3.5 (4.0), 8 x 16 x 2048 x 64 13.7 | 7.6 (8.1).
constexpr int kPermuteRows = 2, kPermuteThreads = 256;
__global__ void __launch_bounds__(kPermuteThreads) permute_rows_kernel(RowTensor t, const int32_t* index, int M, int He, int vec) {
    fa::follow_stream();
    const int h = blockIdx.y, b = blockIdx.z, he = (He == 1) ? 0 : h;
    const int c = threadIdx.x % vec, step = kPermuteThreads / vec;
    const int row0 = blockIdx.x * (step * kPermuteRows) + threadIdx.x / vec;
    const int32_t* idx = index + (int64_t(b) * He + he) * M;
    const uint4* src = t.src + b * t.s_sb + h * t.s_sh + c;
    uint4* dst = t.dst + b * t.d_sb + h * t.d_sh + c;
    int s[kPermuteRows];
    uint4 x[kPermuteRows];
#pragma unroll
    for (int r = 0; r < kPermuteRows; ++r) s[r] = row0 + r * step < M ? idx[row0 + r * step] : 0;
#pragma unroll
    for (int r = 0; r < kPermuteRows; ++r)
        if (row0 + r * step < M) x[r] = src[int64_t(s[r]) * t.s_sl];
#pragma unroll
    for (int r = 0; r < kPermuteRows; ++r)
        if (row0 + r * step < M) dst[int64_t(row0 + r * step) * t.d_sl] = x[r];
}

int elt_bytes(int dtype) { return dtype == FA_FP32 ? 4 : 2; }

// Base 16-byte aligned, last stride 1, the other strides of extents > 1 positive and whole 16-byte units.
int check_rows(const fa_tensor* t, int B, int H, int M, int per16) {
    if (!t || !t->ptr) return FA_ERR_BAD_ARG;
    if (reinterpret_cast<uintptr_t>(t->ptr) % 16 != 0 || t->stride[3] != 1) return FA_ERR_ALIGNMENT;
    const int ext[3] = {B, H, M};
    for (int i = 0; i < 3; ++i)
        if (ext[i] > 1 && (t->stride[i] <= 0 || t->stride[i] % per16 != 0)) return FA_ERR_ALIGNMENT;
    return FA_OK;
}

}  // namespace

extern "C" int fa_group_rows(const fa_problem* p, const fa_ids* eq, int32_t* order, int32_t* inverse,
                             int32_t* grouped_ids, int32_t* status, void* stream) {
    size_t bytes = 0;
    const int rc = fa_plan_bytes(p, &bytes);  // validates the problem as every other entry point does
    if (rc) return rc;
    if (p->mode != FA_MODE1_DOC || !eq || !eq->ptr || !order || !inverse || !grouped_ids || !status) return FA_ERR_BAD_ARG;
    if (eq->dtype != FA_ID_INT32 && eq->dtype != FA_ID_INT64) return FA_ERR_BAD_ARG;
    if (p->M > FA_GROUP_MAX_ROWS) return FA_ERR_UNSUPPORTED;
    const IdRows rows{eq->ptr, eq->stride[0], eq->stride[1], eq->stride[2], eq->dtype == FA_ID_INT64};
    const int64_t n = int64_t(p->id_heads) * p->B * p->M;
    // The counting kernel's blocks read a row while others write its results; the network's block has read its row when it writes.
    const bool apart = !overlaps(rows, p->B, p->id_heads, p->M, order, n) && !overlaps(rows, p->B, p->id_heads, p->M, inverse, n) &&
                       !overlaps(rows, p->B, p->id_heads, p->M, grouped_ids, n);
    if (p->M <= kRankRows && n <= kRankCodes && apart) {
        const dim3 grid(fa::cdiv(p->M, kRankBlock), p->id_heads, p->B);
        return fa::launch_overlapping(group_rank_kernel, grid, kRankThreads, 0, static_cast<cudaStream_t>(stream), rows, p->M, p->id_heads, order,
                                      inverse, grouped_ids, status) == cudaSuccess ? FA_OK : FA_ERR_LAUNCH;
    }
    int P = 1;
    while (P < p->M) P <<= 1;
    const size_t smem = size_t(P) * sizeof(unsigned long long);
    static fa::SmemAllowed allowed;
    if (fa::allow_smem(group_rows_kernel, int(FA_GROUP_MAX_ROWS * sizeof(unsigned long long)), allowed) != cudaSuccess)
        return FA_ERR_LAUNCH;
    const cudaError_t e = fa::launch_overlapping(group_rows_kernel, dim3(p->id_heads, p->B), kSortThreads, int(smem),
                                                 static_cast<cudaStream_t>(stream), rows, p->M, P, p->id_heads, order, inverse, grouped_ids, status);
    return e == cudaSuccess ? FA_OK : FA_ERR_LAUNCH;
}

extern "C" int fa_permute_rows(const fa_problem* p, const fa_tensor* src, const fa_tensor* dst, const int32_t* index,
                               void* stream) {
    size_t bytes = 0;
    int rc = fa_plan_bytes(p, &bytes);
    if (rc) return rc;
    if (!index) return FA_ERR_BAD_ARG;
    const int per16 = 16 / elt_bytes(p->dtype);  // elements per 16 bytes
    if (p->D % per16 != 0) return FA_ERR_UNSUPPORTED;
    if ((rc = check_rows(src, p->B, p->H, p->M, per16))) return rc;
    if ((rc = check_rows(dst, p->B, p->H, p->M, per16))) return rc;
    const int vec = p->D / per16;
    RowTensor t;
    t.src = static_cast<const uint4*>(src->ptr);
    t.dst = static_cast<uint4*>(dst->ptr);
    t.s_sb = src->stride[0] / per16; t.s_sh = src->stride[1] / per16; t.s_sl = src->stride[2] / per16;
    t.d_sb = dst->stride[0] / per16; t.d_sh = dst->stride[1] / per16; t.d_sl = dst->stride[2] / per16;
    // strides of extent-1 dimensions are never multiplied by anything but 0
    const int He = (p->mode == FA_MODE1_DOC) ? p->id_heads : 1;
    const dim3 grid(fa::cdiv(p->M, kPermuteThreads / vec * kPermuteRows), p->H, p->B);
    const cudaError_t e = fa::launch_overlapping(permute_rows_kernel, grid, kPermuteThreads, 0, static_cast<cudaStream_t>(stream), t, index, p->M, He, vec);
    return e == cudaSuccess ? FA_OK : FA_ERR_LAUNCH;
}
