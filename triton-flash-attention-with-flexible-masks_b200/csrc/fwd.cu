// Forward kernel: O = softmax(mask(Q K^T * sm_scale)) V and the row log-sum-exp.
// Replaces `_fwd_kernel` (flash_triton.py:25-141). Same mathematics (base-2 online softmax,
// P rounded to the input dtype before P*V, fp32 accumulation), except that the scale is
// applied in fp32 to the fp32 scores instead of being folded into a rounded Q
// (flash_triton.py:88), and tiles the mask plan proves empty are not visited at all.
//
// Persistent: one CTA per SM walks work items (one item = one block of 128 queries of one
// (batch, head)); items are handed out in an order that puts the query blocks of
// all heads side by side, so that the CTAs of one round carry almost equal work. With document
// masks most items hold only a few tiles, so nothing waits at the border of two items: every role walks the items at
// its own pace, up to NQ of them apart.
//
// 16 warps:
//   warps 0-3  softmax group 0, warps 4-7 softmax group 1 (thread r of a group owns row r)
//   warps 8-11 epilogue group: merges a finished item's two O, stages the result and stores it
//   warp 12    TMA producer (Q per item, K and V rings that run across items; K ahead of V)
//   warps 13,15 tcgen05.mma issuers, of P*V and of S; warp 13 owns the TMEM allocation
//   warp 14    item scheduler: decodes the item, classifies its candidate tiles from the mask plan
//              and compacts the visited ones into a list in shared memory (NQ item slots)
// The CTA's g-th visited tile (counted across its items) belongs to softmax group g & 1: two chains of tiles, each with a
// running maximum, a sum and an accumulator O of its own for the item; the epilogue merges them, the chain of the item's even
// tiles first, so that the result does not depend on which group that was. A chain in which a row had no key stays out of
// the merge: what the values behind its mask are does not matter.
// The next tile's scores are there when a group asks for them, so that it goes from one tile's exponentials straight to the
// next: for D = 128 S has one buffer, free as soon as a group has its scores in registers, and P (input dtype, two values per
// column) columns of its own, one place a chain; for D = 64 there are three buffers, P overwrites the first 64 columns of its
// own, and S(g+3) follows P*V(g) on the pipe.
// Forward kernel, us between events in a graph (some 4 more than the kernel alone): two buffers in which P overwrites S, with
// the exponentials of the groups in turns | one O and one maximum for both chains, three buffers | now. 2 x 32 / 8 heads x
// 3001 x 128 causal 195 | 154 | 152, with q and k of deviation 2 242 | 322 | 198, of 4 229 | 303 | 204 (a shared maximum that
// moves makes either group wait for the other's P*V); 512 queries against 8192 keys, 32 / 8 heads of 128, 77 | 61 | 61, deviation
// 3 86 | 99 | 67; 16 x 8 x 577 x 32 45 | 37 | 37; 4 x 16 x 4096 x 128 in documents 174 | 145 | 151, deviation 3 184 | 206 | 163;
// 32 x 32768 x 128 in 64 documents 908 | 776 | 786; 16 x 32 x 8192 x 128 causal 9520 | 7760 | 7690; 4 x 16 x 4096 x 64 causal
// 249 | 201 | 192; 8 x 8 x 1024 x 8192 x 64, queries of random documents, 94 | 83 | 79. The shared O had errors 1 to 2 %
// larger as well: one entry of a row is an exact 1 in P, not one of each chain.
// Since then the code was made smaller (loops that are not unrolled, masks by a loop, shorter waits) and a block's first item is known at once. Both builds in turn,
// replayed graphs of one launch, some 30 after a pause (so above the power cap but for the last), other documents than above, us, that "now" | at present: 2 x 32 / 8 x
// 3001 153 | 142, 512 against 8192 63.8 | 61.8, 16 x 8 x 577 x 32 36.6 | 33.1, 4 x 16 x 4096 x 128 in documents 146 | 122, 32 x 32768 x 128 in 64 documents
// 484 | 387, 4 x 16 x 4096 x 64 causal 192 | 180, 8 x 8 x 1024 x 8192 x 64 105 | 91.5, 4 x 12 x 1000 x 64 in documents 30.9 | 24.8; long series of
// 16 x 32 x 8192 x 128, under the cap, 8370 | 8150.
// What bounds it: the softmax warps (scores out of TMEM, maximum, 1024 clocks of MUFU for a tile of each group, and fetching their own straight code), at D = 128 the
// 64 KB of K and V that each tile brings from L2 (52 B a clock and SM; half of them would take dense calls 5 % less time), and, in
// dense calls, the clock under the power cap (1.4-1.5 GHz); with short items the drain of two O, which the next item's P*V waits for.
#include <type_traits>
#include "common.cuh"
#include "params.cuh"

namespace fa {

// In an item's list of tiles a flag is one of six bits: TILE_KMANY has the place of TILE_QTAIL, which the forward does not ask for.
constexpr uint32_t LIST_KMANY = TILE_QTAIL;

template <int D>
struct FwdSmem {
    static constexpr int NS = (D == 128) ? 2 : 4;  // depth of the K ring and of the V ring
    // item slots; with more, items are dealt out too far ahead (3 or 4 for D = 64: 8 x 8 x 1024 x 8192 in documents 90, 86 with 2)
    static constexpr int NQ = 2;
    // TMEM columns: D = 128: S [0,128), two P of 64; D = 64: three S of 128, P in the first half of its S. Then the O of each chain.
    // (Three S and two O of 128 do not fit; one S and two P for D = 64, too: 4 x 16 x 4096 x 64 causal 247 us for 223.)
    static constexpr bool POWN = D == 128;   // P has columns of its own
    static constexpr int NP = POWN ? 2 : 3;  // places for P
    static constexpr int tmem_o = POWN ? 256 : 384;
    static_assert(tmem_o + 2 * D <= 512, "TMEM columns");
    static __device__ int tmem_s(int g) { return POWN ? 0 : g % 3 * 128; }
    static __device__ int tmem_p(int g) { return POWN ? 128 + (g & 1) * 64 : g % 3 * 128; }
    static constexpr int TILE = kBlk * D * 2;
    static constexpr int BOX = kBlk * 64 * 2;
    static constexpr int NBOX = D / 64;
    static constexpr int NKC = 8;  // depth of the key-code ring
    static constexpr int off_q = 0;  // NQ Q tiles; a slot also stages its item's O tile for the TMA store
    static constexpr int off_k = NQ * TILE;
    static constexpr int off_v = off_k + NS * TILE;
    static constexpr int off_list = off_v + NS * TILE;           // uint16 [NQ][kListCap]
    static constexpr int off_qc = off_list + NQ * kListCap * 2;  // int32  [NQ][128] query codes
    static constexpr int off_kc = off_qc + NQ * kBlk * 4;        // int32  [NKC][128] key codes, loaded with K on K's barrier
    static constexpr int off_ml = off_kc + NKC * kBlk * 4;       // float  [NQ][2 groups][m, l][128]
    static constexpr int off_info = off_ml + NQ * 4 * kBlk * 4;  // int32 [NQ][8]: T, lo, item (-1: no more items), kv head, query block, head, batch
    static constexpr int off_bar = off_info + NQ * 32;
    // item_full[NQ] item_empty[NQ] q_full[NQ] q_empty[NQ] ml_full[NQ] staged[NQ] k_full[NS] k_empty[NS] v_full[NS] v_empty[NS]
    // s_full[4] s_free[2] p_full[NP] pv_done[NP] o_full[2] o_free[2]
    static constexpr int n_bar = 6 * NQ + 4 * NS + 6 + 2 * NP + 4;
    static constexpr int off_misc = off_bar + n_bar * 8;  // tmem slot, abort flag
    static constexpr int total = off_misc + 16;
};
static_assert(FwdSmem<128>::total <= 232448 && FwdSmem<64>::total <= 232448, "shared memory budget");
// No two blocks of the library's kernels share an SM, and its tensor memory, though the next launch may start while this one ends.
// (Beside a block of head dim 64 another library's may have room; the order in which each of the kernels waits, allocates and lets
// the next one begin keeps that one's allocation from mattering.)
static_assert(FwdSmem<128>::total > 116736 && FwdSmem<64>::total > 116736, "shares an SM");

// SHORT: calls without ids whose items are too few or too empty for one item per (query block, head, batch).
// Two things are added (fwd_pack and fwd_splits in api.cu say when):
//  - p.pack query heads of one kv head share a tile, row g * M + i = query i of the g-th of them (at most 128
//    rows: one decoded token of 4 heads reads the keys and values once instead of four times). The Q and O maps
//    are 5-D, (D, M, G, Hk, B), and a box holds p.rows rows; tile rows past them are never loaded. They
//    start as zeros, may later hold what an earlier item staged there, and only ever reach results that are not stored. Warps without a valid row skip the softmax.
//  - an item's tiles are cut into p.ns runs that are items of their own. With ns > 1 the normalised fp32 rows
//    and their log-sum-exp go to the workspace, and fwd_combine_kernel merges them.
// Such calls are bound by reading K and V (16 tokens of 32 / 8 heads of 128 against 4500 keys: 295 MB, 45 us at the
// copy rate; 127 us with a tile per head, 55 us packed) or, with few heads, by the longest item's chain of tiles.
template <int D, bool BF16, bool SHORT>
__global__ void __launch_bounds__(kFwdThreads, 1)
fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
           const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdParams p) {
    using S = FwdSmem<D>;
    constexpr int NS = S::NS, NQ = S::NQ, NP = S::NP;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;

    const MaskArgs& mk = p.mask;
    const int nQ = mk.L.nQ;
    const int nG = SHORT ? cdiv(p.G, p.pack) : 1;  // tiles' worth of query heads per kv head
    const int HP = SHORT ? p.H / p.G * nG : p.H;   // heads, or packs of heads, per batch
    const int HB = HP * p.B;
    const int ns = SHORT ? p.ns : 1;
    const int n_items = nQ * HB * ns;
    unsigned int* ctr = mk.ctr ? mk.ctr + CTR_FWD : nullptr;

    volatile int* misc = reinterpret_cast<volatile int*>(smem + S::off_misc);  // [0] tmem, [1] abort
    volatile int* info = reinterpret_cast<volatile int*>(smem + S::off_info);
    const uint32_t bar0 = sbase + S::off_bar;
    auto BAR = [&](int i) { return bar0 + 8u * uint32_t(i); };
    constexpr int B_ITEMFULL = 0, B_ITEMEMPTY = NQ, B_QFULL = 2 * NQ, B_QEMPTY = 3 * NQ, B_MLFULL = 4 * NQ, B_STAGED = 5 * NQ, B_KFULL = 6 * NQ,
                  B_KEMPTY = B_KFULL + NS, B_VFULL = B_KEMPTY + NS, B_VEMPTY = B_VFULL + NS, B_SFULL = B_VEMPTY + NS,
                  B_SFREE = B_SFULL + 4, B_PFULL = B_SFREE + 2, B_PVDONE = B_PFULL + NP, B_OFULL = B_PVDONE + NP, B_OFREE = B_OFULL + 2;
    static_assert(B_OFREE + 2 == S::n_bar, "barriers");
    Abort ab{misc + 1, p.status, p.wait_limit};

    // item -> (query block, head, batch). Heads are taken in groups of p.gh; inside a group the query
    // blocks go from the last one down (with a causal mask: long ones first) and the heads of the
    // group vary fastest. The CTAs thus work on neighbouring query blocks of a few heads at a time:
    // few enough that their K / V streams stay in L2, enough that not all CTAs pull the same lines.
    auto decode = [&](int j, int& qb, int& h, int& b) {
        const int per = p.gh * nQ;                 // items of a full group of heads
        const int grp = j / per, rem = j - grp * per;
        const int gsz = min(p.gh, HB - grp * p.gh);  // heads in this group (the last one may be smaller)
        const int pos = rem / gsz, bh = grp * p.gh + (rem - pos * gsz);
        b = bh / HP;
        h = bh - b * HP;
        // few items per CTA: longest first (sorted in the plan), so that no long item is left for the end
        qb = p.by_length ? mk.plan[mk.L.off_ordq + (int64_t(b) * mk.He + (mk.He == 1 ? 0 : h)) * nQ + pos] : nQ - 1 - pos;
    };
    // What the scheduler finds out about item j before it has a slot for it; in `flags` the class of candidate tile lo + lane.
    struct Item {
        int qb, h, b, lo, n;
        uint32_t flags;
        int4 qc;
    };
    auto classify = [&](const Item& it, int i) {
        return i < it.n ? classify_from_plan(mk, it.b, (mk.He == 1) ? 0 : it.h, it.qb, it.lo + i) & (TILE_VISIT | TILE_BOUND | TILE_DOC | TILE_KMONO | TILE_KMANY) : 0u;
    };
    auto prepare = [&](int j) {
        Item it;
        const int sp = SHORT ? j % ns : 0;  // which run of the item's tiles
        decode(SHORT ? j / ns : j, it.qb, it.h, it.b);
        const int he = (mk.He == 1) ? 0 : it.h;
        int lo, hi;
        kv_range(mk, it.b, he, it.qb, lo, hi);
        int n = hi - lo;
        if constexpr (SHORT) {  // no ids: every tile of the range is visited
            const int first = int(int64_t(n) * sp / ns);
            n = int(int64_t(n) * (sp + 1) / ns) - first;
            lo += first;
        }
        it.lo = lo;
        it.n = n < kListCap ? n : kListCap;  // the host refuses problems that could exceed the cap
        it.qc = make_int4(0, 0, 0, 0);
        if (mk.mode == 1)
            it.qc = *reinterpret_cast<const int4*>(mk.plan + mk.L.off_qc + (int64_t(it.b) * mk.He + he) * mk.L.Mpad + int64_t(it.qb) * kBlk + lane * 4);
        it.flags = classify(it, lane);
        return it;
    };

    if (tid == 0) {
        for (int s = 0; s < NQ; ++s) {
            mbar_init(BAR(B_ITEMFULL + s), 1);
            mbar_init(BAR(B_ITEMEMPTY + s), 15);  // producer, two MMA issuers, eight softmax warps, four epilogue warps
            mbar_init(BAR(B_QFULL + s), 1);
            mbar_init(BAR(B_QEMPTY + s), 1);
            mbar_init(BAR(B_MLFULL + s), 8);
            mbar_init(BAR(B_STAGED + s), 4);
        }
        for (int s = 0; s < NS; ++s) {
            mbar_init(BAR(B_KFULL + s), 1);
            mbar_init(BAR(B_KEMPTY + s), 1);
            mbar_init(BAR(B_VFULL + s), 1);
            mbar_init(BAR(B_VEMPTY + s), 1);
        }
        for (int s = 0; s < 4; ++s) mbar_init(BAR(B_SFULL + s), 1);
        for (int s = 0; s < NP; ++s) {
            mbar_init(BAR(B_PFULL + s), 4);  // here and below: one arrival a warp
            mbar_init(BAR(B_PVDONE + s), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(BAR(B_SFREE + s), 4);
            mbar_init(BAR(B_OFULL + s), 1);
            mbar_init(BAR(B_OFREE + s), 4);
        }
        fence_mbar_init();
    }
    if constexpr (SHORT) {
        // Rows without a query are multiplied all the same, and zeros take less power than what lies in shared and tensor memory: 16
        // tokens of 32 / 8 heads of 128 against 4500 keys, call after call under the power cap, 55.8 us -> 53.9 (51.4 without the cap, both).
        for (int i = tid; i < NQ * S::TILE / 16; i += kFwdThreads) reinterpret_cast<uint4*>(smem + S::off_q)[i] = make_uint4(0, 0, 0, 0);
        fence_proxy_async();
    }
    // Without ids the scheduler knows its first item before the kernel may touch memory.
    Item item;
    if (warp == 14 && mk.mode == 0) item = prepare(int(blockIdx.x));
    wait_prerequisites();
    if (warp == 13) {
        tmem_alloc(sbase + S::off_misc, 512);
        tmem_relinquish();
    }
    if (tid == 0) misc[1] = (status_is_fatal(*reinterpret_cast<volatile int*>(p.status)) || (sbase & 1023u) != 0) ? 1 : 0;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    launch_dependents();
    const uint32_t tmem = uint32_t(misc[0]);
    const bool aborted = misc[1] != 0;
    // An earlier launch on this device ran into a time-out that the host has not yet cleared: the CTA fills its items of the fixed order with NaN, and
    // their LSE (see nan_fill_items; with counters any other CTA may have taken all but the first, and if none does they are everybody's. With ns > 1
    // the combine kernel fills the output). By one thread: by a warp, and by the items of the counter, the code cost each launch
    // 0.08 us (8 x 200 x 64 6.52 for 6.44), behind the roles it cost long calls 1 % (32 x 32768 x 128 in 64 documents 395 us for 391; 392 now).
    if (aborted && (sbase & 1023u) == 0 && ns == 1) {
        for (int i = tid; i < S::TILE / 16; i += kFwdThreads) reinterpret_cast<uint4*>(smem + S::off_q)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        fence_proxy_async();
        __syncthreads();
        if (tid == 0) {
#pragma unroll 1
            for (int k = 0, j; (j = item_in_order(k)) < n_items; ++k) {
                int qb, h, b;
                decode(j, qb, h, b);
                const int h0 = SHORT ? h / nG * p.G + (h % nG) * p.pack : h, n_h = SHORT ? min(p.pack, p.G - (h % nG) * p.pack) : 1;
                for (int x = 0; x < S::NBOX; ++x) {
                    if constexpr (SHORT) tma_store_5d(&tmO, sbase + S::off_q + x * S::BOX, x * 64, qb * kBlk, (h % nG) * p.pack, h / nG, b);
                    else tma_store_4d(&tmO, sbase + S::off_q + x * S::BOX, x * 64, qb * kBlk, h, b);
                }
                tma_store_commit();
#pragma unroll 1
                for (int i = 0; i < n_h * kBlk; ++i) {  // the rows past M pad the buffer
                    const int row = qb * kBlk + i % kBlk;
                    p.lse[(int64_t(b) * p.H + h0 + i / kBlk) * mk.L.Mpad + row] = row < mk.M ? __int_as_float(-1) : 0.f;
                }
            }
            tma_store_wait_all();
        }
    }

    auto sQ = [&](int s) { return sbase + S::off_q + uint32_t(s) * S::TILE; };
    auto sK = [&](int s) { return sbase + S::off_k + uint32_t(s) * S::TILE; };
    auto sV = [&](int s) { return sbase + S::off_v + uint32_t(s) * S::TILE; };
    auto list_of = [&](int s) { return reinterpret_cast<const uint16_t*>(smem + S::off_list) + s * kListCap; };
    if (warp >= 12) {
        setmaxnreg_dec<kFwdServiceRegs>();
        if (aborted) {
            // a previous kernel reported an error: do nothing
        } else if (warp == 14) {
            // ------------------------------ item scheduler ------------------------------
            // The first item of a CTA is its own number; the others are handed out in order from a counter in the plan (any CTA
            // takes the next one: the work per item varies with the mask); without counters (no plan given) they are dealt out
            // round robin in alternating direction, which evens out their sorted lengths. us, every item from the counter | the first
            // one known, without ids before the wait: 8 x 200 x 64 7.42 | 7.10, 4 x 12 x 1000 x 64 in documents 24.4 | 22.5, 8 x 8 x 1024 x 8192 x
            // 64 in documents 75.2 | 71.4, 4 x 16 x 4096 x 128 in documents 153 | 148, 16 x 8 x 577 x 32 31.1 | 31.5. An item taken, and what the
            // plan says about it read, while the one before it still holds the slot leaves no pause between items, but is dealt out
            // too far ahead: 28.1 for 27.8, 75.6 for 76.5, 157 for 154. (dK/dV gains nothing from a first item of its own.)
            bool ok = true;
            int j = int(blockIdx.x);
            for (int k = 0;; ++k) {
                const int s = k % NQ, use = k / NQ;
                if (use > 0) ok = mbar_wait_warp(BAR(B_ITEMEMPTY + s), (use - 1) & 1, ab, ST_WAIT_TIMEOUT + 11);
                if (!ok) break;
                if (k > 0) {
                    if (lane == 0) {
                        if (ctr) j = int(gridDim.x + atomicAdd(ctr, 1u));
                        else j = item_in_order(k);
                    }
                    j = __shfl_sync(0xffffffffu, j, 0);
                }
                if ((k > 0 || mk.mode != 0) && j < n_items) item = prepare(j);
                if (j >= n_items) {  // end marker
                    if (lane == 0) {
                        info[s * 8 + 2] = -1;
                        mbar_arrive(BAR(B_ITEMFULL + s));
                    }
                    break;
                }
                uint16_t* list = reinterpret_cast<uint16_t*>(smem + S::off_list) + s * kListCap;
                int T = 0;
                for (int base = 0; base < item.n; base += 32) {
                    const int i = base + lane;
                    const uint32_t f = base == 0 ? item.flags : classify(item, i);
                    const uint32_t m = __ballot_sync(0xffffffffu, (f & TILE_VISIT) != 0);
                    if (f & TILE_VISIT) list[T + __popc(m & ((1u << lane) - 1u))] = uint16_t(uint32_t(i) | ((f & ~TILE_KMANY) | ((f & TILE_KMANY) ? LIST_KMANY : 0u)) << 10);
                    T += __popc(m);
                }
                reinterpret_cast<int4*>(smem + S::off_qc)[s * 32 + lane] = item.qc;
                if (lane == 0) {
                    info[s * 8 + 0] = T;
                    info[s * 8 + 1] = item.lo;
                    info[s * 8 + 2] = j;
                    info[s * 8 + 3] = SHORT ? item.h / nG : item.h / p.G;
                    info[s * 8 + 4] = item.qb;
                    info[s * 8 + 5] = item.h;
                    info[s * 8 + 6] = item.b;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(B_ITEMFULL + s));
            }
        } else if (warp == 12) {
            // ------------------------------ TMA producer ------------------------------
            // Two walks over the CTA's tiles: K (with its item's Q), up to kAhead tiles ahead of V. Into the next item K
            // only goes ahead while its slot is free at once, so that the V tiles of the item at hand never wait for it.
            // The warp runs converged with uniform values (one lane with its numbers in vector registers took 950 clocks
            // from a load to the next, more than half a tile's time).
            tma_prefetch_desc(&tmQ);
            tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmV);
            constexpr int kAhead = 3;
            bool ok = true, last = false;  // last: the K walk has seen the end marker
            int kk = -1, kt = 0, kT = 0, gk = 0, klo = 0, khk = 0, kb = 0, khe = 0;  // K walk: item, its next tile and tiles; tiles issued
            int vk = -1, vt = 0, vT = 0, gv = 0, vlo = 0, vhk = 0, vb = 0;           // V walk
            while (ok) {
                while (vt == vT && vk < kk) {  // the V walk goes on to the next item
                    if (vk >= 0 && lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + vk % NQ));
                    ++vk;
                    const int s = vk % NQ;
                    vt = 0;
                    vT = uniform(info[s * 8 + 0]);
                    vlo = uniform(info[s * 8 + 1]);
                    vhk = uniform(info[s * 8 + 3]);
                    vb = uniform(info[s * 8 + 6]);
                }
                if (last && gv == gk) break;
                bool do_k = !last && gk - gv < kAhead;
                if (do_k && kt == kT) {  // the next item: its slot's last O must have left
                    const int s = (kk + 1) % NQ, use = (kk + 1) / NQ;
                    if (gv < gk && !(mbar_test_warp(BAR(B_ITEMFULL + s), use & 1) &&
                                     (use == 0 || mbar_test_warp(BAR(B_QEMPTY + s), (use - 1) & 1)))) {
                        do_k = false;
                    } else {
                        ok = mbar_wait_warp(BAR(B_ITEMFULL + s), use & 1, ab, ST_WAIT_TIMEOUT + 12);
                        if (!ok) break;
                        if (uniform(info[s * 8 + 2]) < 0) {
                            last = true;
                            continue;
                        }
                        if (use > 0) ok = mbar_wait_warp(BAR(B_QEMPTY + s), (use - 1) & 1, ab, ST_WAIT_TIMEOUT + 13);
                        if (!ok) break;
                        ++kk;
                        kt = 0;
                        kT = uniform(info[s * 8 + 0]);
                        klo = uniform(info[s * 8 + 1]);
                        khk = uniform(info[s * 8 + 3]);
                        const int qb = uniform(info[s * 8 + 4]), h = uniform(info[s * 8 + 5]);
                        kb = uniform(info[s * 8 + 6]);
                        khe = (mk.He == 1) ? 0 : h;
                        if constexpr (SHORT) {
                            mbar_expect_tx_elect(BAR(B_QFULL + s), uint32_t(p.rows) * 128u * S::NBOX);
                            for (int x = 0; x < S::NBOX; ++x)
                                tma_load_5d_elect(sQ(s) + x * S::BOX, &tmQ, BAR(B_QFULL + s), x * 64, qb * kBlk, (h % nG) * p.pack, khk, kb);
                        } else {
                            mbar_expect_tx_elect(BAR(B_QFULL + s), S::TILE);
                            for (int x = 0; x < S::NBOX; ++x)
                                tma_load_4d_elect(sQ(s) + x * S::BOX, &tmQ, BAR(B_QFULL + s), x * 64, qb * kBlk, h, kb);
                        }
                        continue;  // (an item may have no tiles)
                    }
                }
                if (do_k) {
                    const int blk = klo + uniform(list_of(kk % NQ)[kt] & 1023), st = gk % NS, ug = gk / NS;
                    if (ug > 0) ok = mbar_wait_warp(BAR(B_KEMPTY + st), (ug - 1) & 1, ab, ST_WAIT_TIMEOUT + 1);
                    if (!ok) break;
                    // The tile's key codes travel with K: they land in a ring of NKC slots and complete on
                    // K's barrier, so whoever has seen S(g) (computed after that barrier) may read them.
                    // Slot g % NKC was last read by the softmax of tile g - NKC, which is over: S(g - NS), which has just
                    // released K's stage, was issued behind P*V(g - NS - 3) or, where P has columns of its own, when both groups had
                    // read the scores of tiles g - NS - 1 and g - NS - 2, hence were done with those up to g - NS - 3.
                    static_assert(S::NKC >= NS + 3, "key-code ring");
                    mbar_expect_tx_elect(BAR(B_KFULL + st), S::TILE + (mk.mode == 1 ? kBlk * 4 : 0));
                    for (int x = 0; x < S::NBOX; ++x)
                        tma_load_4d_elect(sK(st) + x * S::BOX, &tmK, BAR(B_KFULL + st), x * 64, blk * kBlk, khk, kb);
                    if (mk.mode == 1)
                        bulk_load_1d_elect(sbase + S::off_kc + (gk % S::NKC) * (kBlk * 4),
                                           mk.plan + mk.L.off_kc + (int64_t(kb) * mk.He + khe) * mk.L.Npad + int64_t(blk) * kBlk,
                                           kBlk * 4, BAR(B_KFULL + st));
                    ++kt;
                    ++gk;
                } else {
                    const int blk = vlo + uniform(list_of(vk % NQ)[vt] & 1023), st = gv % NS, ug = gv / NS;
                    if (ug > 0) ok = mbar_wait_warp(BAR(B_VEMPTY + st), (ug - 1) & 1, ab, ST_WAIT_TIMEOUT + 2);
                    if (!ok) break;
                    mbar_expect_tx_elect(BAR(B_VFULL + st), S::TILE);
                    for (int x = 0; x < S::NBOX; ++x)
                        tma_load_4d_elect(sV(st) + x * S::BOX, &tmV, BAR(B_VFULL + st), x * 64, blk * kBlk, vhk, vb);
                    ++vt;
                    ++gv;
                }
            }
        } else {
            // ------------------------------ MMA issuers ------------------------------
            //   warp 13: P*V(g) when P(g) is there
            //   warp 15: S(g) when its buffer is free
            // Two warps, so that S of a later tile (and of the next item's first ones) never waits behind P of this one.
            const uint32_t utmem = uniform(int(tmem));
            constexpr uint32_t idesc_s = make_idesc(BF16, 128, 128, false, false);
            constexpr uint32_t idesc_pv = make_idesc(BF16, 128, D, false, true);
            constexpr uint64_t desc_v = desc_mn_major(S::BOX);
            bool ok = true;
            int G = 0;           // tiles of all earlier items
            int n0 = 0, n1 = 0;  // items in which the chains had tiles
            for (int k = 0;; ++k) {
                const int s = k % NQ, use = k / NQ;
                ok = mbar_wait_warp(BAR(B_ITEMFULL + s), use & 1, ab, ST_WAIT_TIMEOUT + 12);
                if (!ok) break;
                const int T = uniform(info[s * 8 + 0]);
                if (uniform(info[s * 8 + 2]) < 0) break;
                if (warp == 15) {
                    if (T > 0) ok = mbar_wait_warp(BAR(B_QFULL + s), use & 1, ab, ST_WAIT_TIMEOUT + 3);
                    for (int g = G; g < G + T && ok; ++g) {
                        const int st = g % NS;
                        ok = mbar_wait_warp(BAR(B_KFULL + st), (g / NS) & 1, ab, ST_WAIT_TIMEOUT + 4);
                        // the buffer: its scores have been read, or the P that took their place
                        if (S::POWN && ok && g > 0) ok = mbar_wait_warp(BAR(B_SFREE + ((g - 1) & 1)), ((g - 1) >> 1) & 1, ab, ST_WAIT_TIMEOUT + 15);
                        if (!S::POWN && ok && g >= NP) ok = mbar_wait_warp(BAR(B_PVDONE + g % NP), (g / NP - 1) & 1, ab, ST_WAIT_TIMEOUT + 15);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t tS = utmem + uint32_t(S::tmem_s(g)), q_tile = sQ(s), k_tile = sK(st);
#pragma unroll
                        for (int kk = 0; kk < D / 16; ++kk) {
                            const uint32_t off = uint32_t(kk >> 2) * S::BOX + uint32_t(kk & 3) * 32u;
                            umma_ss(tS, smem_desc_at(kDescKMajor, q_tile + off), smem_desc_at(kDescKMajor, k_tile + off), idesc_s, kk > 0);
                        }
                        umma_commit(BAR(B_KEMPTY + st));
                        umma_commit(BAR(B_SFULL + (g & 3)));
                    }
                } else {
                    for (int t = 0; t < T; ++t) {
                        const int g = G + t, st = g % NS, w = g & 1;
                        const uint32_t tO = utmem + uint32_t(S::tmem_o + w * D), tP = utmem + uint32_t(S::tmem_p(g)), v_tile = sV(st);
                        ok = mbar_wait_warp(BAR(B_VFULL + st), (g / NS) & 1, ab, ST_WAIT_TIMEOUT + 5);
                        // The first P*V of a chain in an item overwrites its O: the epilogue of the last item that used it must have
                        // read it. (o_full and o_free count the items in which the chain had tiles, on both sides.)
                        const int n = w ? n1 : n0;
                        if (ok && t < 2 && n > 0) ok = mbar_wait_warp(BAR(B_OFREE + w), (n - 1) & 1, ab, ST_WAIT_TIMEOUT + 14);
                        if (ok) ok = mbar_wait_warp(BAR(B_PFULL + g % NP), (g / NP) & 1, ab, ST_WAIT_TIMEOUT + 6);
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)
                            umma_ts(tO, tP + uint32_t(kk) * 8u, smem_desc_at(desc_v, v_tile + uint32_t(kk) * 2048u), idesc_pv,
                                    (t > 1 || kk > 0) ? 1u : 0u);
                        umma_commit(BAR(B_VEMPTY + st));
                        umma_commit(BAR(B_PVDONE + g % NP));
                        if (t + 2 >= T) {  // the chain's last tile
                            umma_commit(BAR(B_OFULL + w));
                            if (w) ++n1; else ++n0;
                        }
                    }
                }
                if (!ok) break;
                G += T;
                if (lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + s));
                __syncwarp();
            }
        }
        __syncwarp();
    } else if (warp >= 8) {
        // ------------------------------ epilogue group ------------------------------
        setmaxnreg_dec<kFwdEpilogueRegs>();
        const int r = tid & 127;
        const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
        const float c = p.scale_log2;
        bool alive = !aborted;
        int G = 0;           // tiles of all earlier items
        int n0 = 0, n1 = 0;  // items in which the chains of group 0 and 1 had tiles
        for (int k = 0; alive; ++k) {
            const int s = k % NQ, use = k / NQ;
            alive = mbar_wait_warp(BAR(B_ITEMFULL + s), use & 1, ab, ST_WAIT_TIMEOUT + 12);
            if (!alive) break;
            const int T = info[s * 8 + 0], j = info[s * 8 + 2], qb = info[s * 8 + 4], h = info[s * 8 + 5], b = info[s * 8 + 6];
            if (j < 0) break;
            const int g_row = SHORT && p.pack > 1 ? r / mk.M : 0;
            const int row = qb * kBlk + r - g_row * mk.M;
            const int g_own = SHORT ? (h % nG) * p.pack + g_row : 0;
            const bool valid = !SHORT || (row < mk.M && g_row < p.pack && g_own < p.G);
            // the only wait here that lasts as long as an item: it allows each of the tiles what another wait may last
            const Abort item{ab.flag, ab.status, ab.limit * (T + 1)};
            alive = mbar_wait_warp(BAR(B_MLFULL + s), use & 1, item, ST_WAIT_TIMEOUT + 16);
            // an item without tiles: nobody has waited for its Q load yet, and its slot is about to become the staging area
            if (alive && T == 0) alive = mbar_wait_warp(BAR(B_QFULL + s), use & 1, ab, ST_WAIT_TIMEOUT + 17);
            const int we = G & 1;  // the chain that had the item's even tiles: index 0 below, 1 the other one
            const int i0 = we ? n1 : n0, i1 = we ? n0 : n1;
            if (alive && T > 0) alive = mbar_wait_warp(BAR(B_OFULL + we), i0 & 1, ab, ST_WAIT_TIMEOUT + 9);
            if (alive && T > 1) alive = mbar_wait_warp(BAR(B_OFULL + (we ^ 1)), i1 & 1, ab, ST_WAIT_TIMEOUT + 9);
            if (!alive) break;
            tc_fence_after();
            const float* ml = reinterpret_cast<const float*>(smem + S::off_ml) + s * (4 * kBlk);  // [2 groups][m, l][128]
            const int even = we * (2 * kBlk), odd = 2 * kBlk - even;
            const float m0 = ml[even + r], l0 = ml[even + kBlk + r], m1 = ml[odd + r], l1 = ml[odd + kBlk + r];
            const float mt = fmaxf(m0, m1);
            const float a0 = (m0 == -INFINITY) ? 0.f : fast_exp2((m0 - mt) * c);
            const float a1 = (m1 == -INFINITY) ? 0.f : fast_exp2((m1 - mt) * c);
            const float lt = l0 * a0 + l1 * a1;
            const float inv = (lt > 0.f) ? 1.0f / lt : 0.f;
            const float f0 = a0 * inv, f1 = a1 * inv;
            // a chain in which the row had no key takes no part, whatever the values behind its mask are
            const bool use0 = (T > 0) && (f0 != 0.f), use1 = (T > 1) && (f1 != 0.f);
            const bool healthy = misc[1] == 0;
            if (healthy) {
                const float lse = (lt > 0.f) ? fmaf(mt, c, log2f(lt)) : -INFINITY;
                if constexpr (SHORT) {
                    const int64_t bh0 = int64_t(b) * p.H + int64_t(h / nG) * p.G;
                    if (ns > 1) {
                        // a run that went NaN says so: -inf would pass for a run without keys
                        if (valid) p.part_lse[((bh0 + g_own) * mk.M + row) * ns + j % ns] = (lt == lt) ? lse : lt;
                    } else {
                        if (valid) p.lse[(bh0 + g_own) * mk.L.Mpad + row] = lse;
                        // the rows past M that pad the buffer
                        for (int g = (h % nG) * p.pack; g < min(p.G, (h % nG + 1) * p.pack); ++g)
                            if (qb * kBlk + r >= mk.M) p.lse[(bh0 + g) * mk.L.Mpad + qb * kBlk + r] = 0.f;
                    }
                } else {
                    p.lse[(int64_t(b) * p.H + h) * mk.L.Mpad + row] = lse;
                }
            }
            float* part = nullptr;  // this thread's row in the workspace (SHORT, ns > 1)
            if constexpr (SHORT) {
                if (ns > 1 && valid && healthy)
                    part = p.part_o + ((int64_t(j % ns) * p.B * p.H + int64_t(b) * p.H + int64_t(h / nG) * p.G + g_own) * mk.M + row) * D;
            }
            // The O tile is staged in this item's Q slot (Q is dead: every S MMA of the item has completed) in the
            // 128-byte-swizzled layout of the tensor map.
            uint8_t* stage = smem + S::off_q + s * S::TILE;
            const uint32_t tO0 = tmem + lane_base + uint32_t(S::tmem_o + we * D), tO1 = tmem + lane_base + uint32_t(S::tmem_o + (we ^ 1) * D);
            // (rolled: an eighth of the code to fetch for each item. 4 x 16 x 4096 x 128 in documents 152 -> 146 us a forward)
#pragma unroll 1
            for (int q = 0; q < D / 16; ++q) {
                uint32_t x0[16], x1[16];
                // tcgen05.ld is warp-collective: always executed, the values are ignored when unused
                tmem_ld16(tO0 + uint32_t(q) * 16u, x0);
                tmem_ld16(tO1 + uint32_t(q) * 16u, x1);
                tc_wait_ld();
                if (q == D / 16 - 1) {  // O has been read: the MMA issuers may start another item's P*V
                    tc_fence_before();
                    if (T > 0) mbar_arrive_warp(BAR(B_OFREE + we), lane);
                    if (T > 1) mbar_arrive_warp(BAR(B_OFREE + (we ^ 1)), lane);
                }
#pragma unroll
                for (int y = 0; y < 16; ++y) {
                    float v = 0.f;
                    if (use0) v = __uint_as_float(x0[y]) * f0;
                    if (use1) v = fmaf(__uint_as_float(x1[y]), f1, v);
                    x0[y] = __float_as_uint(v);
                }
                if constexpr (SHORT) {
                    if (part) {
#pragma unroll
                        for (int y = 0; y < 4; ++y)
                            *reinterpret_cast<uint4*>(part + 16 * q + 4 * y) = make_uint4(x0[4 * y], x0[4 * y + 1], x0[4 * y + 2], x0[4 * y + 3]);
                    }
                }
                auto two = [&](int y) { return pack2<BF16>(__uint_as_float(x0[y]), __uint_as_float(x0[y + 1])); };
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int cg = 2 * q + i;  // 16-byte chunk of the row
                    uint4* dst = reinterpret_cast<uint4*>(stage + (cg >> 3) * S::BOX + r * 128 + (((cg & 7) ^ (r & 7)) << 4));
                    *dst = make_uint4(two(8 * i), two(8 * i + 2), two(8 * i + 4), two(8 * i + 6));
                }
            }
            G += T;
            n0 += (we ? T > 1 : T > 0) ? 1 : 0;
            n1 += (we ? T > 0 : T > 1) ? 1 : 0;
            fence_proxy_async();
            mbar_arrive_warp(BAR(B_STAGED + s), lane);
            if (warp == 8) alive = mbar_wait_warp(BAR(B_STAGED + s), use & 1, ab, ST_WAIT_TIMEOUT + 18);
            if (!alive) break;
            if (r == 0) {
                if (healthy) {
                    if constexpr (SHORT) {
                        if (ns == 1)  // else the rows went to the workspace
                            for (int x = 0; x < S::NBOX; ++x)
                                tma_store_5d(&tmO, sQ(s) + x * S::BOX, x * 64, qb * kBlk, (h % nG) * p.pack, h / nG, b);
                    } else {
                        for (int x = 0; x < S::NBOX; ++x) tma_store_4d(&tmO, sQ(s) + x * S::BOX, x * 64, qb * kBlk, h, b);
                    }
                    tma_store_commit();
                    tma_store_wait_read();
                }
                mbar_arrive(BAR(B_QEMPTY + s));  // the slot may take another item's Q
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + s));
        }
        if (r == 0) tma_store_wait_all();
        __syncwarp();
    } else {
        setmaxnreg_inc<kFwdSoftmaxRegs>();
        // ------------------------------ softmax groups ------------------------------
        // Every wait is a bounded mbarrier wait: a warp whose wait was given up (alive == false)
        // leaves the item loop at once, and nobody is left waiting for it for longer than the limit.
        const int w = warp >> 2;  // group
        const int r = tid & 127;  // row inside the block
        const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
        const float c = p.scale_log2;
        const uint32_t tO = tmem + lane_base + uint32_t(S::tmem_o + w * D);
        bool alive = !aborted;
        if (SHORT && S::POWN) {  // P of the rows without a query
            uint32_t zero[32] = {};
            tmem_st32(tmem + lane_base + uint32_t(S::tmem_p(w)), zero);
            tmem_st32(tmem + lane_base + uint32_t(S::tmem_p(w)) + 32u, zero);
            tc_wait_st();
            tc_fence_before();
        }
        int G = 0;  // tiles of all earlier items
        for (int k = 0; alive; ++k) {
            const int s = k % NQ, use = k / NQ;
            alive = mbar_wait_warp(BAR(B_ITEMFULL + s), use & 1, ab, ST_WAIT_TIMEOUT + 12);
            if (!alive) break;
            const int T = info[s * 8 + 0];
            const int lo = info[s * 8 + 1];
            if (info[s * 8 + 2] < 0) break;
            const uint16_t* list = list_of(s);
            const int qb = info[s * 8 + 4];
            // this thread's query: row of the head, and (SHORT) which head of the group
            const int g_row = SHORT && p.pack > 1 ? r / mk.M : 0;
            const int row = qb * kBlk + r - g_row * mk.M;
            const bool valid = !SHORT || (row < mk.M && g_row < p.pack && (info[s * 8 + 5] % nG) * p.pack + g_row < p.G);
            const bool active = !SHORT || __any_sync(0xffffffffu, valid);  // does this warp hold a query at all?
            const int qc = reinterpret_cast<const int*>(smem + S::off_qc)[s * kBlk + r];
            const int t0 = (G ^ w) & 1;  // this group's first tile of the item
            float m_run = -INFINITY, l_run = 0.f;

            for (int t = t0; t < T && alive; t += 2) {
                const uint32_t entry = list[t];
                const uint32_t fl = entry >> 10;
                const int k0 = (lo + int(entry & 1023u)) * kBlk;
                const int g = G + t;
                const uint32_t tS = tmem + lane_base + uint32_t(S::tmem_s(g)), tP = tmem + lane_base + uint32_t(S::tmem_p(g));
                // P*V of the group's tile before: it has read its P and added to O
                auto pv_before = [&] { return g < 2 || mbar_wait_warp(BAR(B_PVDONE + (g - 2) % NP), ((g - 2) / NP) & 1, ab, ST_WAIT_TIMEOUT + 8); };
                alive = mbar_wait_warp(BAR(B_SFULL + (g & 3)), (g >> 2) & 1, ab, ST_WAIT_TIMEOUT + 7);
                if (!alive) break;
                tc_fence_after();
                if (SHORT && !active) {  // no row of this warp is a query: its lanes of P and O are never stored
                    if (S::POWN) {
                        mbar_arrive_warp(BAR(B_SFREE + w), lane);
                        alive = pv_before();
                        if (!alive) break;
                    }
                    mbar_arrive_warp(BAR(B_PFULL + g % NP), lane);
                    continue;
                }
                uint32_t sr[128];
#pragma unroll
                for (int q = 0; q < 4; ++q) tmem_ld32(tS + uint32_t(q) * 32u, sr + q * 32);
                tc_wait_ld();
                if (S::POWN) {
                    tc_fence_before();
                    mbar_arrive_warp(BAR(B_SFREE + w), lane);  // the next tile's scores may overwrite these
                }
                float* sc = reinterpret_cast<float*>(sr);

                if (fl & (TILE_BOUND | TILE_DOC)) {
                    // keep(x) = (x <= lim) & (qc >= 0 | kc[x] == qc) as 32-bit masks, one select per entry behind them. The ids' part is worked
                    // out by a loop over the four chunks: unrolled, with a case of its own for each kind of chunk, this was most of
                    // the softmax warps' code, and fetching it cost more than running it. us a forward, so | now: 8 x 8 x 1024 x 8192 x 64 in
                    // documents 72.7 | 62.5, 4 x 12 x 1000 x 64 21.1 | 19.1, 4 x 16 x 4096 x 128 154 | 142, with ids drawn at random from 40 383 | 338,
                    // 32 x 32768 x 128 in 64 documents 870 | 827, 16 x 8 x 577 x 32 without ids 29.1 | 28.1.
                    int lim = kBlk - 1;
                    if (fl & TILE_BOUND) {
                        int jmax = mk.N - 1;
                        if (mk.causal) jmax = min(jmax, row + mk.gap);
                        lim = jmax - k0;
                    }
                    // (the key codes completed on K's barrier, before the S MMA whose result was just read)
                    const int* kcs = reinterpret_cast<const int*>(smem + S::off_kc + (g % S::NKC) * (kBlk * 4));
                    uint32_t same[4] = {~0u, ~0u, ~0u, ~0u};
                    if (fl & TILE_DOC) {
                        if ((fl & TILE_KMONO) && kcs[0] == kcs[kBlk - 1]) {  // one code in the block
                            if (qc < 0 && kcs[0] != qc) same[0] = same[1] = same[2] = same[3] = 0u;
                        } else {
#pragma unroll 1
                            for (int q = 0; q < 4; ++q) {
                                uint32_t m = codes_equal(kcs + 32 * q, kcs[32 * q + lane], qc, (fl & LIST_KMANY) != 0);
                                if (qc >= 0) m = ~0u;  // such a row passes the id check everywhere
                                if (q == 0) same[0] = m; else if (q == 1) same[1] = m; else if (q == 2) same[2] = m; else same[3] = m;
                            }
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t keep = first_bits(lim + 1 - 32 * q) & same[q];
                        if (__any_sync(0xffffffffu, keep != ~0u)) {
#pragma unroll
                            for (int x = 0; x < 32; ++x) sc[32 * q + x] = (keep & (1u << x)) ? sc[32 * q + x] : -INFINITY;
                        }
                    }
                }
                float mxa[8];
#pragma unroll
                for (int a = 0; a < 8; ++a) mxa[a] = max3(sc[a], sc[8 + a], sc[16 + a]);
#pragma unroll
                for (int x = 24; x < 120; x += 16) {
#pragma unroll
                    for (int a = 0; a < 8; ++a) mxa[a] = max3(mxa[a], sc[x + a], sc[x + 8 + a]);
                }
#pragma unroll
                for (int a = 0; a < 8; ++a) mxa[a] = fmaxf(mxa[a], sc[120 + a]);
                const float mx = fmaxf(max3(mxa[0], mxa[1], mxa[2]), max3(max3(mxa[3], mxa[4], mxa[5]), mxa[6], mxa[7]));
                float m_new = fmaxf(m_run, mx);
                // lazy rescale: keep the old reference point while the new maximum is within 2^8 of it
                const bool need = (m_new - m_run) * c > 8.0f;
                if (!need) m_new = m_run;
                if (S::POWN) {  // this tile's P overwrites that one's
                    alive = pv_before();
                    if (!alive) break;
                    tc_fence_after();
                }
                if (__any_sync(0xffffffffu, need)) {
                    const float alpha = need ? fast_exp2((m_run - m_new) * c) : 1.0f;
                    l_run *= alpha;
                    if (t > t0) {
                        if (!S::POWN) {
                            alive = pv_before();
                            if (!alive) break;
                            tc_fence_after();
                        }
                        // (rolled: it lies on the way of every tile and is rarely taken. 4 x 16 x 4096 x 128 in documents 143 -> 136 us a
                        // forward, 2 x 32 / 8 x 3001 x 128 169 -> 163)
#pragma unroll 1
                        for (int q = 0; q < D / 16; ++q) {
                            uint32_t orr[16];
                            tmem_ld16(tO + uint32_t(q) * 16u, orr);
                            tc_wait_ld();
#pragma unroll
                            for (int x = 0; x < 16; ++x) orr[x] = __float_as_uint(__uint_as_float(orr[x]) * alpha);
                            tmem_st16(tO + uint32_t(q) * 16u, orr);
                        }
                        tc_wait_st();
                    }
                }
                m_run = m_new;
                const float mneg = (m_run == -INFINITY) ? 0.f : -m_run * c;
                // exp2(s*c - m*c) on packed pairs
                const uint64_t c2 = pack_f2(c, c), mneg2 = pack_f2(mneg, mneg);
                uint64_t lacc0 = pack_f2(0.f, 0.f), lacc1 = lacc0;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t pk[16];
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        const uint64_t x2 = fma_f2(pack_f2(sc[32 * q + 2 * x], sc[32 * q + 2 * x + 1]), c2, mneg2);
                        float x0, x1;
                        unpack_f2(x2, x0, x1);
                        const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
                        if (x & 1) lacc1 = add_f2(lacc1, pack_f2(p0, p1)); else lacc0 = add_f2(lacc0, pack_f2(p0, p1));
                        pk[x] = pack2<BF16>(p0, p1);
                    }
                    tmem_st16(tP + uint32_t(q) * 16u, pk);
                }
                tc_wait_st();
                tc_fence_before();
                mbar_arrive_warp(BAR(B_PFULL + g % NP), lane);
                {
                    float a0, a1, b0, b1;
                    unpack_f2(lacc0, a0, a1);
                    unpack_f2(lacc1, b0, b1);
                    l_run += (a0 + a1) + (b0 + b1);
                }
            }
            if (!alive) break;
            float* ml = reinterpret_cast<float*>(smem + S::off_ml) + s * (4 * kBlk) + w * (2 * kBlk) + r;
            ml[0] = m_run;
            ml[kBlk] = l_run;
            mbar_arrive_warp(BAR(B_MLFULL + s), lane);
            G += T;
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + s));
        }
    }

    // ------------------------------ tear-down ------------------------------
    tc_fence_before();
    __syncthreads();
    if (warp == 13) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    // the last CTA to leave clears the work counters for the next launch that uses this plan
    if (tid == 0 && ctr) {
        __threadfence();
        if (atomicAdd(ctr + 1, 1u) == gridDim.x - 1) {
            ctr[0] = 0;
            ctr[1] = 0;
        }
    }
}

// Merges the ns partial results of a split forward: O = sum_s w_s O_s with w_s = 2^(lse_s - lse), lse the log2-sum
// over the parts. A part whose lse is NaN or +inf (a NaN or an infinity among its scores) makes the row its own, as in a
// call of one run: zeros or NaN, with an lse of -inf. One warp per row; lane l owns columns l, l + 32, ... (D <= 128), all sums
// in fp32 in the order of the parts. Bound by latency: at most 20 MB are read (fwd_splits in api.cu), mostly from L2, so that eight parts' loads are in flight
// together. A call of one token, 32 / 8 heads of 128, us, four parts behind their own weights | now: 4096 keys in 16 runs 16.1 | 12.7, 16384 in 16 20.7 |
// 17.3; 2 x 64 / 8 heads, 3000 in 8 14.5 | 13.0.
template <bool BF16>
__global__ void __launch_bounds__(256) fwd_combine_kernel(const CombineParams p) {
    follow_stream();
    const int64_t row = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);  // of the [B, H, M] rows
    const int lane = threadIdx.x & 31;
    const int64_t rows = int64_t(p.B) * p.H * p.M;
    if (row >= rows) return;
    const int64_t bh = row / p.M;
    const int i = int(row - bh * p.M);
    float* lse = p.lse + bh * p.Mpad;
    if (i == p.M - 1)  // the rows past M that pad the buffer
        for (int64_t x = p.M + lane; x < p.Mpad; x += 32) lse[x] = 0.f;
    const bool failed = status_is_fatal(*p.status);  // the forward left no parts: NaN, as the other kernels do
    float mx = -INFINITY;
    bool spoilt = false;
    for (int s = lane; s < p.ns; s += 32) {
        const float x = p.part_lse[row * p.ns + s];
        spoilt |= !(x < INFINITY);
        mx = fmaxf(mx, x);
    }
    spoilt = __any_sync(0xffffffffu, spoilt);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float acc[4] = {0.f, 0.f, 0.f, 0.f}, total = 0.f;
    if (mx != -INFINITY || spoilt) {
        for (int s0 = 0; s0 < p.ns; s0 += 32) {
            // a weight a lane; the rows' loads wait for nothing but their turn
            const float x = s0 + lane < p.ns ? p.part_lse[row * p.ns + s0 + lane] : -INFINITY;
            const float own = !spoilt ? fast_exp2(x - mx) : x < INFINITY ? 0.f : 1.f;  // an empty part: 2^-inf = 0
            const int n = min(32, p.ns - s0);
            auto add = [&](auto batch, int t0) {  // parts [t0, t0 + batch), as far as there are any
                constexpr int kBatch = decltype(batch)::value;
                float v[kBatch][4];
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    const float* po = p.part_o + (int64_t(s0 + min(t0 + t, n - 1)) * rows + row) * p.Dk;
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[t][k] = lane + 32 * k < p.D ? po[lane + 32 * k] : 0.f;
                }
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    const float wgt = __shfl_sync(0xffffffffu, own, t0 + t);
                    if (t0 + t >= n || (spoilt && wgt == 0.f)) continue;
                    total += wgt;
#pragma unroll
                    for (int k = 0; k < 4; ++k) acc[k] = fmaf(wgt, v[t][k], acc[k]);
                }
            };
            using std::integral_constant;
            int t0 = 0;
#pragma unroll 1
            for (; t0 + 4 < n; t0 += 8) add(integral_constant<int, 8>{}, t0);
#pragma unroll 1
            for (; t0 < n; t0 += 2) add(integral_constant<int, 2>{}, t0);
        }
    }
    const float inv = total > 0.f ? 1.f / total : 0.f;
    const int b = int(bh / p.H), h = int(bh - int64_t(b) * p.H);
    uint16_t* out = static_cast<uint16_t*>(p.o.ptr) + int64_t(b) * p.o.sb + int64_t(h) * p.o.sh + int64_t(i) * p.o.sl;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (lane + 32 * k < p.D) out[lane + 32 * k] = failed ? uint16_t(0xffff) : uint16_t(pack2<BF16>(acc[k] * inv, 0.f));
    if (lane == 0) lse[i] = (total > 0.f && !spoilt) ? mx + log2f(total) : -INFINITY;
}

cudaError_t launch_fwd_combine(bool bf16, const CombineParams& p, cudaStream_t stream) {
    const unsigned grid = unsigned((int64_t(p.B) * p.H * p.M + 7) / 8);
    return launch_overlapping(bf16 ? fwd_combine_kernel<true> : fwd_combine_kernel<false>, dim3(grid), 256, 0, stream, p);
}

// ---- host launcher (called from api.cu) -------------------------------------------------
template <int D, bool BF16, bool SHORT>
static cudaError_t launch_fwd_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                const CUtensorMap& to, const FwdParams& p, int num_sms, cudaStream_t stream) {
    auto kern = fwd_kernel<D, BF16, SHORT>;
    constexpr int smem = FwdSmem<D>::total;
    static SmemAllowed allowed;
    cudaError_t e = allow_smem(kern, smem, allowed);
    if (e != cudaSuccess) return e;
    const int heads = SHORT ? p.H / p.G * cdiv(p.G, p.pack) : p.H;
    const int n_items = p.mask.L.nQ * heads * p.B * (SHORT ? p.ns : 1);
    dim3 grid(n_items < num_sms ? n_items : num_sms);
    return launch_overlapping(kern, grid, kFwdThreads, smem, stream, tq, tk, tv, to, p);
}


cudaError_t launch_fwd(int D, bool bf16, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                       const CUtensorMap& to, const FwdParams& p, int num_sms, cudaStream_t stream) {
    auto pick = [&](auto d, auto shrt) {
        constexpr int kD = decltype(d)::value;
        constexpr bool kShort = decltype(shrt)::value;
        return bf16 ? launch_fwd_t<kD, true, kShort>(tq, tk, tv, to, p, num_sms, stream)
                    : launch_fwd_t<kD, false, kShort>(tq, tk, tv, to, p, num_sms, stream);
    };
    using std::integral_constant;
    const bool shrt = p.pack > 1 || p.ns > 1;
    if (D == 128) return shrt ? pick(integral_constant<int, 128>{}, std::true_type{}) : pick(integral_constant<int, 128>{}, std::false_type{});
    return shrt ? pick(integral_constant<int, 64>{}, std::true_type{}) : pick(integral_constant<int, 64>{}, std::false_type{});
}

}  // namespace fa
