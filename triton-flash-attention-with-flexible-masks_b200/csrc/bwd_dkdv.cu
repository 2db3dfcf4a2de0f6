// dK / dV kernel. Replaces `_bwd_kv_kernel` (flash_triton.py:175-321) and the grouped-query
// sum that follows it (:635-637): per block of 128 keys, walk the visited query tiles of every
// query head of the group, recompute P, and accumulate dV += P^T dO, dK += dS^T Q in fp32.
//
// The tile is kept transposed (rows = keys, columns = queries): S^T = K Q^T and dP^T = V dO^T
// land in TMEM with one key per lane. P^T (input dtype) takes the place of its scores and dS^T that of dP^T: both are TMEM A
// operands of dV += P^T dO and dK += dS^T Q; dO and Q are read as MN-major B operands from their TMA tiles. No tile of P or dS
// goes through shared memory, which leaves room for a third stage of Q.
//
// Persistent: min(items, SMs) CTAs, item = one key block of one (batch, kv head), taken round
// robin. 19 warps:
//   warps 0-15 compute: warp i owns keys [32 (i % 4), +32) and query columns [32 (i / 4), +32) of every tile. The scores are read in
//              the fragment order of 8 x 8 matrices (four keys and eight queries a thread): a thread then needs the LSE and delta of
//              eight queries only, a quarter of what a key per thread would ask of shared memory for them
//   warp 16    TMA producer (K, V per item; Q ring with the per-row LSE; dO ring) and the TMA stores of the finished item's dK / dV
//   warp 17    tcgen05.mma issuer; owns the TMEM allocation
//   warp 18    scheduler: per item, the range of candidate query blocks and their flags
// The Q / dO rings and all per-tile barriers run across item boundaries, so the next item's K and
// V and first Q / dO tiles are in flight and its first S^T is computed while the compute warps drain
// the accumulators of the finished item (dK and dV are staged in the Q and dO ring stages of the
// item's last tile, which are dead by then; those stages are refilled when the stores have read them).
//
// What bounds it: the chain "scores, exponentials, P, dV, S^T of the next tile" (2935 clocks a dense tile of D = 128 for 2048 of MMA: the
// exponentials' 1024 clocks of MUFU, then two products that the next scores wait for) and that of a compute warp's own steps. With eight warps
// of 64 columns each step of that chain took twice as long, and nothing else ran beside it (3350 clocks). us a launch, eight warps with a key per thread
// and P^T in shared memory | sixteen: 2 x 32 / 8 heads x 3001 x 128 causal 293 | 263; 4 x 16 x 4096 x 128 in documents 211 | 179; 32 x 32768 x 128
// in 64 documents 1351 | 1225; 8 x 8 x 1024 x 8192 x 64, queries of 8 documents, 172 | 135; 16 x 8 x 577 x 32 54 | 45; 4 x 12 x 1000 x 64
// in documents 35 | 30. In between: sixteen warps with P^T in shared memory 273 / 195 / 1267 / 138 / 45 / 31, a tile's shared memory traffic being 2980
// wavefronts then; two MMA warps, so that dK may come between dV and S^T, 305 / 201 / 1320 / 142 / 46 / 30.
// Since then shorter waits, products written once and a shorter walk. Both builds in turn, replayed graphs of one launch, some 30 after a pause (so above the
// power cap), other documents than above, us, that "sixteen" | now: 2 x 32 / 8 x 3001 261 | 264, 4 x 16 x 4096 x 128 in documents 186 | 185, 32 x 32768 x 128
// in 64 documents 588 | 572, 8 x 8 x 1024 x 8192 x 64 143 | 129, 16 x 8 x 577 x 32 47.4 | 45.4, 4 x 12 x 1000 x 64 in documents 33.1 | 32.7, 4 x 16 x 4096 x 64
// causal 309 | 309.
#include "common.cuh"
#include "params.cuh"

namespace fa {

template <int D>
struct DkdvSmem {
    static constexpr int NQ = 3, NDO = (D == 128) ? 2 : 3;  // stages of Q, of dO
    static constexpr int NSB = (D == 128) ? 1 : 2;  // S^T buffers
    // TMEM columns: S^T of tile g at s_col(g), dP^T [128,256), dV [256,256+D), dK [256+D,256+2D)
    static __device__ __forceinline__ uint32_t s_col(int g) { return NSB == 1 || (g & 1) == 0 ? 0u : 384u; }
    static constexpr int TILE = kBlk * D * 2;
    static constexpr int BOX = kBlk * 64 * 2;
    static constexpr int NBOX = D / 64;
    static constexpr int VEC = kBlk * 4;  // lse of one query block
    static constexpr int FLAGS = kListCap / 4;  // one item's candidate flags, 2 bits each
    static constexpr int off_k = 0;
    static constexpr int off_v = TILE;
    static constexpr int off_q = 2 * TILE;
    static constexpr int off_do = off_q + NQ * TILE;
    static constexpr int off_vec = off_do + NDO * TILE;
    static constexpr int off_flags = off_vec + NQ * VEC;  // two item slots
    static constexpr int off_info = off_flags + 2 * FLAGS;  // two item slots x {lo, n, tiles, item, key block, kv head, batch, -}
    static constexpr int off_bar = off_info + 64;
    // k_full, v_full, k_empty, v_empty, q_full[NQ], do_full[NDO], q_empty[NQ], do_empty[NDO], s_full[NSB], p_full[NSB], dp_full,
    // ds_full, dv_done, dk_done, acc_free, staged, stage_free, item_full[2], item_empty[2]
    static constexpr int n_bar = 4 + 2 * NQ + 2 * NDO + 2 * NSB + 7 + 4;
    static constexpr int off_misc = off_bar + n_bar * 8;
    static constexpr int total = off_misc + 16;
};
static_assert(DkdvSmem<128>::total <= 232448 && DkdvSmem<64>::total <= 232448, "shared memory budget");
static_assert(DkdvSmem<128>::total > 116736 && DkdvSmem<64>::total > 116736, "shares an SM with a dQ CTA");

// Per-candidate code kept in shared memory (2 bits): 0 not visited, 1 visited without id check,
// 2 id check, 3 id check with many codes in the query block. Whether a tile needs the range check (causal bound
// and / or query tail) follows from its coordinates alone.
enum : uint32_t { KC_SKIP = 0u, KC_PLAIN = 1u, KC_DOC = 2u, KC_DOCMANY = 3u };

// Flags of tile (qb, kb) for all query heads of one kv head at once. When the heads disagree
// (ids given per head) the id check is forced, entry by entry, which is always exact.
__device__ __forceinline__ uint32_t classify_group(const MaskArgs& mk, int b, int hk, int G, int qb, int kb) {
    if (mk.He == 1 || G == 1) return classify_from_plan(mk, b, mk.He == 1 ? 0 : hk * G, qb, kb);
    uint32_t f = 0;
    bool all = true;
    for (int g = 0; g < G; ++g) {
        const uint32_t fg = classify_from_plan(mk, b, hk * G + g, qb, kb);
        if (fg & TILE_VISIT) f |= fg; else all = false;
    }
    if (f && !all) f |= TILE_DOC;
    return f;
}

// Walks the visited candidates of an item for all heads of the group, head-major:
// (g, c) -> next visited candidate; c == n means "past the end".
struct Walk {
    const uint8_t* fl;
    int n;
    __device__ __forceinline__ uint32_t code(int c) const { return (uint32_t(fl[c >> 2]) >> (2 * (c & 3))) & 3u; }
    __device__ __forceinline__ int first_from(int c) const {
        while (c < n && code(c) == KC_SKIP) ++c;
        return c;
    }
    // The same with the candidate's code, for an item that has tiles: one look at it, and one loop. (All sixteen compute warps of dK/dV walk: with
    // this and dQ's form of it dK/dV of 8 x 8 x 1024 x 8192 x 64 120.7 -> 119.4 us and dQ 102.4 -> 101.1, of 2 x 32 / 8 x 3001 x 128 298 -> 295 and
    // 226.7 -> 225.8.)
    __device__ __forceinline__ void next(int& g, int& c, uint32_t& found) const {
        found = KC_SKIP;
#pragma unroll 1
        do {
            if (++c >= n) { g += 1; c = 0; }
            found = code(c);
        } while (found == KC_SKIP);
    }
    __device__ __forceinline__ void advance(int& g, int& c) const {
        c = first_from(c + 1);
        if (c >= n) { g += 1; c = first_from(0); }
    }
};

template <int D, bool BF16>
__global__ void __launch_bounds__(kDkdvThreads, 1)
bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdK, const __grid_constant__ CUtensorMap tmdV,
                const DkdvParams p) {
    using S = DkdvSmem<D>;
    constexpr int NQ = S::NQ, NDO = S::NDO;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    const int tid = threadIdx.x, warp = uniform(tid >> 5), lane = tid & 31;

    const MaskArgs& mk = p.mask;
    const int G = p.G;
    const int nK = mk.L.nK;
    const int n_items = nK * p.Hk * p.B;
    unsigned int* ctr = mk.ctr ? mk.ctr + CTR_DKDV : nullptr;
    // item -> (key block, kv head, batch). Heads are taken in groups of p.gh; inside a group the key
    // blocks go in order (with a causal mask: long ones first) and the heads of the group vary
    // fastest. The CTAs thus work on neighbouring key blocks of a few heads at a time: few enough
    // that their Q / dO streams stay in L2, enough that not all CTAs pull the same lines.
    auto decode = [&](int j, int& kb, int& hk, int& b, int gh, int nk, int heads, int batches) {
        const int per = gh * nk;
        const int grp = j / per, rem = j - grp * per;
        const int gsz = min(gh, heads * batches - grp * gh);
        const int pos = rem / gsz, bh = grp * gh + (rem - pos * gsz);
        hk = bh % heads;
        b = bh / heads;
        // few items per CTA: longest first (sorted in the plan), so that no long item is left for the end
        kb = p.by_length ? mk.plan[mk.L.off_ordk + (int64_t(b) * mk.He + (mk.He == 1 ? 0 : hk * G)) * nK + pos] : pos;
    };

    volatile int* misc = reinterpret_cast<volatile int*>(smem + S::off_misc);
    volatile int* info = reinterpret_cast<volatile int*>(smem + S::off_info);
    const uint32_t bar0 = sbase + S::off_bar;
    auto BAR = [&](int i) { return bar0 + 8u * uint32_t(i); };
    constexpr int NSB = S::NSB;
    constexpr int B_KFULL = 0, B_VFULL = 1, B_KEMPTY = 2, B_VEMPTY = 3, B_QFULL = 4, B_DOFULL = B_QFULL + NQ, B_QEMPTY = B_DOFULL + NDO,
                  B_DOEMPTY = B_QEMPTY + NQ, B_SFULL = B_DOEMPTY + NDO, B_PFULL = B_SFULL + NSB, B_DPFULL = B_PFULL + NSB, B_DSFULL = B_DPFULL + 1,
                  B_DVDONE = B_DPFULL + 2, B_DKDONE = B_DPFULL + 3, B_ACCFREE = B_DPFULL + 4, B_STAGED = B_DPFULL + 5,
                  B_STAGEFREE = B_DPFULL + 6, B_ITEMFULL = B_DPFULL + 7, B_ITEMEMPTY = B_ITEMFULL + 2;
    static_assert(B_ITEMEMPTY + 2 == S::n_bar, "barriers");
    Abort ab{misc + 1, p.status, p.wait_limit};

    const uint32_t sK = sbase + S::off_k, sV = sbase + S::off_v;
    auto sQ = [&](int s) { return sbase + S::off_q + uint32_t(s) * S::TILE; };
    auto sdO = [&](int s) { return sbase + S::off_do + uint32_t(s) * S::TILE; };
    auto sVec = [&](int s) { return sbase + S::off_vec + uint32_t(s) * S::VEC; };
    auto walk_of = [&](int s, int n) { return Walk{smem + S::off_flags + s * S::FLAGS, n}; };

    if (tid == 0) {
        mbar_init(BAR(B_KFULL), 1); mbar_init(BAR(B_VFULL), 1); mbar_init(BAR(B_KEMPTY), 1); mbar_init(BAR(B_VEMPTY), 1);
        for (int s = 0; s < NQ; ++s) { mbar_init(BAR(B_QFULL + s), 1); mbar_init(BAR(B_QEMPTY + s), 1); }
        for (int s = 0; s < NDO; ++s) { mbar_init(BAR(B_DOFULL + s), 1); mbar_init(BAR(B_DOEMPTY + s), 1); }
        for (int s = 0; s < NSB; ++s) {
            mbar_init(BAR(B_SFULL + s), 1);
            mbar_init(BAR(B_PFULL + s), 16);  // here and below: one arrival a compute warp
        }
        mbar_init(BAR(B_DPFULL), 1);
        mbar_init(BAR(B_DSFULL), 16);
        mbar_init(BAR(B_DVDONE), 1);
        mbar_init(BAR(B_DKDONE), 1);
        mbar_init(BAR(B_ACCFREE), 16);
        mbar_init(BAR(B_STAGED), 16);
        mbar_init(BAR(B_STAGEFREE), 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(BAR(B_ITEMFULL + s), 1);
            mbar_init(BAR(B_ITEMEMPTY + s), 18);  // producer, MMA issuer, sixteen compute warps
        }
        fence_mbar_init();
    }
    wait_prerequisites();
    if (warp == 17) {
        tmem_alloc(sbase + S::off_misc, 512);
        tmem_relinquish();
    }
    if (tid == 0) misc[1] = (status_is_fatal(*reinterpret_cast<volatile int*>(p.status)) || (sbase & 1023u) != 0) ? 1 : 0;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    launch_dependents();  // (fa_bwd's dQ kernel reads nothing that this one writes, but delta, which is complete since the wait)
    const uint32_t tmem = uint32_t(misc[0]);
    const bool aborted = misc[1] != 0;
    // An earlier launch on this device ran into a time-out that the host has not yet cleared: the CTA fills its items of the fixed order with NaN
    // (see nan_fill_items; with counters any other CTA may have taken them, and if none does they are everybody's). The numbers for it are hidden
    // from the compiler, which kept them in registers throughout, 96 for 84 and 28 bytes spilled: 4 x 16 x 4096 x 128 in documents 221 us for 186;
    // with this behind the roles instead 187, 4 x 16 x 4096 x 64 causal 315 for 310.
    if (aborted && (sbase & 1023u) == 0) {
        for (int i = tid; i < S::NBOX * S::BOX / 16; i += kDkdvThreads) reinterpret_cast<uint4*>(smem + S::off_k)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
        fence_proxy_async();
        __syncthreads();
        int gh = p.gh, nk = nK, heads = p.Hk, batches = p.B;
        asm volatile("" : "+r"(gh), "+r"(nk), "+r"(heads), "+r"(batches));
        if (tid == 0) {
            for (int k = 0, j; (j = item_in_order(k)) < n_items; ++k) {
                int kb, hk, b;
                decode(j, kb, hk, b, gh, nk, heads, batches);
                for (int x = 0; x < S::NBOX; ++x) {
                    tma_store_4d(&tmdK, sK + x * S::BOX, x * 64, kb * kBlk, hk, b);
                    tma_store_4d(&tmdV, sK + x * S::BOX, x * 64, kb * kBlk, hk, b);
                }
                tma_store_commit();
            }
            tma_store_wait_all();
        }
    }

    if (warp >= 16) {
        if (aborted) {
        } else if (warp == 18) {
            // ------------------------------ scheduler ------------------------------
            // Item k goes to slot k & 1: range [lo, lo + n) of candidate query blocks (union over the
            // group's heads), a 2-bit code per candidate, and the number of tiles.
            // Items are handed out in order from a counter in the plan (any CTA takes the next one: the
            // work per item varies with the mask); without counters (no plan given) they are
            // dealt out round robin in alternating direction, which evens out their sorted lengths.
            bool ok = true;
            for (int k = 0;; ++k) {
                const int s = k & 1, use = k >> 1;
                if (use > 0) ok = mbar_wait(BAR(B_ITEMEMPTY + s), (use - 1) & 1, ab, ST_WAIT_TIMEOUT + 54);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                int j = 0;
                if (lane == 0) {
                    if (ctr) j = int(atomicAdd(ctr, 1u));
                    else j = item_in_order(k);
                }
                j = __shfl_sync(0xffffffffu, j, 0);
                if (j >= n_items) {  // end marker
                    if (lane == 0) {
                        info[s * 8 + 3] = -1;
                        mbar_arrive(BAR(B_ITEMFULL + s));
                    }
                    break;
                }
                int kb, hk, b;
                decode(j, kb, hk, b, p.gh, nK, p.Hk, p.B);
                int lo = 0x7fffffff, hi = 0;
                {
                    const int ng = (mk.He == 1) ? 1 : G;
                    for (int g = 0; g < ng; ++g) {
                        int l, h2;
                        q_range(mk, b, mk.He == 1 ? 0 : hk * G + g, kb, l, h2);
                        if (h2 > l) { lo = min(lo, l); hi = max(hi, h2); }
                    }
                    if (hi == 0) lo = 0;
                }
                int n = hi - lo;
                if (n > kListCap) n = kListCap;
                uint8_t* fl = smem + S::off_flags + s * S::FLAGS;
                int cnt = 0;
                for (int i = lane; 4 * i < n; i += 32) {
                    uint32_t byte = 0;
                    for (int e = 0; e < 4; ++e) {
                        const int c = 4 * i + e;
                        if (c >= n) break;
                        const uint32_t f = classify_group(mk, b, hk, G, lo + c, kb);
                        uint32_t code = KC_SKIP;
                        if (f & TILE_VISIT) code = !(f & TILE_DOC) ? KC_PLAIN : (f & TILE_QMANY) ? KC_DOCMANY : KC_DOC;
                        cnt += (code != KC_SKIP);
                        byte |= code << (2 * e);
                    }
                    fl[i] = uint8_t(byte);
                }
                for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
                __syncwarp();
                if (lane == 0) {
                    info[s * 8 + 0] = lo;
                    info[s * 8 + 1] = n;
                    info[s * 8 + 2] = cnt * G;  // tiles of all query heads of the group, head-major
                    info[s * 8 + 3] = j;
                    info[s * 8 + 4] = kb;
                    info[s * 8 + 5] = hk;
                    info[s * 8 + 6] = b;
                    mbar_arrive(BAR(B_ITEMFULL + s));
                }
            }
        } else if (warp == 16) {
            // ------------------------------ TMA producer ------------------------------
            // (converged, with uniform values: from a branch of one lane a load takes up to 950 clocks to issue)
            tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmdO); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
            tma_prefetch_desc(&tmdK); tma_prefetch_desc(&tmdV);
            bool ok = true;
            int k = 0, kk = 0;  // items, items with tiles
            int gt = 0;         // tiles of all earlier items (stage / phase of the Q and dO rings)
            int pkb = 0, phk = 0, pb = 0;  // the previous item, whose dK / dV are still to be stored
            // stores the dV / dK of item i, staged in the dO / Q ring stages of tile `last`, and frees the stages
            auto finish_store = [&](int i, int kb, int hk, int b, int last) {
                if (!mbar_wait_warp(BAR(B_STAGED), i & 1, ab, ST_WAIT_TIMEOUT + 55)) return false;
                if (lane == 0) {
                    if (misc[1] == 0) {
                        for (int x = 0; x < S::NBOX; ++x) {
                            tma_store_4d(&tmdV, sdO(last % NDO) + x * S::BOX, x * 64, kb * kBlk, hk, b);
                            tma_store_4d(&tmdK, sQ(last % NQ) + x * S::BOX, x * 64, kb * kBlk, hk, b);
                        }
                        tma_store_commit();
                        tma_store_wait_read();
                    }
                    mbar_arrive(BAR(B_STAGEFREE));
                }
                __syncwarp();
                return true;
            };
            for (;; ++k) {
                const int s = k & 1;
                ok = mbar_wait_warp(BAR(B_ITEMFULL + s), (k >> 1) & 1, ab, ST_WAIT_TIMEOUT + 56);
                if (!ok) break;
                const int lo = uniform(info[s * 8 + 0]), n = uniform(info[s * 8 + 1]), NIT = uniform(info[s * 8 + 2]);
                if (uniform(info[s * 8 + 3]) < 0) break;
                const int kb = uniform(info[s * 8 + 4]), hk = uniform(info[s * 8 + 5]), b = uniform(info[s * 8 + 6]);
                const Walk wk = walk_of(s, n);
                int cg = 0, cc = uniform(wk.first_from(0));
                int qg = 0, qi = cc;  // the walk of Q, which runs a stage ahead of dO where its ring is longer
                auto load_q = [&](int it) {
                    const int h = hk * G + qg, qb = lo + qi;
                    const int gi = gt + it, st = gi % NQ, use = gi / NQ;
                    if (use > 0 && !mbar_wait_warp(BAR(B_QEMPTY + st), (use - 1) & 1, ab, ST_WAIT_TIMEOUT + 41)) return false;
                    mbar_expect_tx_elect(BAR(B_QFULL + st), S::TILE + S::VEC);
                    for (int x = 0; x < S::NBOX; ++x)
                        tma_load_4d_elect(sQ(st) + x * S::BOX, &tmQ, BAR(B_QFULL + st), x * 64, qb * kBlk, h, b);
                    bulk_load_1d_elect(sVec(st), p.lse + (int64_t(b) * p.H + h) * mk.L.Mpad + int64_t(qb) * kBlk, kBlk * 4, BAR(B_QFULL + st));
                    wk.advance(qg, qi);
                    qg = uniform(qg);
                    qi = uniform(qi);
                    return true;
                };
                auto load_do = [&](int it) {
                    const int gi = gt + it, st = gi % NDO, use = gi / NDO;
                    if (use > 0 && !mbar_wait_warp(BAR(B_DOEMPTY + st), (use - 1) & 1, ab, ST_WAIT_TIMEOUT + 42)) return false;
                    mbar_expect_tx_elect(BAR(B_DOFULL + st), S::TILE);
                    for (int x = 0; x < S::NBOX; ++x)
                        tma_load_4d_elect(sdO(st) + x * S::BOX, &tmdO, BAR(B_DOFULL + st), x * 64, (lo + cc) * kBlk, hk * G + cg, b);
                    wk.advance(cg, cc);
                    cg = uniform(cg);
                    cc = uniform(cc);
                    return true;
                };
                // The previous item is staged in the ring stages of its last tile, the next to be loaded behind NQ - 1 tiles of Q
                // and NDO - 1 of dO. K, V and those do not wait for its epilogue.
                const int nq = NIT < NQ - 1 ? NIT : NQ - 1, ndo = NIT < NDO - 1 ? NIT : NDO - 1;
                if (NIT > 0) {
                    if (kk > 0) ok = mbar_wait_warp(BAR(B_KEMPTY), (kk - 1) & 1, ab, ST_WAIT_TIMEOUT + 57);
                    if (!ok) break;
                    mbar_expect_tx_elect(BAR(B_KFULL), S::TILE);
                    for (int x = 0; x < S::NBOX; ++x) tma_load_4d_elect(sK + x * S::BOX, &tmK, BAR(B_KFULL), x * 64, kb * kBlk, hk, b);
                    if (kk > 0) ok = mbar_wait_warp(BAR(B_VEMPTY), (kk - 1) & 1, ab, ST_WAIT_TIMEOUT + 60);
                    if (!ok) break;
                    mbar_expect_tx_elect(BAR(B_VFULL), S::TILE);
                    for (int x = 0; x < S::NBOX; ++x) tma_load_4d_elect(sV + x * S::BOX, &tmV, BAR(B_VFULL), x * 64, kb * kBlk, hk, b);
                    for (int it = 0; it < nq && ok; ++it) {
                        ok = load_q(it);
                        if (ok && it < ndo) ok = load_do(it);
                    }
                    if (!ok) break;
                }
                if (k > 0) ok = finish_store(k - 1, pkb, phk, pb, gt + NQ * NDO - 1);
                if (!ok) break;
                if (NIT > 0) {
                    for (int it = ndo; it < NIT && ok; ++it) {
                        const int q = it + NQ - NDO;
                        if (q < NIT) ok = load_q(q);
                        if (ok) ok = load_do(it);
                    }
                    if (!ok) break;
                    ++kk;
                }
                gt += NIT;
                pkb = kb; phk = hk; pb = b;
                if (lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + s));
                __syncwarp();
            }
            if (ok && k > 0) finish_store(k - 1, pkb, phk, pb, gt + NQ * NDO - 1);
        } else if (warp == 17) {
            // ------------------------------ MMA issuer (warp 17) ------------------------------
            // One warp and one order, the pipe's: S^T of a later tile directly behind dV, whose P^T it overwrites, and dP^T of the next
            // one behind dK, whose dS^T it overwrites.
            {
                const uint32_t utmem = uniform(int(tmem));
                constexpr uint32_t idesc_s = make_idesc(BF16, 128, 128, false, false);
                constexpr uint32_t idesc_d = make_idesc(BF16, 128, D, false, true);
                constexpr uint64_t desc_mn = desc_mn_major(S::BOX);
                auto q_ready = [&](int gi) { return mbar_wait_warp(BAR(B_QFULL + gi % NQ), (gi / NQ) & 1, ab, ST_WAIT_TIMEOUT + 44); };
                auto do_ready = [&](int gi) { return mbar_wait_warp(BAR(B_DOFULL + gi % NDO), (gi / NDO) & 1, ab, ST_WAIT_TIMEOUT + 45); };
                auto ss_mmas = [&](uint32_t d, uint32_t a_tile, uint32_t b_tile) {
#pragma unroll
                    for (int kk2 = 0; kk2 < D / 16; ++kk2) {
                        if (D == 64 && kk2 >= p.ksteps) break;
                        const uint32_t off = uint32_t(kk2 >> 2) * S::BOX + uint32_t(kk2 & 3) * 32u;
                        umma_ss(d, smem_desc_at(kDescKMajor, a_tile + off), smem_desc_at(kDescKMajor, b_tile + off),
                                idesc_s, kk2 > 0);
                    }
                };
                bool ok = true;
                int k = 0, kk = 0, gt = 0;
                for (;; ++k) {
                    const int s = k & 1;
                    ok = mbar_wait_warp(BAR(B_ITEMFULL + s), (k >> 1) & 1, ab, ST_WAIT_TIMEOUT + 56);
                    if (!ok) break;
                    const int NIT = uniform(info[s * 8 + 2]);
                    if (uniform(info[s * 8 + 3]) < 0) break;
                    if (NIT > 0) {
                        // Steps before tile 0 issue what the first tiles' dV and dK stand behind: each product is written once, for the sake of
                        // the instruction caches.
                        ok = mbar_wait_warp(BAR(B_KFULL), kk & 1, ab, ST_WAIT_TIMEOUT + 43);
                        for (int it = -NSB; it < NIT && ok; ++it) {
                            const int gi = gt + it;
                            if (it >= 0) {
                                // dV(0) and dK(0) overwrite the accumulators: the previous item's epilogue must have read them
                                if (it == 0 && kk > 0) ok = mbar_wait_warp(BAR(B_ACCFREE), (kk - 1) & 1, ab, ST_WAIT_TIMEOUT + 58);
                                // dV += P^T dO: A = P^T from TMEM (a warp's P lies over its own S), B = dO (MN-major)
                                if (ok) ok = mbar_wait_warp(BAR(B_PFULL + gi % NSB), (gi / NSB) & 1, ab, ST_WAIT_TIMEOUT + 47);
                                if (!ok) break;
                                tc_fence_after();
#pragma unroll
                                for (int kk2 = 0; kk2 < kBlk / 16; ++kk2) {
                                    const uint32_t acol = uint32_t(kk2 >> 1) * 32u + uint32_t(kk2 & 1) * 8u;
                                    umma_ts(utmem + 256u, utmem + S::s_col(gi) + acol, smem_desc_at(desc_mn, sdO(gi % NDO) + uint32_t(kk2) * 2048u),
                                            idesc_d, (it > 0 || kk2 > 0) ? 1u : 0u);
                                }
                                umma_commit(BAR(B_DOEMPTY + gi % NDO));
                                if (it + 1 == NIT) umma_commit(BAR(B_DVDONE));
                            }
                            if (it + NSB < NIT) {  // S^T(it + NSB)
                                const int gs = gi + NSB;
                                ok = q_ready(gs);
                                if (!ok) break;
                                tc_fence_after();
                                ss_mmas(utmem + S::s_col(gs), sK, sQ(gs % NQ));
                                umma_commit(BAR(B_SFULL + gs % NSB));
                                if (it + NSB + 1 == NIT) umma_commit(BAR(B_KEMPTY));
                            }
                            if (it >= 0) {
                                // dK += dS^T Q: A = dS^T from TMEM (a warp's dS lies over its own dP), B = Q (MN-major)
                                ok = mbar_wait_warp(BAR(B_DSFULL), gi & 1, ab, ST_WAIT_TIMEOUT + 48);
                                if (!ok) break;
                                tc_fence_after();
#pragma unroll
                                for (int kk2 = 0; kk2 < kBlk / 16; ++kk2) {
                                    const uint32_t acol = uint32_t(kk2 >> 1) * 32u + uint32_t(kk2 & 1) * 8u;
                                    umma_ts(utmem + 256u + uint32_t(D), utmem + 128u + acol, smem_desc_at(desc_mn, sQ(gi % NQ) + uint32_t(kk2) * 2048u),
                                            idesc_d, (it > 0 || kk2 > 0) ? 1u : 0u);
                                }
                                umma_commit(BAR(B_QEMPTY + gi % NQ));
                            }
                            if (it >= -1 && it + 1 < NIT) {  // dP^T(it + 1)
                                if (it < 0) ok = mbar_wait_warp(BAR(B_VFULL), kk & 1, ab, ST_WAIT_TIMEOUT + 43);
                                if (ok) ok = do_ready(gi + 1);
                                if (!ok) break;
                                tc_fence_after();
                                ss_mmas(utmem + 128u, sV, sdO((gi + 1) % NDO));
                                umma_commit(BAR(B_DPFULL));
                                if (it + 2 == NIT) umma_commit(BAR(B_VEMPTY));
                            }
                        }
                        if (!ok) break;
                        umma_commit(BAR(B_DKDONE));
                    }
                    if (NIT > 0) ++kk;
                    gt += NIT;
                    if (lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + s));
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------ compute groups ------------------------------
        const int w = warp >> 2;
        const int r = tid & 127;
        const uint32_t lane_base = uint32_t((warp & 3) * 32) << 16;
        const int cbase = 32 * w;  // first query column of this warp inside a tile
        const float c = p.scale_log2;
        bool ok = !aborted;
        const uint32_t tdP = tmem + lane_base + 128u + uint32_t(cbase);
        constexpr uint32_t kHalfLanes = 16u << 16;  // the upper 16 lanes of a warp's 32
        int k = 0, kk = 0, gt = 0;
        for (; ok; ++k) {
            const int s = k & 1;
            ok = mbar_wait(BAR(B_ITEMFULL + s), (k >> 1) & 1, ab, ST_WAIT_TIMEOUT + 56);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const int lo = info[s * 8 + 0], n = info[s * 8 + 1], NIT = info[s * 8 + 2], jt = info[s * 8 + 3];
            if (jt < 0) break;
            const int kb = info[s * 8 + 4], hk = info[s * 8 + 5], b = info[s * 8 + 6];
            const Walk wk = walk_of(s, n);
            const int j = kb * kBlk + r;  // this thread's key
            const int k0 = kb * kBlk, k1 = min(k0 + kBlk, mk.N);

            int cg = 0, cc = -1;
            uint32_t code = KC_SKIP;
            int kc = 0, kc_g = -1;  // this key's code for the current query head
            const float* const delta0 = p.delta + (int64_t(b) * p.H + hk * G) * mk.L.Mpad + cbase + 2 * (lane & 3);
            for (int it = 0; it < NIT && ok; ++it) {
                wk.next(cg, cc, code);
                const bool fl_doc = code >= KC_DOC, many = code == KC_DOCMANY;
                const int qb0 = (lo + cc) * kBlk;
                const bool fl_range = (mk.causal && (k0 + kBlk > mk.N || k1 - 1 > qb0 + mk.gap)) || (qb0 + kBlk > mk.M);
                const int q0 = qb0 + cbase;  // first query row of this warp's columns
                const int gi = gt + it;
                // the rows' LSE came with Q, which S^T has been computed from; their delta is asked for here
                const float* vlse = reinterpret_cast<const float*>(smem + S::off_vec + gi % NQ * S::VEC) + cbase + 2 * (lane & 3);
                const float2* vdelta = reinterpret_cast<const float2*>(delta0 + cg * mk.L.Mpad + qb0);
                float2 delta[4];
#pragma unroll
                for (int n = 0; n < 4; ++n) delta[n] = vdelta[4 * n];

                // keep(x) = (cmin <= x < cmax) & (qc[x] >= 0 | qc[x] == kc) as a 32-bit mask, worked out before the
                // scores are there
                const bool flagged = fl_range || fl_doc;
                uint32_t keep = ~0u;
                if (flagged) {
                    if (fl_doc) {
                        const int64_t bh_ids = int64_t(b) * mk.He + ((mk.He == 1) ? 0 : hk * G + cg);
                        if (kc_g != cg) { kc = mk.plan[mk.L.off_kc + bh_ids * mk.L.Npad + j]; kc_g = cg; }
                        const int* qcs = mk.plan + mk.L.off_qc + bh_ids * mk.L.Mpad + q0;
                        const int qc = qcs[lane];
                        keep = codes_equal(qcs, qc, kc, many) | __ballot_sync(0xffffffffu, qc >= 0);
                    }
                    if (fl_range) {
                        const int cmin = mk.causal ? (j - mk.gap) - q0 : 0, cmax = mk.M - q0;
                        keep &= first_bits(cmax) & ~first_bits(cmin);
                    }
                }

                const uint32_t tS = tmem + lane_base + S::s_col(gi) + uint32_t(cbase);
                ok = mbar_wait_warp(BAR(B_SFULL + gi % NSB), (gi / NSB) & 1, ab, ST_WAIT_TIMEOUT + 50);
                if (!ok) break;
                tc_fence_after();
                uint32_t sr[32];
                tmem_ld_frag32(tS, sr);
                tmem_ld_frag32(tS + kHalfLanes, sr + 16);
                tc_wait_ld();
                float* pr = reinterpret_cast<float*>(sr);  // [2 halves of 16 keys][4 chunks of 8 queries][2 keys][2 queries]
                // P^T = exp2(S^T*c - LSE) on packed pairs, 0 where masked. A fully masked row has LSE = -inf and only
                // occurs in flagged tiles.
                if (flagged && !__any_sync(0xffffffffu, keep != 0u)) {
#pragma unroll
                    for (int x = 0; x < 32; ++x) pr[x] = 0.f;
                } else {
                    const uint64_t c2 = pack_f2(c, c);
#pragma unroll
                    for (int n = 0; n < 4; ++n) {
                        const float2 l2 = *reinterpret_cast<const float2*>(vlse + 8 * n);
                        const uint64_t nl2 = pack_f2(-l2.x, -l2.y);
#pragma unroll
                        for (int y = 0; y < 4; ++y) {
                            float* x = pr + 16 * (y >> 1) + 4 * n + 2 * (y & 1);
                            float x0, x1;
                            unpack_f2(fma_f2(pack_f2(x[0], x[1]), c2, nl2), x0, x1);
                            x[0] = fast_exp2(x0);
                            x[1] = fast_exp2(x1);
                        }
                    }
                    if (flagged && __any_sync(0xffffffffu, keep != ~0u)) {
#pragma unroll
                        for (int y = 0; y < 4; ++y) {
                            // keep holds this lane's key: the word of the key whose scores these are comes from its lane
                            const uint32_t bits = __shfl_sync(0xffffffffu, keep, 8 * y + (lane >> 2)) >> (2 * (lane & 3));
#pragma unroll
                            for (int n = 0; n < 4; ++n) {
                                float* x = pr + 16 * (y >> 1) + 4 * n + 2 * (y & 1);
                                x[0] = (bits & (1u << (8 * n))) ? x[0] : 0.f;
                                x[1] = (bits & (2u << (8 * n))) ? x[1] : 0.f;
                            }
                        }
                    }
                }
                // P^T (input dtype) takes the place of its scores
                uint32_t pk[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) pk[x] = pack2<BF16>(pr[2 * x], pr[2 * x + 1]);
                tmem_st_frag16(tS, pk);
                tmem_st_frag16(tS + kHalfLanes, pk + 8);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive_warp(BAR(B_PFULL + gi % NSB), lane);

                ok = mbar_wait_warp(BAR(B_DPFULL), gi & 1, ab, ST_WAIT_TIMEOUT + 52);
                if (!ok) break;
                tc_fence_after();
                uint32_t dp[32];
                tmem_ld_frag32(tdP, dp);
                tmem_ld_frag32(tdP + kHalfLanes, dp + 16);
                tc_wait_ld();
                // masked entries have P == 0 exactly and dP - delta is finite, so dS is 0 there
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const uint64_t nd2 = pack_f2(-delta[n].x, -delta[n].y);
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const int x = 16 * (y >> 1) + 4 * n + 2 * (y & 1);
                        float d0, d1;
                        unpack_f2(mul_f2(pack_f2(pr[x], pr[x + 1]),
                                         add_f2(pack_f2(__uint_as_float(dp[x]), __uint_as_float(dp[x + 1])), nd2)), d0, d1);
                        pk[8 * (y >> 1) + 2 * n + (y & 1)] = pack2<BF16>(d0, d1);
                    }
                }
                // dS^T (input dtype) takes the place of dP^T
                tmem_st_frag16(tdP, pk);
                tmem_st_frag16(tdP + kHalfLanes, pk + 8);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive_warp(BAR(B_DSFULL), lane);
            }
            if (!ok) break;

            // ------------------------------ item epilogue ------------------------------
            // the previous item's stores have read their staging stage (it may be the same one)
            if (k > 0) ok = mbar_wait(BAR(B_STAGEFREE), (k - 1) & 1, ab, ST_WAIT_TIMEOUT + 59);
            // dV is final (and the last dO tile dead) when the last dV MMAs are complete: it is drained
            // while the last dK MMAs still run
            if (ok && NIT > 0) ok = mbar_wait(BAR(B_DVDONE), kk & 1, ab, ST_WAIT_TIMEOUT + 51);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            {
                // dV and dK * sm_scale (flash_triton.py:313) go out through shared memory: each thread writes its quarter of a
                // row of dV into the dO ring stage of the item's last tile, and of dK into the Q ring stage (dead: the last dV,
                // and then the last dK, MMAs are complete) in the tensor maps' 128-byte-swizzled layout; the producer warp issues
                // the TMA stores, which clip rows >= N.
                const int last = gt + NIT + NQ * NDO - 1;  // (of an earlier item, if this one has no tiles)
                constexpr int COLS = D / 4;  // of a warp
                const uint32_t c0 = uint32_t(w) * COLS;
#pragma unroll
                for (int which = 0; which < 2; ++which) {  // 0: dV, 1: dK
                    if (which == 1 && NIT > 0) {
                        ok = mbar_wait(BAR(B_DKDONE), kk & 1, ab, ST_WAIT_TIMEOUT + 53);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const float mul = which ? p.sm_scale : 1.0f;
                    uint8_t* stage = smem + (which ? S::off_q + last % NQ * S::TILE : S::off_do + last % NDO * S::TILE);
                    // (rolled, D = 128: 2 x 32 / 8 x 3001 x 128 301 -> 296 us, 32 x 32768 x 128 in 64 documents 1414 -> 1398)
#pragma unroll 1
                    for (int q = 0; q < COLS / 16; ++q) {
                        uint32_t x[16];
                        // tcgen05.ld is warp-collective: always executed, the values are ignored for an item without tiles
                        tmem_ld16(tmem + lane_base + 256u + uint32_t(which * D) + c0 + uint32_t(q) * 16u, x);
                        tc_wait_ld();
                        uint32_t o16[8];
#pragma unroll
                        for (int y = 0; y < 8; ++y) {
                            const float v0 = (NIT > 0) ? __uint_as_float(x[2 * y]) * mul : 0.f;
                            const float v1 = (NIT > 0) ? __uint_as_float(x[2 * y + 1]) * mul : 0.f;
                            o16[y] = pack2<BF16>(v0, v1);
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int cgk = int(c0) / 8 + 2 * q + i;  // 16-byte chunk of the row
                            const int box = cgk >> 3, ch = cgk & 7;
                            uint4* dst = reinterpret_cast<uint4*>(stage + box * S::BOX + r * 128 + ((ch ^ (r & 7)) << 4));
                            *dst = make_uint4(o16[4 * i], o16[4 * i + 1], o16[4 * i + 2], o16[4 * i + 3]);
                        }
                    }
                }
            }
            if (!ok) break;
            // both accumulators have been read: warp 17 may start the next item's dV / dK
            tc_fence_before();
            if (NIT > 0) {
                mbar_arrive_warp(BAR(B_ACCFREE), lane);
                ++kk;
            }
            fence_proxy_async();
            mbar_arrive_warp(BAR(B_STAGED), lane);  // the producer warp issues the TMA stores
            gt += NIT;
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(B_ITEMEMPTY + s));
        }
    }

    // ------------------------------ tear-down ------------------------------
    tc_fence_before();
    __syncthreads();
    if (warp == 17) {
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

template <int D, bool BF16>
static cudaError_t launch_dkdv_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                 const CUtensorMap& tdo, const CUtensorMap& tdk, const CUtensorMap& tdv,
                                 const DkdvParams& p, int num_sms, cudaStream_t stream) {
    auto kern = bwd_dkdv_kernel<D, BF16>;
    constexpr int smem = DkdvSmem<D>::total;
    static SmemAllowed allowed;
    cudaError_t e = allow_smem(kern, smem, allowed);
    if (e != cudaSuccess) return e;
    const int n_items = p.mask.L.nK * p.Hk * p.B;
    const int grid = n_items < num_sms ? n_items : num_sms;
    return launch_overlapping(kern, dim3(grid), kDkdvThreads, smem, stream, tq, tk, tv, tdo, tdk, tdv, p);
}


cudaError_t launch_bwd_dkdv(int D, bool bf16, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                            const CUtensorMap& tdo, const CUtensorMap& tdk, const CUtensorMap& tdv,
                            const DkdvParams& p, int num_sms, cudaStream_t stream) {
    if (D == 128) return bf16 ? launch_dkdv_t<128, true>(tq, tk, tv, tdo, tdk, tdv, p, num_sms, stream)
                              : launch_dkdv_t<128, false>(tq, tk, tv, tdo, tdk, tdv, p, num_sms, stream);
    return bf16 ? launch_dkdv_t<64, true>(tq, tk, tv, tdo, tdk, tdv, p, num_sms, stream)
                : launch_dkdv_t<64, false>(tq, tk, tv, tdo, tdk, tdv, p, num_sms, stream);
}

}  // namespace fa
