// The products of sd_gemm.cu for launches with many tiles, by CTA pairs (tcgen05.mma.cta_group::2).
//
// An SM takes operands in at ~75 bytes per clock, whichever way they come.  The single-CTA kernel's 128x256 tile needs 48 KB
// for every 512 cycles of tensor-core work and therefore runs its main loop at 655 cycles per 64-wide K stage.  A pair of
// CTAs shares operands: each SM holds its own half of the one operand and half of the other.  A 256x256 tile would share
// both, but with masked 128x128 blocks two row blocks keep different K tiles.  So the pair's tile is ONE row block of the
// masked operand against 512 rows of the dense one, with the operands exchanged: the dense operand is the MMA's A (M = 256, a
// 128-row slab per CTA), the masked row block its B (N = 128, 64 rows per CTA), and two such MMAs share that B.  A CTA then
// takes in 40 KB for the same 512 cycles: 2 slabs of 16 KB and 8 KB of the row block.
//
// The accumulator holds the result transposed (TMEM lane = row of the dense operand, column = row of the masked one), which
// the epilogue turns round on its way through shared memory where the result wants it.
//
// One product is a list of entries, each a row block and one or two "duos" (a duo: two slabs, one M256 MMA):
//   dense / DSD : two consecutive duos; the last one alone when the dense operand has an odd number of them
//   SDD         : up to four kept tiles of a row block; one duo when one or two are left over
// Full entries are dealt first, heaviest row block first, then the single duos.  A last wave that would occupy at most half of
// the pairs is dealt as single duos (24 KB per 256 cycles of tensor work: 0.6 of a full entry).
#pragma once

namespace sd {

constexpr int P_STAGES = 5;
constexpr int P_EPI_WARPS = 4;                                // one per TMEM lane quadrant, each with one staging buffer
constexpr int P_THREADS = 96 + 32 * P_EPI_WARPS;
constexpr int P_W_BYTES = 128 * BK * 2;                       // one slab of the dense operand, 16 KiB
constexpr int P_S_BYTES = 64 * BK * 2;                        // this CTA's half of the row block, 8 KiB
constexpr int P_STAGE_BYTES = 2 * P_W_BYTES + P_S_BYTES;      // 40 KiB
constexpr int P_TILE_SMEM = P_STAGES * P_STAGE_BYTES;
constexpr int P_STAGING_BYTES = P_EPI_WARPS * 4096;
constexpr int P_TAB_MAX = 160;                                // entries of one pair
constexpr int P_MAX_ROW_BLOCKS = 1024;                        // SDD: row blocks whose entry counts fit shared memory
constexpr int P_TAB_BYTES = P_TAB_MAX * 32;
constexpr int P_PREFIX_BYTES = (P_MAX_ROW_BLOCKS + 4) * 4;
constexpr int P_SMEM = P_TILE_SMEM + P_STAGING_BYTES + P_TAB_BYTES + P_PREFIX_BYTES + 1024 /*align*/ + 256 /*barriers*/;
static_assert(P_SMEM <= 227 * 1024, "over the shared memory of one CTA");

struct __align__(16) PairEntry {
    int sp_row;          // first row of the masked operand; < 0: no entry
    int list_beg;        // its kept K tiles: list_idx[list_beg .. list_beg + nk)
    int nk;
    int shape;           // duos | stages << 2
    int slab[4];         // first rows of the dense operand's slabs, duo by duo; < 0: absent
};
static_assert(sizeof(PairEntry) == 32, "P_TAB_BYTES");

// How the entries of a launch are dealt to its pairs (see the file header).
struct PairDeal {
    int full, single;    // entries with two duos and with one
    int whole, halves;   // full entries dealt as they are; those after them, if any, are dealt as two single duos each
    int entries, passes;
    __host__ __device__ void init(int full_, int single_, int pairs) {
        full = full_;
        single = single_;
        const int rest = full % pairs;
        const bool cut = 2 * rest + single <= pairs;
        whole = cut ? full - rest : full;
        halves = 2 * (full - whole);
        entries = whole + halves + single;
        passes = (entries + pairs - 1) / pairs;
    }
    // full entry and duo of it (0, 1, or -1: both), or full + index of a single entry
    __host__ __device__ int pick(int entry, int* duo) const {
        *duo = -1;
        if (entry < whole) return entry;
        entry -= whole;
        if (entry < halves) { *duo = entry & 1; return whole + (entry >> 1); }
        return full + entry - halves;
    }
};

// SDD: a row block with n kept tiles has (n + 1) / 4 full entries (the last of three tiles at n % 4 == 3) and a single one for
// one or two tiles left over.
__host__ __device__ __forceinline__ int sdd_full(int n) { return (n + 1) >> 2; }
__host__ __device__ __forceinline__ int sdd_single(int n) { return ((n & 3) == 1 || (n & 3) == 2) ? 1 : 0; }

// Entry `entry` of a launch.  prefix (SDD): full entries | single entries << 16 of the row blocks before each one.
__device__ __forceinline__ PairEntry pair_entry(const GemmArgs& g, const PairDeal& d, int entry, const int* prefix, bool ordered) {
    PairEntry e;
    int duo;
    const int i = d.pick(entry, &duo);
    const bool single = i >= d.full;
    int rb, nk = (g.KK + 127) >> 7, beg = 0;
    const int n_duos = (single || duo >= 0) ? 1 : 2;
    bool last_kept = true;
    if (g.mode == MODE_SDD) {
        const int want = single ? i - d.full : i, shift = single ? 16 : 0;
        int lo = 0, hi = g.n_row_blocks - 1;                  // last row block with at most `want` entries before it
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (((prefix[mid] >> shift) & 0xffff) <= want) lo = mid; else hi = mid - 1;
        }
        rb = lo;
        const int b = __ldg(g.list_ptr + rb), n = __ldg(g.list_ptr + rb + 1) - b;
        const int first = 4 * (single ? sdd_full(n) : want - ((prefix[rb] >> shift) & 0xffff)) + (duo > 0 ? 2 : 0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            e.slab[j] = (j < 2 * n_duos && first + j < n) ? __ldg(g.list_idx + b + first + j) * 128 : -1;
    } else {
        const int duos = (g.NN + 255) >> 8, fpr = duos >> 1;
        int rbi, d0;
        if (single) { rbi = i - d.full; d0 = duos - 1; }
        else { rbi = i / fpr; d0 = 2 * (i - rbi * fpr) + (duo > 0 ? 1 : 0); }
        rb = ordered && g.order ? __ldg(g.order + rbi) : rbi;
#pragma unroll
        for (int j = 0; j < 4; ++j) e.slab[j] = (j < 2 * n_duos && d0 * 256 + j * 128 < g.NN) ? d0 * 256 + j * 128 : -1;
        if (g.mode == MODE_DSD) {
            beg = __ldg(g.list_ptr + rb);
            const int end = __ldg(g.list_ptr + rb + 1);
            if (((g.KK - 1) & 127) < BK && end > beg) last_kept = __ldg(g.list_idx + end - 1) == nk - 1;
            nk = end - beg;
        }
    }
    const int stages = 2 * nk - ((((g.KK - 1) & 127) < BK && last_kept && nk) ? 1 : 0);
    e.sp_row = stages ? rb * 128 : -1;                        // empty row blocks are zero-filled by the epilogue warps
    e.list_beg = beg;
    e.nk = nk;
    e.shape = n_duos | (stages << 2);
    return e;
}

template <bool W_MN, bool S_MN>
__global__ void __launch_bounds__(P_THREADS, 1)
sparsedrop_pair_kernel(const __grid_constant__ CUtensorMap tmapW, const __grid_constant__ CUtensorMap tmapS,
                       const __grid_constant__ CUtensorMap tmapC, const GemmArgs g) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t tiles = (raw_addr + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (tiles - raw_addr);
    uint8_t* staging = aligned + P_TILE_SMEM;
    PairEntry* tab = reinterpret_cast<PairEntry*>(staging + P_STAGING_BYTES);
    int* prefix = reinterpret_cast<int*>(staging + P_STAGING_BYTES + P_TAB_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(staging + P_STAGING_BYTES + P_TAB_BYTES + P_PREFIX_BYTES);
    // full, empty: one per ring slot; tmem_full, tmem_empty: one per accumulator.  `full` and `tmem_empty` are used in the
    // leading CTA only, `empty` and `tmem_full` in both.
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * P_STAGES;
    const uint32_t bar_tfull = bar_empty + 8 * P_STAGES, bar_tempty = bar_tfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * P_STAGES + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * P_STAGES + 5);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int n_warps = P_THREADS / 32;
    const uint32_t rank = cluster_rank();
    if (threadIdx.x == 0) {
        for (int s = 0; s < P_STAGES; ++s) {
            mbar_init(bar_full + 8 * s, 2);                    // the leader's two producers, for the bytes of both CTAs
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(bar_tfull + 8 * a, 1);
            mbar_init(bar_tempty + 8 * a, 2 * P_EPI_WARPS);    // one arrival per epilogue warp of both CTAs
        }
        *abort_flag = 0;
        fence_mbar_init();
        tma_prefetch_desc(&tmapW);
        tma_prefetch_desc(&tmapS);
        tma_prefetch_desc(&tmapC);
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(tmem_slot), TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync();                                            // barriers of both CTAs exist, both have their TMEM
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_launch();
    grid_dep_wait();

    // ---- this pair's entries
    const int pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
    PairDeal deal;
    bool snake = false, ordered = false;
    if (g.mode == MODE_SDD) {
        for (int r = threadIdx.x; r < g.n_row_blocks; r += P_THREADS) {
            const int n = __ldg(g.list_ptr + r + 1) - __ldg(g.list_ptr + r);
            prefix[r + 1] = sdd_full(n) | (sdd_single(n) << 16);
        }
        if (threadIdx.x == 0) prefix[0] = 0;
        __syncthreads();
        if (warp == 0) {
            int carry = 0;
            for (int r0 = 1; r0 <= g.n_row_blocks; r0 += 32) {
                int v = r0 + lane <= g.n_row_blocks ? prefix[r0 + lane] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                if (r0 + lane <= g.n_row_blocks) prefix[r0 + lane] = v + carry;
                carry += __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        const int total = prefix[g.n_row_blocks];
        deal.init(total & 0xffff, total >> 16, pairs);
    } else {
        const int duos = (g.NN + 255) >> 8;
        deal.init(g.n_row_blocks * (duos >> 1), g.n_row_blocks * (duos & 1), pairs);
        // with one pass the order of the entries does not matter; forwards and backwards in turn only where row blocks differ
        ordered = deal.passes > 1;
        if (g.mode == MODE_DSD && ordered) snake = __ldg(g.h_nnz) != g.n_row_blocks * __ldg(g.h_max);
    }
    for (int ps = threadIdx.x; ps < deal.passes; ps += P_THREADS) {
        const int entry = ps * pairs + (((ps & 1) && snake) ? pairs - 1 - pair : pair);
        if (entry < deal.entries) tab[ps] = pair_entry(g, deal, entry, prefix, ordered);
        else tab[ps].sp_row = -1;
    }
    __syncthreads();

    if (warp == 0 || warp == n_warps - 1) {
        // ============================== producers: warp 0 the first slab of the dense operand, the last warp the second one and
        // the row block (one thread issues a load only every ~110 cycles, and a slab whose rows are contiguous takes two)
        const bool first = warp == 0;
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int ps = 0; ok && ps < deal.passes; ++ps) {
                const int sp = tab[ps].sp_row + int(rank) * 64;
                if (tab[ps].sp_row < 0) continue;
                const bool has_slab = first || (tab[ps].shape & 3) == 2;
                const uint32_t tx = (has_slab ? 2u * P_W_BYTES : 0u) + (first ? 0u : 2u * P_S_BYTES);   // of both CTAs
                int slab = tab[ps].slab[(first ? 0 : 2) + int(rank)];
                if (slab < 0) slab = tab[ps].slab[0];         // an absent slab is loaded from one that exists, and not stored
                Seg w;
                w.klist = g.mode == MODE_DSD ? g.list_idx + tab[ps].list_beg : nullptr;
                w.i0 = 0; w.i1 = tab[ps].nk; w.bits = 0; w.use_bits = false;
                KIter kit;
                kit.init(w);
                int kb;
                while (ok && kit.next(kb)) {
                    for (int h = 0; h < 2; ++h) {
                        const int k = kb * 128 + h * BK;
                        if (k >= g.KK) break;
                        if (!mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, g.status, ST_PRODUCER)) { ok = false; break; }
                        const uint32_t full = cluster_map(bar_full + 8 * stage, 0);
                        if (rank == 0) mbar_arrive_expect_tx(bar_full + 8 * stage, tx);
                        const uint32_t slot = tiles + stage * P_STAGE_BYTES, sW = slot + (first ? 0 : P_W_BYTES);
                        const uint32_t sS = slot + 2 * P_W_BYTES;
                        if (!first) {
                            if (!S_MN) tma_load_2d_pair(sS, &tmapS, full, k, sp);
                            else tma_load_2d_pair(sS, &tmapS, full, sp, k);
                        }
                        if (has_slab) {
                            if (!W_MN) {
                                tma_load_2d_pair(sW, &tmapW, full, k, slab);
                            } else {
                                tma_load_2d_pair(sW, &tmapW, full, slab, k);
                                tma_load_2d_pair(sW + MN_ATOM_BYTES, &tmapW, full, slab + 64, k);
                            }
                        }
                        if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ============================== MMA issuer: the leading CTA's, for both
        if (rank == 0) {
            constexpr uint64_t W_HI = W_MN ? make_smem_desc_hi(MN_ATOM_BYTES, 1024) : make_smem_desc_hi(16, 1024);
            constexpr uint64_t S_HI = S_MN ? make_smem_desc_hi(MN_ATOM_BYTES, 1024) : make_smem_desc_hi(16, 1024);
            constexpr uint32_t W_KSTEP = W_MN ? 2048 : 32, S_KSTEP = S_MN ? 2048 : 32;
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int ps = 0; ok && ps < deal.passes; ++ps) {
                if (tab[ps].sp_row < 0) continue;
                const int shape = tab[ps].shape, n_duos = shape & 3, n_stages = shape >> 2;
                if (!mbar_wait_cluster(bar_tempty + 8 * acc, acc_phase ^ 1, abort_flag, g.status, ST_MMA_ACC)) break;
                uint32_t accumulate = 0;
                tc_fence_after();
                const uint32_t d = tmem_base + acc * 256;
                for (int st = 0; st < n_stages; ++st) {
                    if (!mbar_wait(bar_full + 8 * stage, phase, abort_flag, g.status, ST_MMA_FULL)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t sW = tiles + stage * P_STAGE_BYTES, sS = sW + 2 * P_W_BYTES;
                    if (elect_one()) {
#pragma unroll
                        for (int j = 0; j < BK / 16; ++j) {
                            umma_f16_pair(d, make_smem_desc(sW + j * W_KSTEP, W_HI), make_smem_desc(sS + j * S_KSTEP, S_HI),
                                          g.idesc256, j ? 1u : accumulate);
                            if (n_duos == 2)
                                umma_f16_pair(d + 128, make_smem_desc(sW + P_W_BYTES + j * W_KSTEP, W_HI),
                                              make_smem_desc(sS + j * S_KSTEP, S_HI), g.idesc256, j ? 1u : accumulate);
                        }
                        umma_commit_pair(bar_empty + 8 * stage);
                    }
                    accumulate = 1;
                    if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                if (elect_one()) umma_commit_pair(bar_tfull + 8 * acc);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
        __syncwarp();
    } else {
        // ============================== epilogue
        const int quad = warp & 3;
        const int etid = quad * 32 + lane;
        const bool aligned16 = (reinterpret_cast<uintptr_t>(g.C) & 15) == 0;
        const bool vec_ok = g.c_cs == 1 && (g.c_rs & 7) == 0 && aligned16, vec_t_ok = g.c_rs == 1 && (g.c_cs & 7) == 0 && aligned16;
        zero_uncovered(g, vec_ok, vec_t_ok, etid, lane, int(blockIdx.x), int(gridDim.x));
        const uint32_t buf = smem_u32(staging) + uint32_t(warp - 2) * 4096u;
        int acc = 0, n_stores = 0;
        uint32_t acc_phase = 0;
        for (int ps = 0; ps < deal.passes; ++ps) {
            const PairEntry e = tab[ps];
            if (e.sp_row < 0) continue;
            const bool ok = mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag, g.status, ST_EPILOGUE);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + acc * 256 + (uint32_t(quad * 32) << 16);
            // 32 rows of the dense operand (lanes) x 32 rows of the masked one (registers) at a time; chunk c of a duo covers
            // its rows [32 c, 32 c + 32).  Two chunks share a staging buffer and a store of 16-bit results.
            auto process = [&](const int u, const int c, uint32_t (&r)[32]) {
                const int slab = u ? (rank ? e.slab[3] : e.slab[2]) : (rank ? e.slab[1] : e.slab[0]);
                const int wrow = slab + quad * 32, srow = e.sp_row + c * 32;
                const bool store = slab >= 0 && wrow < g.NN;   // (a box may hang over the edge, but not start beyond it)
                if (g.act == 1) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = int(r[j]) < 0 ? 0u : r[j];
                }
                if (g.tma_store == 1) {                       // masked rows contiguous in memory: [lane][64], SWIZZLE_128B
                    if (!(c & 1)) wait_staging_free(false, n_stores, lane);
                    const uint32_t rowaddr = buf + lane * 128, sw = lane & 7, piece0 = (c & 1) << 2;
                    uint32_t p[16];
                    convert_chunk(r, g.scale, g.is_bf16, p);
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((piece0 + v) ^ sw) << 4)),
                                     "r"(p[4 * v]), "r"(p[4 * v + 1]), "r"(p[4 * v + 2]), "r"(p[4 * v + 3])
                                     : "memory");
                    if (c & 1) {
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            if (store && srow - 32 < g.MM) tma_store_2d(&tmapC, buf, srow - 32, wrow);
                            bulk_commit();
                        }
                        ++n_stores;
                    }
                } else if (g.tma_store == 2) {                // dense rows contiguous: [64 masked rows][32 lanes], SWIZZLE_64B
                    if (!(c & 1)) wait_staging_free(false, n_stores, lane);
                    const uint32_t hbuf = buf + ((c & 1) << 11), lane_off = ((lane & 7) << 1), chunk = lane >> 3;
                    uint32_t p[16];
                    convert_chunk(r, g.scale, g.is_bf16, p);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const uint32_t addr = hbuf + j * 64 + (((chunk ^ ((j >> 1) & 3))) << 4) + lane_off;
                        asm volatile("st.shared.b16 [%0], %1;" ::"r"(addr), "h"((unsigned short)(p[j >> 1] >> (16 * (j & 1))))
                                     : "memory");
                    }
                    if (c & 1) {
                        fence_proxy_async();
                        __syncwarp();
                        if (lane == 0) {
                            if (store && srow - 32 < g.MM) tma_store_2d(&tmapC, buf, wrow, srow - 32);
                            bulk_commit();
                        }
                        ++n_stores;
                    }
                } else {                                       // fp32, a chunk per store, SWIZZLE_128B
                    wait_staging_free(false, n_stores, lane);
                    if (g.tma_store == 3) {                    // dense rows contiguous: [32 masked rows][32 lanes]
                        const uint32_t piece = uint32_t(lane) >> 2, within = (uint32_t(lane) & 3u) << 2;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            asm volatile("st.shared.b32 [%0], %1;" ::"r"(buf + j * 128 + ((piece ^ (uint32_t(j) & 7u)) << 4) + within),
                                         "f"(__uint_as_float(r[j]) * g.scale)
                                         : "memory");
                    } else {                                   // masked rows contiguous: [lane][32]
                        const uint32_t rowaddr = buf + lane * 128, sw = lane & 7;
#pragma unroll
                        for (int v = 0; v < 8; ++v)
                            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + ((v ^ sw) << 4)),
                                         "f"(__uint_as_float(r[4 * v]) * g.scale), "f"(__uint_as_float(r[4 * v + 1]) * g.scale),
                                         "f"(__uint_as_float(r[4 * v + 2]) * g.scale), "f"(__uint_as_float(r[4 * v + 3]) * g.scale)
                                         : "memory");
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) {
                        if (store && srow < g.MM) {
                            if (g.tma_store == 3) tma_store_2d(&tmapC, buf, wrow, srow); else tma_store_2d(&tmapC, buf, srow, wrow);
                        }
                        bulk_commit();
                    }
                    ++n_stores;
                }
            };
            // the next chunk is in flight from TMEM while one is converted and stored
            const int n_chunks = 4 * (e.shape & 3);
            uint32_t rbuf[2][32];
            tmem_ld_32x32(taddr, rbuf[0]);
            tmem_ld_wait();
            for (int c = 0; c < n_chunks; c += 2) {
                tmem_ld_32x32(taddr + (c + 1) * 32, rbuf[1]);
                process(c >> 2, c & 3, rbuf[0]);
                tmem_ld_wait();
                if (c + 2 < n_chunks) tmem_ld_32x32(taddr + (c + 2) * 32, rbuf[0]);
                process(c >> 2, (c & 3) + 1, rbuf[1]);
                tmem_ld_wait();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_map(bar_tempty + 8 * acc, 0));
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
        if (lane == 0) bulk_wait_all();
        __syncwarp();
    }

    tc_fence_before();
    cluster_sync();                                            // nothing of the pair is in flight towards a CTA that has left
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
}

}  // namespace sd
