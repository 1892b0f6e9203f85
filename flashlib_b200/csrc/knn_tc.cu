// Tensor-core candidate pass of the exact kNN: a persistent, warp-specialised sm_100a
// kernel.  Per work item (one tile of 128 queries x one contiguous range of database
// tiles) it keeps the bf16 query tile resident in shared memory, streams bf16 database
// tiles of 256 rows through a TMA ring, multiplies them with tcgen05.mma into two
// 128 x 256 fp32 accumulators in tensor memory (so the next tile's MMAs overlap the
// current tile's epilogue).  The operand planes carry 16 extra columns (ones on the query
// side, -||x||^2/2 split into three bf16 terms on the database side), so one extra K=16 MMA
// step makes every accumulator element the score
//     s = <q, x> - ||x||^2 / 2          (larger = closer)
// and the epilogue only compares: column groups with a score above a row's threshold go to a queue of
// that row's thread, and from there the scores that still pass to the row's candidate list, both
// in scratch that stays in the L2.  Nothing of the 128 x 256 score tile is stored; per query and
// range only the four warpgroups' lists (16 entries each; deeper or other pools in the modes
// described below) and their final thresholds are published, unsorted.
//
// Warp roles of the list modes (608 threads): warps 0-15 epilogue in four warpgroups (group g takes
// columns 64g..64g+63 of every accumulator; warp w reads TMEM lanes 32(w%4)..32(w%4)+31, one query
// row per thread, and keeps a list per row), warp 16 TMA producer, warps 17 and 18 MMA issuers (every
// other tile each; warp 17 owns the TMEM allocation).  The other modes (352 threads) have two epilogue
// warpgroups of 128 columns.  What bounds the list modes, 10 000 x 1M x 128, k = 10 (scoring pass 2.56 ms
// with two warpgroups, pools in shared memory and one issuing lane): 1 152 cycles of tensor core a tile,
// which run at about 1.6 PFLOP/s before the power limit, and the epilogue's ALU pipe beside it
// (half a three-input maximum a score, 16 lanes a cycle): 2.05 ms; its screening alone would allow 1.74,
// the MMAs alone 1.63.  Four warpgroups because two warps a scheduler leave half of that pipe idle; the queue
// because a flagged group costs a warp 10 instructions that way, and 40 when its scores are compared and
// appended on the spot (2.36 ms), wherever its lanes' scores then go.
// Every wait is bounded; a wait that gives up raises a CTA-wide abort flag, records where
// it happened in the status words and every role falls through to the common exit.
#include "knn_internal.h"
#include "pool.cuh"
#include "tc_ptx.cuh"
#include <stdlib.h>

namespace fl {

using namespace tc;

constexpr int TC_BM = 128;            // queries per tile (MMA M)
constexpr int TC_BN = 256;            // database rows per tile (MMA N)
constexpr int TC_BK = 64;             // bf16 features per shared-memory chunk (128 bytes)
constexpr int TC_NWG = 2;             // epilogue warpgroups; group g owns columns 128g.. of every tile
constexpr int TC_LIST_NWG = 4;        // ... of the list modes: columns 64g..
constexpr int TC_LIST_PUB = 16, TC_LIST_K1 = 16, TC_LIST_CAP = 32;            // list modes: entries published, kept at a
constexpr int TC_BIG_PUB = 128, TC_BIG_K1 = 128, TC_BIG_CAP = 256;            // compaction, working capacity (k <= 16; beyond)
// List modes: queue of flagged column groups of an epilogue thread, slots of 8 scores and a row number (48 bytes).  Emptied by
// all warps of the CTA at every TC_QUEUE_EVERY-th tile, and by a warp that could overflow with the next tile's 8.
constexpr int TC_QUEUE_EVERY = 64, TC_QUEUE_SLOTS = 24, TC_QUEUE_SLOT_BYTES = 48, TC_QUEUE_FULL = TC_QUEUE_SLOTS - 8;
constexpr int TC_QUEUE_BYTES = TC_QUEUE_SLOTS * TC_QUEUE_SLOT_BYTES;
constexpr int TC_MID_K1 = 24;         // deep-pool mode: a query has few pools (inverted-file scan: two per
constexpr int TC_MID_CAP = 48;        // probed list), so each must reach further below the k-th neighbour
constexpr int TC_MID_PUB = 64;        // published entries per pool in that mode (padded)
constexpr int TC_MMA_WARPS = 2;       // MMA issuers; issuer j owns accumulator j, i.e. every other tile
constexpr int TC_THREADS = (4 * TC_NWG + 1 + TC_MMA_WARPS) * 32;
constexpr int TC_LIST_THREADS = (4 * TC_LIST_NWG + 1 + TC_MMA_WARPS) * 32;
constexpr int TC_A_CHUNK = TC_BM * 128;   // bytes of one K-chunk of the query tile
constexpr int TC_A_AUG = TC_BM * 32;      // bytes of the query tile's 16 norm columns
constexpr int TC_B_CHUNK = TC_BN * 128;   // bytes of one K-chunk of a database tile
constexpr int TC_B_AUG = TC_BN * 32;      // bytes of a database tile's 16 norm columns
constexpr int TC_B_STAGE = TC_B_CHUNK + TC_B_AUG;   // ring slot: a K-chunk, plus the norm
                                                    // columns when it is the tile's last chunk
// Streamed query tile (more than 512 features): a slot also holds the query tile's chunk and, for the
// tile's last chunk, its norm columns.
constexpr int TC_STREAM_A = TC_A_CHUNK + TC_A_AUG;
constexpr int TC_MAX_STAGES = 6;
constexpr uint64_t TC_WAIT_DEFAULT_NS = 2000000000ull;   // 2 s per wait unless the launch says otherwise

struct TcSmemPlan {
    int nkc, nstage;
    int off_a, off_b, off_pool_sc, off_pool_id, off_hbuf, off_bar, bytes;
};

// nabuf: query-tile buffers (2: the next item's tile is loaded while the current item is scored).
static TcSmemPlan tc_smem_plan(int d_pad, int smem_limit, int pool_stride, int slot_bytes = TC_B_STAGE, int nabuf = 1) {
    TcSmemPlan s{};
    s.nkc = d_pad / TC_BK;
    int cur = 0;
    s.off_a = cur; cur += nabuf * (s.nkc * TC_A_CHUNK + TC_A_AUG);
    const int pool = TC_NWG * TC_BM * pool_stride * 4;   // 0: no pools in shared memory
    const int fixed = cur + 2 * pool + 256 + 1024 /* alignment slack */;
    int ns = (smem_limit - fixed) / slot_bytes;
    if (ns > TC_MAX_STAGES) ns = TC_MAX_STAGES;
    s.nstage = ns;
    s.off_b = cur; cur += (ns > 0 ? ns : 0) * slot_bytes;
    s.off_pool_sc = cur; cur += pool;
    s.off_pool_id = cur; cur += pool;
    s.off_hbuf = cur;
    s.off_bar = cur; cur += 256;
    s.bytes = cur + 1024;
    return s;
}

// Per-CTA cycle counters of the last launch (debug aid, read by fl_debug_tc_prof_read):
// [0] producer waiting for a free slot, [1] MMA waiting for operands, [2] MMA waiting for a
// free accumulator, [3] epilogue waiting for an accumulator, [4] cycles in the epilogue's
// second pass, [5] column groups revisited there, [6] pool compactions, [7] scores appended
// (warp 0 / lane 0 views), [8] kernel cycles, [9] tiles.
// The counters cost registers in the epilogue warps, so they are compiled in only with -DFL_TC_PROF
// (FLASHLIB_B200_NVCC_FLAGS=-DFL_TC_PROF python -m flashlib_b200._build --force); otherwise
// fl_debug_tc_prof_read returns zeros.
constexpr int TC_PROF_WORDS = 16;
__device__ unsigned long long g_tc_prof[160 * TC_PROF_WORDS];
#ifdef FL_TC_PROF
#define TC_PROF(...) __VA_ARGS__
#else
#define TC_PROF(...)
#endif

struct TcKernelParams {
    int n_qtiles, n_tiles, nsplit, tiles_per_split, nkc, nstage;
    const uint32_t* fmt;     // operand format of the feature columns (FMT_*; null: bf16)
    int last_steps;          // K = 16 steps of a tile's last chunk that hold features at all (1 to 4)
    int nabuf;               // query-tile buffers in shared memory (1 or 2)
    int stream_a;            // 1: the query tile is not resident; its chunk travels with every database chunk
    int off_b, off_pool_sc, off_pool_id, off_bar;
    int64_t nq_pad;
    float* part_sc; uint32_t* part_id;
    float* tau;
    float* part_tau;
    int* part_cnt;           // large-k mode: entries of every published pool
    const int* nq_dev;       // optional: live query rows, counted on the device by an earlier kernel
    const int* row_query;    // optional: query of every (gathered) query row, -1 for rows without one, and
    float* tau_q;            //   a running threshold per query shared by all rows of that query
    const int* item_t0;      // optional (one range per query tile): first / one-past-last database
    const int* item_t1;      //   tile of query tile `it`, instead of the uniform ranges
    int item_tile_cap;       // > 0: at most this many tiles of every table range (seeding over item tables)
    const int* item_order;   // optional, with item tables: the CTAs walk item item_order[i] in place of item i
                             //   (longest ranges first, so that the round-robin deal comes out even)
    float* seed_cls;         // seeding output: [nq_pad][nsplit][TC_NWG][16] class maxima
    void* lists;             // list modes: working lists of every CTA, tc_list_bytes()
    float2* gpool;           // global-pool modes: (score, row) pairs, [nq_pad][nsplit][TC_NWG][CAP]
    float* asg_sc; uint32_t* asg_id;   // assignment mode outputs: [rows][TC_NWG] x (best, second) / centroid
    const int* asg_rows;     // optional, with nq_dev: output row of every (gathered) live query row
    int32_t* status;
    uint32_t wait_hint_ns;   // suspend-time hint of the barrier waits
    uint64_t wait_ns;        // limit of the MMA lane's barrier waits; a wait that runs out aborts the CTA
                             // (FL_ETIMEOUT).  The producer and the epilogue warps, which can only starve
                             // after the MMA lane has, wait twice as long, so the status names the wait
                             // nearest to the cause.
    int tile_stride;         // database tile actually read for loop index t is t * tile_stride (1 outside seeding)
    int dbg_flags;           // timing experiments (results invalid): 1 flag nothing, 4 skip the
                             // screening too, 8 skip the
                             // norm-column MMA step, 16 issue no MMA at all (operand streaming only);
                             // 32 the producer leaves out its fourth operand load, so the MMA lane's
                             // wait for it runs out (host-visible test of the bounded-wait exit)
    float* dbg_scores;       // optional: [128][n_tiles*256] scores of query tile 0
    int64_t dbg_ld;
};

// Database tiles [t0, t1) of work item `it`: a uniform range of the whole plane, or the item's own
// range from the tables (cut to item_tile_cap tiles when that is set).
__device__ __forceinline__ void tc_item_range(const TcKernelParams& p, int it, int split, int& t0, int& t1) {
    if (p.item_t0 != nullptr) {
        t0 = __ldg(p.item_t0 + it);
        t1 = __ldg(p.item_t1 + it);
        if (p.item_tile_cap > 0) t1 = min(t1, t0 + p.item_tile_cap);
    } else {
        t0 = split * p.tiles_per_split;
        t1 = min(p.n_tiles, t0 + p.tiles_per_split);
    }
}

__device__ __forceinline__ void tc_report_timeout(int32_t* status, int role, int which) {
    if (status) {
        if (atomicCAS(status + FL_STATUS_ERROR, 0, FL_ETIMEOUT) == 0) status[FL_STATUS_WHERE] = (role << 16) | which;
    }
}

// Compacts the pools of the rows named in `need` (one bit per lane = row of this warp): (score, row) pairs of 8 bytes,
// `stride` pairs from row to row.  Kept out of line: compaction is rare and the sorting network is large.
template <int CAP, int K1>
static __device__ __noinline__ float2 tc_compact_rows_pairs(unsigned need, float2* warp_pool, int stride, int cnt, float tau) {
    constexpr int NPL = (CAP + 31) / 32;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    while (need) {
        const int src = __ffs(need) - 1;
        need &= need - 1;
        const int n = __shfl_sync(FULL_MASK, cnt, src);
        float2* pool = warp_pool + src * stride;
        float key[NPL];
        uint32_t id[NPL];
#pragma unroll
        for (int r = 0; r < NPL; ++r) {
            const int e = (r << 5) | lane;
            const float2 v = e < n ? pool[e] : make_float2(neg_inf(), __uint_as_float(INVALID_ID));
            key[r] = v.x;
            id[r] = __float_as_uint(v.y);
        }
        warp_sort_desc<NPL, false>(key, id);
        float thr = neg_inf();
#pragma unroll
        for (int r = 0; r < NPL; ++r) {
            const int e = (r << 5) | lane;
            if (e < K1) pool[e] = make_float2(key[r], __uint_as_float(id[r]));
            if (((K1 - 1) >> 5) == r) thr = __shfl_sync(FULL_MASK, key[r], (K1 - 1) & 31);
        }
        __syncwarp();
        if (lane == src) { cnt = min(n, K1); tau = fmaxf(tau, n >= K1 ? thr : neg_inf()); }
    }
    return make_float2(__int_as_float(cnt), tau);
}

// Appends the scores of x[0..7] (rows col0 ..) that exceed tau at ADDR, which moves on: the 8 comparisons first
// (independent), then the predicated stores, so that only the address increments form a chain.
#define FL_APPEND(ST, ADD, C, ADDR)                                                                                    \
    asm volatile(                                                                                                      \
        "{\n\t.reg .pred p0, p1, p2, p3, p4, p5, p6, p7;\n\t.reg .b32 c;\n\t"                                         \
        "setp.gt.f32 p0, %3, %1;\n\tsetp.gt.f32 p1, %4, %1;\n\tsetp.gt.f32 p2, %5, %1;\n\tsetp.gt.f32 p3, %6, %1;\n\t" \
        "setp.gt.f32 p4, %7, %1;\n\tsetp.gt.f32 p5, %8, %1;\n\tsetp.gt.f32 p6, %9, %1;\n\tsetp.gt.f32 p7, %10, %1;\n\t" \
        "@p0 " ST " [%0], {%3, %2};\n\t@p0 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 1;\n\t"                              \
        "@p1 " ST " [%0], {%4, c};\n\t@p1 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 2;\n\t"                               \
        "@p2 " ST " [%0], {%5, c};\n\t@p2 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 3;\n\t"                               \
        "@p3 " ST " [%0], {%6, c};\n\t@p3 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 4;\n\t"                               \
        "@p4 " ST " [%0], {%7, c};\n\t@p4 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 5;\n\t"                               \
        "@p5 " ST " [%0], {%8, c};\n\t@p5 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 6;\n\t"                               \
        "@p6 " ST " [%0], {%9, c};\n\t@p6 " ADD " %0, %0, 8;\n\tadd.u32 c, %2, 7;\n\t"                               \
        "@p7 " ST " [%0], {%10, c};\n\t@p7 " ADD " %0, %0, 8;\n\t}"                                                  \
        : "+" C(ADDR)                                                                                                  \
        : "r"(__float_as_uint(tau)), "r"(col0), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]),      \
          "r"(x[6]), "r"(x[7])                                                                                         \
        : "memory")

// MODE 1 (TC_MODE_SEED) turns the kernel into the threshold-seeding pass: it scans a strided sample of
// the database tiles and, instead of pools, keeps 16 running maxima per query row over
// disjoint column classes; their minimum is a score that 16 distinct rows reach, i.e. a valid
// starting threshold that spares the main pass most of its cold-start appends.
//
// MODE 2 (TC_MODE_ASSIGN) is the k-means assignment: the "database" is the (small) centroid
// set, every row only needs its best centroid, so each thread keeps the best and second-best
// score of its row in registers (the column index rides in the low 7 mantissa bits of the
// score) and no pool is touched.
//
// MODE 3 (TC_MODE_KNN_BIG) is MODE 0 for 16 < k <= 112 (lists of 256, 128 kept and published).
//
// MODE 4 (TC_MODE_KNN_MID) is MODE 0 with deeper pools in shared memory (24 of 48 kept, 64
// published): for callers whose queries have only a few pools each (a small database scored as
// one range; the inverted-file scan, where a query row meets only the tiles of one list).  There a
// row has a candidate in most tiles, so queueing whole groups would store most of the scores; this mode
// compares the scores of flagged groups against the row's threshold on the spot and appends the passing
// ones with predicated 8-byte stores.
//
// MODE 5 (TC_MODE_KNN_GPOOL) is MODE 4 with the pools in global memory, as (score, row) pairs in
// the buffer the finalisation reads (64 slots per (query row, warpgroup), 24 kept at a
// compaction, entry counts published): no pool takes shared memory, so the TMA ring is four
// slots deep -- two whole tiles, where MODE 4 has room for one and stalls on every load -- and
// nothing is copied out when an item ends.  The inverted-file scan runs in this mode.
//
// MODE 7 (TC_MODE_KNN_GPOOL_BIG) is MODE 5 with 256 slots, 128 kept, for 16 < k <= 112.
constexpr int TC_MODE_KNN = 0, TC_MODE_SEED = 1, TC_MODE_ASSIGN = 2, TC_MODE_KNN_BIG = 3, TC_MODE_KNN_MID = 4,
              TC_MODE_KNN_GPOOL = 5, TC_MODE_KNN_GPOOL_BIG = 7;
constexpr bool tc_list_mode(int mode) { return mode == TC_MODE_KNN || mode == TC_MODE_KNN_BIG; }
constexpr int TC_GP_K1 = 24, TC_GP_CAP = 64;
//
// PAIR: two CTAs of a cluster work as one (tcgen05 cta_group::2).  CTA r of the pair owns query
// tile 2 i + r of pair-item i, loads its own query tile and rows 128 r .. 128 r + 127 of every
// 256-row database tile (half the L2 and shared-memory traffic per CTA), the leader (r = 0)
// issues one M = 256 MMA per step that reads both halves and writes each CTA's 128 x 256
// accumulator into that CTA's tensor memory; both CTAs run the epilogue on their own rows.
// Operand and accumulator barriers live in the leader; "slot free", "query tile free" and
// "accumulator full" are committed to both CTAs.
template <bool DBG, int MODE, bool PAIR = false>
__global__ void __launch_bounds__(tc_list_mode(MODE) ? TC_LIST_THREADS : TC_THREADS, 1)
knn_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_q_aug,
              const __grid_constant__ CUtensorMap map_db, const __grid_constant__ CUtensorMap map_db_aug,
              const TcKernelParams p) {
    constexpr bool LIST = tc_list_mode(MODE);
    constexpr int NWG = LIST ? TC_LIST_NWG : TC_NWG, COLS = TC_BN / NWG;
    extern __shared__ uint8_t smem_raw[];
    // the swizzled operand tiles need 1024-byte aligned shared memory
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = smem_u32(smem);
    const uint32_t a_addr = sbase;                                // nkc chunks of 16 KB
    const uint32_t a_aug_addr = sbase + p.nkc * TC_A_CHUNK;       // 4 KB: the query tile's norm columns
    const uint32_t b_addr = sbase + p.off_b;                      // nstage slots of 40 KB
    float* pool_sc = reinterpret_cast<float*>(smem + p.off_pool_sc);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.off_bar);
    // barrier slots: [0, 6) full, [6, 12) empty, 12 a_full, 13 a_empty, 14-15 tmem_full, 16-17 tmem_empty,
    // 18 a_full / 19 a_empty of the second query-tile buffer, 22-23 turn of MMA warp 0 / 1
    const uint32_t bar0 = smem_u32(bars);
    auto BAR = [&](int i) { return bar0 + 8u * i; };
    constexpr int B_FULL = 0, B_EMPTY = 6, B_AFULL = 12, B_AEMPTY = 13, B_TFULL = 14, B_TEMPTY = 16, B_TURN = 22;
    // Query-tile buffer of item number i of this CTA: buffer i % nabuf, used for the (i / nabuf)-th time.
    const uint32_t a_stride = (uint32_t)(p.nkc * TC_A_CHUNK + TC_A_AUG);
    const bool two_a = !PAIR && p.nabuf == 2;
    auto a_buf = [&](uint32_t item) { return two_a ? (item & 1u) : 0u; };
    auto a_phase = [&](uint32_t item) { return two_a ? ((item >> 1) & 1u) : (item & 1u); };
    auto a_full_bar = [&](uint32_t buf) { return BAR(buf ? 18 : B_AFULL); };
    auto a_empty_bar = [&](uint32_t buf) { return BAR(buf ? 19 : B_AEMPTY); };
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 20);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    // a timing experiment leaves work out: whoever reads the status words learns that the
    // neighbours of this launch are not to be used
    if (DBG && (p.dbg_flags & 31) && blockIdx.x == 0 && tid == 0 && p.status != nullptr) {
        if (atomicCAS(p.status + FL_STATUS_ERROR, 0, FL_EUNSUPPORTED) == 0) p.status[FL_STATUS_WHERE] = 0xDB600 | p.dbg_flags;
    }
    const uint32_t cta_rank = PAIR ? cluster_ctarank() : 0u;
    const bool leader = cta_rank == 0;
    // geometry of one ring slot and of the work split
    constexpr int B_ROWS = PAIR ? TC_BN / 2 : TC_BN;          // database rows this CTA loads per tile
    constexpr int SLOT_CHUNK = B_ROWS * 128, SLOT_B_BYTES = B_ROWS * 128 + B_ROWS * 32;
    constexpr bool CAN_STREAM = MODE == TC_MODE_KNN_GPOOL || MODE == TC_MODE_KNN_GPOOL_BIG || MODE == TC_MODE_SEED;
    const bool stream_a = CAN_STREAM && p.stream_a != 0;
    const uint32_t slot_bytes = stream_a ? (uint32_t)(SLOT_B_BYTES + TC_STREAM_A) : (uint32_t)SLOT_B_BYTES;
    constexpr uint32_t OPERAND_CTAS = PAIR ? 2u : 1u;         // CTAs whose loads one operand barrier counts

    if (tid == 0) {
        for (int i = 0; i < TC_MAX_STAGES; ++i) { mbar_init(BAR(B_FULL + i), 1); mbar_init(BAR(B_EMPTY + i), 1); }
        mbar_init(BAR(B_AFULL), 1);
        mbar_init(BAR(B_AEMPTY), TC_MMA_WARPS);
        mbar_init(BAR(18), 1);
        mbar_init(BAR(19), TC_MMA_WARPS);
        for (int i = 0; i < TC_MMA_WARPS; ++i) mbar_init(BAR(B_TURN + i), 1);
        for (int i = 0; i < 2; ++i) { mbar_init(BAR(B_TFULL + i), 1); mbar_init(BAR(B_TEMPTY + i), 4 * NWG * OPERAND_CTAS); }
        *abort_flag = 0;
        fence_barrier_init();
    }
    constexpr int W_PRODUCER = 4 * NWG, W_MMA = 4 * NWG + 1;
    if (warp == W_PRODUCER && lane == 0) {
        prefetch_tensormap(&map_q); prefetch_tensormap(&map_q_aug);
        prefetch_tensormap(&map_db); prefetch_tensormap(&map_db_aug);
    }
    if (warp == W_MMA) {
        if (PAIR) { tmem_alloc_pair(smem_u32(tmem_slot), 512); tmem_relinquish_pair(); }
        else { tmem_alloc(smem_u32(tmem_slot), 512); tmem_relinquish(); }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();      // the peer's barriers exist before anyone signals them
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    // query tiles: fixed by the launch, or (nq_dev) cut down to the live rows counted on the device
    int n_qtiles = p.n_qtiles;
    if (p.nq_dev != nullptr) {
        const int live = (__ldcg(p.nq_dev) + TC_BM - 1) / TC_BM;
        n_qtiles = live < n_qtiles ? live : n_qtiles;
    }
    // item = (range, query tile) or, for CTA pairs, (range, pair of query tiles); a pair walks the
    // items together
    const int n_units = PAIR ? n_qtiles / 2 : n_qtiles;
    const int n_items = n_units * p.nsplit;
    const int it_first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int it_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int d_pad = p.nkc * TC_BK;

    if (warp == W_PRODUCER) {
        // ------------------------------ TMA producer --------------------------------------
        // (the whole warp walks the loop and an elected lane issues, as in the MMA warps: from a `lane == 0`
        // branch a 128-feature tile's three loads and two waits took 1 500 cycles)
        const uint32_t elected = elect_one();
        int s = 0;             // ring slot and its phase
        uint32_t ph = 0;
        int fill = 0;
        uint32_t item_no = 0;
        bool ok = true;
        TC_PROF(long long prof_a = 0;)
        // loads of a pair are credited to the leader's barrier, which expects both CTAs' bytes
        auto load = [&](uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
            if (PAIR) tma_load_2d_pair(dst, map, c0, c1, bar); else tma_load_2d(dst, map, c0, c1, bar);
        };
        auto wait = [&](uint32_t bar, int name, uint32_t parity) {
            const bool got = __all_sync(FULL_MASK, mbar_wait(bar, parity, abort_flag, 2 * p.wait_ns, p.wait_hint_ns));
            if (!got && lane == 0) tc_report_timeout(p.status, 4, name);
            return got;
        };
        for (int it = it_first; it < n_items && ok; it += it_step, ++item_no) {
            const int itp = p.item_order != nullptr ? __ldg(p.item_order + it) : it;
            const int split = itp / n_units, unit = itp - split * n_units;
            const int qt = PAIR ? 2 * unit + (int)cta_rank : unit;
            int t0, t1;
            tc_item_range(p, itp, split, t0, t1);
            const uint32_t ab = a_buf(item_no), a_off = ab * a_stride;
            if (!stream_a) {
                ok = wait(a_empty_bar(ab), ab ? 19 : B_AEMPTY, a_phase(item_no) ^ 1u);
                if (!ok) break;
                if (elected) {
                    if (leader) mbar_expect_tx(a_full_bar(ab), (p.nkc * TC_A_CHUNK + TC_A_AUG) * OPERAND_CTAS);
                    for (int kc = 0; kc < p.nkc; ++kc)
                        load(a_addr + a_off + kc * TC_A_CHUNK, &map_q, kc * TC_BK, qt * TC_BM, a_full_bar(ab));
                    load(a_aug_addr + a_off, &map_q_aug, d_pad, qt * TC_BM, a_full_bar(ab));
                }
                __syncwarp();
            }
            const int nt = t1 - t0;
            const int rot = (int)(((int64_t)unit * nt) / n_units);
            for (int i = 0; i < nt && ok; ++i) {
                // Query tiles walk their range from different starting tiles, so the CTAs of a
                // wave do not all ask the L2 for the same lines at the same moment.
                const int t = t0 + (i + rot < nt ? i + rot : i + rot - nt);
                const int row0 = t * p.tile_stride * TC_BN + (int)cta_rank * B_ROWS;
                for (int kc = 0; kc < p.nkc; ++kc, ++fill) {
                    TC_PROF(const long long c0 = clock64();)
                    ok = wait(BAR(B_EMPTY + s), B_EMPTY + s, ph ^ 1u);
                    if (!ok) break;
                    TC_PROF(prof_a += clock64() - c0;)
                    if (elected && !(DBG && (p.dbg_flags & 32) && fill == 3)) {       // (32: this slot never fills)
                        const bool last = (kc == p.nkc - 1);
                        const uint32_t slot = b_addr + s * slot_bytes, full = BAR(B_FULL + s);
                        if (leader) {
                            uint32_t bytes = last ? SLOT_B_BYTES : SLOT_CHUNK;
                            if (stream_a) bytes += TC_A_CHUNK + (last ? TC_A_AUG : 0);
                            mbar_expect_tx(full, bytes * OPERAND_CTAS);
                        }
                        load(slot, &map_db, kc * TC_BK, row0, full);
                        if (last) load(slot + SLOT_CHUNK, &map_db_aug, d_pad, row0, full);
                        if (stream_a) {
                            load(slot + SLOT_B_BYTES, &map_q, kc * TC_BK, qt * TC_BM, full);
                            if (last) load(slot + SLOT_B_BYTES + TC_A_CHUNK, &map_q_aug, d_pad, qt * TC_BM, full);
                        }
                    }
                    __syncwarp();
                    if (++s == p.nstage) { s = 0; ph ^= 1u; }
                }
            }
        }
        TC_PROF(if (lane == 0 && blockIdx.x < 160) g_tc_prof[blockIdx.x * TC_PROF_WORDS + 0] = prof_a;)
        if (!ok) {
            // give copies already in flight a bounded time to land before the CTA exits
            const uint64_t t_start = globaltimer_ns();
            while (globaltimer_ns() - t_start < 2000000ull) { }
        }
    } else if (warp >= W_MMA && warp < W_MMA + TC_MMA_WARPS) {
        // ------------------------------ MMA issuer -----------------------------------------
        // Bound by the serial cost of issuing, which must stay below the tensor core's 128 cycles a K = 16 step.
        // Two things keep it there.  A whole warp walks the loop and one elected lane issues: from a `lane == 0`
        // branch a chunk of four MMAs took 682 cycles however narrow they were (operands moved to uniform
        // registers under divergence), elected and unrolled 410.  And two warps take turns by tile: a wait that
        // succeeds at once and a commit cost about 200 cycles each, so one warp needs 1 450 cycles for the nine
        // steps of a 128-feature tile (1 152 cycles of tensor core).  A warp hands the turn on with its last MMA: its
        // commits and its wait for the accumulator fall into the other's turn.  (The turn also keeps the waits on
        // the ring in order: a slot's barrier is only asked about a phase when the one before has completed.)
        // Scoring of 10 000 x 1M x 128, one CTA a tile and the epilogue of before: 2.55 ms -> 2.22.
        if (leader) {
            // the norm columns are bf16 whatever the features are (a step of their own: one format within an MMA)
            constexpr uint32_t idesc_norm = umma_idesc_bf16(PAIR ? 2 * TC_BM : TC_BM, TC_BN);
            const uint32_t idesc_feat = p.fmt != nullptr && __ldg(p.fmt) == FMT_F16 ? umma_idesc_f16(PAIR ? 2 * TC_BM : TC_BM, TC_BN) : idesc_norm;
            const uint32_t elected = elect_one();
            auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t acc, uint32_t idesc) {
                if (DBG && (p.dbg_flags & 16)) return;     // timing experiment: operand streaming only
                if (PAIR) umma_bf16_pair(d, a, b, idesc, acc); else umma_bf16(d, a, b, idesc, acc);
            };
            auto commit = [&](uint32_t bar) { if (PAIR) umma_commit_pair(bar); else umma_commit(bar); };
            // all lanes wait; a lane that gave up takes the others with it
            auto wait = [&](int bar, uint32_t parity) {
                const bool got = __all_sync(FULL_MASK, mbar_wait(BAR(bar), parity, abort_flag, p.wait_ns, p.wait_hint_ns));
                if (!got && lane == 0) tc_report_timeout(p.status, 5, bar);
                return got;
            };
            const int b = warp - W_MMA;            // this warp's accumulator and tiles
            const uint32_t d_tmem = tmem_base + b * TC_BN;
            int s = 0;             // ring slot of the current tile's first chunk and its phase
            uint32_t ph = 0;
            uint32_t tile_no = 0;  // tiles so far, the other warp's included
            uint32_t item_no = 0;
            uint32_t turn = b == 0 ? 1u : 0u;      // the first turn is warp 0's without being handed to it
            bool ok = true;
            auto skip = [&](int chunks) { for (s += chunks; s >= p.nstage; s -= p.nstage) ph ^= 1u; };
            TC_PROF(long long prof_full = 0; long long prof_tempty = 0;)
            for (int it = it_first; it < n_items && ok; it += it_step, ++item_no) {
                const int itp = p.item_order != nullptr ? __ldg(p.item_order + it) : it;
                const int split = itp / n_units;
                int t0, t1;
                tc_item_range(p, itp, split, t0, t1);
                const uint32_t ab = a_buf(item_no), a_off = ab * a_stride;
                if (!stream_a) {
                    ok = wait(ab ? 18 : B_AFULL, a_phase(item_no));
                    if (!ok) break;
                }
                for (int t = t0; t < t1 && ok; ++t, ++tile_no) {
                    if ((int)(tile_no & 1) != b) { skip(p.nkc); continue; }
                    TC_PROF(const long long c0 = clock64();)
                    ok = wait(B_TEMPTY + b, ((tile_no >> 1) & 1) ^ 1);
                    if (!ok) break;
                    TC_PROF(prof_tempty += clock64() - c0;)
                    ok = wait(B_TURN + b, turn);
                    if (!ok) break;
                    turn ^= 1u;
                    for (int kc = 0; kc < p.nkc; ++kc) {
                        TC_PROF(const long long c1 = clock64();)
                        ok = wait(B_FULL + s, ph);
                        if (!ok) break;
                        TC_PROF(prof_full += clock64() - c1;)
                        tc_fence_after_sync();
                        if (elected) {
                            const uint32_t slot = b_addr + s * slot_bytes;
                            const bool last = kc == p.nkc - 1;
                            const uint64_t da = umma_desc(stream_a ? slot + SLOT_B_BYTES : a_addr + a_off + kc * TC_A_CHUNK);
                            const uint64_t db = umma_desc(slot);
                            // +32 bytes per 16-feature step inside the 128-byte swizzled row
                            mma(d_tmem, da, db, kc != 0 ? 1u : 0u, idesc_feat);
                            if (!last || p.last_steps == TC_BK / 16) {
#pragma unroll
                                for (int k4 = 1; k4 < TC_BK / 16; ++k4) mma(d_tmem, da + 2 * k4, db + 2 * k4, 1u, idesc_feat);
                            } else {
                                // columns of zeros beyond the last feature: 96 features take 7 steps with the norm
                                // columns in place of 9
                                for (int k4 = 1; k4 < p.last_steps; ++k4) mma(d_tmem, da + 2 * k4, db + 2 * k4, 1u, idesc_feat);
                            }
                            if (last && !(DBG && (p.dbg_flags & 8))) {
                                // norm columns: ones x split(-||x||^2/2), 32-byte rows, 32-byte swizzle
                                const uint32_t a_aug = stream_a ? slot + SLOT_B_BYTES + TC_A_CHUNK : a_aug_addr + a_off;
                                mma(d_tmem, umma_desc_sw32(a_aug), umma_desc_sw32(slot + SLOT_CHUNK), 1u, idesc_norm);
                            }
                            if (last) mbar_arrive(BAR(B_TURN + (b ^ 1)));
                            commit(BAR(B_EMPTY + s));   // slot reusable once these MMAs retire
                            if (last) commit(BAR(B_TFULL + b));
                        }
                        __syncwarp();
                        skip(1);
                    }
                }
                if (ok && !stream_a && elected) commit(a_empty_bar(ab));     // query tile buffer reusable (both warps' word)
                __syncwarp();
            }
            TC_PROF(if (lane == 0 && b == 0 && blockIdx.x < 160) {
                g_tc_prof[blockIdx.x * TC_PROF_WORDS + 1] = prof_full;
                g_tc_prof[blockIdx.x * TC_PROF_WORDS + 2] = prof_tempty;
            })
        }
    } else if (warp < W_PRODUCER) {
        // ------------------------------ epilogue warps --------------------------------------
        // warp = 4 * warpgroup + TMEM lane quarter; warpgroup g reads columns COLS g .. COLS (g + 1) - 1 of
        // every accumulator and keeps its own pool per query row.
        const int wg = warp >> 2, quarter = warp & 3;
        constexpr bool BIG = (MODE == TC_MODE_KNN_BIG);
        constexpr bool MID = (MODE == TC_MODE_KNN_MID);
        constexpr bool GPB = (MODE == TC_MODE_KNN_GPOOL_BIG);
        constexpr bool GP = (MODE == TC_MODE_KNN_GPOOL) || GPB;
        constexpr int CAP = (BIG || GPB) ? TC_BIG_CAP : LIST ? TC_LIST_CAP : MID ? TC_MID_CAP : TC_GP_CAP;
        constexpr int K1 = (BIG || GPB) ? TC_BIG_K1 : LIST ? TC_LIST_K1 : MID ? TC_MID_K1 : TC_GP_K1;
        constexpr int PSTR = CAP + 1;                    // shared pools: padded stride
        constexpr int PUB = BIG ? TC_BIG_PUB : LIST ? TC_LIST_PUB : TC_MID_PUB;   // published entries per pool
        const uint32_t lane_taddr = tmem_base + (uint32_t(quarter * 32) << 16);
        uint32_t tile_no = 0;
        bool ok = true;
        TC_PROF(long long prof_tfull = 0; long long prof_rare = 0; long long prof_cc = 0; long long prof_flush = 0;
                unsigned prof_groups = 0; unsigned prof_compact = 0; unsigned prof_append = 0;
                const long long prof_t0 = clock64();)
        // hands accumulator b back to the MMA lane (of the leader, for a pair)
        auto release_acc = [&](int b) {
            if (PAIR) mbar_arrive_cluster(BAR(B_TEMPTY + b), 0u); else mbar_arrive(BAR(B_TEMPTY + b));
        };
        // List modes: this thread's queue of flagged groups and its row's working list, both its CTA's own scratch.
        float tau = neg_inf();
        int cnt = 0;
        char* const scratch = static_cast<char*>(p.lists) + ((int64_t)blockIdx.x * (4 * NWG) + warp) * (32 * (TC_QUEUE_BYTES + CAP * 8));
        float2* const warp_list = reinterpret_cast<float2*>(scratch + 32 * TC_QUEUE_BYTES);
        const uint64_t queue = reinterpret_cast<uint64_t>(scratch + lane * TC_QUEUE_BYTES);
        uint64_t queue_end = queue;
        // The queued scores that still pass move to the lists, every lane its own group a step.
        auto flush = [&]() {
            TC_PROF(const long long cf0 = clock64();)
            const uint32_t bytes = (uint32_t)(queue_end - queue), most = __reduce_max_sync(FULL_MASK, bytes);
            float2* const list = warp_list + lane * CAP;
#pragma unroll 1
            for (uint32_t o0 = 0; o0 < most; o0 += 2 * TC_QUEUE_SLOT_BYTES) {
                float4 x[2][2];
                uint32_t first[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t o = o0 + u * TC_QUEUE_SLOT_BYTES;
                    x[u][0] = x[u][1] = make_float4(neg_inf(), neg_inf(), neg_inf(), neg_inf());
                    first[u] = 0;
                    if (o < bytes) {
                        const float4* slot = reinterpret_cast<const float4*>(queue + o);
                        x[u][0] = slot[0];
                        x[u][1] = slot[1];
                        first[u] = *reinterpret_cast<const uint32_t*>(slot + 2);
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (u > 0 && o0 + u * TC_QUEUE_SLOT_BYTES >= most) break;
                    const unsigned need = __ballot_sync(FULL_MASK, cnt > CAP - 8);
                    if (need) {
                        TC_PROF(prof_compact += __popc(need); const long long cc0 = clock64();)
                        const float2 cr = tc_compact_rows_pairs<CAP, K1>(need, warp_list, CAP, cnt, tau);
                        TC_PROF(prof_cc += clock64() - cc0;)
                        cnt = __float_as_int(cr.x);
                        tau = cr.y;
                    }
                    const float sv[8] = {x[u][0].x, x[u][0].y, x[u][0].z, x[u][0].w, x[u][1].x, x[u][1].y, x[u][1].z, x[u][1].w};
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (sv[j] > tau) list[cnt++] = make_float2(sv[j], __uint_as_float(first[u] + j));
                }
            }
            queue_end = queue;
            TC_PROF(prof_flush += clock64() - cf0;)
        };
        for (int it = it_first; it < n_items && ok; it += it_step) {
            const int itp = p.item_order != nullptr ? __ldg(p.item_order + it) : it;
            const int split = itp / n_units, unit = itp - split * n_units;
            const int qt = PAIR ? 2 * unit + (int)cta_rank : unit;
            int t0, t1;
            tc_item_range(p, itp, split, t0, t1);
            const int64_t qrow = (int64_t)qt * TC_BM + quarter * 32 + lane;
            float tau_in = MODE == TC_MODE_ASSIGN ? neg_inf() : __ldcg(p.tau + qrow);
            int qidx = -1;
            if (p.row_query != nullptr) {
                // rows that belong to the same query (one per probed list) pass their thresholds on:
                // a score below what 24 rows of another probed list reach cannot be among the k best
                qidx = __ldg(p.row_query + qrow);
                if (qidx >= 0) tau_in = fmaxf(tau_in, __ldcg(p.tau_q + qidx));
            }
            tau = tau_in;
            cnt = 0;
            float cls[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) cls[c] = neg_inf();
            float b1 = neg_inf(), b2 = neg_inf();   // assignment mode: best / second-best packed score
            int tbest = 0;                           // tile that produced b1
            const int nt = t1 - t0;
            const int rot = (int)(((int64_t)unit * nt) / n_units);
            for (int i = 0; i < nt; ++i, ++tile_no) {
                const int t = t0 + (i + rot < nt ? i + rot : i + rot - nt);
                const int b = tile_no & 1;
                TC_PROF(const long long c0 = clock64();)
                if (!__all_sync(FULL_MASK, mbar_wait(BAR(B_TFULL + b), (tile_no >> 1) & 1, abort_flag, 2 * p.wait_ns, p.wait_hint_ns))) {
                    if (lane == 0) tc_report_timeout(p.status, warp, B_TFULL + b);
                    ok = false;
                    break;
                }
                TC_PROF(prof_tfull += clock64() - c0;)
                tc_fence_after_sync();
                // this warpgroup's half of the accumulator columns / of the tile's database rows
                const uint32_t tile_taddr = lane_taddr + b * TC_BN + wg * COLS;
                const uint32_t row_base = (uint32_t)t * TC_BN + wg * COLS;

                // Pass 1, branch free: stream the 256 scores of this thread's query row through
                // registers, 64 columns per wait, and note which groups of 8 columns hold a score
                // above the row's threshold (bit g of `hits` = columns 8g .. 8g+7).
                // tcgen05.wait::ld waits for every load in flight, so while one batch of 64
                // columns is reduced the next one is already on its way.
                uint32_t va[32], vb[32], vc[32], vd[32];
                constexpr bool SEED = (MODE == TC_MODE_SEED);
                if (MODE == TC_MODE_ASSIGN) {
                    const float b1_before = b1;
                    // column index into the low 7 mantissa bits: one three-input logic instruction per
                    // score, (v & mask) | column, with the mask held in a register
                    uint32_t idx_mask;
                    asm volatile("mov.u32 %0, 0xFFFFFF80;" : "=r"(idx_mask));
                    auto pack = [&](uint32_t v, uint32_t col) {
                        uint32_t r;
                        asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(idx_mask), "r"(col));
                        return r;
                    };
                    auto top2 = [&](uint32_t (&v)[32], int slice) {
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            const float x = __uint_as_float(pack(v[j], (uint32_t)(slice * 32 + j)));
                            const float y = __uint_as_float(pack(v[j + 1], (uint32_t)(slice * 32 + j + 1)));
                            const float hi = fmaxf(x, y), lo = fminf(x, y);
                            b2 = fmax3(b2, lo, fminf(b1, hi));
                            b1 = fmaxf(b1, hi);
                        }
                    };
                    tmem_ld_32x32b_x32(tile_taddr, va);
                    tmem_ld_32x32b_x32(tile_taddr + 32, vb);
                    tmem_ld_wait();
                    reg_fence32(va);
                    reg_fence32(vb);
                    tmem_ld_32x32b_x32(tile_taddr + 64, vc);
                    tmem_ld_32x32b_x32(tile_taddr + 96, vd);
                    top2(va, 0);
                    top2(vb, 1);
                    tmem_ld_wait();
                    reg_fence32(vc);
                    reg_fence32(vd);
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) release_acc(b);
                    top2(vc, 2);
                    top2(vd, 3);
                    if (b1 != b1_before) tbest = t;
                    continue;
                }
                if (SEED) {
                    auto fold = [&](uint32_t (&v)[32]) {
#pragma unroll
                        for (int c = 0; c < 16; ++c)
                            cls[c] = fmax3(cls[c], __uint_as_float(v[c]), __uint_as_float(v[c + 16]));
                    };
                    tmem_ld_32x32b_x32(tile_taddr, va);
                    tmem_ld_32x32b_x32(tile_taddr + 32, vb);
                    tmem_ld_wait();
                    reg_fence32(va);
                    reg_fence32(vb);
                    tmem_ld_32x32b_x32(tile_taddr + 64, vc);
                    tmem_ld_32x32b_x32(tile_taddr + 96, vd);
                    fold(va);
                    fold(vb);
                    tmem_ld_wait();
                    reg_fence32(vc);
                    reg_fence32(vd);
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) release_acc(b);
                    fold(vc);
                    fold(vd);
                    continue;
                }
                if (GP || MID) {
                    // This row's pool of (score, row) pairs -- in global memory (GP) or shared memory (MID) --
                    // and the address of its next free slot.
                    float2* warp_pool = GP ? p.gpool + (((int64_t)(qt * TC_BM + quarter * 32) * p.nsplit + split) * NWG + wg) * CAP
                                           : reinterpret_cast<float2*>(pool_sc) + warp * 32 * PSTR;
                    const int gstride = GP ? p.nsplit * NWG * CAP : PSTR;      // pairs between the pools of consecutive rows
                    const uint64_t my_addr = reinterpret_cast<uint64_t>(warp_pool + (int64_t)lane * gstride);
                    const uint32_t my_saddr = MID ? smem_u32(warp_pool + lane * gstride) : 0u;
                    tmem_ld_32x32b_x32(tile_taddr, va);
                    tmem_ld_32x32b_x32(tile_taddr + 32, vb);
                    tmem_ld_32x32b_x32(tile_taddr + 64, vc);
                    tmem_ld_32x32b_x32(tile_taddr + 96, vd);
                    tmem_ld_wait();
                    reg_fence32(va);
                    reg_fence32(vb);
                    reg_fence32(vc);
                    reg_fence32(vd);
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) release_acc(b);
                    // Which groups of 8 columns hold a score above the threshold of any row of the warp:
                    // branch-free maxima, one vote for the tile.  Only those are compared score by score --
                    // appending every group costs a chain of 128 address increments, 2.6 us per tile.
                    unsigned wm = 0;
                    auto screen = [&](uint32_t (&v)[32], int slice) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const float x = fmax3(__uint_as_float(v[g * 8 + 0]), __uint_as_float(v[g * 8 + 1]), __uint_as_float(v[g * 8 + 2]));
                            const float y = fmax3(__uint_as_float(v[g * 8 + 3]), __uint_as_float(v[g * 8 + 4]), __uint_as_float(v[g * 8 + 5]));
                            const float z = fmax3(__uint_as_float(v[g * 8 + 6]), __uint_as_float(v[g * 8 + 7]), x);
                            wm |= (fmaxf(y, z) > tau) ? (1u << (slice * 4 + g)) : 0u;
                        }
                    };
                    screen(va, 0);
                    screen(vb, 1);
                    screen(vc, 2);
                    screen(vd, 3);
                    wm = __reduce_or_sync(FULL_MASK, wm);
                    if (wm) {
                        uint64_t waddr = my_addr + 8ull * (uint64_t)cnt;
                        uint32_t saddr = my_saddr + 8u * (uint32_t)cnt;
                        auto append = [&](uint32_t (&v)[32], int slice) {
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                if (!((wm >> (slice * 4 + g)) & 1u)) continue;
                                // every lane's pool has room for the 8 scores of the group
                                const int now = MID ? (int)((saddr - my_saddr) >> 3) : (int)((waddr - my_addr) >> 3);
                                const unsigned need = __ballot_sync(FULL_MASK, now > CAP - 8);
                                if (need) {
                                    TC_PROF(prof_compact += __popc(need);)
                                    const float2 cr = tc_compact_rows_pairs<CAP, K1>(need, warp_pool, gstride, now, tau);
                                    tau = cr.y;
                                    waddr = my_addr + 8ull * (uint64_t)__float_as_int(cr.x);
                                    saddr = my_saddr + 8u * (uint32_t)__float_as_int(cr.x);
                                }
                                // the 8 comparisons first (independent), then the predicated stores: only
                                // the address increments form a chain
                                const uint32_t col0 = row_base + slice * 32 + g * 8;
                                const uint32_t* x = v + g * 8;
                                if (MID) FL_APPEND("st.shared.v2.b32", "add.u32", "r", saddr);
                                else FL_APPEND("st.global.v2.b32", "add.u64", "l", waddr);
                            }
                        };
                        append(va, 0);
                        append(vb, 1);
                        append(vc, 2);
                        append(vd, 3);
                        const int now = MID ? (int)((saddr - my_saddr) >> 3) : (int)((waddr - my_addr) >> 3);
                        TC_PROF(prof_append += now - cnt;)
                        cnt = now;
                    }
                    continue;
                }
                // All 128 scores of this thread's query row into registers, and the accumulator back to the MMA warps
                // at once: it is theirs again after about 300 cycles, where reading it in two halves, screening
                // and coming back for the flagged groups held it for 1 000 to 1 500 -- with two accumulators and 1 152
                // cycles of MMA a tile, that was what paced the kernel.
                // List modes.  All 64 scores of this thread's row into registers and the accumulator back to the MMA
                // warps at once; then which groups of 8 columns hold a score above the row's threshold (branch free).
                // A flagged group goes to the thread's queue as it is, without a look at the single scores.
                tmem_ld_32x32b_x32(tile_taddr, va);
                tmem_ld_32x32b_x32(tile_taddr + 32, vb);
                tmem_ld_wait();
                reg_fence32(va);
                reg_fence32(vb);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) release_acc(b);
                unsigned hits = 0;
                auto scan = [&](uint32_t (&v)[32], int slice) {
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const float x = fmax3(__uint_as_float(v[g * 8 + 0]), __uint_as_float(v[g * 8 + 1]),
                                              __uint_as_float(v[g * 8 + 2]));
                        const float y = fmax3(__uint_as_float(v[g * 8 + 3]), __uint_as_float(v[g * 8 + 4]),
                                              __uint_as_float(v[g * 8 + 5]));
                        const float z = fmax3(__uint_as_float(v[g * 8 + 6]), __uint_as_float(v[g * 8 + 7]), x);
                        hits |= (fmaxf(y, z) > tau) ? (1u << (slice * 4 + g)) : 0u;
                    }
                    if (DBG) {
                        if (p.dbg_scores != nullptr && qt == 0) {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                p.dbg_scores[(int64_t)(quarter * 32 + lane) * p.dbg_ld + row_base + slice * 32 + j] =
                                    __uint_as_float(v[j]);
                        }
                    }
                };
                if (!DBG || !(p.dbg_flags & 4)) {
                    scan(va, 0);
                    scan(vb, 1);
                }
                if (DBG && (p.dbg_flags & 1)) hits = 0;
                const unsigned wm = __reduce_or_sync(FULL_MASK, hits);
                if (wm) {
                    TC_PROF(const long long cr0 = clock64(); prof_groups += __popc(wm);)
                    auto enqueue = [&](uint32_t (&v)[32], int slice) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const unsigned bit = 1u << (slice * 4 + g);
                            if (!(wm & bit)) continue;                        // (uniform)
                            const uint32_t* x = v + g * 8;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t"
                                "@p st.global.v4.b32 [%0], {%3, %4, %5, %6};\n\t"
                                "@p st.global.v4.b32 [%0+16], {%7, %8, %9, %10};\n\t"
                                "@p st.global.b32 [%0+32], %2;\n\t@p add.u64 %0, %0, %11;\n\t}"
                                : "+l"(queue_end)
                                : "r"(hits & bit), "r"(row_base + slice * 32 + g * 8), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]),
                                  "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "n"(TC_QUEUE_SLOT_BYTES)
                                : "memory");
                        }
                    };
                    enqueue(va, 0);
                    enqueue(vb, 1);
                    TC_PROF(prof_rare += clock64() - cr0;)
                }
                const bool full = (uint32_t)(queue_end - queue) > (uint32_t)(TC_QUEUE_FULL * TC_QUEUE_SLOT_BYTES);
                if ((tile_no & (TC_QUEUE_EVERY - 1)) == TC_QUEUE_EVERY - 1 || __any_sync(FULL_MASK, full)) flush();
            }
            if (LIST) flush();
            if (!ok) break;
            if (MODE == TC_MODE_ASSIGN) {
                if (p.asg_rows != nullptr && qrow >= __ldcg(p.nq_dev)) continue;
                const int64_t o = (p.asg_rows != nullptr ? (int64_t)__ldg(p.asg_rows + qrow) : qrow) * NWG + wg;
                p.asg_sc[2 * o] = b1;
                p.asg_sc[2 * o + 1] = b2;
                p.asg_id[o] = (uint32_t)tbest * TC_BN + wg * (TC_BN / NWG) + (__float_as_uint(b1) & 0x7Fu);
                continue;
            }
            if (MODE == TC_MODE_SEED) {
                float4* o = reinterpret_cast<float4*>(p.seed_cls + ((qrow * p.nsplit + split) * NWG + wg) * 16);
#pragma unroll
                for (int c = 0; c < 4; ++c) o[c] = make_float4(cls[4 * c], cls[4 * c + 1], cls[4 * c + 2], cls[4 * c + 3]);
                continue;
            }
            // end of the item: publish every row's pool (the rest of its slots padded, or its entry count beside it) and
            // the row's threshold.  Nothing is sorted here: the finalisation merges the published entries anyway.
            if (LIST) {
                const unsigned need = __ballot_sync(FULL_MASK, cnt > PUB);
                if (need) {
                    const float2 cr = tc_compact_rows_pairs<CAP, K1>(need, warp_list, CAP, cnt, tau);
                    cnt = __float_as_int(cr.x);
                    tau = cr.y;
                }
                __syncwarp();
                const int64_t o = (qrow * p.nsplit + split) * NWG + wg;
                p.part_tau[o] = tau;
                if (BIG) p.part_cnt[o] = cnt;
                constexpr int PER = PUB < 32 ? PUB : 32, ROWS = 32 / PER;        // lanes a row, rows a step
#pragma unroll 2
                for (int r0 = 0; r0 < 32; r0 += ROWS) {
                    const int src = r0 + lane / PER;
                    const int n = __shfl_sync(FULL_MASK, cnt, src);
                    const int64_t q = (int64_t)qt * TC_BM + quarter * 32 + src;
                    const int64_t to = ((q * p.nsplit + split) * NWG + wg) * PUB;
#pragma unroll
                    for (int e = lane % PER; e < PUB; e += PER) {
                        if (BIG && e >= n) break;
                        const float2 v = e < n ? warp_list[src * CAP + e] : make_float2(neg_inf(), __uint_as_float(INVALID_ID));
                        p.part_sc[to + e] = v.x;
                        p.part_id[to + e] = __float_as_uint(v.y);
                    }
                }
                __syncwarp();
                if (tau > tau_in) __stcg(p.tau + qrow, tau);
                continue;
            }
            if (GP) {
                // the pools already are the published buffers
                p.part_cnt[(qrow * p.nsplit + split) * NWG + wg] = cnt;
                p.part_tau[(qrow * p.nsplit + split) * NWG + wg] = tau;
                if (tau > tau_in) __stcg(p.tau + qrow, tau);
                if (qidx >= 0 && tau > tau_in) atomic_max_f32(p.tau_q + qidx, tau);
                continue;
            }
            __syncwarp();
            const float2* warp_pool = reinterpret_cast<const float2*>(pool_sc) + warp * 32 * PSTR;
#pragma unroll 1
            for (int src = 0; src < 32; ++src) {
                const int n = __shfl_sync(FULL_MASK, cnt, src);
                const float2* row = warp_pool + src * PSTR;
                const int64_t q = (int64_t)qt * TC_BM + quarter * 32 + src;
                const int64_t o = ((q * p.nsplit + split) * NWG + wg) * PUB;
#pragma unroll
                for (int e = lane; e < PUB; e += 32) {
                    const float2 v = e < n ? row[e] : make_float2(neg_inf(), __uint_as_float(INVALID_ID));
                    p.part_sc[o + e] = v.x;
                    p.part_id[o + e] = __float_as_uint(v.y);
                }
            }
            p.part_tau[(qrow * p.nsplit + split) * NWG + wg] = tau;
            if (tau > tau_in) __stcg(p.tau + qrow, tau);
            if (qidx >= 0 && tau > tau_in) atomic_max_f32(p.tau_q + qidx, tau);
        }
        TC_PROF(
        if (warp == 0 && lane == 0 && blockIdx.x < 160) {
            unsigned long long* pr = g_tc_prof + blockIdx.x * TC_PROF_WORDS;
            pr[3] = prof_tfull; pr[4] = prof_rare; pr[5] = prof_groups; pr[6] = prof_compact; pr[7] = prof_append;
            pr[8] = clock64() - prof_t0; pr[9] = tile_no;
            pr[10] = prof_flush; pr[11] = prof_cc;
        }
        )
    }

    // ------------------------------ common exit ----------------------------------------------
    tc_fence_before_sync();
    __syncthreads();
    if (PAIR) cluster_sync_all();      // neither CTA leaves while the other may still touch its memory
    if (warp == W_MMA) {
        tc_fence_after_sync();
        if (PAIR) tmem_dealloc_pair(tmem_base, 512); else tmem_dealloc(tmem_base, 512);
    }
}

// What a seeded threshold is lowered by (all lanes of a warp): twice the scoring error bound plus the proof's slack.
__device__ __forceinline__ float tc_seed_margin(const TcSeedMargin& mg, int64_t row) {
    float qsq = 0.f, lost = 0.f;
    const void* qp = row_at(mg.q, row, mg.ldq, mg.dt);
    for (int c = threadIdx.x & 31; c < mg.d; c += 32) {
        const float x = ld_elem(qp, c, mg.dt), l = bf16_lost(x);
        qsq += x * x;
        lost += l * l;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        qsq += __shfl_xor_sync(FULL_MASK, qsq, o);
        lost += __shfl_xor_sync(FULL_MASK, lost, o);
    }
    return 2.f * score_eps(OPERANDS_BF16, qsq, lost, 0.f, mg.norms, mg.acc) + proof_slack(qsq, __ldg(mg.norms + NORM_ROW), mg.d);
}

// Starting threshold of every query row from the seeding pass: the `rank`-th largest of the
// row's 32 class maxima (16 column classes x 2 warpgroups, disjoint sets of database rows).  At
// least `rank` distinct rows reach it, and being an order statistic of many classes it scatters
// far less than the smallest of a few maxima.  One warp per row, lane = class.
//
// With a margin (row-sharded databases: the class maxima are the element-wise maximum over all
// shards, so the `rank` rows may live on other shards) the threshold is lowered by twice the
// scoring error bound plus the fp32 slack: a row whose score stays at or below
//     cert = pick - 2 score_eps - slack
// is at least as far from the query as each of those `rank` rows, whichever shard holds them,
// so a shard that re-scores every row above `cert` cannot miss a global neighbour.  `cert` is
// also written to mg.cert_out, where the finalisation reads it.
__global__ void __launch_bounds__(256) tc_seed_select_kernel(const float* __restrict__ seed_cls, float* __restrict__ tau,
                                                             int64_t nq, int rank, const TcSeedMargin mg) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= nq) return;                                 // padding rows keep their +inf
    const float v = __ldg(seed_cls + row * (TC_NWG * 16) + lane);
    // rank of each value among the 32 (ties broken by position): a permutation
    int r = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const float o = __shfl_sync(FULL_MASK, v, j);
        r += (o > v || (o == v && j < lane)) ? 1 : 0;
    }
    const unsigned sel = __ballot_sync(FULL_MASK, r == rank - 1);
    float pick = __shfl_sync(FULL_MASK, v, __ffs(sel) - 1);
    if (mg.q != nullptr) {
        const float margin = tc_seed_margin(mg, row);
        if (pick > neg_inf()) pick -= margin;
        if (lane == 0 && mg.cert_out != nullptr) mg.cert_out[row] = pick;
    }
    if (lane == 0 && pick > neg_inf()) tau[row] = pick;
}

// The same from a sample whose tiles were dealt to several CTAs: every row has nsplit x 32 class maxima of
// disjoint sets of rows, folded to at most 512 (the maximum of several disjoint classes is the maximum
// of their union), and the threshold is a value that at least `rank` of them reach, close to the
// largest such -- so `rank` may go beyond 32, where the one-CTA form above has to make do with 32
// classes.  One warp per query row; rows without a query keep their +inf.
__global__ void __launch_bounds__(256) tc_seed_select_split_kernel(const float* __restrict__ seed_cls, float* __restrict__ tau,
                                                                   int64_t nq, int nsplit, int rank, const TcSeedMargin mg) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= nq) return;
    constexpr int R = 16;
    float v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = neg_inf();
    const float* base = seed_cls + row * (int64_t)nsplit * (TC_NWG * 16) + lane;
    for (int s0 = 0; s0 < nsplit; s0 += R) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (s0 + r < nsplit) v[r] = fmaxf(v[r], __ldg(base + (int64_t)(s0 + r) * (TC_NWG * 16)));
    }
    int b[R], lo = 0x7fffffff, hi = (int)0x80000000, have = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int x = __float_as_int(v[r]);
        b[r] = x >= 0 ? x : (x ^ 0x7fffffff);              // orders like the float
        const bool real = v[r] > -1e37f;                   // neither empty nor padding rows
        have += __popc(__ballot_sync(FULL_MASK, real));
        if (real) { lo = min(lo, b[r]); hi = max(hi, b[r]); }
    }
    if (have < rank) return;
    lo = __reduce_min_sync(FULL_MASK, lo);
    hi = __reduce_max_sync(FULL_MASK, hi);
    for (int it = 0; it < 32 && lo < hi; ++it) {
        const int mid = (int)(((long long)lo + hi + 1) >> 1);
        int c = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) c += __popc(__ballot_sync(FULL_MASK, b[r] >= mid));
        if (c >= rank) lo = mid; else hi = mid - 1;
        if (c >= rank && c <= rank + (rank >> 3) + 1) break;
    }
    float pick = __int_as_float(lo >= 0 ? lo : (lo ^ 0x7fffffff));
    if (mg.q != nullptr) pick -= tc_seed_margin(mg, row);
    // A score equal to the threshold is not kept: one step below it, so that the `rank` rows are.  A norm of NaN or
    // infinity among the rows makes the margin, and an infinite score the step, NaN: no score exceeds that, so
    // the row keeps its -inf.
    pick -= fabsf(pick) * 1.2e-7f;
    if (lane == 0 && pick > neg_inf()) tau[row] = pick;
}

// ---- host side ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess)
            return nullptr;
        fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// 2-D bf16 row-major tensor [rows][cols]; box = box_cols columns x box_rows rows.  box_cols is
// 64 (128-byte rows in shared memory, 128-byte swizzle) or 16 (32-byte rows, 32-byte swizzle).
static int make_map_bf16(CUtensorMap* map, const void* base, int64_t rows, int cols, int box_cols, int box_rows) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) { set_error("cuTensorMapEncodeTiled is not available from the driver"); return FL_ECUDA; }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE,
                    box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_32B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed with code %d", (int)r); return FL_ECUDA; }
    return FL_OK;
}

// Scratch of the list modes: a working list per epilogue thread of every CTA that `items` work items can occupy.
int64_t tc_list_bytes(int64_t items, int k) {
    const int64_t ctas = items < sm_count() ? items : sm_count();
    return ctas * 4 * TC_LIST_NWG * 32 * (TC_QUEUE_BYTES + (tc_knn_big(k) ? TC_BIG_CAP : TC_LIST_CAP) * 8);
}
int tc_knn_big(int k) { return k > 16 ? 1 : 0; }
int tc_pool_size(int k) { return tc_knn_big(k) ? TC_BIG_K1 : TC_LIST_K1; }
int tc_partial_len(int k) { return TC_LIST_NWG * (tc_knn_big(k) ? TC_BIG_PUB : TC_LIST_PUB); }
static int tc_pair_requested();
// Deep pools for plain k <= 16 scoring when the whole database is one range, i.e. a query ends up
// with just two pools: the larger of two 12th-best scores sits too close to the k-th neighbour
// for the proof (a quarter of the rows of a 1M x 1M self-kNN failed it).  With three ranges the
// shallow pools prove every row of the benchmark mixture and are faster.  Needs the 128-feature
// shared-memory budget.
int tc_use_deep_pools(int k, int d_pad, int nsplit) {
    return !tc_knn_big(k) && d_pad <= 128 && nsplit == 1 && tc_pair_requested() <= 0;
}
int tc_deep_pool_size() { return TC_MID_K1; }
int tc_deep_partial_len() { return TC_NWG * TC_MID_PUB; }
int tc_pair_pools_per_range() { return TC_NWG; }
int tc_lists_per_range() { return TC_LIST_NWG; }
int tc_pair_pool_cap(int k) { return tc_knn_big(k) ? TC_BIG_CAP : TC_GP_CAP; }

int tc_knn_supported(int64_t nq, int64_t m, int d, int k) {
    if (nq < 1 || m < 1) return FL_EUNSUPPORTED;
    if (k > 112) return FL_EUNSUPPORTED;            // pools keep 12 (k <= 16) or 128 entries: leave the proof a margin
    if (d > 512) return FL_EUNSUPPORTED;            // resident query tile: up to 8 chunks of 64 features (beyond 4:
                                                    // pools in global memory only, two ring slots at d = 512)
    if (round_up(m, 256) / 256 > (1 << 23)) return FL_EUNSUPPORTED;
    return FL_OK;
}

// (the streamed query tile has no limit of its own; 8 192 features keep the accumulation's part of the error bound at 2^-10)
int tc_wide_supported(int64_t nq, int64_t m, int d, int k) {
    if (d <= 512 || d > 8192 || nq < 1 || k > 112) return 0;
    if (m < 512 || round_up(m, 256) / 256 > (1 << 23)) return 0;
    if (!direct_possible(nq, m, d, k)) return nq * m >= (int64_t(1) << 20);
    return direct_estimate_us(nq, m, d) > 60.0 + (double)m * (double)(round_up(d, 64) + PLANE_AUG_COLS) * 2.0 / 5.5e6;
}

// Auto mode takes the tensor-core path where it is the faster one.  Its dozen launches cost about 60 us
// whatever the size, then a few queries stream the bf16 plane from HBM; the CUDA-core scan for few
// queries has two launches and reads the stored rows once per four queries.
int tc_knn_auto(int64_t nq, int64_t m, int d, int k) {
    if (tc_knn_supported(nq, m, d, k) != FL_OK || m < 512) return 0;
    if (!direct_possible(nq, m, d, k)) return nq * m >= (int64_t(1) << 20);
    const double tc = 60.0 + (double)m * (double)(round_up(d, 64) + PLANE_AUG_COLS) * 2.0 / 5.5e6;
    return direct_estimate_us(nq, m, d) > tc;
}

// CTA pairs (cta_group::2) in the list modes: each CTA of a pair loads half of every database tile, which halves what the
// L2 delivers to the SMs -- one CTA alone asks for 64 bytes a cycle, about all there is (10 000 x 1M x 128: scoring
// 2.16 ms alone, 2.05 in pairs; with an epilogue that only reads the accumulators 1.87 and 1.63).  They need an even
// number of query tiles, so an odd one is padded: 11 % more work at nine tiles, the fewest that come here
// (tc_small), and less from there on.  FLASHLIB_B200_TC_PAIR=0/1 overrides.
static int tc_pair_requested() {
    static int v = -2;
    if (v == -2) { const char* e = getenv("FLASHLIB_B200_TC_PAIR"); v = e ? (atoi(e) != 0 ? 1 : 0) : -1; }
    return v;
}
int tc_pair_enabled(int64_t nq_pad) { return tc_pair_requested() != 0 && (nq_pad / TC_BM) % 2 == 0; }
int64_t tc_query_rows_padded(int64_t nq) {
    const bool even = tc_pair_requested() < 0 ? nq > 8 * TC_BM : tc_pair_requested() != 0;
    return round_up(nq, even ? 2 * TC_BM : TC_BM);
}

void tc_split_plan(int64_t nq_pad, int64_t m_pad, int k, int* nsplit, int64_t* tiles_per_split) {
    const bool pair = tc_pair_enabled(nq_pad) != 0;
    // work units that walk a range together, and how many of them the GPU runs at once
    const int64_t n_qtiles = pair ? nq_pad / TC_BM / 2 : nq_pad / TC_BM;
    const int64_t n_tiles = m_pad / TC_BN;
    const int sms = pair ? sm_count() / 2 : sm_count();
    int64_t max_s = n_tiles / 8;
    if (max_s > 64) max_s = 64;
    if (max_s < 1) max_s = 1;
    // Estimated run time in tile units: every SM works through `waves` items of `tps` tiles plus
    // a fixed cost per item (query tile load, pipeline fill and drain, pool publication).
    constexpr int64_t ITEM_OVERHEAD_TILES = 8;
    int64_t best_cost = -1;
    int64_t best_s = 1;
    for (int64_t s = 1; s <= max_s; ++s) {
        const int64_t tps = ceil_div(n_tiles, s);
        const int64_t s_eff = ceil_div(n_tiles, tps);
        const int64_t items = n_qtiles * s_eff;
        const int64_t grid = items < sms ? items : sms;
        const int64_t waves = ceil_div(items, grid);
        const int64_t cost = waves * (tps + ITEM_OVERHEAD_TILES);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best_s = s_eff; }
    }
    *tiles_per_split = ceil_div(n_tiles, best_s);
    *nsplit = (int)ceil_div(n_tiles, *tiles_per_split);
}

// ---- experiment controls ------------------------------------------------------------------
// Timing experiments and seeding overrides.  The environment is read once, when the first
// tensor-core launch is prepared; fl_debug_tc_experiment changes the flags and the wait limit
// afterwards (tests of the bounded-wait exit).  Launches with experiment flags 1..16 set mark
// the status words (FL_EUNSUPPORTED): their neighbours are not to be used.
struct TcExperiment {
    int flags = 0;
    uint32_t hint_ns = 1000u;
    uint64_t wait_ns = TC_WAIT_DEFAULT_NS;
    int noseed = 0, seed_tiles = -1, seed_rank = -1;
};
static TcExperiment& tc_experiment() {
    static TcExperiment e = [] {
        TcExperiment x;
        if (const char* v = getenv("FLASHLIB_B200_TC_DEBUG")) x.flags = atoi(v);
        if (const char* v = getenv("FLASHLIB_B200_TC_HINT")) x.hint_ns = (uint32_t)atoi(v);
        if (const char* v = getenv("FLASHLIB_B200_TC_NOSEED")) x.noseed = atoi(v) != 0;
        if (const char* v = getenv("FLASHLIB_B200_TC_SEED_TILES")) x.seed_tiles = atoi(v);
        if (const char* v = getenv("FLASHLIB_B200_TC_SEED_RANK")) x.seed_rank = atoi(v);
        return x;
    }();
    return e;
}
int tc_debug_active() { return tc_experiment().flags != 0; }
void tc_debug_set(int flags, unsigned wait_us) {
    TcExperiment& e = tc_experiment();
    e.flags = flags;
    e.wait_ns = wait_us ? (uint64_t)wait_us * 1000ull : TC_WAIT_DEFAULT_NS;
}

// Few query tiles or a small database: such calls are bound by latencies and by the fixed cost of their
// launches, not by the tensor pipe.  They keep their pools in global memory as pairs (mode KNN_GPOOL: no
// pool in shared memory, four ring slots, nothing published at the end of an item), cut the database
// into row ranges so that every SM has one, and finalise with a block per query.  The line, measured
// with k = 10: up to eight query tiles whatever the database (300 queries x 1M rows 402 -> 241 us,
// 1 000 554 -> 460; 3 000 1 240 -> 1 265), beyond that up to 64 tiles of work per SM (10 000 x 100 000
// x 64, 208 tiles per SM: 507 -> 771).
int tc_small(int64_t nq_pad, int64_t m_pad) {
    if (tc_pair_requested() > 0) return 0;
    const int64_t n_qtiles = nq_pad / TC_BM;
    return n_qtiles <= 8 || n_qtiles * (m_pad / TC_BN) <= 64 * (int64_t)sm_count();
}

// Row ranges of such a call: every item costs about four tiles of latency on top of its own.
void tc_small_split(int64_t nq_pad, int64_t m_pad, int* nsplit, int64_t* tiles_per_split) {
    const int64_t n_qtiles = nq_pad / TC_BM, n_tiles = m_pad / TC_BN;
    const int sms = sm_count();
    int64_t max_s = n_tiles / 2;
    if (max_s > sms) max_s = sms;
    if (max_s < 1) max_s = 1;
    int64_t best_cost = -1, best_s = 1;
    for (int64_t s = 1; s <= max_s; ++s) {
        const int64_t tps = ceil_div(n_tiles, s), se = ceil_div(n_tiles, tps);
        const int64_t cost = ceil_div(n_qtiles * se, sms) * (tps + 4);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best_s = se; }
    }
    *tiles_per_split = ceil_div(n_tiles, best_s);
    *nsplit = (int)ceil_div(n_tiles, *tiles_per_split);
}

// Seeding sample of a call that is not part of a row-sharded search: `tiles` tiles dealt to `splits` CTAs per
// query tile (32 class maxima each), and the threshold is a value that `rank` sampled rows reach -- about
// rank n_tiles / tiles rows of the whole database.  The aim is 10 k + 200 of them (k > 16: 6 k + 50): enough that
// the k-th neighbour's error band stays inside, few enough that the pools hardly ever fill.  Rank 24
// holds that figure within a fifth; k + 6 rows are enough for small k.
// `dense`: the sample is an eighth of the database or more, so the threshold cuts close to the k-th
// neighbour: k + 6 rows must reach it, and it is lowered by twice the scoring error bound
// (tc_seed_select_split_kernel).
void tc_seed_plan(int64_t nq_pad, int64_t m_pad, int k, TcSeedPlan* w) {
    const int64_t n_qtiles = nq_pad / TC_BM, n_tiles = m_pad / TC_BN;
    const int sms = sm_count();
    *w = TcSeedPlan{};
    if (tc_experiment().noseed || tc_experiment().seed_tiles >= 0 || tc_experiment().seed_rank >= 0) return;
    w->rank = k + 6 < 24 ? k + 6 : 24;
    const int64_t aim = k <= 16 ? 10 * k + 200 : 6 * k + 50 > 250 ? 6 * k + 50 : 250;
    int64_t tiles = ceil_div(w->rank * n_tiles, aim);
    if (tiles < 16) tiles = 16;
    if (n_qtiles > 8 && k <= 16 && tiles > 192) tiles = 192;      // (the scoring pass of many query tiles tightens them itself)
    if (tiles > n_tiles) tiles = n_tiles;
    w->dense = tiles * 8 >= n_tiles;
    if (w->dense) w->rank = k + 6;
    const int64_t need = ceil_div(w->rank, 2 * 16);              // classes enough for the rank
    int64_t best = -1, best_s = 0;
    for (int64_t s = need > 2 ? need : 2; s <= tiles && s <= sms; ++s) {
        const int64_t per = ceil_div(tiles, s), se = ceil_div(tiles, per);
        if (se < need || se < 2) continue;
        const int64_t cost = ceil_div(n_qtiles * se, sms) * (per + 4);
        if (best < 0 || cost < best) { best = cost; best_s = se; }
    }
    if (best_s == 0) return;                                     // a database of one tile: no seeding
    w->tiles = (int)tiles;
    w->splits = (int)best_s;
}

// Tensor maps are encoded once per (buffer, shape, box) and kept in a small per-thread cache:
// a serving loop calls with the same plane and the same workspace over and over.
struct MapKey { const void* base; int64_t rows; int cols, box_cols, box_rows; };
static int cached_map_bf16(CUtensorMap* map, const void* base, int64_t rows, int cols, int box_cols, int box_rows) {
    constexpr int SLOTS = 16;
    thread_local MapKey keys[SLOTS];
    thread_local CUtensorMap maps[SLOTS];
    thread_local int used = 0, next = 0;
    for (int i = 0; i < used; ++i) {
        const MapKey& k = keys[i];
        if (k.base == base && k.rows == rows && k.cols == cols && k.box_cols == box_cols && k.box_rows == box_rows) {
            *map = maps[i];
            return FL_OK;
        }
    }
    const int rc = make_map_bf16(map, base, rows, cols, box_cols, box_rows);
    if (rc != FL_OK) return rc;
    const int slot = used < SLOTS ? used++ : (next++ % SLOTS);
    keys[slot] = MapKey{base, rows, cols, box_cols, box_rows};
    maps[slot] = *map;
    return FL_OK;
}

int tc_seed_tiles(int64_t m_pad, int k);
struct TcLaunch {
    CUtensorMap map_q, map_q_aug, map_db, map_db_aug;
    TcSmemPlan sp;
    TcKernelParams kp;
    int seed_tiles, seed_rank;
    bool big, mid, gpb;
};

static int tc_last_steps(const TcKnnParams& p) {
    if (p.d_used <= 0) return TC_BK / 16;
    const int rest = p.d_used - (p.d_pad - TC_BK);                 // features in the last chunk
    return rest <= 16 ? 1 : (rest + 15) / 16;
}

// Everything a launch needs: tensor maps, shared-memory plan, kernel parameters and the size of
// the seeding sample.
static int tc_prepare(const TcKnnParams& p, float* dbg, int64_t dbg_ld, TcLaunch* L) {
    FL_CHECK_ARG(p.qplane && p.dbrows && p.tau, "tensor-core kNN launch with a null buffer");
    L->big = (tc_knn_big(p.k) != 0 || p.big_pools != 0) && p.pair_pools == nullptr;
    L->gpb = p.pair_pools != nullptr && tc_knn_big(p.k) != 0;
    L->mid = p.deep_pools != 0;
    const int pitch = p.d_pad + PLANE_AUG_COLS;
    int rc = cached_map_bf16(&L->map_q, p.qplane, p.nq_pad, pitch, TC_BK, TC_BM);
    if (rc == FL_OK) rc = cached_map_bf16(&L->map_q_aug, p.qplane, p.nq_pad, pitch, PLANE_AUG_COLS, TC_BM);
    if (rc == FL_OK) rc = cached_map_bf16(&L->map_db, p.dbrows, p.m_pad, pitch, TC_BK, TC_BN);
    if (rc == FL_OK) rc = cached_map_bf16(&L->map_db_aug, p.dbrows, p.m_pad, pitch, PLANE_AUG_COLS, TC_BN);
    if (rc != FL_OK) return rc;
    FL_CHECK_ARG(!(L->mid && (L->big || dbg)), "tensor-core kNN launch: deep pools go with k <= 16");
    // a query tile of more than 512 features is streamed with the database chunks
    const bool stream = p.d_pad > 512;
    FL_CHECK_ARG(!stream || p.pair_pools != nullptr, "tensor-core kNN launch: more than 512 features go with pair pools");
    L->sp = tc_smem_plan(p.d_pad, smem_optin_bytes(), L->mid ? TC_MID_CAP + 1 : 0,
                         stream ? TC_B_STAGE + TC_STREAM_A : TC_B_STAGE, stream ? 0 : 1);
    if (L->sp.nstage < 2) { set_error("tensor-core kNN: feature dimension %d leaves no room for the TMA ring", p.d_pad); return FL_EUNSUPPORTED; }
    const TcExperiment& ex = tc_experiment();
    TcKernelParams& kp = L->kp;
    kp = TcKernelParams{};
    kp.n_qtiles = (int)(p.nq_pad / TC_BM);
    kp.n_tiles = (int)(p.m_pad / TC_BN);
    kp.nsplit = p.nsplit;
    kp.tiles_per_split = (int)p.tiles_per_split;
    kp.last_steps = tc_last_steps(p); kp.fmt = p.fmt;
    kp.nkc = L->sp.nkc; kp.nstage = L->sp.nstage;
    kp.stream_a = stream ? 1 : 0;
    kp.off_b = L->sp.off_b; kp.off_pool_sc = L->sp.off_pool_sc; kp.off_pool_id = L->sp.off_pool_id;
    kp.off_bar = L->sp.off_bar;
    kp.nq_pad = p.nq_pad; kp.part_sc = p.part_sc; kp.part_id = p.part_id;
    kp.tau = p.tau; kp.part_tau = p.part_tau; kp.status = p.status; kp.dbg_scores = dbg; kp.dbg_ld = dbg_ld;
    kp.part_cnt = p.part_cnt;
    kp.gpool = reinterpret_cast<float2*>(p.pair_pools);
    kp.lists = p.lists;
    kp.seed_cls = p.seed_cls;
    kp.nq_dev = p.nq_dev; kp.item_t0 = p.item_t0; kp.item_t1 = p.item_t1; kp.item_order = p.item_order;
    kp.row_query = p.row_query; kp.tau_q = p.tau_q;
    kp.dbg_flags = ex.flags;
    kp.wait_hint_ns = ex.hint_ns;
    kp.wait_ns = ex.wait_ns;
    kp.tile_stride = 1;
    // Seeding sample.  The threshold is the seed_rank-th largest of 32 class maxima, which sits
    // near rank 32 ln(32 / (32 - seed_rank)) of the sample, hence near that figure times
    // n_tiles / seed_tiles of the whole database.
    //  k <= 16: the pools tighten the threshold quickly; one tile in 16 (at most 64 tiles, 192 for the
    //           largest databases), k + 6 rows guaranteed.
    //  large k: the pools seldom fill, so the seeded threshold is what filters.  Aim at about
    //           rank 6 k of the database: loose enough that the k-th neighbour's error band
    //           stays inside, tight enough that a few hundred rows per query are published.
    int seed_rank = p.k + 6 < 32 ? p.k + 6 : 32;
    if (L->big) seed_rank = p.k >= 64 ? 16 : 8;
    if (ex.seed_rank >= 0) seed_rank = ex.seed_rank;
    if (seed_rank < 1) seed_rank = 1;
    if (seed_rank > 32) seed_rank = 32;
    const int seed_tiles = tc_seed_tiles(p.m_pad, p.k);
    L->seed_tiles = seed_tiles;
    L->seed_rank = seed_rank;
    return FL_OK;
}

// Database tiles the seeding pass samples (0: no seeding for this shape).
int tc_seed_tiles(int64_t m_pad, int k) {
    const int n_tiles = (int)(m_pad / TC_BN);
    const TcExperiment& ex = tc_experiment();
    // one tile in 16, at most 64 -- 192 for the largest databases (measured on 3 907 tiles x 10 000
    // queries: 64 tiles 2.490 ms per step, 96 2.455, 128 2.385, 192 2.361, 256 2.391; on 489-tile shards x 80 000
    // queries, with the epilogue of before, the 30 tiles of the rule beat 16 and 48)
    int seed_tiles = n_tiles >= 3072 ? 192 : n_tiles >= 1024 ? 64 : n_tiles / 16;

    if (tc_knn_big(k)) {
        const double sample_rank = k >= 64 ? 22.2 : 9.2;
        seed_tiles = (int)((double)n_tiles * sample_rank / (6.0 * k));
        if (seed_tiles > n_tiles / 8) seed_tiles = n_tiles / 8;
        if (seed_tiles > n_tiles / 2) seed_tiles = n_tiles / 2;
        if (seed_tiles < 16) seed_tiles = 0;
    } else if (n_tiles < 256) {
        // Small databases (k <= 16): a cold pool costs a fixed few dozen insertions and compactions
        // per query row, which dwarfs the scoring of a handful of tiles (the coarse probe of an
        // inverted-file search scores 4).  Sample 16 tiles, or simply all of them: the threshold
        // is then tight, so the selection lowers it by the proof's margin (tc_seed_dense).
        seed_tiles = n_tiles < 16 ? n_tiles : 16;
    }
    if (ex.seed_tiles >= 0) seed_tiles = ex.seed_tiles < n_tiles ? ex.seed_tiles : n_tiles;
    if (ex.noseed) seed_tiles = 0;
    return seed_tiles;
}
// 1 when the seeding sample is a large share of the database: a threshold that k + 6 sampled rows
// reach then cuts close to the k-th neighbour, and must be lowered by twice the scoring error bound
// for the finalisation's proof to hold (see tc_seed_select_kernel).
int tc_seed_dense(int64_t m_pad, int k) {
    const int n_tiles = (int)(m_pad / TC_BN);
    return !tc_knn_big(k) && n_tiles < 256 && tc_seed_tiles(m_pad, k) > 0;
}

// Seeding pass: class maxima of a strided sample of the database tiles into p.seed_cls
// ([nq_pad][32]).  Without a sample (database too small) the maxima are set to -inf.
int launch_knn_tc_seed(const TcKnnParams& p, cudaStream_t st) {
    FL_CHECK_ARG(p.seed_cls != nullptr, "tensor-core seeding pass without a class buffer");
    TcLaunch L;
    int rc = tc_prepare(p, nullptr, 0, &L);
    if (rc != FL_OK) return rc;
    TcKernelParams sk = L.kp;
    sk.dbg_scores = nullptr;
    sk.row_query = nullptr; sk.tau_q = nullptr;
    if (p.item_t0 != nullptr) {
        // item tables (inverted-file scan): the first item_tile_cap tiles of every item's own range
        FL_CHECK_ARG(p.item_tile_cap > 0 && p.nsplit == 1, "tensor-core seeding over item tables needs a tile cap");
        sk.item_tile_cap = p.item_tile_cap;
    } else {
        const int tiles = p.seed_tiles > 0 ? p.seed_tiles : L.seed_tiles;
        if (tiles == 0) return launch_fill_f32(p.seed_cls, p.nq_pad * (TC_NWG * 16), -INFINITY, st);
        sk.nsplit = p.seed_splits > 1 ? p.seed_splits : 1;
        sk.tiles_per_split = (int)ceil_div(tiles, sk.nsplit);
        sk.tile_stride = L.kp.n_tiles / tiles;
        sk.n_tiles = tiles;
        sk.nq_dev = nullptr;
    }
    // the seeding kernel keeps no pools: the ring gets the shared memory the pools would take
    const TcSmemPlan sp = L.sp;
    const int sitems = sk.n_qtiles * sk.nsplit;
    const int sgrid = sitems < sm_count() ? sitems : sm_count();
    FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_SEED>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
    knn_tc_kernel<false, TC_MODE_SEED><<<sgrid, TC_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, sk);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

// Starting thresholds from class maxima (this shard's, or the element-wise maximum over all
// shards of a sharded database): see tc_seed_select_kernel.
int launch_knn_tc_seed_select(const TcKnnParams& p, const TcSeedMargin& mg, cudaStream_t st) {
    FL_CHECK_ARG(p.seed_cls != nullptr && p.tau != nullptr, "tensor-core threshold selection without buffers");
    if (p.seed_splits > 1) {
        tc_seed_select_split_kernel<<<(unsigned)ceil_div(p.nq, 8), 256, 0, st>>>(p.seed_cls, p.tau, p.nq, p.seed_splits, p.seed_rank, mg);
        FL_CHECK_LAUNCH();
        return FL_OK;
    }
    TcLaunch L;
    int rc = tc_prepare(p, nullptr, 0, &L);
    if (rc != FL_OK) return rc;
    tc_seed_select_kernel<<<(unsigned)ceil_div(p.nq, 8), 256, 0, st>>>(p.seed_cls, p.tau, p.nq, L.seed_rank, mg);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

// Main scoring launch (thresholds in p.tau as they stand).
static int launch_tc_main(const TcKnnParams& p, float* dbg, int64_t dbg_ld, cudaStream_t st) {
    const bool gp = p.pair_pools != nullptr;
    FL_CHECK_ARG(p.part_tau && (gp ? p.part_cnt != nullptr : (p.part_sc && p.part_id && (p.lists || p.deep_pools))), "tensor-core kNN launch with a null buffer");
    TcLaunch L;
    int rc = tc_prepare(p, dbg, dbg_ld, &L);
    if (rc != FL_OK) return rc;
    const bool big = L.big, mid = L.mid;
    FL_CHECK_ARG(!gp || !dbg, "tensor-core kNN launch: no score dump with global pair pools");
    FL_CHECK_ARG(!big || (p.part_cnt && !dbg), "tensor-core kNN launch (large k) without a count buffer");
    FL_CHECK_ARG((p.row_query == nullptr) == (p.tau_q == nullptr), "tensor-core kNN launch: row_query and tau_q go together");
    FL_CHECK_ARG((p.item_t0 == nullptr) == (p.item_t1 == nullptr) && (p.item_t0 == nullptr || (p.nsplit == 1 && !big)),
                 "tensor-core kNN launch: per-tile ranges need one range per query tile and k <= 16");
    const TcKernelParams& kp = L.kp;
    const TcSmemPlan& sp = L.sp;
    const int pitch = p.d_pad + PLANE_AUG_COLS;
    const int items = kp.n_qtiles * kp.nsplit;
    const int grid = items < sm_count() ? items : sm_count();
    // CTA pairs (cta_group::2): list modes and streamed query tiles over uniform ranges, an even number of query tiles.  A
    // streamed chunk of 64 features is 48 KB for 512 cycles of MMA; in a pair each CTA loads 32, which leaves room for
    // five ring slots in place of three (2 000 x 200 000 x 768 in bf16: 996 -> 662 us, scoring 814 -> 493).
    const bool stream = kp.stream_a != 0;
    const bool pair = (!gp || stream) && !mid && dbg == nullptr && p.item_t0 == nullptr && p.nq_dev == nullptr &&
                      tc_pair_enabled(p.nq_pad);
    if (pair) {
        CUtensorMap map_db_h, map_db_aug_h;
        rc = cached_map_bf16(&map_db_h, p.dbrows, p.m_pad, pitch, TC_BK, TC_BN / 2);
        if (rc == FL_OK) rc = cached_map_bf16(&map_db_aug_h, p.dbrows, p.m_pad, pitch, PLANE_AUG_COLS, TC_BN / 2);
        if (rc != FL_OK) return rc;
        const TcSmemPlan spp = tc_smem_plan(p.d_pad, smem_optin_bytes(), 0, TC_B_STAGE / 2 + (stream ? TC_STREAM_A : 0), stream ? 0 : 1);
        TcKernelParams kq = kp;
        kq.nstage = spp.nstage; kq.off_b = spp.off_b; kq.off_pool_sc = spp.off_pool_sc; kq.off_pool_id = spp.off_pool_id;
        kq.off_bar = spp.off_bar;
        const int pair_items = (kp.n_qtiles / 2) * kp.nsplit;
        int clusters = sm_count() / 2;
        if (clusters > pair_items) clusters = pair_items;
        auto kern = L.gpb ? knn_tc_kernel<false, TC_MODE_KNN_GPOOL_BIG, true>
                  : gp  ? knn_tc_kernel<false, TC_MODE_KNN_GPOOL, true>
                  : big ? knn_tc_kernel<false, TC_MODE_KNN_BIG, true>
                        : kp.dbg_flags != 0 ? knn_tc_kernel<true, TC_MODE_KNN, true> : knn_tc_kernel<false, TC_MODE_KNN, true>;
        FL_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, spp.bytes));
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(2 * clusters));
        cfg.blockDim = dim3(gp ? TC_THREADS : TC_LIST_THREADS);
        cfg.dynamicSmemBytes = (size_t)spp.bytes;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        FL_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, L.map_q, L.map_q_aug, map_db_h, map_db_aug_h, kq));
    } else if (L.gpb) {
        FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_KNN_GPOOL_BIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
        knn_tc_kernel<false, TC_MODE_KNN_GPOOL_BIG><<<grid, TC_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, kp);
    } else if (gp) {
        FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_KNN_GPOOL>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
        knn_tc_kernel<false, TC_MODE_KNN_GPOOL><<<grid, TC_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, kp);
    } else if (mid) {
        FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_KNN_MID>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
        knn_tc_kernel<false, TC_MODE_KNN_MID><<<grid, TC_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, kp);
    } else if (big) {
        FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_KNN_BIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
        knn_tc_kernel<false, TC_MODE_KNN_BIG><<<grid, TC_LIST_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, kp);
    } else if (dbg != nullptr || kp.dbg_flags != 0) {
        FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<true, TC_MODE_KNN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
        knn_tc_kernel<true, TC_MODE_KNN><<<grid, TC_LIST_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, kp);
    } else {
        FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_KNN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
        knn_tc_kernel<false, TC_MODE_KNN><<<grid, TC_LIST_THREADS, sp.bytes, st>>>(L.map_q, L.map_q_aug, L.map_db, L.map_db_aug, kp);
    }
    FL_CHECK_LAUNCH();
    return FL_OK;
}

// Seeding (when p.seed_cls is given and the database is large enough for it to matter), threshold
// selection and the main scoring launch.
static int launch_tc_impl(const TcKnnParams& p, float* dbg, int64_t dbg_ld, cudaStream_t st) {
    if (p.seed_cls != nullptr && tc_seed_tiles(p.m_pad, p.k) > 0) {
        int rc = launch_knn_tc_seed(p, st);
        if (rc != FL_OK) return rc;
        rc = launch_knn_tc_seed_select(p, TcSeedMargin{}, st);
        if (rc != FL_OK) return rc;
    }
    return launch_tc_main(p, dbg, dbg_ld, st);
}
int launch_knn_tc_scoring(const TcKnnParams& p, cudaStream_t st) { return launch_tc_main(p, nullptr, 0, st); }

// FLASHLIB_B200_ASSIGN_SINGLE_A=1: one query-tile buffer in the assignment launches (measurements).
static int tc_assign_single_a() {
    static int v = -1;
    if (v < 0) { const char* e = getenv("FLASHLIB_B200_ASSIGN_SINGLE_A"); v = (e && atoi(e) != 0) ? 1 : 0; }
    return v;
}

int tc_prof_read(unsigned long long* host_out, int words) {
    const size_t n = sizeof(unsigned long long) * (size_t)(words < 160 * TC_PROF_WORDS ? words : 160 * TC_PROF_WORDS);
    FL_CHECK_CUDA(cudaMemcpyFromSymbol(host_out, g_tc_prof, n));
    return FL_OK;
}

// Assignment launch: queries = sample rows, database = centroids; writes per (row, warpgroup)
// the best and second-best score and the best centroid.
int launch_assign_tc(const TcKnnParams& p, float* asg_sc, uint32_t* asg_id, const int* nq_dev, cudaStream_t st,
                     const int* asg_rows) {
    FL_CHECK_ARG(p.qplane && p.dbrows && asg_sc && asg_id && (nq_dev || !asg_rows), "tensor-core assignment launch with a null buffer");
    CUtensorMap map_q, map_q_aug, map_db, map_db_aug;
    const int pitch = p.d_pad + PLANE_AUG_COLS;
    int rc = make_map_bf16(&map_q, p.qplane, p.nq_pad, pitch, TC_BK, TC_BM);
    if (rc == FL_OK) rc = make_map_bf16(&map_q_aug, p.qplane, p.nq_pad, pitch, PLANE_AUG_COLS, TC_BM);
    if (rc == FL_OK) rc = make_map_bf16(&map_db, p.dbrows, p.m_pad, pitch, TC_BK, TC_BN);
    if (rc == FL_OK) rc = make_map_bf16(&map_db_aug, p.dbrows, p.m_pad, pitch, PLANE_AUG_COLS, TC_BN);
    if (rc != FL_OK) return rc;
    // Items are short here (a query tile against a handful of centroid tiles): with room for a second
    // query-tile buffer beside a three-slot ring the next item's tile is loaded while this one is scored.
    TcSmemPlan sp = tc_smem_plan(p.d_pad, smem_optin_bytes(), 0, TC_B_STAGE, 2);
    int nabuf = 2;
    if (sp.nstage < 3 || tc_assign_single_a()) { sp = tc_smem_plan(p.d_pad, smem_optin_bytes(), 0); nabuf = 1; }
    if (sp.nstage < 2) { set_error("tensor-core assignment: feature dimension %d leaves no room for the TMA ring", p.d_pad); return FL_EUNSUPPORTED; }
    TcKernelParams kp{};
    kp.nabuf = nabuf;
    kp.n_qtiles = (int)(p.nq_pad / TC_BM);
    kp.n_tiles = (int)(p.m_pad / TC_BN);
    kp.nsplit = 1;
    kp.tiles_per_split = kp.n_tiles;
    kp.last_steps = tc_last_steps(p); kp.fmt = p.fmt;
    kp.nkc = sp.nkc; kp.nstage = sp.nstage;
    kp.off_b = sp.off_b; kp.off_pool_sc = sp.off_pool_sc; kp.off_pool_id = sp.off_pool_id; kp.off_bar = sp.off_bar;
    kp.nq_pad = p.nq_pad; kp.status = p.status;
    kp.asg_rows = asg_rows; kp.asg_sc = asg_sc; kp.asg_id = asg_id;
    kp.nq_dev = nq_dev;
    kp.tile_stride = 1; kp.wait_hint_ns = tc_experiment().hint_ns;
    kp.wait_ns = tc_experiment().wait_ns;      // (a limit of zero gives up after a few microseconds of waiting)
    const int grid = kp.n_qtiles < sm_count() ? kp.n_qtiles : sm_count();
    FL_CHECK_CUDA(cudaFuncSetAttribute(knn_tc_kernel<false, TC_MODE_ASSIGN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp.bytes));
    knn_tc_kernel<false, TC_MODE_ASSIGN><<<grid, TC_THREADS, sp.bytes, st>>>(map_q, map_q_aug, map_db, map_db_aug, kp);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

int launch_knn_tc(const TcKnnParams& p, cudaStream_t st) { return launch_tc_impl(p, nullptr, 0, st); }
int launch_knn_tc_debug(const TcKnnParams& p, float* dbg, int64_t dbg_ld, cudaStream_t st) {
    return launch_tc_impl(p, dbg, dbg_ld, st);
}

}  // namespace fl
