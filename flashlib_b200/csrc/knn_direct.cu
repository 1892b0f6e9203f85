// Exact kNN for few queries: every database row is read once per group of up to four queries and
// scored by its fp32 sum (q - x)^2 straight from the stored values -- no norms, no operand plane,
// no error bound.  Two launches: a scan that leaves the k best of every (query, row range) and a
// merge that orders them and writes the answer.  The same scan, one query per block over the rows
// of one inverted list, serves small inverted-file searches.
//
// Bound: HBM for one query (the rows are read once: 1M x 128 in 134 us, 3.8 TB/s), the FP32 pipe from two groups on.
// The CUDA-core tile kernel (knn_simt.cu) works in tiles of 64 queries: one query costs it as much as
// 64, and its row ranges stop at 64 blocks.
#include "knn_internal.h"
#include "pool.cuh"
#include <math.h>

namespace fl {

constexpr int DIR_WARPS = 8, DIR_THREADS = 32 * DIR_WARPS;

// VEC consecutive elements of a row as fp32 (VEC: 4 or 1 for fp32 rows, 8 or 1 for 16-bit rows).
template <bool F32, int VEC>
__device__ __forceinline__ void dir_load(const char* row, int f, int dt, float (&v)[VEC]) {
    if (F32) {
        if (VEC == 4) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(row + (int64_t)f * 4));
            v[0] = t.x; v[1 % VEC] = t.y; v[2 % VEC] = t.z; v[3 % VEC] = t.w;
        } else {
            v[0] = __ldg(reinterpret_cast<const float*>(row) + f);
        }
    } else {
        if (VEC == 8) {
            const uint4 t = __ldg(reinterpret_cast<const uint4*>(row + (int64_t)f * 2));
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (dt == DT_BF16) {
                    v[(2 * i) % VEC] = __uint_as_float(w[i] << 16);
                    v[(2 * i + 1) % VEC] = __uint_as_float(w[i] & 0xffff0000u);
                } else {
                    v[(2 * i) % VEC] = f16_bits_to_f32((unsigned short)(w[i] & 0xffffu));
                    v[(2 * i + 1) % VEC] = f16_bits_to_f32((unsigned short)(w[i] >> 16));
                }
            }
        } else {
            v[0] = ld_elem(row, f, dt);
        }
    }
}

// The next float below a key <= 0: a threshold that keys equal to t still pass.
__device__ __forceinline__ float dir_step_below(float t) {
    return __int_as_float(t == 0.f ? (int)0x80000001 : __float_as_int(t) + 1);
}

// Cuts a pool to its k best (equal keys: lowest rows first) and returns the k-th key, -inf while there
// are fewer.  Out of line: rare, and the sorting network is large.
template <int N>
static __device__ __noinline__ float dir_compact(float* sc, uint32_t* id, int cnt, int k) {
    const int lane = threadIdx.x & 31;
    float key[N];
    uint32_t row[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const int e = (r << 5) | lane;
        key[r] = e < cnt ? sc[e] : neg_inf();
        row[r] = e < cnt ? id[e] : INVALID_ID;
    }
    warp_sort_desc<N, true>(key, row);
    float kth = neg_inf();
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const int e = (r << 5) | lane;
        if (e < k) { sc[e] = key[r]; id[e] = row[r]; }
        if (((k - 1) >> 5) == r) kth = __shfl_sync(FULL_MASK, key[r], (k - 1) & 31);
    }
    __syncwarp();
    return kth;
}

// The k best of the eight pools of a query (`stride` entries apart, counts cstride apart, `total` entries
// in all), sorted by one warp and written out (-inf / INVALID_ID padded).
template <int N>
__device__ __forceinline__ void dir_sort_out(const float* key, const uint32_t* id, int stride, const int* cnt, int cstride,
                                             int total, int k, float* out_key, uint32_t* out_id) {
    const int lane = threadIdx.x & 31;
    float ka[N];
    uint32_t ia[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        int e = (r << 5) | lane, w = 0;
        const bool in = e < total;
        while (in && e >= cnt[w * cstride]) { e -= cnt[w * cstride]; ++w; }
        ka[r] = in ? key[w * stride + e] : neg_inf();
        ia[r] = in ? id[w * stride + e] : INVALID_ID;
    }
    warp_sort_desc<N, true>(ka, ia);
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const int e = (r << 5) | lane;
        if (e < k) { out_key[e] = ka[r]; out_id[e] = ia[r]; }
    }
}

template <int NPL>
static __device__ __noinline__ void dir_collect(float* key, uint32_t* id, int stride, const int* cnt, int cstride, int total,
                                                int k, float* out_key, uint32_t* out_id) {
    const int lane = threadIdx.x & 31;
    if (total <= 32 * NPL) { dir_sort_out<NPL>(key, id, stride, cnt, cstride, total, k, out_key, out_id); return; }
    if (total <= 64 * NPL) { dir_sort_out<2 * NPL>(key, id, stride, cnt, cstride, total, k, out_key, out_id); return; }
    // too many for one sort: pool after pool
    float ka[NPL];
    uint32_t ia[NPL];
#pragma unroll
    for (int r = 0; r < NPL; ++r) { ka[r] = neg_inf(); ia[r] = INVALID_ID; }
    for (int w = 0; w < DIR_WARPS; ++w) {
        dir_compact<2 * NPL>(key + w * stride, id + w * stride, cnt[w * cstride], k);
        float kb[NPL];
        uint32_t ib[NPL];
#pragma unroll
        for (int r = 0; r < NPL; ++r) {
            const int e = (r << 5) | lane;
            kb[r] = e < k ? key[w * stride + e] : neg_inf();
            ib[r] = e < k ? id[w * stride + e] : INVALID_ID;
        }
        warp_merge_desc<NPL, true>(ka, ia, kb, ib);
    }
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
        const int e = (r << 5) | lane;
        if (e < k) { out_key[e] = ka[r]; out_id[e] = ia[r]; }
    }
}

// A key that at least k of the up to 256 keys (eight per lane, -inf where there is none) reach, close
// to the largest such: bisection over the keys' order-preserving integer image.  -inf when fewer
// than k keys exist.  Keys of -inf and NaN do not count.
static __device__ __noinline__ float dir_first_threshold(const float* keys, int k) {
    const int lane = threadIdx.x & 31;
    int v[8], lo = 0x7fffffff, hi = (int)0x80000000, have = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const float x = keys[r * 32 + lane];
        const int b = __float_as_int(x);
        const bool real = x > neg_inf();                  // (a NaN would order by its sign: not counted below either)
        v[r] = real ? (b >= 0 ? b : (b ^ 0x7fffffff)) : (int)0x80000000;      // orders like the float
        have += __popc(__ballot_sync(FULL_MASK, real));
        if (real) { lo = min(lo, v[r]); hi = max(hi, v[r]); }
    }
    if (have < k) return neg_inf();
    lo = __reduce_min_sync(FULL_MASK, lo);
    hi = __reduce_max_sync(FULL_MASK, hi);
    // count(>= lo) >= k throughout; stop when the count is close to k or the interval is closed
    for (int it = 0; it < 32 && lo < hi; ++it) {
        const int mid = (int)(((long long)lo + hi + 1) >> 1);
        int c = 0;
#pragma unroll
        for (int r = 0; r < 8; ++r) c += __popc(__ballot_sync(FULL_MASK, v[r] >= mid));
        if (c >= k) lo = mid; else hi = mid - 1;
        if (c >= k && c <= k + (k >> 3) + 1) break;
    }
    return __int_as_float(lo >= 0 ? lo : (lo ^ 0x7fffffff));
}

// Scan.  Eight lanes share a row (lane % 8 = 16-byte piece of a 128-byte stretch), so a warp reads four
// rows per load instruction and 32 rows per pass over the features with eight loads in flight; the
// partial sums of the eight lanes are folded by recursive halving (seven shuffles for eight rows),
// which leaves one row's distance per lane.  A (warp, query) keeps a pool of 64 NPL entries in
// shared memory (k <= 32 NPL): a distance below the threshold is appended, a full pool is cut to its
// k best and the threshold (shared by the block's warps) rises to the k-th.  The block's first 256
// keys are looked at together before any is kept: a key that k of them reach is the threshold
// from then on, so that the pools hardly ever fill -- without it every warp sorts its way
// down from an empty pool, and four queries over 1M x 128 rows took 176 us in place of 133.
//
// Blocks an SM holds: four of one query and rows read four values at a time, whose eight loads a thread are then 128 KB in
// flight (1M x 128: scan 124 us with two blocks and the next eight loads hoisted over the folding, 117 so; 4.4 TB/s).
constexpr int dir_blocks(int nq, int npl, int vec) { return nq == 1 && npl == 1 && vec <= 4 ? 4 : 2; }
template <int NQ, int NPL, bool F32, int VEC>
__global__ void __launch_bounds__(DIR_THREADS, dir_blocks(NQ, NPL, VEC)) direct_scan_kernel(const DirectParams p) {
    extern __shared__ __align__(16) float dir_smem[];
    constexpr int STEP = 8 * VEC;
    const int dq = (p.d + STEP - 1) / STEP * STEP;         // query pitch in shared memory, zero padded
    float* s_q = dir_smem;
    float* s_sc = s_q + NQ * dq;                           // [warp][query][cap]
    constexpr int cap = NPL * 64;
    uint32_t* s_id = reinterpret_cast<uint32_t*>(s_sc + DIR_WARPS * NQ * cap);
    __shared__ float s_thr[NQ];
    __shared__ int s_cnt[DIR_WARPS][NQ];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sl = lane & 7, g = lane >> 3;

    const char* db = static_cast<const char*>(p.db);
    const char* q = static_cast<const char*>(p.q);
    int64_t r0, r1, list;          // rows of this block; list = output list of query 0 (queries p.nlists apart)
    int64_t q0;
    int nqb;
    constexpr int ES = F32 ? 4 : 2;
    if (p.probed != nullptr) {
        const int64_t pair = blockIdx.x / p.nchunk;
        const int chunk = (int)(blockIdx.x - pair * p.nchunk);
        q0 = pair / p.nprobe;
        nqb = 1;
        list = pair * p.nchunk + chunk;
        const int c = __ldg(p.probed + pair);
        r0 = r1 = 0;
        if (c >= 0 && c < p.ivf_nlist) {
            const int64_t a = __ldg(p.list_offsets + c), b = __ldg(p.list_offsets + c + 1);
            const int64_t per = ((b - a + p.nchunk - 1) / p.nchunk + 31) / 32 * 32;
            r0 = a + chunk * per < b ? a + chunk * per : b;
            r1 = r0 + per < b ? r0 + per : b;
        }
    } else {
        const int64_t groups = (p.nq + NQ - 1) / NQ;
        const int chunk = (int)(blockIdx.x / groups);
        q0 = (int64_t)(blockIdx.x - chunk * groups) * NQ;
        nqb = (int)(p.nq - q0 < NQ ? p.nq - q0 : NQ);
        r0 = (int64_t)chunk * p.rows_per_chunk;
        r1 = r0 + p.rows_per_chunk < p.m ? r0 + p.rows_per_chunk : p.m;
        list = q0 * p.nchunk + chunk;
    }
    for (int i = tid; i < NQ * dq; i += DIR_THREADS) {
        const int qi = i / dq, f = i - qi * dq;
        float v = 0.f;
        if (qi < nqb && f < p.d) v = ld_elem(q + (q0 + qi) * p.ldq * ES, f, p.dt);
        s_q[i] = v;
    }
    if (tid < NQ) s_thr[tid] = neg_inf();
    __syncthreads();

    float thr[NQ];
    int cnt[NQ];
#pragma unroll
    for (int qi = 0; qi < NQ; ++qi) { thr[qi] = neg_inf(); cnt[qi] = 0; }
    float* my_sc = s_sc + warp * NQ * cap;
    uint32_t* my_id = s_id + warp * NQ * cap;
    const int64_t rstep = 4 * p.ldb * ES;                  // bytes between the rows of consecutive loads
    const unsigned below = (1u << lane) - 1u;

    // (every warp makes the first pass, rows or not: the block meets there)
    bool first = true;
    for (int64_t base = r0 + warp * 32; first || base < r1; base += DIR_THREADS) {
        float acc[8][NQ];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int qi = 0; qi < NQ; ++qi) acc[j][qi] = 0.f;
        const char* row = db + (base + g) * p.ldb * ES;
        const int left = (int)(r1 - base < 32 ? r1 - base : 32);   // rows of this pass (none: <= 0)
#pragma unroll (NQ <= 2 && dir_blocks(NQ, NPL, VEC) == 2 ? 2 : 1)
        for (int f0 = 0; f0 < dq; f0 += STEP) {
            const int f = f0 + sl * VEC;
            const bool in = f < p.d;
            float x[8][VEC];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
#pragma unroll
                for (int t = 0; t < VEC; ++t) x[j][t] = 0.f;
                if (in && j * 4 + g < left) dir_load<F32, VEC>(row + j * rstep, f, p.dt, x[j]);
            }
#pragma unroll
            for (int qi = 0; qi < NQ; ++qi) {
                float qv[VEC];
#pragma unroll
                for (int t = 0; t < VEC; ++t) qv[t] = s_q[qi * dq + f + t];
#pragma unroll
                for (int j = 0; j < 8; ++j)
#pragma unroll
                    for (int t = 0; t < VEC; ++t) {
                        const float df = qv[t] - x[j][t];
                        acc[j][qi] = fmaf(df, df, acc[j][qi]);
                    }
            }
        }
        const int off = sl * 4 + g;                        // row of this lane after the fold
        const bool valid = off < left;
        float key[NQ];
#pragma unroll
        for (int qi = 0; qi < NQ; ++qi) {
            // fold the eight lanes of a row: lane sl ends with the sum of load sl
            float a4[4], a2[2];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float give = (sl & 4) ? acc[j][qi] : acc[j + 4][qi];
                const float keep = (sl & 4) ? acc[j + 4][qi] : acc[j][qi];
                a4[j] = keep + __shfl_xor_sync(FULL_MASK, give, 4);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float give = (sl & 2) ? a4[j] : a4[j + 2];
                const float keep = (sl & 2) ? a4[j + 2] : a4[j];
                a2[j] = keep + __shfl_xor_sync(FULL_MASK, give, 2);
            }
            const float give = (sl & 1) ? a2[0] : a2[1];
            const float keep = (sl & 1) ? a2[1] : a2[0];
            key[qi] = -(keep + __shfl_xor_sync(FULL_MASK, give, 1));
            key[qi] = valid && qi < nqb ? key[qi] : neg_inf();
        }
        if (first) {
            first = false;
            float* s_first = s_sc;                         // [query][256]: the pools are still empty
#pragma unroll
            for (int qi = 0; qi < NQ; ++qi) s_first[qi * DIR_THREADS + tid] = key[qi];
            __syncthreads();
            if (warp < NQ) {
                const float t = dir_first_threshold(s_first + warp * DIR_THREADS, p.k);
                if (lane == 0 && t > neg_inf()) s_thr[warp] = dir_step_below(t);
            }
            __syncthreads();
        }
#pragma unroll
        for (int qi = 0; qi < NQ; ++qi) {
            const float t = fmaxf(thr[qi], *reinterpret_cast<volatile float*>(s_thr + qi));
            const bool pass = key[qi] > t;
            const unsigned mask = __ballot_sync(FULL_MASK, pass);
            if (mask) {
                float* sc = my_sc + qi * cap;
                uint32_t* id = my_id + qi * cap;
                if (pass) {
                    const int pos = cnt[qi] + __popc(mask & below);
                    sc[pos] = key[qi];
                    id[pos] = (uint32_t)(base + off);
                }
                cnt[qi] += __popc(mask);
                if (cnt[qi] > cap - 32) {
                    __syncwarp();
                    const float nt = dir_compact<2 * NPL>(sc, id, cnt[qi], p.k);
                    cnt[qi] = cnt[qi] < p.k ? cnt[qi] : p.k;
                    // (this warp meets its rows in ascending order, so for itself equal keys no longer count)
                    thr[qi] = fmaxf(t, nt);
                    if (lane == 0 && nt > neg_inf()) atomic_max_f32(s_thr + qi, dir_step_below(nt));
                }
            }
        }
    }
#pragma unroll
    for (int qi = 0; qi < NQ; ++qi)
        if (lane == 0) s_cnt[warp][qi] = cnt[qi];
    __syncthreads();
    // The block's pools of a query together usually hold little more than k entries: one warp sorts them.
    for (int qi = warp; qi < nqb; qi += DIR_WARPS) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < DIR_WARPS; ++w) total += s_cnt[w][qi];
        const int64_t o = (list + qi * (int64_t)p.nchunk) * p.k;
        dir_collect<NPL>(s_sc + qi * cap, s_id + qi * cap, NQ * cap, &s_cnt[0][qi], NQ, total, p.k, p.part_key + o, p.part_id + o);
    }
}

// Merge: one block per query.  At least k of the candidates reach the k-th best of the lists' heads, so
// only entries at or above that enter a list in shared memory (a little more than k of them), which one
// block sort orders; up to DIR_MERGE_CAP candidates are sorted as they are.  Where neither holds (fewer
// lists than k, or many ties) the warps walk the lists with a merge step each.  A single block is bound by
// latency: the walk alone, one dependent load after the other, took 28 us on 296 lists of 10; this takes 6.
// The k survivors are scored once more in the summation order of the pool finalisation, so that a
// row's distance does not depend on which path found it.
constexpr int DIR_MERGE_CAP = 1024;
template <int NPL>
__global__ void __launch_bounds__(DIR_THREADS) direct_merge_kernel(const DirectParams p) {
    __shared__ float s_key[DIR_MERGE_CAP];
    __shared__ uint32_t s_id[DIR_MERGE_CAP];
    __shared__ int s_n;
    __shared__ float s_cut;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t qi = blockIdx.x;
    const int lists = p.lists_per_query, k = p.k;
    const int cand = lists * k;
    const float* pk = p.part_key + qi * (int64_t)cand;
    const uint32_t* pi = p.part_id + qi * (int64_t)cand;
    float ka[NPL];
    uint32_t ia[NPL];
    bool sorted = false;
    if (cand <= DIR_MERGE_CAP || lists >= k) {
        float cut = neg_inf();
        if (tid == 0) s_n = 0;
        if (cand > DIR_MERGE_CAP) {
            float head = neg_inf();
            for (int l = tid; l < lists; l += DIR_THREADS) head = fmaxf(head, __ldg(pk + (int64_t)l * k));
            s_key[tid] = head;
            __syncthreads();
            if (warp == 0) {
                const float t = dir_first_threshold(s_key, k);
                if (lane == 0) s_cut = t;
            }
            __syncthreads();
            cut = s_cut;
        }
        __syncthreads();
        for (int i = tid; i < cand; i += DIR_THREADS) {
            const float key = __ldg(pk + i);
            if (key >= cut && key > neg_inf()) {
                const int pos = atomicAdd(&s_n, 1);
                if (pos < DIR_MERGE_CAP) { s_key[pos] = key; s_id[pos] = __ldg(pi + i); }
            }
        }
        __syncthreads();
        const int n = s_n;
        if (n <= DIR_MERGE_CAP) {
            sorted = true;
            int P = pow2_ceil_dev(n > k ? n : k);
            for (int i = n + tid; i < P; i += DIR_THREADS) { s_key[i] = neg_inf(); s_id[i] = INVALID_ID; }
            block_sort_desc<DIR_THREADS>(s_key, s_id, P);
        }
    }
    if (!sorted) {
#pragma unroll
        for (int r = 0; r < NPL; ++r) { ka[r] = neg_inf(); ia[r] = INVALID_ID; }
        float kth = neg_inf();
        for (int l0 = warp * 32; l0 < lists; l0 += DIR_THREADS) {
            const int l = l0 + lane;
            const float head = l < lists ? __ldg(pk + (int64_t)l * k) : neg_inf();
            unsigned live = __ballot_sync(FULL_MASK, head >= kth && head > neg_inf());
            while (live) {
                const int src = __ffs(live) - 1;
                live &= live - 1;
                const int64_t o = (int64_t)(l0 + src) * k;
                float kb[NPL];
                uint32_t ib[NPL];
#pragma unroll
                for (int r = 0; r < NPL; ++r) {
                    const int e = (r << 5) | lane;
                    kb[r] = e < k ? __ldg(pk + o + e) : neg_inf();
                    ib[r] = e < k ? __ldg(pi + o + e) : INVALID_ID;
                }
                warp_merge_desc<NPL, true>(ka, ia, kb, ib);
#pragma unroll
                for (int r = 0; r < NPL; ++r)
                    if (((k - 1) >> 5) == r) kth = __shfl_sync(FULL_MASK, ka[r], (k - 1) & 31);
                live &= __ballot_sync(FULL_MASK, head >= kth && head > neg_inf());
            }
        }
        __syncthreads();
        static_assert(DIR_WARPS * NPL * 32 <= DIR_MERGE_CAP, "the warps' lists fit the merge list");
#pragma unroll
        for (int r = 0; r < NPL; ++r) {
            const int e = (r << 5) | lane;
            s_key[warp * NPL * 32 + e] = ka[r];
            s_id[warp * NPL * 32 + e] = ia[r];
        }
        block_sort_desc<DIR_THREADS>(s_key, s_id, DIR_WARPS * NPL * 32);
    }
    const void* qp = row_at(p.q, qi, p.ldq, p.dt);
    for (int e0 = warp * 4; e0 < k; e0 += DIR_WARPS * 4) {
        uint32_t cid[4];
        float a[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) { cid[t] = e0 + t < k ? s_id[e0 + t] : INVALID_ID; a[t] = 0.f; }
        if (p.vec) {
            for (int c = lane * 4; c < p.d; c += 128) {
                const float4 qv = ld_elem4(qp, c, p.dt);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (cid[t] != INVALID_ID) {
                        const float4 xv = ld_elem4(row_at(p.db, cid[t], p.ldb, p.dt), c, p.dt);
                        const float d0 = qv.x - xv.x, d1 = qv.y - xv.y, d2 = qv.z - xv.z, d3 = qv.w - xv.w;
                        a[t] += d0 * d0 + d1 * d1 + d2 * d2 + d3 * d3;
                    }
                }
            }
        } else {
            for (int c = lane; c < p.d; c += 32) {
                const float qv = ld_elem(qp, c, p.dt);
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (cid[t] != INVALID_ID) {
                        const float df = qv - ld_elem(row_at(p.db, cid[t], p.ldb, p.dt), c, p.dt);
                        a[t] += df * df;
                    }
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a[t] += __shfl_xor_sync(FULL_MASK, a[t], o);
            if (lane == 0 && cid[t] != INVALID_ID) s_key[e0 + t] = -a[t];
        }
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
        const int e = (r << 5) | lane;
        const bool have = e < k && s_id[e] != INVALID_ID;
        ka[r] = have ? s_key[e] : neg_inf();
        ia[r] = have ? s_id[e] : INVALID_ID;
    }
    warp_sort_desc<NPL, true>(ka, ia);
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
        const int e = (r << 5) | lane;
        if (e < k) {
            const bool ok = ia[r] != INVALID_ID;
            p.out_dist[qi * k + e] = ok ? -ka[r] : pos_inf();
            p.out_idx[qi * k + e] = ok ? (int32_t)((int64_t)ia[r] + p.row_offset) : -1;
        }
    }
    if (qi == 0 && p.status != nullptr && lane < FL_STATUS_WORDS) p.status[lane] = lane == FL_STATUS_POOL ? k : 0;
}

// ---- host side ---------------------------------------------------------------------------
// Pool classes of the scan: k <= 32 and k <= 128.
constexpr int DIR_MAX_K = 128, DIR_MAX_QUERIES = 4;
static int dir_npl(int k) { return k <= 32 ? 1 : 4; }
static size_t dir_smem_bytes(int nq, int d, int step, int npl) {
    return sizeof(float) * ((size_t)nq * round_up(d, step) + (size_t)2 * DIR_WARPS * nq * npl * 64);
}

// Queries per block and row ranges.  Four queries share a row read while that leaves a block for every SM and their rows
// and pools take 100 KB at most, otherwise two or one; two ranges per SM (four for one query), but no more than the database has passes of
// a block (256 rows), dealt evenly (257 rows: 160 and 97).
static void dir_geometry(int64_t nq, int64_t m, int d, int k, int* nqb, int* nchunk, int64_t* rows_per_chunk) {
    const int npl = dir_npl(k);
    const int64_t max_chunks = ceil_div(m, DIR_THREADS);
    int n = DIR_MAX_QUERIES;
    while (n > 1 && (n / 2 >= nq || ceil_div(nq, n) * max_chunks < sm_count() || dir_smem_bytes(n, d, 64, npl) > 100 * 1024)) n >>= 1;
    const int64_t groups = ceil_div(nq, n);
    const int64_t fit = (int64_t)dir_blocks(n, npl, 4) * sm_count();
    int64_t c = ceil_div(fit, groups);
    if (groups < fit && groups * c > fit && c > 1 && groups * (c - 1) >= fit * 3 / 4) --c;
    if (c > max_chunks) c = max_chunks;
    if (c < 1) c = 1;
    *rows_per_chunk = round_up(ceil_div(m, c), 32);
    *nchunk = (int)ceil_div(m, *rows_per_chunk);
    *nqb = n;
}

int direct_supported(int64_t nq, int64_t m, int d, int k) {
    if (nq < 1 || m < 1 || k < 1 || k > DIR_MAX_K || m >= (1ll << 31)) return 0;
    return dir_smem_bytes(1, d, 64, dir_npl(k)) <= (size_t)(160 * 1024) ? 1 : 0;
}

// Estimated time in us of the scan, fitted to measurements (1 to 64 queries, 10 000 to 1M rows, 16 to 128
// features: within a third of each): a row read by a group of queries costs a fixed part for folding and
// comparing, and its bytes.
double direct_estimate_us(int64_t nq, int64_t m, int d) {
    const double row = (2.65e-5 + 5.1e-7 * d) * (d % 4 == 0 ? 1.0 : 1.5);
    return 14.0 + (double)ceil_div(nq, DIR_MAX_QUERIES) * (double)m * row;
}

int direct_possible(int64_t nq, int64_t m, int d, int k) { return nq <= 512 && direct_supported(nq, m, d, k); }

int direct_wide(const void* db, int64_t ldb, int d, int dt) {
    const int v = dt == DT_F32 ? 4 : 8;
    return d % v == 0 && ldb % v == 0 && (reinterpret_cast<uintptr_t>(db) & 15) == 0;
}

// Estimated us of this scan and of the tile kernel (knn_simt.cu) for one element type, fitted to 1 260 shapes (1 to 512
// queries, 1 000 to 200 000 rows, 16 to 1 024 features, k = 10, 40 and 100, fp32 and bf16).  Here four queries
// share a read, features are padded to the stretch of eight lanes, rows that 16-byte reads do not fit cost twice
// (fp32) to five times (16 bits) as much, and from k = 33 on a range's pool is sorted several times.  The tile kernel takes
// 64 queries at once in up to 64 row ranges: a walk over the tiles of one range, or all tiles over the SMs.
static double direct_scan_us(int64_t nq, int64_t m, int d, int k, int dt, int wide) {
    const bool f32 = dt == DT_F32;
    double row;
    if (f32) row = 1.6e-5 + (wide ? 5.5e-7 * (double)round_up(d, 32) * (d > 512 ? 1.15 : 1.0) : (d <= 64 ? 6.5e-7 : 1e-6) * (double)round_up(d, 8));
    else if (wide) row = 1.5e-5 + 7.2e-7 * (double)round_up(d, 64) * (d > 512 ? 1.5 : 1.0);
    else row = 4e-6 * d - 3e-5 > 6e-5 ? 4e-6 * d - 3e-5 : 6e-5;
    const double groups = (double)ceil_div(nq, DIR_MAX_QUERIES);
    double ranges = 2.0 * sm_count() / groups;
    if (ranges > m / 256.0) ranges = m / 256.0;
    if (ranges < 1) ranges = 1;
    const double least = 256.0 * sm_count(), rows = groups * (double)m;
    double t = 18 + (rows > least ? rows : least) * row + 0.04 * (double)nq;
    if (k > 32) t += 4.6 * pow(k / 100.0, 0.6) * pow((double)m / ranges, 0.52) * (nq > 8 ? 1.0 : 0.9) * (f32 || nq < 32 ? 1.0 : 1.5);
    return t;
}
static double tile_scan_us(int64_t nq, int64_t m, int d, int k, int dt) {
    const int c = k <= 24 ? 0 : k <= 56 ? 1 : 2;           // pools of 32, 64, 128 entries
    const double alone[3] = {112, 160, 243}, shared[3] = {88, 100, 175}, walk[3] = {0, 4, 12}, work[3] = {0, 2, 9.7};
    const double sms = sm_count(), groups = (double)ceil_div(nq, 64), tiles = (double)ceil_div(m, 128);
    double ranges = (double)ceil_div(2 * (int64_t)sms, (int64_t)groups);
    if (ranges > tiles / 4) ranges = tiles / 4;
    if (ranges > 64) ranges = 64;
    if (ranges < 1) ranges = 1;
    const double dp = (double)round_up(d, 32) * (dt == DT_F32 || d <= 128 ? 1.0 : 1.65);
    const double blocks = groups * ranges, per = tiles / ranges;
    const double one = ceil(per) * (14 + 0.089 * dp + walk[c]);
    if (blocks <= sms) return alone[c] + one * (nq < 8 ? 0.85 : 1.0);
    const double both = (blocks <= 2 * sms ? 2 * per : tiles * groups / sms) * (8 + 0.08 * dp + work[c]);
    const double second = blocks >= 2 * sms ? 1.0 : (blocks - sms) / sms;
    return alone[c] + shared[c] * second + (one > both ? one : both);
}
// 1: the exact mode takes this scan.  Measured, this and the tile kernel: 1 x 1M x 128: 132 and 1 844 us; 300 x 20 000 x 64:
// 147 and 322; 512 x 200 000 x 128: 2 329 and 1 687; 256 x 20 000 x 64, k = 100: 664 and 408; 512 x 20 000 x 100 in
// bf16 (no 16-byte reads): 936 and 405; 512 x 200 000 x 333 in bf16: 38 600 and 6 350.
int direct_pick(int64_t nq, int64_t m, int d, int k, int dt, int wide) {
    return direct_possible(nq, m, d, k) && direct_scan_us(nq, m, d, k, dt, wide) <= tile_scan_us(nq, m, d, k, dt);
}

int64_t direct_workspace_bytes(int64_t nq, int64_t m, int d, int k) {
    int nqb, nchunk;
    int64_t rpc;
    dir_geometry(nq, m, d, k, &nqb, &nchunk, &rpc);
    return 2 * round_up(nq * nchunk * (int64_t)k * 4, 1024);
}

int64_t direct_ivf_workspace_bytes(int64_t npairs, int nchunk, int k) { return 2 * round_up(npairs * nchunk * (int64_t)k * 4, 1024); }

// Row ranges per (query, probed list) pair: enough for eight blocks per SM, at most eight ranges.
int direct_ivf_chunks(int64_t npairs) {
    int64_t c = ceil_div((int64_t)8 * sm_count(), npairs > 0 ? npairs : 1);
    return (int)(c > 8 ? 8 : c < 1 ? 1 : c);
}

template <int NQ, int NPL, bool F32, int VEC>
static int dir_launch_scan(const DirectParams& p, unsigned grid, cudaStream_t st) {
    const size_t smem = dir_smem_bytes(NQ, p.d, 8 * VEC, NPL);
    if (smem > 40 * 1024)
        FL_CHECK_CUDA(cudaFuncSetAttribute(direct_scan_kernel<NQ, NPL, F32, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    direct_scan_kernel<NQ, NPL, F32, VEC><<<grid, DIR_THREADS, smem, st>>>(p);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

template <bool F32, int VEC>
static int dir_launch_nq(const DirectParams& p, int nqb, unsigned grid, cudaStream_t st) {
    if (p.npl == 4) {
        switch (nqb) {
            case 1: return dir_launch_scan<1, 4, F32, VEC>(p, grid, st);
            case 2: return dir_launch_scan<2, 4, F32, VEC>(p, grid, st);
            default: return dir_launch_scan<4, 4, F32, VEC>(p, grid, st);
        }
    }
    switch (nqb) {
        case 1: return dir_launch_scan<1, 1, F32, VEC>(p, grid, st);
        case 2: return dir_launch_scan<2, 1, F32, VEC>(p, grid, st);
        default: return dir_launch_scan<4, 1, F32, VEC>(p, grid, st);
    }
}

static int dir_launch(DirectParams& p, int nqb, int64_t grid, void* ws, cudaStream_t st) {
    p.npl = dir_npl(p.k);
    const int64_t nlists = p.nq * (int64_t)p.lists_per_query;
    p.part_key = static_cast<float*>(ws);
    p.part_id = reinterpret_cast<uint32_t*>(static_cast<char*>(ws) + round_up(nlists * p.k * 4, 1024));
    FL_CHECK_ARG(grid < (1ll << 31) && p.nq < (1ll << 31), "few-query scan: too many blocks");
    const int wide = direct_wide(p.db, p.ldb, p.d, p.dt);
    int rc;
    if (p.dt == DT_F32)
        rc = wide ? dir_launch_nq<true, 4>(p, nqb, (unsigned)grid, st) : dir_launch_nq<true, 1>(p, nqb, (unsigned)grid, st);
    else
        rc = wide ? dir_launch_nq<false, 8>(p, nqb, (unsigned)grid, st) : dir_launch_nq<false, 1>(p, nqb, (unsigned)grid, st);
    if (rc != FL_OK) return rc;
    const int mn = pow2_ceil((p.k + 31) / 32);
    switch (mn) {
        case 1: direct_merge_kernel<1><<<(unsigned)p.nq, DIR_THREADS, 0, st>>>(p); break;
        case 2: direct_merge_kernel<2><<<(unsigned)p.nq, DIR_THREADS, 0, st>>>(p); break;
        default: direct_merge_kernel<4><<<(unsigned)p.nq, DIR_THREADS, 0, st>>>(p); break;
    }
    FL_CHECK_LAUNCH();
    return FL_OK;
}

int launch_knn_direct(DirectParams p, void* ws, cudaStream_t st) {
    int nqb;
    dir_geometry(p.nq, p.m, p.d, p.k, &nqb, &p.nchunk, &p.rows_per_chunk);
    p.lists_per_query = p.nchunk;
    p.probed = nullptr;
    profile_begin(st);
    const int rc = dir_launch(p, nqb, ceil_div(p.nq, nqb) * p.nchunk, ws, st);
    profile_end(st);
    return rc;
}

int launch_ivf_direct(DirectParams p, void* ws, cudaStream_t st) {
    const int64_t npairs = p.nq * (int64_t)p.nprobe;
    p.nchunk = direct_ivf_chunks(npairs);
    p.lists_per_query = p.nprobe * p.nchunk;
    profile_begin(st);
    const int rc = dir_launch(p, 1, npairs * p.nchunk, ws, st);
    profile_end(st);
    return rc;
}

}  // namespace fl
