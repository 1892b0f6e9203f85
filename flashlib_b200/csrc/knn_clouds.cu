// Exact kNN of many small problems with few features (point clouds): d <= 16, k <= 40.  A thread (or several) per
// query, the rows of a problem pass through shared memory, and a distance is the fp32 sum (q - x)^2 itself.
// Two passes over the rows: the first leaves the smallest distance of each of G interleaved groups of
// rows (row r belongs to group r % G); the k-th smallest of those is reached by at least k rows, and by
// hardly more (k = 16 of 64 groups: 18 +- 2), so the second pass keeps what does not exceed it and a warp
// sorts each query's list.  A list that overflows -- many equal distances, or an order of the rows that
// resonates with the groups -- is answered by a warp that scans the rows with a sorted pool.
//
// The rows lie feature by feature in shared memory and a thread takes four at a time in packed pairs: a
// shared-memory read returns 128 bytes a cycle and SM however many lanes want the same word, so rows padded
// to four features, one at a time, cost 16 such cycles a warp and row of the four sub-cores (317 us for
// the batch below), three features of four rows 12, and no sum has to be folded.
//
// Bound: dependent instructions with few warps to hide them (3.5 a scheduler; issue slots 53 % busy).  The tile kernel (knn_simt.cu) pads 3 features to 32 and
// keeps a pool per query in shared memory: 32 problems of 2 048 x 2 048 x 3, k = 16, took it 1 710 us; here 232.
#include "knn_internal.h"
#include "packed.cuh"

namespace fl {

constexpr int CLOUD_THREADS = 128, CLOUD_WARPS = CLOUD_THREADS / 32;
constexpr int CLOUD_LIST = 32;                    // entries a thread keeps

// Squared distances of four consecutive rows, two packed pairs of rows at a time: the rows lie feature by feature
// (negated) in shared memory, CP floats apart, so nothing is padded but the features to DP and no sum
// has to be folded.
template <int DP, int CP>
__device__ __forceinline__ void cloud_dist4(const unsigned long long (&q)[DP], const float* rows, float (&s)[4]) {
    unsigned long long s01 = 0ull, s23 = 0ull;
#pragma unroll
    for (int f = 0; f < DP; ++f) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(rows + f * CP);
        s01 = sqadd2(add2(q[f], v.x), s01);
        s23 = sqadd2(add2(q[f], v.y), s23);
    }
    unpk2(s01, s[0], s[1]);
    unpk2(s23, s[2], s[3]);
}

// Rows [c0, c0 + kc) of the problem, and NaN up to a multiple of four rows: no comparison lets those pass.
template <int DP, int CP>
__device__ __forceinline__ void cloud_stage(float* rows, const float* db, int64_t ldb, int d, int c0, int kc) {
    const int kp = (kc + 3) & ~3;
    for (int e = threadIdx.x; e < kp * DP; e += CLOUD_THREADS) {
        const int j = e / DP, f = e - j * DP;
        rows[f * CP + j] = j >= kc ? __int_as_float(0x7fc00000) : f < d ? -__ldg(db + (int64_t)(c0 + j) * ldb + f) : 0.f;
    }
}

// One query's answer by a warp: 32 rows at a time, sorted and merged into the pool when one of them
// belongs there.  Out of line: rare.
template <int NPL>
static __device__ __noinline__ void cloud_scan_query(const float* q, const float* db, int m, int64_t ldb, int d, int k,
                                                     float (&ka)[NPL], uint32_t (&ia)[NPL]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < NPL; ++r) { ka[r] = neg_inf(); ia[r] = INVALID_ID; }
    float kth = neg_inf();
    int have = 0;
    for (int base = 0; base < m; base += 32) {
        const int row = base + lane;
        const float* p = db + (int64_t)(row < m ? row : m - 1) * ldb;
        float s = 0.f;
        for (int f = 0; f < d; ++f) {
            const float df = __ldg(q + f) - __ldg(p + f);
            s = fmaf(df, df, s);
        }
        const bool real = row < m && s == s;
        float kb[NPL];
        uint32_t ib[NPL];
#pragma unroll
        for (int r = 0; r < NPL; ++r) { kb[r] = neg_inf(); ib[r] = INVALID_ID; }
        kb[0] = real ? -s : neg_inf();
        ib[0] = real ? (uint32_t)row : INVALID_ID;
        const unsigned live = __ballot_sync(FULL_MASK, real);
        if (!__any_sync(FULL_MASK, real && (have < k || kb[0] > kth))) continue;
        have += __popc(live);
        warp_sort_desc<NPL, true>(kb, ib);
        warp_merge_desc<NPL, true>(ka, ia, kb, ib);
#pragma unroll
        for (int r = 0; r < NPL; ++r)
            if (((k - 1) >> 5) == r) kth = __shfl_sync(FULL_MASK, ka[r], (k - 1) & 31);
    }
}

struct CloudParams {
    const float* q; int64_t nq, ldq, q_bstride;
    const float* db; int m; int64_t ldb, db_bstride;
    int d, k;
    float* out_dist; int32_t* out_idx;
    int splits;              // threads per query: 1, 2 or 4, each with its share of the rows
};

// G groups; answers of up to 32 NPL entries are sorted.  Every thread lists what it meets on its own --
// no counter is shared and only a row group with a candidate branches in the second pass.
template <int DP, int G, int NPL>
__global__ void __launch_bounds__(CLOUD_THREADS) knn_clouds_kernel(const CloudParams p) {
    extern __shared__ __align__(16) float cloud_smem[];
    constexpr int CH = DP <= 4 ? 1024 : DP <= 8 ? 512 : 256, CP = CH + 4, LP = CLOUD_LIST + 1;
    static_assert(CH % G == 0, "a chunk holds whole rounds of the groups");
    __shared__ int s_cnt[CLOUD_THREADS];
    __shared__ float s_thr[CLOUD_THREADS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Q = CLOUD_THREADS / p.splits;        // queries of this block
    const int ql = tid % Q, split = tid / Q;
    float* rows = cloud_smem;                      // [DP][CP]
    float* mins = rows + DP * CP;                  // [G][Q], then the lists [thread][LP]
    float* l_key = mins;
    uint32_t* l_id = reinterpret_cast<uint32_t*>(l_key + CLOUD_THREADS * LP);
    const float* q = p.q + blockIdx.y * p.q_bstride;
    const float* db = p.db + blockIdx.y * p.db_bstride;
    const int64_t q0 = (int64_t)blockIdx.x * Q;
    const int64_t qi = q0 + ql;
    const int m = p.m, k = p.k;

    unsigned long long xr[DP];                     // every feature twice
#pragma unroll
    for (int f = 0; f < DP; ++f) {
        const float v = (qi < p.nq && f < p.d) ? __ldg(q + qi * p.ldq + f) : 0.f;
        xr[f] = pk2(v, v);
    }
    for (int c0 = 0; c0 < m; c0 += CH) {
        const int kc = min(CH, m - c0);
        if (c0 > 0) __syncthreads();
        cloud_stage<DP, CP>(rows, db, p.ldb, p.d, c0, kc);
        __syncthreads();
        for (int g = split * 4; g < G; g += p.splits * 4) {
            float mn[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) mn[i] = c0 > 0 ? mins[(g + i) * Q + ql] : pos_inf();
#pragma unroll 2
            for (int j = g; j < kc; j += G) {      // (fminf takes the number where the other is NaN)
                float s[4];
                cloud_dist4<DP, CP>(xr, rows + j, s);
#pragma unroll
                for (int i = 0; i < 4; ++i) mn[i] = fminf(mn[i], s[i]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) mins[(g + i) * Q + ql] = mn[i];
        }
    }
    __syncthreads();
    if (tid < Q) {
        // A value that at least k of the minima do not exceed, close to the smallest such: bisection over
        // their bits, which order like the values (none is negative).  +inf where fewer than k are finite.
        unsigned lo = 0xffffffffu, hi = 0u;
#pragma unroll 8
        for (int g = 0; g < G; ++g) {
            const unsigned v = __float_as_uint(mins[g * Q + tid]);
            lo = min(lo, v);
            hi = max(hi, v);
        }
        // count(<= hi) >= k throughout
        while (lo < hi) {
            const unsigned mid = lo + ((hi - lo) >> 1);
            int c = 0;
#pragma unroll 8
            for (int g = 0; g < G; ++g) c += __float_as_uint(mins[g * Q + tid]) <= mid ? 1 : 0;
            if (c >= k) hi = mid; else lo = mid + 1;
            if (c >= k && c <= k + (k >> 4)) break;
        }
        s_thr[tid] = __uint_as_float(hi);
    }
    __syncthreads();
    const float thr = s_thr[ql];
    float* my_key = l_key + tid * LP;
    uint32_t* my_id = l_id + tid * LP;
    int cnt = 0;
    for (int c0 = 0; c0 < m; c0 += CH) {
        const int kc = min(CH, m - c0);
        if (m > CH) {
            if (c0 > 0) __syncthreads();
            cloud_stage<DP, CP>(rows, db, p.ldb, p.d, c0, kc);
            __syncthreads();
        }
#pragma unroll 2
        for (int j = split * 4; j < kc; j += p.splits * 4) {
            float s[4];
            cloud_dist4<DP, CP>(xr, rows + j, s);
            if (fminf(fminf(s[0], s[1]), fminf(s[2], s[3])) <= thr) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool in = s[i] <= thr;
                    if (in && cnt < CLOUD_LIST) { my_key[cnt] = -s[i]; my_id[cnt] = (uint32_t)(c0 + j + i); }
                    cnt += in ? 1 : 0;
                }
            }
        }
    }
    s_cnt[tid] = cnt;
    __syncthreads();
    for (int t = warp; t < Q && q0 + t < p.nq; t += CLOUD_WARPS) {
        int total = 0;
        bool fits = true;
        for (int w = 0; w < p.splits; ++w) {
            const int c = s_cnt[w * Q + t];
            fits = fits && c <= CLOUD_LIST;
            total += c;
        }
        float ka[NPL];
        uint32_t ia[NPL];
        if (fits && total <= 32 * NPL) {
#pragma unroll
            for (int r = 0; r < NPL; ++r) {
                int e = (r << 5) | lane, w = t;
                const bool in = e < total;
                while (in && e >= s_cnt[w]) { e -= s_cnt[w]; w += Q; }
                ka[r] = in ? l_key[w * LP + e] : neg_inf();
                ia[r] = in ? l_id[w * LP + e] : INVALID_ID;
            }
            warp_sort_desc<NPL, true>(ka, ia);
        } else {
            cloud_scan_query<NPL>(q + (q0 + t) * p.ldq, db, m, p.ldb, p.d, k, ka, ia);
        }
        const int64_t o = (blockIdx.y * p.nq + q0 + t) * k;
#pragma unroll
        for (int r = 0; r < NPL; ++r) {
            const int e = (r << 5) | lane;
            if (e < k) {
                const bool ok = ia[r] != INVALID_ID;
                p.out_dist[o + e] = ok ? -ka[r] : pos_inf();
                p.out_idx[o + e] = ok ? (int32_t)ia[r] : -1;
            }
        }
    }
}

template <int DP, int G, int NPL>
static int clouds_launch(CloudParams p, int batch, cudaStream_t st) {
    // Several threads a query while the queries alone do not give every SM its four blocks, and for the larger
    // group counts, whose minima would otherwise leave room for one or two blocks.
    p.splits = G > 64 ? 4 : 1;
    while (p.splits < 4 && batch * ceil_div(p.nq, CLOUD_THREADS / p.splits) < 4 * (int64_t)sm_count()) p.splits *= 2;
    const int Q = CLOUD_THREADS / p.splits;
    const size_t lists = (size_t)CLOUD_THREADS * (CLOUD_LIST + 1) * 2, mins = (size_t)G * Q;
    const size_t smem = sizeof(float) * (DP * ((DP <= 4 ? 1024 : DP <= 8 ? 512 : 256) + 4) + (lists > mins ? lists : mins));
    FL_CHECK_CUDA(cudaFuncSetAttribute(knn_clouds_kernel<DP, G, NPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    knn_clouds_kernel<DP, G, NPL><<<dim3((unsigned)ceil_div(p.nq, Q), (unsigned)batch), CLOUD_THREADS, smem, st>>>(p);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

template <int DP>
static int clouds_dispatch(const CloudParams& p, int batch, cudaStream_t st) {
    // groups enough that the k-th smallest minimum lets little more than k rows pass, and the lists hold them
    // with six standard deviations to spare: 16 of 64, 32 of 128, 40 of 256
    if (p.k <= 16) return clouds_launch<DP, 64, 1>(p, batch, st);
    if (p.k <= 32) return clouds_launch<DP, 128, 2>(p, batch, st);
    return clouds_launch<DP, 256, 2>(p, batch, st);
}

// Estimated us of a batch by this kernel and by the tile kernel (knn_simt.cu), fitted to 900 shapes (2 to 64
// problems, 1 to 4 096 queries, 512 to 1M rows, 3 to 16 features, k = 16 to 40).  A block here walks every row of its
// problem twice and no other block helps it: 16 ns a row with 3 features, 24 with 8, 40 with 16, 1.6 times that once
// the problems outgrow the L2, whatever the number of queries -- then the pairs.  The tile kernel deals the rows of a
// problem to up to 64 blocks of 64 queries.
static double clouds_estimate_us(int batch, int64_t nq, int64_t m, int d, int k) {
    const double dp = d <= 3 ? 3 : d <= 4 ? 4 : d <= 8 ? 8 : 16;
    const double walk = (double)m * (1.02e-2 + 2.0e-3 * dp) * ((double)batch * m * d * 4 > 90e6 ? 1.6 : 1.0);
    const double pairs = (double)batch * nq * m * (0.3e-6 + 0.17e-6 * dp) * (k > 16 ? 1.25 : 1.0);
    return 12 + (k <= 16 ? (nq < 2 ? 6 : 10) : (nq < 2 ? 14 : 32)) + (walk > pairs ? walk : pairs);
}
static double tile_batch_estimate_us(int batch, int64_t nq, int64_t m, int k) {
    const double per_row = nq <= 16 ? 1.0e-3 : nq <= 64 ? 1.25e-3 : 0.9e-3;
    return (nq < 8 ? 46 : 95) + (k > 16 ? (nq < 8 ? 12 : 36) : 0) + (m < 16384 ? 2.9e-3 * m : 31.0 + 1e-3 * m) +
           (double)(batch - 1) * ceil_div(nq, 64) * m * per_row;
}
static int clouds_supported(int64_t nq, int64_t m, int d, int k) {
    return nq >= 1 && d <= 16 && k <= 40 && nq * m <= ((int64_t)1 << (d <= 8 && k <= 32 ? 26 : 24));
}
// Measured, this against the tile kernel: 32 x 2 048^2 x 3, k = 16: 232 and 1 704 us; 64 x 64 x 4 096 x 3: 87 and 564;
// 2 x 16 x 65 536 x 3: 1 050 and 308; 8 x 16 x 1 000 000 x 3: 24 600 and 9 100; 2 x 64 x 8 192 x 16: 367 and 156.
int clouds_pick(int batch, int64_t nq, int64_t m, int d, int k) {
    return clouds_supported(nq, m, d, k) && clouds_estimate_us(batch, nq, m, d, k) <= tile_batch_estimate_us(batch, nq, m, k);
}

// One problem after the other on the tensor cores costs 130 us and its scoring, and for more problems than operand planes
// are kept (four) the building of its planes (2 x 8 192^2 x 8, k = 32: 377 us in the batch and 483 one by one; 4 x
// 8 192^2 x 3, k = 16: 387 and 831; 4 x 8 192^2 x 16, k = 40: 1 618 and 996; 32 x 64 x 262 144 x 3: 5.8 and 17.9 ms).
int clouds_beat_single(int batch, int64_t nq, int64_t m, int d, int k) {
    return clouds_supported(nq, m, d, k) && clouds_estimate_us(batch, nq, m, d, k) <= batch * (130 + (double)nq * m * 1e-6 + (batch > 4 ? 8e-4 * m : 0.0));
}

int launch_knn_clouds(const float* q, int batch, int64_t nq, int64_t ldq, int64_t q_bstride, const float* db, int64_t m,
                      int64_t ldb, int64_t db_bstride, int d, int k, float* out_dist, int32_t* out_idx, cudaStream_t st) {
    CloudParams p{};
    p.q = q; p.nq = nq; p.ldq = ldq; p.q_bstride = q_bstride;
    p.db = db; p.m = (int)m; p.ldb = ldb; p.db_bstride = db_bstride;
    p.d = d; p.k = k; p.out_dist = out_dist; p.out_idx = out_idx;
    if (d <= 3) return clouds_dispatch<3>(p, batch, st);
    if (d == 4) return clouds_dispatch<4>(p, batch, st);
    if (d <= 8) return clouds_dispatch<8>(p, batch, st);
    return clouds_dispatch<16>(p, batch, st);
}

}  // namespace fl
