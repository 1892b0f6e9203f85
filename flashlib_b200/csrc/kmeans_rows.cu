// k-means on the CUDA cores, one sample row per thread: the row sits in registers, the centroids in
// shared memory, and every pair costs d subtractions and d FMAs in packed fp32 pairs -- the fp32 sum
// (x - c)^2 itself, so the nearest centroid needs no norms, no second candidate and no re-scoring.
// Nothing is padded but the features (to a multiple of 4, 8, 16 or 32); the tile kernel of kmeans.cu pads
// to 32 features and 128 centroids.  The same kernel moves the rows between the clusters' sums
// while it still holds them, and fl_kmeans_lloyd_f32 below runs whole Lloyd loops with two launches an
// iteration.
//
// Bound: the FP32 pipe (2 d lanes per pair) for many rows, launch latency for few.
#include "kmeans_rows.h"
#include "packed.cuh"
#include <climits>
#include <sched.h>

namespace fl {

constexpr int ROWS_THREADS = 128, ROWS_WARPS = ROWS_THREADS / 32;
constexpr int ROWS_MAX_D = 128;
constexpr int ROWS_CHUNK_BYTES = 16 * 1024;     // centroids held in shared memory at a time

struct RowsParams {
    const float* x; int64_t n, ldx, xbs; int d;
    const float* c; int K; int64_t ldc, cbs;
    int32_t* labels;                // [batch][n]
    // Sums (contiguous [batch][K][d]) and counts, or null.  add_all: every row is added to its cluster's sum.
    // Otherwise `labels` holds the labels the sums stand for, and only rows that change sides are moved.
    float* sums; int32_t* cnts; int add_all;
    const int* done;                // optional: nothing is left to do once *done != 0
    int vec;                        // rows of x allow 16-byte reads and d is a multiple of 4
    int vec_sums;                   // so do the rows of `sums`
    int chunk;                      // centroids per shared-memory chunk
    int splits;                     // threads per row: 1, 2 or 4 (R = 1), each with its share of the centroids
};

// A row none of whose squared distances is finite (overflow, infinities): ranked by <x,c> - ||c||^2/2, the
// nearer of the best two by the distance, the lower index on ties -- what the tile kernel of
// kmeans.cu answers.  INT_MAX when every score is NaN.
static __device__ __noinline__ int rows_label_by_score(const float* x, int d, const float* c, int K, int64_t ldc) {
    float best = neg_inf(), sec = neg_inf();
    int bi = INT_MAX, si = INT_MAX;
    for (int j = 0; j < K; ++j) {
        const float* cj = c + (int64_t)j * ldc;
        float dot = 0.f, h = 0.f;
        for (int t = 0; t < d; ++t) { const float v = cj[t]; dot = fmaf(x[t], v, dot); h += v * v; }
        const float s = dot - 0.5f * h;
        if (s > best || (s == best && j < bi)) { sec = best; si = bi; best = s; bi = j; }
        else if (s > sec || (s == sec && j < si)) { sec = s; si = j; }
    }
    if (si != INT_MAX) {
        float d1 = 0.f, d2 = 0.f;
        for (int t = 0; t < d; ++t) {
            const float e1 = x[t] - c[(int64_t)bi * ldc + t], e2 = x[t] - c[(int64_t)si * ldc + t];
            d1 += e1 * e1;
            d2 += e2 * e2;
        }
        if (d2 < d1 || (d2 == d1 && si < bi)) return si;
    }
    return bi;
}

// Sum over a warp of DP values a lane, by recursive halving (DP + 4 - log2 DP shuffles in place of 5 DP): the lane whose
// low bits are zero ends with feature rows_fold_feature().
template <int DP>
__device__ __forceinline__ float rows_fold(float (&v)[DP]) {
    const int lane = threadIdx.x & 31;
    int n = DP;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
#pragma unroll
            for (int j = 0; j < DP / 2; ++j) {
                if (j < n) {
                    const float give = (lane & o) ? v[j] : v[j + n];
                    const float keep = (lane & o) ? v[j + n] : v[j];
                    v[j] = keep + __shfl_xor_sync(FULL_MASK, give, o);
                }
            }
        } else {
            v[0] += __shfl_xor_sync(FULL_MASK, v[0], o);
        }
    }
    return v[0];
}
template <int DP>
__device__ __forceinline__ int rows_fold_feature() {       // -1: another lane has it
    const int lane = threadIdx.x & 31;
    return (lane & (32 / DP - 1)) ? -1 : lane / (32 / DP);
}

// Up to this many labels among the 32 rows of a warp, the rows of each are added up before they meet the sums: few
// clusters, rows in their order.  Otherwise 32 lanes meet on a handful of addresses -- 10 iterations on 8 x 100 000 x 16 rows
// took 13.9 ms with 2 clusters (0.53 so), 4.0 with 16 (1.15), 11.3 with 4 and rows in order (0.33).  With 32
// clusters a warp mostly meets more, and one atomic per row and four features is as fast (2.5).
constexpr int ROWS_FOLD_LABELS = 16;

// R rows per thread: a centroid read from shared memory then serves R rows.
template <int DP, int R>
__global__ void __launch_bounds__(ROWS_THREADS) kmeans_rows_kernel(const RowsParams p) {
    extern __shared__ __align__(16) float rows_smem[];
    constexpr int P2 = DP / 2;
    constexpr bool STAGED = DP > 16;            // rows come through shared memory, a warp's 32 at a time,
    constexpr int PITCH = 33;                   // 32 features at a time; odd: lanes reading down a column do not conflict
    if (p.done != nullptr && *p.done != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = ROWS_THREADS / p.splits;      // threads that hold different rows
    const int rt = tid & (T - 1), split = tid / T;
    const int rwarp = rt >> 5;
    const int64_t b = blockIdx.y;
    const float* x = p.x + b * p.xbs;
    const float* c = p.c + b * p.cbs;
    int32_t* labels = p.labels + b * p.n;
    const int64_t row0 = (int64_t)blockIdx.x * (T * R);
    float* cs = rows_smem;
    float* xs = rows_smem + p.chunk * DP + warp * 32 * PITCH;

    unsigned long long xr[R][P2];
    if (STAGED) {
        const int64_t w0 = row0 + rwarp * 32;
        const int live = (int)min((int64_t)32, p.n - w0);       // <= 0: none
#pragma unroll
        for (int f0 = 0; f0 < DP; f0 += 32) {
            const int w = min(32, p.d - f0);
            if (f0 > 0) __syncwarp();
            if (w > 0) {
                // element e of the warp's rows: (row, column) walked without a division per element
                int r = lane / w, col = lane - r * w;
                const int dr = 32 / w, dc = 32 - dr * w;
                for (int e = lane; e < live * w; e += 32) {
                    xs[r * PITCH + col] = __ldg(x + (w0 + r) * p.ldx + f0 + col);
                    r += dr;
                    col += dc;
                    if (col >= w) { col -= w; ++r; }
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < (DP - f0 < 32 ? DP - f0 : 32) / 2; ++i) {
                const float a = (lane < live && 2 * i < w) ? xs[lane * PITCH + 2 * i] : 0.f;
                const float v = (lane < live && 2 * i + 1 < w) ? xs[lane * PITCH + 2 * i + 1] : 0.f;
                xr[0][f0 / 2 + i] = pk2(a, v);
            }
        }
    } else {
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int64_t r = row0 + q * T + rt;
            const float* src = x + r * p.ldx;
            if (p.vec) {
#pragma unroll
                for (int i = 0; i < DP / 4; ++i) {
                    const float4 v = (r < p.n && 4 * i < p.d) ? __ldg(reinterpret_cast<const float4*>(src) + i)
                                                             : make_float4(0.f, 0.f, 0.f, 0.f);
                    xr[q][2 * i] = pk2(v.x, v.y);
                    xr[q][2 * i + 1] = pk2(v.z, v.w);
                }
            } else {
#pragma unroll
                for (int i = 0; i < P2; ++i) {
                    const float a = (r < p.n && 2 * i < p.d) ? __ldg(src + 2 * i) : 0.f;
                    const float v = (r < p.n && 2 * i + 1 < p.d) ? __ldg(src + 2 * i + 1) : 0.f;
                    xr[q][i] = pk2(a, v);
                }
            }
        }
    }

    float best[R];
    int bi[R];
#pragma unroll
    for (int q = 0; q < R; ++q) { best[q] = pos_inf(); bi[q] = INT_MAX; }
    for (int k0 = 0; k0 < p.K; k0 += p.chunk) {
        const int kc = min(p.chunk, p.K - k0);
        if (k0 > 0) __syncthreads();
        // negated, so that a difference is one packed addition
        for (int e = tid; e < kc * DP; e += ROWS_THREADS) {
            const int j = e / DP, f = e - j * DP;
            cs[e] = f < p.d ? -__ldg(c + (int64_t)(k0 + j) * p.ldc + f) : 0.f;
        }
        __syncthreads();
#pragma unroll 2
        for (int j = split; j < kc; j += p.splits) {
            const ulonglong2* cp = reinterpret_cast<const ulonglong2*>(cs + j * DP);
            unsigned long long s0[R], s1[R];
#pragma unroll
            for (int q = 0; q < R; ++q) s0[q] = s1[q] = 0ull;
#pragma unroll
            for (int i = 0; i < DP / 4; ++i) {
                const ulonglong2 v = cp[i];
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    s0[q] = sqadd2(add2(xr[q][2 * i], v.x), s0[q]);
                    s1[q] = sqadd2(add2(xr[q][2 * i + 1], v.y), s1[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const float s = fold2(add2(s0[q], s1[q]));
                if (s < best[q]) { best[q] = s; bi[q] = k0 + j; }       // ascending j: the lowest index wins ties
            }
        }
    }

    if (R == 1 && p.splits > 1) {
        // the splits of a row meet; the first of them carries on
        __shared__ float s_best[ROWS_THREADS];
        __shared__ int s_bi[ROWS_THREADS];
        s_best[tid] = best[0];
        s_bi[tid] = bi[0];
        __syncthreads();
        if (split != 0) return;
        for (int t = rt + T; t < ROWS_THREADS; t += T)
            if (s_best[t] < best[0] || (s_best[t] == best[0] && s_bi[t] < bi[0])) { best[0] = s_best[t]; bi[0] = s_bi[t]; }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int64_t r = row0 + q * T + rt;
        int lab = bi[q], from = -1;
        if (r < p.n) {
            if (lab == INT_MAX) lab = rows_label_by_score(x + r * p.ldx, p.d, c, p.K, p.ldc);
            if (p.sums != nullptr && !p.add_all) from = labels[r];
            if (from != lab) labels[r] = lab;
        }
        if (p.sums == nullptr) continue;
        float* sums = p.sums + b * p.K * p.d;
        int32_t* cnts = p.cnts + b * p.K;
        int to = (r < p.n && lab < p.K) ? lab : -1;
        if (from < 0 || from >= p.K) from = -1;
        if (from == to) from = to = -1;
        const unsigned same = __match_any_sync(FULL_MASK, to);
        const bool leader = to >= 0 && lane == __ffs(same) - 1;
        if (leader) atomicAdd(cnts + to, __popc(same));
        if (from >= 0) atomicAdd(cnts + from, -1);
        if (STAGED) {
            // the warp's lanes across one moved row after another: whole sectors per atomic; consecutive rows of one
            // cluster are added up first
            constexpr int NF = (DP + 31) / 32;
            float run[NF];
            int cur = -1;
            unsigned moved = __ballot_sync(FULL_MASK, to >= 0 || from >= 0);
            while (moved) {
                const int src = __ffs(moved) - 1;
                moved &= moved - 1;
                const int t = __shfl_sync(FULL_MASK, to, src), f = __shfl_sync(FULL_MASK, from, src);
                const float* xm = x + (row0 + rwarp * 32 + src) * p.ldx;
                if (t != cur) {
#pragma unroll
                    for (int i = 0; i < NF; ++i) {
                        if (cur >= 0 && lane + 32 * i < p.d) atomicAdd(sums + (int64_t)cur * p.d + lane + 32 * i, run[i]);
                        run[i] = 0.f;
                    }
                    cur = t;
                }
#pragma unroll
                for (int i = 0; i < NF; ++i) {
                    if (lane + 32 * i < p.d) {
                        const float v = __ldg(xm + lane + 32 * i);
                        run[i] += v;
                        if (f >= 0) atomicAdd(sums + (int64_t)f * p.d + lane + 32 * i, -v);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < NF; ++i)
                if (cur >= 0 && lane + 32 * i < p.d) atomicAdd(sums + (int64_t)cur * p.d + lane + 32 * i, run[i]);
        } else if (unsigned leaders = p.add_all ? __ballot_sync(FULL_MASK, leader) : FULL_MASK; __popc(leaders) <= ROWS_FOLD_LABELS) {
            while (leaders) {
                const int src = __ffs(leaders) - 1;
                leaders &= leaders - 1;
                const int t = __shfl_sync(FULL_MASK, to, src);
                float v[DP];
#pragma unroll
                for (int i = 0; i < P2; ++i) {
                    unpk2(xr[q][i], v[2 * i], v[2 * i + 1]);
                    if (to != t) v[2 * i] = v[2 * i + 1] = 0.f;
                }
                const float s = rows_fold<DP>(v);
                const int f = rows_fold_feature<DP>();
                if (f >= 0 && f < p.d) atomicAdd(sums + (int64_t)t * p.d + f, s);
            }
        } else {
#pragma unroll
            for (int i = 0; i < DP / 4; ++i) {
                float v0, v1, v2, v3;
                unpk2(xr[q][2 * i], v0, v1);
                unpk2(xr[q][2 * i + 1], v2, v3);
                if (4 * i >= p.d) break;
                if (p.vec_sums) {
                    if (to >= 0) atomicAdd(reinterpret_cast<float4*>(sums + (int64_t)to * p.d) + i, make_float4(v0, v1, v2, v3));
                    if (from >= 0) atomicAdd(reinterpret_cast<float4*>(sums + (int64_t)from * p.d) + i, make_float4(-v0, -v1, -v2, -v3));
                } else {
                    const float v[4] = {v0, v1, v2, v3};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (4 * i + e < p.d) {
                            if (to >= 0) atomicAdd(sums + (int64_t)to * p.d + 4 * i + e, v[e]);
                            if (from >= 0) atomicAdd(sums + (int64_t)from * p.d + 4 * i + e, -v[e]);
                        }
                    }
                }
            }
        }
    }
}

template <int DP, int R>
static int rows_launch(const RowsParams& in, int batch, cudaStream_t st) {
    RowsParams p = in;
    int chunk = ROWS_CHUNK_BYTES / (DP * 4);
    if (chunk > p.K) chunk = p.K;
    p.chunk = chunk;
    // several threads a row while the rows alone do not give every SM a block (2 000 rows of 128 features, 200
    // centroids: 91 -> 64 us; at 50 000 rows the shorter walk no longer pays for loading each row twice)
    p.splits = 1;
    if (R == 1)
        while (p.splits < 4 && batch * p.n * p.splits < (int64_t)ROWS_THREADS * sm_count()) p.splits *= 2;
    const size_t smem = sizeof(float) * ((size_t)chunk * DP + (DP > 16 ? (size_t)ROWS_WARPS * 32 * 33 : 0));
    FL_CHECK_CUDA(cudaFuncSetAttribute(kmeans_rows_kernel<DP, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kmeans_rows_kernel<DP, R><<<dim3((unsigned)ceil_div(p.n, ROWS_THREADS / p.splits * R), (unsigned)batch), ROWS_THREADS, smem, st>>>(p);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

static int rows_dispatch(RowsParams p, int batch, cudaStream_t st) {
    p.vec = p.d % 4 == 0 && p.ldx % 4 == 0 && p.xbs % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
    p.vec_sums = p.sums != nullptr && p.d % 4 == 0 && (reinterpret_cast<uintptr_t>(p.sums) & 15) == 0;
    // four rows a thread once that still leaves every SM several blocks: a quarter of the shared-memory reads
    const bool many = batch * p.n >= (int64_t)4 * ROWS_THREADS * 4 * sm_count();
    const int d = p.d;
    if (d <= 4) return many ? rows_launch<4, 4>(p, batch, st) : rows_launch<4, 1>(p, batch, st);
    if (d <= 8) return many ? rows_launch<8, 4>(p, batch, st) : rows_launch<8, 1>(p, batch, st);
    if (d <= 16) return many ? rows_launch<16, 4>(p, batch, st) : rows_launch<16, 1>(p, batch, st);
    if (d <= 24) return rows_launch<24, 1>(p, batch, st);
    if (d <= 32) return rows_launch<32, 1>(p, batch, st);
    if (d <= 40) return rows_launch<40, 1>(p, batch, st);
    if (d <= 48) return rows_launch<48, 1>(p, batch, st);
    if (d <= 64) return rows_launch<64, 1>(p, batch, st);
    if (d <= 96) return rows_launch<96, 1>(p, batch, st);
    return rows_launch<128, 1>(p, batch, st);
}

// Estimated us of an assignment by this kernel and by the tile kernel (kmeans.cu), fitted to measurements (2 000
// to 1M rows, 10 to 2 000 centroids, 4 to 128 features): the larger of the time that the pairs take on the
// whole GPU and one thread's (block's) walk over the centroids.
static double rows_estimate_us(int64_t rows, int K, int d) {
    const double dp = d <= 4 ? 4 : d <= 8 ? 8 : d <= 16 ? 16 : (double)round_up(d, d <= 48 ? 8 : 32);
    const double gain = rows < (int64_t)ROWS_THREADS / 2 * sm_count() ? 2.0 : rows < (int64_t)ROWS_THREADS * sm_count() ? 1.4 : 1.0;
    const double walk = K * dp * 3.1e-3 / gain, all = (double)rows * (K * dp / 11.5e6 + d * 2.3e-6);
    return walk > all ? walk : all;
}
static double tile_estimate_us(int64_t rows, int K, int d) {
    const double ct = (double)ceil_div(K, 128), tiles = ct * (double)ceil_div(d, 32);
    const double walk = tiles * 4.6, all = (double)rows * (ct * 2.4e-4 + tiles * 3.4e-4);
    return walk > all ? walk : all;
}

// 1: this kernel is the faster one.  Measured, this against the tile kernel: 1M x 8, K = 256: 190 and 1 110 us;
// 50 001 x 33, K = 50: 24 and 53; 1M x 128, K = 10: 425 and 1 179; 200 000 x 128, K = 200: 455 and 509;
// 2 000 x 128, K = 200: 64 and 41; 20 000 x 128, K = 500: 230 and 154.
int kmeans_rows_pick(int64_t rows, int K, int d) {
    return d <= ROWS_MAX_D && rows_estimate_us(rows, K, d) <= tile_estimate_us(rows, K, d);
}

int launch_kmeans_rows(const float* x, int batch, int64_t n, int64_t ldx, int64_t xbs, const float* c, int K, int64_t ldc,
                       int64_t cbs, int d, int32_t* labels, cudaStream_t st) {
    RowsParams p{};
    p.x = x; p.n = n; p.ldx = ldx; p.xbs = xbs; p.d = d;
    p.c = c; p.K = K; p.ldc = ldc; p.cbs = cbs; p.labels = labels;
    return rows_dispatch(p, batch, st);
}

// Control words of a Lloyd loop on the device: converged flag, blocks finished, largest shift (float bits).

// New centroids, one warp per centroid (and, with `shift`, how far each moved); clears the sums when the next iteration adds
// every row again.  With
// tol > 0 the last block to finish compares the largest shift with it and tells the host, in pinned
// memory, how many iterations are finished; negated when the loop has converged.
__global__ void __launch_bounds__(256) kmeans_step_kernel(float* __restrict__ sums, int32_t* __restrict__ cnts,
                                                          const float* __restrict__ old_c, float* __restrict__ new_c,
                                                          int64_t KB, int d, int clear, float tol, int it,
                                                          unsigned* __restrict__ ctl, volatile int32_t* host,
                                                          float* __restrict__ shift_out) {
    if (tol > 0.f && ctl[LLOYD_DONE] != 0) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t j = (int64_t)blockIdx.x * 8 + warp;
    float s = 0.f;
    if (j < KB) {
        const int cnt = cnts[j];
        const float fc = (float)cnt;
        for (int t = lane; t < d; t += 32) {
            const float o = old_c[j * d + t];
            const float v = cnt > 0 ? sums[j * d + t] / fc : o;
            new_c[j * d + t] = v;
            s += (v - o) * (v - o);
            if (clear) sums[j * d + t] = 0.f;
        }
        __syncwarp();
        if (clear && lane == 0) cnts[j] = 0;
    }
    if (!(tol > 0.f) && shift_out == nullptr) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
    if (shift_out != nullptr && lane == 0 && j < KB) shift_out[j] = sqrtf(s);
    if (!(tol > 0.f)) return;
    __shared__ unsigned shift[8];
    if (lane == 0) shift[warp] = __float_as_uint(fabsf(sqrtf(s)));      // NaN orders above every number
    __syncthreads();
    if (threadIdx.x != 0) return;
    unsigned m = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) m = max(m, shift[w]);
    atomicMax(ctl + LLOYD_SHIFT, m);
    __threadfence();
    if (atomicAdd(ctl + LLOYD_BLOCKS, 1u) != gridDim.x - 1) return;
    __threadfence();
    m = atomicExch(ctl + LLOYD_SHIFT, 0u);
    ctl[LLOYD_BLOCKS] = 0;
    const int done = __uint_as_float(m) < tol;
    if (done) ctl[LLOYD_DONE] = 1;
    __threadfence_system();
    host[0] = done ? -(it + 1) : it + 1;
}

int launch_kmeans_step(float* sums, int32_t* cnts, const float* old_c, float* new_c, int64_t KB, int d, int clear, float tol, int it,
                       int32_t* ctl, int32_t* host, float* shift, cudaStream_t st) {
    kmeans_step_kernel<<<(unsigned)ceil_div(KB, 8), 256, 0, st>>>(sums, cnts, old_c, new_c, KB, d, clear, tol, it,
                                                                  reinterpret_cast<unsigned*>(ctl), host, shift);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

// Waits until the device has finished `want` iterations or converged, or the stream has stopped.
void lloyd_wait(const int32_t* host, int want, cudaStream_t st) {
    for (unsigned spin = 1;; ++spin) {
        const int v = __atomic_load_n(host, __ATOMIC_ACQUIRE);
        if (v < 0 || v >= want) return;
        if ((spin & 1023u) == 0) {
            if (cudaStreamQuery(st) != cudaErrorNotReady) return;
            sched_yield();
        }
    }
}

}  // namespace fl

using namespace fl;

// Which kernel an assignment of `rows` rows is for: a batch counts with all its rows.  0: the tensor cores,
// 1: the CUDA cores.  A tensor-core call (problem by problem) costs 105 us plus 0.2 ns a row and 0.0002 ns a
// pair whatever the features (up to 128): 1M x 8, K = 256: 320 us against 190 here; 1M x 8, K = 1 024: 626 and
// 726; 65 536 x 8, K = 256: 147 and 29; 200 000 x 64, K = 200: 167 and 215.
extern "C" int fl_kmeans_assign_pick(int batch, int64_t n, int K, int d) {
    if (batch < 1 || n < 1 || K < 1 || d < 1 || d > ROWS_MAX_D) return 0;
    const double tc = batch * (105.0 + 2e-4 * (double)n + 2e-7 * (double)n * K);
    return rows_estimate_us((int64_t)batch * n, K, d) <= tc;
}

// 1 where a Lloyd loop through fl_kmeans_lloyd_f32 beats one of single steps with the tile kernel, whose launches
// and host work take some 100 us an iteration (50 001 x 33, K = 50: 120 us against 36).
extern "C" int fl_kmeans_lloyd_pick(int batch, int64_t n, int K, int d) {
    if (batch < 1 || n < 1 || K < 1 || d < 1 || d > ROWS_MAX_D) return 0;
    return rows_estimate_us((int64_t)batch * n, K, d) <= tile_estimate_us((int64_t)batch * n, K, d) + 60.0;
}

extern "C" int fl_kmeans_lloyd_words(void) { return LLOYD_WORDS; }

extern "C" int fl_kmeans_lloyd_f32(const float* x, int batch, int64_t n, int64_t ldx, int64_t x_batch_stride, int d, int K,
                                   float* cents_a, float* cents_b, float* sums, int32_t* cnts, int32_t* labels, int iters,
                                   float tol, int refresh, int32_t* ctl, int32_t* host, int* n_iter, void* stream) {
    FL_CHECK_ARG(batch >= 1 && batch <= 65535 && n >= 1 && K >= 1 && d >= 1 && ldx >= d && iters >= 1 && refresh >= 1,
                 "fl_kmeans_lloyd_f32: bad shape");
    FL_CHECK_ARG(x && cents_a && cents_b && sums && cnts && labels && ctl && n_iter && (host || !(tol > 0.f)),
                 "fl_kmeans_lloyd_f32: null pointer");
    FL_CHECK_ARG((int64_t)batch * K < (1ll << 31), "fl_kmeans_lloyd_f32: too large");
    if (d > ROWS_MAX_D) { set_error("fl_kmeans_lloyd_f32: d=%d > %d", d, ROWS_MAX_D); return FL_EUNSUPPORTED; }
    cudaStream_t st = (cudaStream_t)stream;
    const bool test = tol > 0.f;
    if (test) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        FL_CHECK_CUDA(cudaStreamIsCapturing(st, &cap));
        FL_CHECK_ARG(cap == cudaStreamCaptureStatusNone, "fl_kmeans_lloyd_f32: a loop that tests convergence cannot be captured");
        *host = 0;
    }
    const int64_t KB = (int64_t)batch * K;
    FL_CHECK_CUDA(cudaMemsetAsync(sums, 0, sizeof(float) * (size_t)KB * d, st));
    FL_CHECK_CUDA(cudaMemsetAsync(cnts, 0, sizeof(int32_t) * (size_t)KB, st));
    FL_CHECK_CUDA(cudaMemsetAsync(ctl, 0, sizeof(int32_t) * LLOYD_WORDS, st));
    float* cur = cents_a;
    float* nxt = cents_b;
    for (int it = 0; it < iters; ++it) {
        // The host stays at most three iterations ahead: launches after the one that converges do nothing.
        if (test && it >= 3) {
            lloyd_wait(host, it - 2, st);
            if (__atomic_load_n(host, __ATOMIC_ACQUIRE) < 0) break;
        }
        RowsParams p{};
        p.x = x; p.n = n; p.ldx = ldx; p.xbs = x_batch_stride; p.d = d;
        p.c = cur; p.K = K; p.ldc = d; p.cbs = (int64_t)K * d; p.labels = labels;
        p.sums = sums; p.cnts = cnts; p.add_all = it % refresh == 0;
        p.done = test ? ctl + LLOYD_DONE : nullptr;
        const int rc = rows_dispatch(p, batch, st);
        if (rc != FL_OK) {
            if (test) cudaStreamSynchronize(st);       // launched steps still write to `host`
            return rc;
        }
        const int rs = launch_kmeans_step(sums, cnts, cur, nxt, KB, d, (it + 1) % refresh == 0, tol, it, ctl, host, nullptr, st);
        if (rs != FL_OK) {
            if (test) cudaStreamSynchronize(st);
            return rs;
        }
        float* t = cur; cur = nxt; nxt = t;
    }
    *n_iter = iters;
    if (test) {
        lloyd_wait(host, iters, st);
        int v = __atomic_load_n(host, __ATOMIC_ACQUIRE);
        if (v >= 0 && v < iters) {
            FL_CHECK_CUDA(cudaStreamSynchronize(st));      // the stream stopped early: reports its error
            v = __atomic_load_n(host, __ATOMIC_ACQUIRE);
        }
        *n_iter = v < 0 ? -v : v;
    }
    return FL_OK;
}
