// Tensor-core k-means assignment: the sample rows play the queries and the centroids the
// database of the kNN candidate kernel (knn_tc.cu); a lean per-point kernel then re-scores
// the few best candidates exactly, proves the winner against the scoring error bound and
// queues the points it cannot prove for the exact CUDA-core path.
#include "knn_internal.h"
#include "pool.cuh"
#include "kmeans_rows.h"
#include <cuda_bf16.h>

namespace fl {

// Split operand planes.  An fp32 value v is carried as hi = bf16(v) and lo = bf16(v - hi); the
// plane rows hold [hi | lo | hi | ones] (samples) and [lo | hi | hi | norm terms] (centroids), so one bf16 product
// over 3 d_pad columns yields  hi.lo + lo.hi + hi.hi,  i.e. the fp32 inner product up to the
// dropped lo.lo term and the second-order residuals: an error of about 10^-5 ||x|| ||c|| on ordinary data, at
// most 2^-15, where one rounding errs by 0.0037 and at most 2^-7.  (The large term comes last: fp32 roundings of the
// small ones do not count, see score_acc_split.)  Used when 3 d_pad columns of a 128-row tile fit in shared
// memory (d <= 128).
__device__ __forceinline__ void bf16_split(float v, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(v);
    lo = __float2bfloat16_rn(v - __bfloat162float(hi));
}

// The two halves of four values, and the squares of what the first and both of them miss added to lost and lost2.
__device__ __forceinline__ void bf16_split4(float4 v, uint2& hi, uint2& lo, float& lost, float& lost2) {
    const float4 rest = bf16_lost4(v);
    lost += sq4(rest);
    lost2 += sq4(bf16_lost4(rest));
    __nv_bfloat16 h[4], l[4];
    bf16_split(v.x, h[0], l[0]);
    bf16_split(v.y, h[1], l[1]);
    bf16_split(v.z, h[2], l[2]);
    bf16_split(v.w, h[3], l[3]);
    auto bits = [](__nv_bfloat16 a, __nv_bfloat16 b) {
        return (uint32_t)__bfloat16_as_ushort(a) | (uint32_t)__bfloat16_as_ushort(b) << 16;
    };
    hi = make_uint2(bits(h[0], h[1]), bits(h[2], h[3]));
    lo = make_uint2(bits(l[0], l[1]), bits(l[2], l[3]));
}

// Centroid side, one warp per row (four columns a lane: wide reads where `vec` allows, 8-byte writes): [m_pad][3 d_pad + 16] rows, ||c||^2/2 per row and the
// largest norms (of the rows, of what hi and hi + lo miss of them).  Padding rows score -3e38.
__global__ void split_c_plane_kernel(const float* __restrict__ c, int64_t m, int d, int64_t ld,
                                     __nv_bfloat16* __restrict__ rows, float* __restrict__ hnorm,
                                     unsigned int* __restrict__ norm_bits, int64_t m_pad, int d_pad, int vec) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int pitch = 3 * d_pad + PLANE_AUG_COLS;
    __nv_bfloat16* o = rows + row * pitch;
    float sq[3] = {0.f, 0.f, 0.f};              // NORM_ROW, NORM_LOST, NORM_LOST2
    if (row >= m) {
        for (int t = lane; t < pitch; t += 32) o[t] = __float2bfloat16_rn(t == 3 * d_pad ? -3.0e38f : 0.f);
        if (lane == 0) hnorm[row] = pos_inf();
    } else {
        const float* p = c + row * ld;
        for (int t = lane * 4; t < d_pad; t += 128) {
            const float4 v = ld_row4(p, t, d, vec, DT_F32);
            sq[0] += sq4(v);
            uint2 hi, lo;
            bf16_split4(v, hi, lo, sq[1], sq[2]);
            *reinterpret_cast<uint2*>(o + t) = lo;
            *reinterpret_cast<uint2*>(o + d_pad + t) = hi;
            *reinterpret_cast<uint2*>(o + 2 * d_pad + t) = hi;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
            for (int i = 0; i < 3; ++i) sq[i] += __shfl_xor_sync(FULL_MASK, sq[i], off);
        }
        if (lane == 0) hnorm[row] = 0.5f * sq[0];
        write_norm_columns(o + 3 * d_pad, sq[0], PLANE_AUG_COLS);
    }
    block_norms_update(norm_bits, sq);
}

// Sample side of the second stage: the points listed in `rows` (live count on the device, at most
// `cap`), one warp per row in a grid-stride loop, written as split rows [hi | lo | hi | ones].
// With `tau_out` (kNN second stage) row r also gets its starting threshold: the exact k-th distance
// d_k found so far (prev_dist [point][k]) bounds the true one from above, so every true neighbour
// scores at least (||x||^2 - d_k) / 2 exactly and at most eps (score_eps of split operands) less in
// this stage; the threshold sits 2 eps and the proof's slack below that, so that a pool that never
// overflowed proves its row.
__global__ void split_x_gather_kernel(const float* __restrict__ x, int64_t ldx, int d, const int* __restrict__ rows,
                                      const int* __restrict__ rows_count, int cap, __nv_bfloat16* __restrict__ out,
                                      int d_pad, const float* __restrict__ prev_dist, int k,
                                      const float* __restrict__ norms, float acc, float* __restrict__ tau_out, int vec) {
    const int lane = threadIdx.x & 31;
    const int pitch = 3 * d_pad + PLANE_AUG_COLS;
    int count = *rows_count;
    count = count < cap ? count : cap;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    if (tau_out != nullptr) {
        // rows of the last live tile beyond the list's end hold stale memory: they must never append
        const int tile_end = (count + 127) & ~127;
        for (int r = count + blockIdx.x * blockDim.x + threadIdx.x; r < tile_end; r += gridDim.x * blockDim.x) tau_out[r] = pos_inf();
    }
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < count; r += nwarps) {
        const int64_t pt = rows[r];
        const float* src = x + pt * ldx;
        __nv_bfloat16* o = out + (int64_t)r * pitch;
        float qsq = 0.f, lost = 0.f, lost2 = 0.f;
        for (int t = lane * 4; t < d_pad; t += 128) {
            uint2 hi, lo;
            const float4 v = ld_row4(src, t, d, vec, DT_F32);
            qsq += sq4(v);
            bf16_split4(v, hi, lo, lost, lost2);
            *reinterpret_cast<uint2*>(o + t) = hi;
            *reinterpret_cast<uint2*>(o + d_pad + t) = lo;
            *reinterpret_cast<uint2*>(o + 2 * d_pad + t) = hi;
        }
        if (lane < PLANE_AUG_COLS) o[3 * d_pad + lane] = __float2bfloat16_rn(lane < 3 ? 1.f : 0.f);
        if (tau_out != nullptr) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                qsq += __shfl_xor_sync(FULL_MASK, qsq, off);
                lost += __shfl_xor_sync(FULL_MASK, lost, off);
                lost2 += __shfl_xor_sync(FULL_MASK, lost2, off);
            }
            if (lane == 0) {
                const float dk = prev_dist[pt * k + (k - 1)];
                float tau = neg_inf();
                if (dk < pos_inf())
                    tau = 0.5f * (qsq - dk) - 2.f * score_eps(OPERANDS_SPLIT, qsq, lost, lost2, norms, acc) -
                          proof_slack(qsq, __ldg(norms + NORM_ROW), d);
                tau_out[r] = tau > neg_inf() ? tau : neg_inf();
            }
        }
    }
}

// Eight lanes per point, four points per warp, grid-stride.  The scoring pass left, for each half
// of the centroid columns, the best and second-best score and the best centroid of scoring row r.
// Row r is point r (first stage) or point rows[r] (second stage, live count on the device).
// Both best centroids are re-scored with exact fp32 sum (x - c)^2; the closer one wins (lower
// index on exact ties).  Every other centroid scored at most `bound` = the larger of the two
// second-best scores (plus the 2^-16 relative perturbation of carrying the column index in the
// score's low mantissa bits), so the label is proven when its exact distance is below
// ||x||^2 - 2 (bound + eps); otherwise the point goes to the `next` list (the next, more precise
// stage) or, when that is absent or full, to the exact-path list.
//
// SPLIT: the scores are those of the split planes, and what their roundings took of the point is summed up here; for plain
// bf16 operands that comes with ||x||^2 from the pass that rounded the points (xsq).
template <bool SPLIT>
__global__ void __launch_bounds__(128) assign_finalize_kernel(
    const float* __restrict__ x, int64_t n, int64_t ldx, const float* __restrict__ c, int K, int64_t ldc, int d,
    int vec, const float* __restrict__ asg_sc, const uint32_t* __restrict__ asg_id, const float2* __restrict__ xsq, float acc,
    const float* __restrict__ norms, int32_t* __restrict__ labels, const int* __restrict__ rows,
    const int* __restrict__ rows_count, int* __restrict__ next_count, int* __restrict__ next_list, int next_cap,
    int* __restrict__ fb_count, int* __restrict__ fb_list, int fb_cap, int scores_by_point) {
    const int sl = threadIdx.x & 7;
    int64_t live = n;
    if (rows_count != nullptr) { const int64_t cnt = *rows_count; live = cnt < n ? cnt : n; }
    const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) >> 3;
    const int64_t rounds = (live + ngroups - 1) / ngroups;
    for (int64_t it = 0; it < rounds; ++it) {
        const int64_t r_raw = it * ngroups + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3);
        const bool alive = r_raw < live;
        const int64_t r = alive ? r_raw : live - 1;          // idle groups shadow the last row
        const int64_t pt = rows != nullptr ? (int64_t)rows[r] : r;
        // the scores sit at the scoring row: the list position (points gathered for their own scoring
        // pass) or the point itself (a list of points that were scored in place)
        const int64_t sr = scores_by_point ? pt : r;
        const float4 sc = __ldg(reinterpret_cast<const float4*>(asg_sc + sr * 4));   // b1_0, b2_0, b1_1, b2_1
        const uint2 ids = __ldg(reinterpret_cast<const uint2*>(asg_id + sr * 2));
        const bool v0 = ids.x < (uint32_t)K && sc.x > -1e37f;   // false: no real centroid in that half
        const bool v1 = ids.y < (uint32_t)K && sc.z > -1e37f;
        const float* xp = x + pt * ldx;
        const float* c0 = c + (int64_t)(v0 ? ids.x : 0u) * ldc;
        const float* c1 = c + (int64_t)(v1 ? ids.y : 0u) * ldc;
        float qsq = 0.f, lost = 0.f, lost2 = 0.f, a0 = 0.f, a1 = 0.f;
        if (vec) {
#pragma unroll 4
            for (int t = sl * 4; t < d; t += 32) {
                const float4 xv = __ldg(reinterpret_cast<const float4*>(xp + t));
                const float4 p0 = __ldg(reinterpret_cast<const float4*>(c0 + t));
                const float4 p1 = __ldg(reinterpret_cast<const float4*>(c1 + t));
                if (SPLIT) {
                    qsq += sq4(xv);
                    const float4 l = bf16_lost4(xv);
                    lost += sq4(l);
                    lost2 += sq4(bf16_lost4(l));
                }
                float e0 = xv.x - p0.x, e1 = xv.y - p0.y, e2 = xv.z - p0.z, e3 = xv.w - p0.w;
                a0 += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
                e0 = xv.x - p1.x; e1 = xv.y - p1.y; e2 = xv.z - p1.z; e3 = xv.w - p1.w;
                a1 += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
            }
        } else {
            for (int t = sl; t < d; t += 8) {
                const float xv = __ldg(xp + t);
                const float e0 = xv - __ldg(c0 + t), e1 = xv - __ldg(c1 + t);
                if (SPLIT) {
                    const float l = bf16_lost(xv), l2 = bf16_lost(l);
                    qsq += xv * xv; lost += l * l; lost2 += l2 * l2;
                }
                a0 += e0 * e0; a1 += e1 * e1;
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            if (SPLIT) {
                qsq += __shfl_xor_sync(FULL_MASK, qsq, o);
                lost += __shfl_xor_sync(FULL_MASK, lost, o);
                lost2 += __shfl_xor_sync(FULL_MASK, lost2, o);
            }
            a0 += __shfl_xor_sync(FULL_MASK, a0, o);
            a1 += __shfl_xor_sync(FULL_MASK, a1, o);
        }
        if (!alive || sl != 0) continue;
        float best_d = pos_inf();
        uint32_t best_i = INVALID_ID;
        if (v0) { best_d = a0; best_i = ids.x; }
        if (v1 && (a1 < best_d || (a1 == best_d && ids.y < best_i))) { best_d = a1; best_i = ids.y; }
        float bound = fmaxf(sc.y, sc.w);
        bool ok = best_i != INVALID_ID;
        if (ok && bound > -1e37f) {
            bound += fabsf(bound) * 3.1e-5f;                       // index bits in the mantissa: 2^-15 relative
            if (!SPLIT) {
                const float2 x2 = __ldg(xsq + pt);
                qsq = x2.x;
                lost = x2.y;
            }
            ok = list_proven(best_d, qsq, bound, score_eps(SPLIT ? OPERANDS_SPLIT : OPERANDS_BF16, qsq, lost, lost2, norms, acc),
                             proof_slack(qsq, __ldg(norms + NORM_ROW), d));
        }
        labels[pt] = ok ? (int32_t)best_i : 0;
        if (!ok) {
            bool queued = false;
            if (next_count != nullptr) {
                const int i = atomicAdd(next_count, 1);
                if (i < next_cap) { next_list[i] = (int)pt; queued = true; }
            }
            if (!queued) {
                const int i = atomicAdd(fb_count, 1);
                if (i < fb_cap) fb_list[i] = (int)pt;
            }
        }
    }
}

// First-stage proof from the scores alone, one thread per point: the best-scoring centroid is the
// nearest one if its score leads the runner-up's by more than twice the scoring error bound (every
// score is within eps of the exact <x,c> - ||c||^2/2, so the exact scores keep that order).  No
// sample row and no centroid is read -- 32 bytes per point instead of its 4 d -- at the price of a
// lead of 2 eps where the exact re-scoring of assign_finalize_kernel needs eps; what the lead does
// not decide goes to the `next` list (the second stage, whose bound is a hundred times smaller).
//
// Inside a Lloyd loop (live.rows: the points this iteration scores at all, or all of them) a proven point also gets its
// bounds for the next iterations: at most `x` from its centroid, at least `y` from every other one.
struct LivePoints {
    const int* rows;         // listed points and their number (device), or, when *count is negative, all n of them
    const int* count;
    float2* bounds;
};
__global__ void __launch_bounds__(256) assign_by_lead_kernel(
    int64_t n, int K, int d, const float* __restrict__ asg_sc, const uint32_t* __restrict__ asg_id, const float2* __restrict__ xsq,
    float acc, const float* __restrict__ norms, int32_t* __restrict__ labels, int* __restrict__ next_count,
    int* __restrict__ next_list, int next_cap, int* __restrict__ fb_count, int* __restrict__ fb_list, int fb_cap,
    const LivePoints live) {
    int64_t pt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pt >= n) return;
    const int listed = live.count != nullptr ? __ldg(live.count) : -1;
    if (listed >= 0) {
        if (pt >= listed) return;
        pt = __ldg(live.rows + pt);
    }
    const float4 sc = __ldg(reinterpret_cast<const float4*>(asg_sc + pt * 4));   // b1_0, b2_0, b1_1, b2_1
    const uint2 ids = __ldg(reinterpret_cast<const uint2*>(asg_id + pt * 2));
    const bool v0 = ids.x < (uint32_t)K && sc.x > -1e37f;   // false: no real centroid in that half
    const bool v1 = ids.y < (uint32_t)K && sc.z > -1e37f;
    const bool first = v0 && (!v1 || sc.x >= sc.z);
    const float best = first ? sc.x : sc.z;
    const uint32_t best_i = first ? ids.x : ids.y;
    float second = first ? sc.y : sc.w;                      // runner-up of the winner's half ...
    if (v0 && v1) second = fmaxf(second, first ? sc.z : sc.x);   // ... or the other half's best
    bool ok = v0 || v1;
    if (ok && second > -1e37f) {
        const float2 x2 = __ldg(xsq + pt);
        const float q2 = x2.x, eps = score_eps(OPERANDS_BF16, q2, x2.y, 0.f, norms, acc);
        // the column index rides in the low mantissa bits of both scores: 2^-15 relative each
        const float lo = best - fabsf(best) * 3.1e-5f, hi = second + fabsf(second) * 3.1e-5f;
        const float slack = proof_slack(q2, __ldg(norms + NORM_ROW), d);
        ok = lo - hi > 2.f * eps + slack;
        if (live.bounds != nullptr) {
            // squared distances from the scores, both ends of the error band (no bounds for a point that is not proven)
            const float du = q2 - 2.f * (lo - eps) + slack, dl = q2 - 2.f * (hi + eps) - slack;
            live.bounds[pt] = ok ? make_float2(__fsqrt_ru(fmaxf(du, 0.f)), dl > 0.f ? __fsqrt_rd(dl) : 0.f) : make_float2(pos_inf(), 0.f);
        }
    } else if (live.bounds != nullptr) {
        live.bounds[pt] = make_float2(pos_inf(), 0.f);
    }
    labels[pt] = ok ? (int32_t)best_i : 0;
    if (!ok) {
        bool queued = false;
        if (next_count != nullptr) {
            const int i = atomicAdd(next_count, 1);
            if (i < next_cap) { next_list[i] = (int)pt; queued = true; }
        }
        if (!queued) {
            const int i = atomicAdd(fb_count, 1);
            if (i < fb_cap) fb_list[i] = (int)pt;
        }
    }
}

// Which points of a Lloyd iteration need their scores at all (Hamerly, "Making k-means even faster", SDM 2010).  Since the
// bounds of a point were taken its own centroid has moved by shift[label] and no other by more than the largest shift of
// the others: while the upper bound so widened stays below the lower one, the label cannot have changed.  The sums are
// rounded against the point, and `shift` -- an fp32 norm of up to 128 differences -- counts 2 10^-5 more than it says.
// The rest is listed; when that is more than `most`, all points are scored in place instead (count[0] < 0) and nothing
// is gathered.  count: [0] points listed or -1, [1] rows of the gathered pass, [2] rows of the pass in place, [3] blocks
// done, [4] points found (cleared by the caller).
// Bound by HBM: 20 bytes a point.
constexpr int BOUNDS_THREADS = 256, BOUNDS_PER = 4;
__global__ void __launch_bounds__(BOUNDS_THREADS) lloyd_bounds_kernel(int64_t n, int K, const int32_t* __restrict__ labels,
                                                                      float2* __restrict__ bounds, const float* __restrict__ shift,
                                                                      const int32_t* __restrict__ done, int most,
                                                                      int* __restrict__ list, int* __restrict__ count) {
    __shared__ float s_m1[BOUNDS_THREADS / 32], s_m2[BOUNDS_THREADS / 32];
    __shared__ int s_at[BOUNDS_THREADS / 32], s_n[BOUNDS_THREADS / 32], s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the largest shift, whose it is, and the largest of the others; a shift that is no number counts as infinite
    float m1 = -1.f, m2 = -1.f;
    int at = -1;
    auto fold = [&](float a1, int aa, float a2) {
        if (a1 > m1) { m2 = fmaxf(m1, a2); m1 = a1; at = aa; } else m2 = fmaxf(m2, a1);
    };
    auto moved = [&](int j) { const float s = __ldg(shift + j); return s >= 0.f ? s : pos_inf(); };
    for (int j = tid; j < K; j += BOUNDS_THREADS) fold(moved(j), j, -1.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float a1 = __shfl_xor_sync(FULL_MASK, m1, o), a2 = __shfl_xor_sync(FULL_MASK, m2, o);
        const int aa = __shfl_xor_sync(FULL_MASK, at, o);
        fold(a1, aa, a2);
    }
    if (lane == 0) { s_m1[warp] = m1; s_m2[warp] = m2; s_at[warp] = at; }
    __syncthreads();
    m1 = m2 = -1.f;
    at = -1;
    for (int w = 0; w < BOUNDS_THREADS / 32; ++w) fold(s_m1[w], s_at[w], s_m2[w]);
    constexpr float MORE = 1.00002f;
    m1 = __fmul_ru(fmaxf(m1, 0.f), MORE);
    m2 = __fmul_ru(fmaxf(m2, 0.f), MORE);
    const bool stop = done != nullptr && *done != 0;
    for (int64_t base = (int64_t)blockIdx.x * (BOUNDS_THREADS * BOUNDS_PER); base < n && !stop;
         base += (int64_t)gridDim.x * (BOUNDS_THREADS * BOUNDS_PER)) {
        bool live[BOUNDS_PER];
        int mine = 0;
#pragma unroll
        for (int i = 0; i < BOUNDS_PER; ++i) {
            const int64_t pt = base + i * BOUNDS_THREADS + tid;
            live[i] = false;
            if (pt < n) {
                const int lab = __ldg(labels + pt);               // (-1 where no distance is a number)
                float2 b = bounds[pt];
                b.x = __fadd_ru(b.x, lab >= 0 ? __fmul_ru(moved(lab), MORE) : pos_inf());
                b.y = __fsub_rd(b.y, lab == at ? m2 : m1);
                live[i] = !(b.x < b.y);
                if (!live[i]) bounds[pt] = b;         // (a listed point gets new ones, or none)
            }
            mine += live[i] ? 1 : 0;
        }
        int before = mine;                            // of this warp's lanes, then of the block's warps
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL_MASK, before, o);
            if (lane >= o) before += t;
        }
        if (lane == 31) s_n[warp] = before;
        __syncthreads();
        if (tid == 0) {
            int total = 0;
            for (int w = 0; w < BOUNDS_THREADS / 32; ++w) { const int t = s_n[w]; s_n[w] = total; total += t; }
            s_base = total > 0 ? atomicAdd(count + 4, total) : 0;
        }
        __syncthreads();
        int pos = s_base + s_n[warp] + before - mine;
#pragma unroll
        for (int i = 0; i < BOUNDS_PER; ++i)
            if (live[i]) list[pos++] = (int)(base + i * BOUNDS_THREADS + tid);
        __syncthreads();
    }
    if (tid != 0) return;
    __threadfence();
    if (atomicAdd(count + 3, 1) != (int)gridDim.x - 1) return;
    const int found = atomicAdd(count + 4, 0);
    const bool all = found > most;
    count[0] = all ? -1 : found;
    count[1] = all ? 0 : found;
    count[2] = all ? (int)n : 0;
}

// Plane rows of the listed points side by side (a warp copies one, 16 bytes a lane; rows are multiples of 32 bytes).
__global__ void __launch_bounds__(256) gather_rows_kernel(const uint4* __restrict__ plane, int words, const int* __restrict__ list,
                                                          const int* __restrict__ count, uint4* __restrict__ out) {
    const int lane = threadIdx.x & 31, live = __ldg(count), warps = (gridDim.x * blockDim.x) >> 5;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < live; r += warps) {
        const uint4* src = plane + (int64_t)__ldg(list + r) * words;
        for (int c = lane; c < words; c += 32) out[(int64_t)r * words + c] = __ldg(src + c);
    }
}

// Points whose label could not be proven, when they are few: one block per listed point, eight lanes per centroid,
// the fp32 sum (x - c)^2 to every centroid; the lowest index wins exact ties.  Left to the tile pass (`rest`,
// whose counter starts at zero): longer lists as a whole, where the tiles' reuse of the centroids pays, and
// points without a finite distance.  Bound by latency -- a block walks K / 64 dependent loads: for the few dozen points
// of the 1M x 128, K = 1 024 loop 24 us (and 7 for the empty tile pass) where the tile pass and its finalisation took 78 + 20.
constexpr int ASSIGN_DIRECT_MAX = 2048, ASSIGN_DIRECT_MAX_K = 4096;
__global__ void __launch_bounds__(256) assign_direct_kernel(
    const float* __restrict__ x, int64_t ldx, const float* __restrict__ c, int K, int64_t ldc, int d, int vec,
    const int* __restrict__ list, const int* __restrict__ list_count, int32_t* __restrict__ labels,
    int* __restrict__ rest_list, int* __restrict__ rest_count) {
    __shared__ __align__(16) float xs[256];
    __shared__ float s_best[8];
    __shared__ int s_idx[8];
    const int tid = threadIdx.x, lane = tid & 31, sl = tid & 7, g = tid >> 3;
    const int count = *list_count;
    if (count > ASSIGN_DIRECT_MAX) {
        for (int i = blockIdx.x * 256 + tid; i < count; i += gridDim.x * 256) rest_list[i] = list[i];
        if (blockIdx.x == 0 && tid == 0) *rest_count = count;
        return;
    }
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int pt = list[i];
        if (tid < d) xs[tid] = __ldg(x + (int64_t)pt * ldx + tid);
        __syncthreads();
        float best = pos_inf();
        int bi = 0x7fffffff;
        for (int base = 0; base < K; base += 64) {
            const int j0 = base + g, j1 = base + 32 + g;
            const float* c0 = c + (int64_t)(j0 < K ? j0 : K - 1) * ldc;
            const float* c1 = c + (int64_t)(j1 < K ? j1 : K - 1) * ldc;
            float a0 = 0.f, a1 = 0.f;
            if (vec) {
#pragma unroll 4
                for (int t = sl * 4; t < d; t += 32) {
                    const float4 xv = *reinterpret_cast<const float4*>(xs + t);
                    const float4 p0 = __ldg(reinterpret_cast<const float4*>(c0 + t));
                    const float4 p1 = __ldg(reinterpret_cast<const float4*>(c1 + t));
                    float e0 = xv.x - p0.x, e1 = xv.y - p0.y, e2 = xv.z - p0.z, e3 = xv.w - p0.w;
                    a0 += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
                    e0 = xv.x - p1.x; e1 = xv.y - p1.y; e2 = xv.z - p1.z; e3 = xv.w - p1.w;
                    a1 += e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
                }
            } else {
#pragma unroll 4
                for (int t = sl; t < d; t += 8) {
                    const float e0 = xs[t] - __ldg(c0 + t), e1 = xs[t] - __ldg(c1 + t);
                    a0 += e0 * e0;
                    a1 += e1 * e1;
                }
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                a0 += __shfl_xor_sync(FULL_MASK, a0, o);
                a1 += __shfl_xor_sync(FULL_MASK, a1, o);
            }
            if (j0 < K && a0 < best) { best = a0; bi = j0; }       // ascending: the lower index stays on ties
            if (j1 < K && a1 < best) { best = a1; bi = j1; }
        }
#pragma unroll
        for (int o = 16; o >= 8; o >>= 1) {
            const float ob = __shfl_xor_sync(FULL_MASK, best, o);
            const int oi = __shfl_xor_sync(FULL_MASK, bi, o);
            if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) { s_best[tid >> 5] = best; s_idx[tid >> 5] = bi; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < 8; ++w)
                if (s_best[w] < best || (s_best[w] == best && s_idx[w] < bi)) { best = s_best[w]; bi = s_idx[w]; }
            if (bi != 0x7fffffff) labels[pt] = bi;
            else rest_list[atomicAdd(rest_count, 1)] = pt;
        }
        __syncthreads();
    }
}

struct AssignTcWs {
    int64_t n_pad; int d_pad, pitch; int fb_cap;
    int split;          // 1: a second stage with split (hi/lo) operand planes of 3 d_pad columns
    int l1_cap; int64_t l1_pad; int pitch3;
    int nsplit_fb; int64_t rows_per_split_fb; int fb_bq, fb_blocks;
    PlaneLayout cl, cl3;
    int64_t off_cplane, off_cplane3, off_xplane, off_xsq, off_xfmt, off_xsplit, off_asg_sc, off_asg_id, off_cnt, off_l0list, off_l1list,
        off_fblist, off_fblist2, off_fbpart_sc, off_fbpart_id, off_fbdist, bytes;
};

// Split planes need the 128-row sample tile of 3 d_pad columns resident in shared memory
// beside a three-slot TMA ring: d <= 128.
static int assign_tc_split(int d) { return d <= 128; }

static int64_t take(int64_t& cur, int64_t bytes) {
    const int64_t o = cur;
    cur += round_up(bytes > 0 ? bytes : 1, 1024);
    return o;
}

static AssignTcWs assign_tc_plan(int64_t n, int K, int d, int have_xplane) {
    AssignTcWs w{};
    w.n_pad = round_up(n, 128);
    w.split = assign_tc_split(d);
    w.d_pad = (int)round_up(d, 64);
    w.pitch = w.d_pad + PLANE_AUG_COLS;
    w.pitch3 = 3 * w.d_pad + PLANE_AUG_COLS;
    w.cl = plane_layout(K, w.d_pad);
    w.cl3 = plane_layout(K, 3 * w.d_pad);     // same row count, hnorm and meta blocks; 3 d_pad feature columns
    w.fb_cap = (int)n;   // every point may take the exact path: no overflow case to report
    // second stage: room for half of the points (more unproven points than that take the exact path)
    w.l1_cap = w.split ? (int)((n + 1) / 2) : 0;
    w.l1_pad = round_up(w.l1_cap > 0 ? w.l1_cap : 1, 128);
    simt_split_plan(w.fb_cap, K, 32, d, &w.nsplit_fb, &w.rows_per_split_fb);
    // the exact pass spreads a fixed grid over the live points (simt_dyn_split): one pool per
    // (block, query slot) at most
    w.fb_bq = simt_block_queries(32);
    w.fb_blocks = (int)(ceil_div(w.fb_cap, w.fb_bq > 0 ? w.fb_bq : 1) * w.nsplit_fb);
    if (w.fb_blocks < 4 * sm_count()) w.fb_blocks = 4 * sm_count();
    const int64_t fb_pools = (int64_t)w.fb_blocks * (w.fb_bq > 0 ? w.fb_bq : 1);
    int64_t cur = 0;
    w.off_cplane = take(cur, w.cl.bytes);
    w.off_cplane3 = w.split ? take(cur, w.cl3.bytes) : -1;
    w.off_xplane = have_xplane ? -1 : take(cur, w.n_pad * w.pitch * 2);
    w.off_xsq = have_xplane ? -1 : take(cur, w.n_pad * 8);
    w.off_xfmt = have_xplane ? -1 : take(cur, 4);
    w.off_xsplit = w.split ? take(cur, w.l1_pad * w.pitch3 * 2) : -1;
    w.off_asg_sc = take(cur, w.n_pad * 4 * 4);
    w.off_asg_id = take(cur, w.n_pad * 2 * 4);
    w.off_cnt = take(cur, 1024);
    w.off_l0list = take(cur, (w.split ? n : 1) * 4);
    w.off_l1list = take(cur, (int64_t)(w.l1_cap > 0 ? w.l1_cap : 1) * 4);
    w.off_fblist = take(cur, (int64_t)w.fb_cap * 4);
    w.off_fblist2 = take(cur, (int64_t)w.fb_cap * 4);
    w.off_fbpart_sc = take(cur, fb_pools * 32 * 4);
    w.off_fbpart_id = take(cur, fb_pools * 32 * 4);
    w.off_fbdist = take(cur, n * 4);
    w.bytes = cur;
    return w;
}

int split_plane_supported(int d) { return assign_tc_split(d); }

// Split database plane [lo | hi | hi | norm terms] in the layout plane_layout(m, 3 d_pad).
int launch_split_db_plane(const float* c, int64_t m, int d, int64_t ldc, void* plane, cudaStream_t st) {
    const int d_pad = (int)round_up(d, 64);
    const PlaneLayout L = plane_layout(m, 3 * d_pad);
    char* pl = static_cast<char*>(plane);
    FL_CHECK_CUDA(cudaMemsetAsync(pl + L.off_meta, 0, 1024, st));
    const int wpb = 8;
    split_c_plane_kernel<<<(unsigned)ceil_div(L.m_pad, wpb), wpb * 32, 0, st>>>(
        c, m, d, ldc, reinterpret_cast<__nv_bfloat16*>(pl + L.off_rows), reinterpret_cast<float*>(pl + L.off_hnorm),
        reinterpret_cast<unsigned int*>(pl + L.off_meta), L.m_pad, d_pad, dt_vec_ok(c, ldc, DT_F32) && d % 4 == 0);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

int launch_split_query_gather(const float* x, int64_t ldx, int d, const int* rows, const int* rows_count, int cap,
                              void* out, int d_pad, const float* prev_dist, int k, const float* norms, float acc,
                              float* tau_out, cudaStream_t st) {
    split_x_gather_kernel<<<(unsigned)(8 * sm_count()), 256, 0, st>>>(x, ldx, d, rows, rows_count, cap,
                                                                     static_cast<__nv_bfloat16*>(out), d_pad, prev_dist, k,
                                                                     norms, acc, tau_out,
                                                                     dt_vec_ok(x, ldx, DT_F32) && d % 4 == 0);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

int assign_tc_supported(int64_t n, int K, int d) {
    if (n < 1 || K < 1 || d > 256) return 0;
    return 1;
}

}  // namespace fl

using namespace fl;

static int64_t xplane_fmt_offset(int64_t n, int d) {
    return round_up(round_up(n, 128) * (round_up(d, 64) + PLANE_AUG_COLS) * 2, 1024) + round_up(n, 128) * 8;
}

extern "C" int64_t fl_kmeans_xplane_bytes(int64_t n, int d) {
    if (n < 1 || d < 1) return 0;
    // the 16-bit rows, then ||x||^2 of every row and the square of the norm of what rounding took of it (f32 [n_pad][2]), then
    // the operand format
    return xplane_fmt_offset(n, d) + 1024;
}

extern "C" int fl_kmeans_prepare_x_f32(const float* x, int64_t n, int d, int64_t ldx, void* xplane,
                                       int64_t xplane_bytes, void* stream) {
    FL_CHECK_ARG(x && xplane && n >= 1 && d >= 1 && ldx >= d, "fl_kmeans_prepare_x_f32: bad arguments");
    if (xplane_bytes < fl_kmeans_xplane_bytes(n, d)) { set_error("fl_kmeans_prepare_x_f32: plane buffer too small"); return FL_EWORKSPACE; }
    const int64_t n_pad = round_up(n, 128);
    // the rows' norms (the scoring error bound of a point needs its own) come from the same read
    float2* xsq = reinterpret_cast<float2*>(static_cast<char*>(xplane) + round_up(n_pad * (round_up(d, 64) + PLANE_AUG_COLS) * 2, 1024));
    uint32_t* fmt = reinterpret_cast<uint32_t*>(static_cast<char*>(xplane) + xplane_fmt_offset(n, d));
    const int rc = launch_operand_format(x, n, ldx, d, fmt, (cudaStream_t)stream);
    if (rc != FL_OK) return rc;
    return launch_query_plane(x, n, ldx, d, xplane, n_pad, (int)round_up(d, 64), (cudaStream_t)stream, DT_F32, xsq, fmt);
}

extern "C" int64_t fl_kmeans_assign_tc_workspace_bytes(int64_t n, int K, int d, int have_xplane) {
    if (!assign_tc_supported(n, K, d)) return 0;
    return assign_tc_plan(n, K, d, have_xplane).bytes;
}

// Two stages.  (1) planes of one rounding: every point is scored against every centroid; labels the
// proof accepts (scoring error about 0.0005 ||x|| max||c|| in fp16, which almost all data takes, 0.0037 in bf16) are final.  (2) d <= 128: the unproven points
// (a device-side list) are gathered into split planes and scored again, error about 6e-5: nearly all of
// the rest is proven.  What is left takes the exact CUDA-core path.
//
// live: inside a Lloyd loop, the points to score (n in place, or the listed ones through `gathered`, room for
// gathered_rows plane rows); needs the second stage (d <= 128) and a sample plane.
static int assign_tc_run(const float* x, int64_t n, int64_t ldx, const char* xpl, const float2* xsq, const uint32_t* fmt, const float* c,
                         int K, int64_t ldc, int d, int32_t* labels, char* base, const AssignTcWs& w, const LivePoints& live,
                         void* gathered, int64_t gathered_rows, int32_t* status, cudaStream_t st) {
    int rc;
    // centroid planes (database side): plain, and split for the second stage
    char* cpl = base + w.off_cplane;
    rc = launch_plane_build(c, K, d, ldc, cpl, st, DT_F32, fmt);
    if (rc != FL_OK) return rc;
    char* cpl3 = nullptr;
    if (w.split) {
        cpl3 = base + w.off_cplane3;
        rc = launch_split_db_plane(c, K, d, ldc, cpl3, st);
        if (rc != FL_OK) return rc;
    }
    int* counters = reinterpret_cast<int*>(base + w.off_cnt);
    int* fb_count = counters;          // points for the exact path
    int* l1_count = counters + 64;     // points for the second stage
    int* fb_list = reinterpret_cast<int*>(base + w.off_fblist);
    int* l1_list = reinterpret_cast<int*>(base + w.off_l1list);
    int* l0_count = counters + 128;    // points the scores' lead did not decide
    int* l0_list = reinterpret_cast<int*>(base + w.off_l0list);
    FL_CHECK_CUDA(cudaMemsetAsync(counters, 0, 1024, st));
    const int vecx = (ldx % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const int vecc = (ldc % 4 == 0) && ((reinterpret_cast<uintptr_t>(c) & 15) == 0);
    const int vec = vecx && vecc && (d % 4 == 0);
    float* asg_sc = reinterpret_cast<float*>(base + w.off_asg_sc);
    uint32_t* asg_id = reinterpret_cast<uint32_t*>(base + w.off_asg_id);
    const unsigned fin_grid = (unsigned)(4 * sm_count());      // grid-stride finalisation
    const float* norms = reinterpret_cast<const float*>(cpl + w.cl.off_meta);
    const float acc1 = score_acc(d + PLANE_AUG_COLS);

    // ---- stage 1: one rounding, to the samples' operand format ---------------------------------------------------------------
    {
        TcKnnParams tp{};
        tp.qplane = xpl; tp.nq = n; tp.nq_pad = w.n_pad;
        tp.dbrows = cpl + w.cl.off_rows; tp.hnorm = reinterpret_cast<const float*>(cpl + w.cl.off_hnorm);
        tp.fmt = fmt;
        tp.m = K; tp.m_pad = w.cl.m_pad; tp.d_pad = w.cl.d_pad; tp.d_used = d;
        tp.status = status;
        profile_begin(st);
        rc = launch_assign_tc(tp, asg_sc, asg_id, live.count != nullptr ? live.count + 2 : nullptr, st);
        if (rc == FL_OK && live.count != nullptr) {
            // the listed points, gathered; their scores go where the pass in place would have put them
            gather_rows_kernel<<<(unsigned)(8 * sm_count()), 256, 0, st>>>(reinterpret_cast<const uint4*>(xpl), w.pitch / 8, live.rows,
                                                                          live.count + 1, static_cast<uint4*>(gathered));
            FL_CHECK_LAUNCH();
            TcKnnParams tg = tp;
            tg.qplane = gathered; tg.nq = gathered_rows; tg.nq_pad = round_up(gathered_rows, 128);
            rc = launch_assign_tc(tg, asg_sc, asg_id, live.count + 1, st, live.rows);
        }
        profile_end(st);
        if (rc != FL_OK) return rc;
        if (w.split) {
            // a second, far more precise stage follows: decide what the scores' lead decides
            // without touching the rows
            assign_by_lead_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(
                n, K, d, asg_sc, asg_id, xsq, acc1, norms, labels, l0_count, l0_list, (int)n, fb_count, fb_list, w.fb_cap, live);
            FL_CHECK_LAUNCH();
            // ... then, for the undecided ones only, the exact distances to the two half-winners, which
            // need half the lead; what is still open goes to the second stage
            assign_finalize_kernel<false><<<fin_grid, 128, 0, st>>>(
                x, n, ldx, c, K, ldc, d, vec, asg_sc, asg_id, xsq, acc1, norms, labels, l0_list, l0_count,
                l1_count, l1_list, w.l1_cap, fb_count, fb_list, w.fb_cap, 1);
        } else {
            assign_finalize_kernel<false><<<fin_grid, 128, 0, st>>>(
                x, n, ldx, c, K, ldc, d, vec, asg_sc, asg_id, xsq, acc1, norms, labels, nullptr, nullptr,
                nullptr, l1_list, w.l1_cap, fb_count, fb_list, w.fb_cap, 0);
        }
        FL_CHECK_LAUNCH();
    }
    // ---- stage 2: split planes for the unproven points --------------------------------------
    if (w.split) {
        __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(base + w.off_xsplit);
        split_x_gather_kernel<<<(unsigned)(8 * sm_count()), 256, 0, st>>>(x, ldx, d, l1_list, l1_count, w.l1_cap, xs, w.d_pad,
                                                                         nullptr, 0, nullptr, 0.f, nullptr, vecx && d % 4 == 0);
        FL_CHECK_LAUNCH();
        TcKnnParams tp{};
        tp.qplane = xs; tp.nq = w.l1_cap; tp.nq_pad = w.l1_pad;
        tp.dbrows = cpl3 + w.cl3.off_rows; tp.hnorm = reinterpret_cast<const float*>(cpl3 + w.cl3.off_hnorm);
        tp.m = K; tp.m_pad = w.cl3.m_pad; tp.d_pad = w.cl3.d_pad; tp.d_used = 2 * w.d_pad + d;
        tp.status = status;
        rc = launch_assign_tc(tp, asg_sc, asg_id, l1_count, st);
        if (rc != FL_OK) return rc;
        assign_finalize_kernel<true><<<fin_grid, 128, 0, st>>>(
            x, w.l1_cap, ldx, c, K, ldc, d, vec, asg_sc, asg_id, nullptr, score_acc_split(d),
            reinterpret_cast<const float*>(cpl3 + w.cl3.off_meta), labels, l1_list, l1_count,
            nullptr, nullptr, 0, fb_count, fb_list, w.fb_cap, 0);
        FL_CHECK_LAUNCH();
    }
    rc = launch_fallback_fixup(fb_count, w.fb_cap, status, tc_pool_size(1), st);
    if (rc != FL_OK) return rc;

    // points whose label could not be proven: a few directly, otherwise exact CUDA-core scoring + exact re-rank, k = 1
    if (K <= ASSIGN_DIRECT_MAX_K) {
        int* rest_count = counters + 192;                          // (cleared with the others)
        int* rest_list = reinterpret_cast<int*>(base + w.off_fblist2);
        assign_direct_kernel<<<(unsigned)(4 * sm_count()), 256, 0, st>>>(x, ldx, c, K, ldc, d, vec, fb_list, fb_count, labels,
                                                                        rest_list, rest_count);
        FL_CHECK_LAUNCH();
        fb_list = rest_list;
        fb_count = rest_count;
    }
    SimtKnnParams sp{};
    sp.q = x; sp.ldq = ldx; sp.qlist = fb_list; sp.count_dev = fb_count; sp.count = 0;
    sp.db = c; sp.m = K; sp.ldb = ldc; sp.d = d;
    sp.hnorm = reinterpret_cast<const float*>(cpl + w.cl.off_hnorm);
    sp.K1 = 32; sp.cap = simt_pool_cap(32); sp.npl = sp.cap / 32; sp.keep = simt_pool_keep(32, 1);
    sp.nsplit = w.nsplit_fb; sp.rows_per_split = w.rows_per_split_fb;
    sp.dyn_blocks = w.fb_blocks; sp.dyn_bq = w.fb_bq;
    sp.part_sc = reinterpret_cast<float*>(base + w.off_fbpart_sc);
    sp.part_id = reinterpret_cast<uint32_t*>(base + w.off_fbpart_id);
    sp.vecq = vecx; sp.vecd = vecc;
    rc = launch_knn_simt(sp, w.fb_cap, st);
    if (rc != FL_OK) return rc;
    FinalizeParams fp{};
    fp.q = x; fp.ldq = ldx; fp.qlist = fb_list; fp.count_dev = fb_count; fp.count = 0;
    fp.db = c; fp.m = K; fp.ldb = ldc; fp.d = d; fp.vec = vec;
    fp.part_sc = sp.part_sc; fp.part_id = sp.part_id; fp.nsplit = w.nsplit_fb; fp.K1 = 32;
    fp.dyn_blocks = w.fb_blocks; fp.dyn_bq = w.fb_bq;
    fp.k = 1; fp.rerank = 9; fp.row_offset = 0;
    fp.out_dist = reinterpret_cast<float*>(base + w.off_fbdist); fp.out_idx = labels; fp.verify = 0;
    return launch_knn_finalize(fp, w.fb_cap, st);
}

extern "C" int fl_kmeans_assign_tc_f32(const float* x, int64_t n, int64_t ldx, const void* xplane, const float* c,
                                       int K, int64_t ldc, int d, int32_t* labels, void* ws, int64_t ws_bytes,
                                       int32_t* status, void* stream) {
    FL_CHECK_ARG(n >= 0 && K >= 1 && d >= 1 && ldx >= d && ldc >= d, "fl_kmeans_assign_tc_f32: bad shape");
    if (!assign_tc_supported(n > 0 ? n : 1, K, d)) { set_error("fl_kmeans_assign_tc_f32: d=%d > 256 is not supported", d); return FL_EUNSUPPORTED; }
    if (n == 0) return FL_OK;
    FL_CHECK_ARG(x && c && labels && ws, "fl_kmeans_assign_tc_f32: null pointer");
    FL_CHECK_ARG((reinterpret_cast<uintptr_t>(ws) & 255) == 0, "fl_kmeans_assign_tc_f32: workspace must be 256-byte aligned");
    FL_CHECK_ARG(n < (1ll << 31), "fl_kmeans_assign_tc_f32: more than 2^31 rows");
    const AssignTcWs w = assign_tc_plan(n, K, d, xplane != nullptr);
    if (ws_bytes < w.bytes) { set_error("fl_kmeans_assign_tc_f32: workspace %lld < %lld bytes", (long long)ws_bytes, (long long)w.bytes); return FL_EWORKSPACE; }
    cudaStream_t st = (cudaStream_t)stream;
    char* base = static_cast<char*>(ws);
    if (status) FL_CHECK_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t) * FL_STATUS_WORDS, st));

    // sample plane (query side), whose operand format the plain centroid plane shares
    const char* xpl = static_cast<const char*>(xplane);
    const float2* xsq;
    const uint32_t* fmt;
    int rc;
    if (!xpl) {
        float2* xs = reinterpret_cast<float2*>(base + w.off_xsq);
        uint32_t* f = reinterpret_cast<uint32_t*>(base + w.off_xfmt);
        rc = launch_operand_format(x, n, ldx, d, f, st);
        if (rc == FL_OK) rc = launch_query_plane(x, n, ldx, d, base + w.off_xplane, w.n_pad, w.d_pad, st, DT_F32, xs, f);
        if (rc != FL_OK) return rc;
        xpl = base + w.off_xplane;
        xsq = xs;
        fmt = f;
    } else {
        xsq = reinterpret_cast<const float2*>(xpl + round_up(w.n_pad * w.pitch * 2, 1024));
        fmt = reinterpret_cast<const uint32_t*>(xpl + xplane_fmt_offset(n, d));
    }
    return assign_tc_run(x, n, ldx, xpl, xsq, fmt, c, K, ldc, d, labels, base, w, LivePoints{}, nullptr, 0, status, st);
}

// ---------------------------------------------------------------------------------------
// Whole Lloyd loops on the tensor cores.  An iteration scores only the points whose bounds no longer prove their label
// (lloyd_bounds_kernel): all of them in the first few, a tenth later on -- and moves only the rows that change sides between
// the sums.  1M x 128 in 1 024 clusters, 20 iterations: 9.4 ms with every point scored in every iteration, 6.4 so.
struct LloydTcWs { AssignTcWs a; int64_t most, off_bounds, off_list, off_gather, off_count, off_prev, off_shift, bytes; };
static LloydTcWs lloyd_tc_plan(int64_t n, int K, int d) {
    LloydTcWs w{};
    w.a = assign_tc_plan(n, K, d, 1);
    // Up to this many listed points are gathered; beyond, scoring all in place is as cheap (a gathered row is read and
    // written once more, 0.1 ns of the 0.2 that its scores take).
    w.most = n / 2;
    int64_t cur = w.a.bytes;
    w.off_bounds = take(cur, n * 8);
    w.off_list = take(cur, n * 4);
    w.off_gather = take(cur, round_up(w.most > 0 ? w.most : 1, 128) * w.a.pitch * 2);
    w.off_count = take(cur, 32);
    w.off_prev = take(cur, n * 4);
    w.off_shift = take(cur, (int64_t)K * 4);
    w.bytes = cur;
    return w;
}

extern "C" int fl_kmeans_lloyd_tc_supported(int64_t n, int K, int d) {
    return n >= 1 && n < (1ll << 31) && K >= 1 && d >= 1 && assign_tc_split(d) ? 1 : 0;
}
extern "C" int64_t fl_kmeans_lloyd_tc_workspace_bytes(int64_t n, int K, int d) {
    return fl_kmeans_lloyd_tc_supported(n, K, d) ? lloyd_tc_plan(n, K, d).bytes : 0;
}

extern "C" int fl_kmeans_lloyd_tc_f32(const float* x, int64_t n, int64_t ldx, const void* xplane, int d, int K, float* cents_a,
                                      float* cents_b, float* sums, int32_t* cnts, int32_t* labels, int iters, float tol, int refresh,
                                      int32_t* ctl, int32_t* host, int* n_iter, void* ws, int64_t ws_bytes, int32_t* status,
                                      void* stream) {
    FL_CHECK_ARG(n >= 1 && K >= 1 && d >= 1 && ldx >= d && iters >= 1 && refresh >= 1, "fl_kmeans_lloyd_tc_f32: bad shape");
    FL_CHECK_ARG(x && xplane && cents_a && cents_b && sums && cnts && labels && ctl && n_iter && ws && (host || !(tol > 0.f)),
                 "fl_kmeans_lloyd_tc_f32: null pointer");
    FL_CHECK_ARG((reinterpret_cast<uintptr_t>(ws) & 255) == 0 && (reinterpret_cast<uintptr_t>(xplane) & 255) == 0,
                 "fl_kmeans_lloyd_tc_f32: workspace and sample plane must be 256-byte aligned");
    if (!fl_kmeans_lloyd_tc_supported(n, K, d)) { set_error("fl_kmeans_lloyd_tc_f32: n=%lld, d=%d not supported", (long long)n, d); return FL_EUNSUPPORTED; }
    const LloydTcWs w = lloyd_tc_plan(n, K, d);
    if (ws_bytes < w.bytes) { set_error("fl_kmeans_lloyd_tc_f32: workspace %lld < %lld bytes", (long long)ws_bytes, (long long)w.bytes); return FL_EWORKSPACE; }
    cudaStream_t st = (cudaStream_t)stream;
    const bool test = tol > 0.f;
    if (test) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        FL_CHECK_CUDA(cudaStreamIsCapturing(st, &cap));
        FL_CHECK_ARG(cap == cudaStreamCaptureStatusNone, "fl_kmeans_lloyd_tc_f32: a loop that tests convergence cannot be captured");
        *host = 0;
    }
    char* base = static_cast<char*>(ws);
    const char* xpl = static_cast<const char*>(xplane);
    const float2* xsq = reinterpret_cast<const float2*>(xpl + round_up(w.a.n_pad * w.a.pitch * 2, 1024));
    const uint32_t* fmt = reinterpret_cast<const uint32_t*>(xpl + xplane_fmt_offset(n, d));
    int* count = reinterpret_cast<int*>(base + w.off_count);
    int* list = reinterpret_cast<int*>(base + w.off_list);
    int32_t* prev = reinterpret_cast<int32_t*>(base + w.off_prev);
    float* shift = reinterpret_cast<float*>(base + w.off_shift);
    float2* bounds = reinterpret_cast<float2*>(base + w.off_bounds);
    const int32_t* done = test ? ctl + LLOYD_DONE : nullptr;
    if (status) FL_CHECK_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t) * FL_STATUS_WORDS, st));
    FL_CHECK_CUDA(cudaMemsetAsync(ctl, 0, sizeof(int32_t) * LLOYD_WORDS, st));
    float* cur = cents_a;
    float* nxt = cents_b;
    auto step = [&](int it) -> int {
        LivePoints live{};
        live.bounds = bounds;
        if (it > 0) {
            FL_CHECK_CUDA(cudaMemsetAsync(count, 0, 32, st));
            int64_t blocks = ceil_div(n, BOUNDS_THREADS * BOUNDS_PER);
            if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
            lloyd_bounds_kernel<<<(unsigned)blocks, BOUNDS_THREADS, 0, st>>>(n, K, labels, bounds, shift, done, (int)w.most, list, count);
            FL_CHECK_LAUNCH();
            live.rows = list;
            live.count = count;
        }
        int rc = assign_tc_run(x, n, ldx, xpl, xsq, fmt, cur, K, d, d, labels, base, w.a, live, base + w.off_gather,
                               w.most > 0 ? w.most : 1, status, st);
        if (rc != FL_OK) return rc;
        if (it % refresh == 0) {
            rc = fl_kmeans_update_f32(x, n, ldx, d, labels, K, sums, cnts, st);
            if (rc != FL_OK) return rc;
            FL_CHECK_CUDA(cudaMemcpyAsync(prev, labels, (size_t)n * 4, cudaMemcpyDeviceToDevice, st));
        } else {
            rc = fl_kmeans_update_delta_f32(x, n, ldx, d, labels, prev, K, sums, cnts, st);
            if (rc != FL_OK) return rc;
        }
        return launch_kmeans_step(sums, cnts, cur, nxt, K, d, 0, tol, it, ctl, host, shift, st);
    };
    for (int it = 0; it < iters; ++it) {
        // The host stays at most three iterations ahead: launches after the one that converges change nothing.
        if (test && it >= 3) {
            lloyd_wait(host, it - 2, st);
            if (__atomic_load_n(host, __ATOMIC_ACQUIRE) < 0) break;
        }
        const int rc = step(it);
        if (rc != FL_OK) {
            if (test) cudaStreamSynchronize(st);           // launched steps still write to `host`
            return rc;
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
