// Finalisation of the candidate pools that the dense epilogues of the scoring kernel keep in global
// memory as (score, row) pairs: one block per query gathers the entries above every pool's final
// threshold, orders them by score, re-scores the best with exact fp32 sum (q - x)^2 and proves the k
// nearest against the scoring error bound, or queues the query for the next stage.
//
// Four warps per query read the pools' counts at once, copy their entries as one list and re-score 32
// rows per round trip; nothing is sorted but the handful of re-scored rows.  (The one-warp form, which
// walks pool after pool, sorts by score and re-scores four rows per trip, took 54 us for 32 queries x 128
// pools.)
#include "knn_internal.h"
#include "pool.cuh"

namespace fl {

constexpr int PF_THREADS = 128, PF_WARPS = PF_THREADS / 32, PF_CAND = 1024, PF_RERANK = 256;

// A value that at least k of the R * 32 keys (R per lane, -inf where there is none) reach, close to the
// largest such; -inf when fewer than k exist.  All lanes of a warp call it.
template <int R>
__device__ __forceinline__ float pf_kth_reached(const float (&key)[R], int k) {
    int v[R], lo = 0x7fffffff, hi = (int)0x80000000, have = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int b = __float_as_int(key[r]);
        const bool real = key[r] > neg_inf();
        v[r] = real ? (b >= 0 ? b : (b ^ 0x7fffffff)) : (int)0x80000000;      // orders like the float
        have += __popc(__ballot_sync(FULL_MASK, real));
        if (real) { lo = min(lo, v[r]); hi = max(hi, v[r]); }
    }
    if (have < k) return neg_inf();
    lo = __reduce_min_sync(FULL_MASK, lo);
    hi = __reduce_max_sync(FULL_MASK, hi);
    for (int it = 0; it < 32 && lo < hi; ++it) {
        const int mid = (int)(((long long)lo + hi + 1) >> 1);
        int c = 0;
#pragma unroll
        for (int r = 0; r < R; ++r) c += __popc(__ballot_sync(FULL_MASK, v[r] >= mid));
        if (c >= k) lo = mid; else hi = mid - 1;
        if (c == k) break;
    }
    return __int_as_float(lo >= 0 ? lo : (lo ^ 0x7fffffff));
}

__global__ void __launch_bounds__(PF_THREADS) pairs_finalize_kernel(const PairFinalizeParams p) {
    __shared__ float s_key[PF_CAND];
    __shared__ uint32_t s_id[PF_CAND];
    __shared__ float s_dist[PF_RERANK];        // -distance of the re-scored rows, and their ids
    __shared__ uint32_t s_rid[PF_RERANK];
    __shared__ float s_max[PF_THREADS];
    __shared__ int s_off[PF_THREADS + 1];
    __shared__ int s_pool[PF_THREADS];
    __shared__ float s_f[3 * PF_WARPS];
    __shared__ int s_w[PF_WARPS];
    __shared__ int s_n, s_m;
    __shared__ float s_pick;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t qi = blockIdx.x;
    const void* qp = row_at(p.q, qi, p.ldq, p.dt);
    auto pool_of = [&](int i) -> int64_t { return i < p.npool ? qi * p.npool + i : -1; };
    // u = the largest final threshold: every row in no pool scored at most that much
    float u = neg_inf(), qs = 0.f, ls = 0.f;
    for (int i = tid; i < p.npool; i += PF_THREADS) {
        const int64_t pl = pool_of(i);
        if (pl >= 0) u = fmaxf(u, __ldg(p.pool_tau + pl));
    }
    for (int c = tid; c < p.d; c += PF_THREADS) {
        const float v = ld_elem(qp, c, p.dt), l = bf16_lost(v);
        qs += v * v;
        ls += l * l;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        u = fmaxf(u, __shfl_xor_sync(FULL_MASK, u, o));
        qs += __shfl_xor_sync(FULL_MASK, qs, o);
        ls += __shfl_xor_sync(FULL_MASK, ls, o);
    }
    if (lane == 0) { s_f[warp] = u; s_f[PF_WARPS + warp] = qs; s_f[2 * PF_WARPS + warp] = ls; }
    __syncthreads();
    float qsq = 0.f, lost = 0.f;
#pragma unroll
    for (int w = 0; w < PF_WARPS; ++w) { u = fmaxf(u, s_f[w]); qsq += s_f[PF_WARPS + w]; lost += s_f[2 * PF_WARPS + w]; }
    const float mn = __ldg(p.norms + NORM_ROW);
    const float eps = score_eps(OPERANDS_BF16, qsq, lost, 0.f, p.norms, p.acc);
    const float slack = proof_slack(qsq, mn, p.d);

    // Gather what scored above `cut`.  More than fit: the cut rises to the score at the first quarter of
    // those stored (an arbitrary subset) and the gather starts over; everything below is covered by `bound`.
    float cut = u, tmax = neg_inf();
    int total = 0;
    for (int round = 0; round < 4; ++round) {
        __syncthreads();
        if (tid == 0) s_n = 0;
        tmax = neg_inf();
        for (int base = 0; base < p.npool; base += PF_THREADS) {
            const int64_t pl = pool_of(base + tid);
            int n = 0;
            if (pl >= 0) { n = __ldg(p.pool_cnt + pl); n = n < p.cap ? n : p.cap; }
            int inc = n;                                   // inclusive prefix sum over the block
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(FULL_MASK, inc, o);
                if (lane >= o) inc += t;
            }
            __syncthreads();
            if (lane == 31) s_w[warp] = inc;
            s_pool[tid] = (int)(pl >= 0 ? pl : 0);
            __syncthreads();
            int before = 0;
#pragma unroll
            for (int w = 0; w < PF_WARPS; ++w) before += w < warp ? s_w[w] : 0;
            s_off[tid] = before + inc - n;
            if (tid == PF_THREADS - 1) s_off[PF_THREADS] = before + inc;
            __syncthreads();
            const int chunk = s_off[PF_THREADS];
            for (int i0 = 0; i0 < chunk; i0 += PF_THREADS) {
                const int idx = i0 + tid;
                float sc = neg_inf();
                uint32_t id = INVALID_ID;
                if (idx < chunk) {
                    int lo = 0, hi = PF_THREADS - 1;       // last pool whose offset is <= idx
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (s_off[mid] <= idx) lo = mid; else hi = mid - 1;
                    }
                    const float2 v = __ldg(p.pools + (int64_t)s_pool[lo] * p.cap + (idx - s_off[lo]));
                    if (v.x > cut) {
                        const uint32_t raw = __float_as_uint(v.y);
                        if (raw < (uint32_t)p.m) { sc = v.x; id = raw; tmax = fmaxf(tmax, sc); }
                    }
                }
                const unsigned mask = __ballot_sync(FULL_MASK, id != INVALID_ID);
                if (mask) {
                    int at = 0;
                    if (lane == 0) at = atomicAdd(&s_n, __popc(mask));
                    at = __shfl_sync(FULL_MASK, at, 0) + __popc(mask & ((1u << lane) - 1u));
                    if (id != INVALID_ID && at < PF_CAND) { s_key[at] = sc; s_id[at] = id; }
                }
            }
        }
        __syncthreads();
        total = s_n;
        if (total <= PF_CAND) break;
        block_sort_desc<PF_THREADS>(s_key, s_id, PF_CAND);
        cut = fmaxf(cut, s_key[PF_CAND / 4 - 1]);
    }
    const bool overflow = total > PF_CAND;
    const int n = overflow ? PF_CAND : total;

    // Re-scoring in two steps.  At least k entries reach `pick`, the k-th best of the threads' maxima (every
    // entry if fewer exist): their exact distances bound the k-th distance by D.  A row closer than D has a
    // score of at least f = (qsq - D - slack) / 2 - eps, so the entries between f and `pick` come next, and
    // no other row matters as long as f lies above the cut.
    s_max[tid] = tmax;
    if (tid == 0) s_m = 0;
    __syncthreads();
    if (warp == 0) {
        float v[PF_WARPS];
#pragma unroll
        for (int r = 0; r < PF_WARPS; ++r) v[r] = s_max[r * 32 + lane];
        const float t = pf_kth_reached<PF_WARPS>(v, p.k);
        if (lane == 0) s_pick = t;
    }
    __syncthreads();
    const float pick = s_pick;
    // entries with lo <= score < hi join the list of rows to re-score
    auto collect = [&](float lo, float hi) {
        for (int i0 = 0; i0 < n; i0 += PF_THREADS) {
            const int i = i0 + tid;
            const bool take = i < n && s_key[i] >= lo && s_key[i] < hi;
            const unsigned mask = __ballot_sync(FULL_MASK, take);
            if (mask) {
                int at = 0;
                if (lane == 0) at = atomicAdd(&s_m, __popc(mask));
                at = __shfl_sync(FULL_MASK, at, 0) + __popc(mask & ((1u << lane) - 1u));
                if (take && at < PF_RERANK) s_rid[at] = s_id[i];
            }
        }
        __syncthreads();
    };
    auto rescore = [&](int from, int to) {
        for (int c0 = from + warp * 8; c0 < to; c0 += PF_WARPS * 8) {
            uint32_t cid[8];
            float a[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) { cid[t] = c0 + t < to ? s_rid[c0 + t] : INVALID_ID; a[t] = 0.f; }
            if (p.vec) {
                for (int c = lane * 4; c < p.d; c += 128) {
                    const float4 qv = ld_elem4(qp, c, p.dt);
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
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
                    for (int t = 0; t < 8; ++t) {
                        if (cid[t] != INVALID_ID) {
                            const float df = qv - ld_elem(row_at(p.db, cid[t], p.ldb, p.dt), c, p.dt);
                            a[t] += df * df;
                        }
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < 8; ++t) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) a[t] += __shfl_xor_sync(FULL_MASK, a[t], o);
                if (lane == 0 && c0 + t < to) s_dist[c0 + t] = -a[t];
            }
        }
        __syncthreads();
    };
    collect(pick, pos_inf());
    int m = s_m < PF_RERANK ? s_m : PF_RERANK;
    bool fits = s_m <= PF_RERANK;
    rescore(0, m);
    float bound = pick;
    if (pick > neg_inf() && fits) {
        if (warp == 0) {
            float v[PF_RERANK / 32];
#pragma unroll
            for (int r = 0; r < PF_RERANK / 32; ++r) v[r] = r * 32 + lane < m ? s_dist[r * 32 + lane] : neg_inf();
            const float t = pf_kth_reached<PF_RERANK / 32>(v, p.k);
            if (lane == 0) s_pick = t;
        }
        __syncthreads();
        float f = 0.5f * (qsq + s_pick - slack) - eps;     // s_pick = -D
        f -= 2e-6f * (qsq + mn * mn);                      // the proof below compares the same sum: stay clear of its rounding
        bound = fminf(f, pick);
        collect(bound, pick);
        fits = s_m <= PF_RERANK;
        const int m2 = fits ? s_m : PF_RERANK;
        rescore(m, m2);
        m = m2;
    }
    bound = fits ? fmaxf(bound, cut) : pos_inf();
    // order the re-scored rows by (distance, row)
    const int P2 = pow2_ceil_dev(m > p.k ? m : p.k);
    for (int i = tid; i < P2; i += PF_THREADS) {
        s_key[i] = i < m ? s_dist[i] : neg_inf();
        s_id[i] = i < m ? s_rid[i] : INVALID_ID;
    }
    block_sort_desc<PF_THREADS>(s_key, s_id, P2);
    for (int e = tid; e < p.k; e += PF_THREADS) {
        const bool ok = s_id[e] != INVALID_ID && s_key[e] > neg_inf();
        p.out_dist[qi * p.k + e] = ok ? -s_key[e] : pos_inf();
        p.out_idx[qi * p.k + e] = ok ? (int32_t)((int64_t)s_id[e] + p.row_offset) : -1;
    }
    if (tid == 0) {
        const float dk = s_id[p.k - 1] != INVALID_ID ? -s_key[p.k - 1] : pos_inf();
        if (overflow || !fits || !list_proven(dk, qsq, bound, eps, slack)) {
            bool queued = false;
            if (p.next_count != nullptr) {
                const int i = atomicAdd(p.next_count, 1);
                if (i < p.next_cap) { p.next_list[i] = (int)qi; queued = true; }
            }
            if (!queued) {
                const int i = atomicAdd(p.fb_count, 1);
                if (i < p.fb_cap) p.fb_list[i] = (int)qi;
            }
        }
    }
}

int launch_pairs_finalize(const PairFinalizeParams& p, cudaStream_t st) {
    if (p.nq <= 0) return FL_OK;
    FL_CHECK_ARG(p.pools && p.pool_cnt && p.pool_tau && p.norms && p.fb_count && p.k >= 1 && p.k <= PF_RERANK && p.npool >= 1,
                 "pair-pool finalisation: bad parameters");
    pairs_finalize_kernel<<<(unsigned)p.nq, PF_THREADS, 0, st>>>(p);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

}  // namespace fl
