// Shared helpers for the flashlib_b200 kernels: error plumbing for the C ABI and the
// warp-level sorting network used by every top-k pool in this library.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdarg.h>
#include <stdio.h>
#include <math.h>

#include "../../include/flashlib_b200.h"

namespace fl {

// ---- host-side error plumbing ------------------------------------------------------
void set_error(const char* fmt, ...);
void count_launch();
// Profiling hooks (no-ops unless fl_profile_enable(1) was called): bracket the dominant
// kernel of an entry point with CUDA events recorded on the caller's stream.
void profile_begin(cudaStream_t st);
void profile_end(cudaStream_t st);
// fl_profile_enable(2): one event per mark along an entry point's launch sequence.
void profile_mark(cudaStream_t st);

#define FL_CHECK_ARG(cond, ...)                                                         \
    do {                                                                                \
        if (!(cond)) {                                                                  \
            ::fl::set_error(__VA_ARGS__);                                               \
            return FL_EINVAL;                                                           \
        }                                                                               \
    } while (0)

#define FL_CHECK_CUDA(expr)                                                             \
    do {                                                                                \
        cudaError_t e__ = (expr);                                                       \
        if (e__ != cudaSuccess) {                                                       \
            ::fl::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__),    \
                            __FILE__, __LINE__);                                        \
            return FL_ECUDA;                                                            \
        }                                                                               \
    } while (0)

// Every kernel launch in the library goes through this macro: it counts the launch
// (fl_launch_count) and surfaces launch-configuration errors.
#define FL_CHECK_LAUNCH()                                                               \
    do {                                                                                \
        ::fl::count_launch();                                                           \
        FL_CHECK_CUDA(cudaGetLastError());                                              \
    } while (0)

static inline int64_t round_up(int64_t a, int64_t b) { return (a + b - 1) / b * b; }
static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
static inline int pow2_ceil(int v) { int p = 1; while (p < v) p <<= 1; return p; }

// Number of SMs of the current device (cached per device).
int sm_count();
// Opt-in dynamic shared memory limit of the current device in bytes.
int smem_optin_bytes();

// ---- device-side helpers -----------------------------------------------------------
constexpr unsigned FULL_MASK = 0xffffffffu;
constexpr uint32_t INVALID_ID = 0xffffffffu;

// Element types of the caller's rows (FL_DTYPE_* of the C ABI): fp32, or 16-bit storage that is
// widened to fp32 on load (exactly: every bf16 / fp16 value is an fp32 value).
constexpr int DT_F32 = FL_DTYPE_F32, DT_BF16 = FL_DTYPE_BF16, DT_F16 = FL_DTYPE_F16;
static inline int dt_size(int dt) { return dt == DT_F32 ? 4 : 2; }
// Four consecutive elements can be fetched with one load: 16 bytes of fp32, 8 bytes of 16-bit values.
static inline bool dt_vec_ok(const void* p, int64_t ld, int dt) {
    return (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(p) & (dt == DT_F32 ? 15 : 7)) == 0);
}

// fp32 accumulation of `terms` products in a tensor-core score, relative to ||q|| ||x||: one rounding of 2^-23 each
// (truncation; the products themselves are exact), raised by the 2^-7 by which rounded operands may be longer.
// Measured with operands of one sign: at most 0.016 of it (64 to 256 features).
static inline float score_acc(int terms) { return 1.25e-7f * (float)terms; }
// Split planes of d features: the 2 d products with a low half come first, while the sum is 2^-7 of ||q|| ||x|| at most.
static inline float score_acc_split(int d) { return score_acc(d + 16 + d / 64 + 1); }

#if defined(__CUDACC__)

__device__ __forceinline__ float neg_inf() { return __int_as_float(0xff800000); }
__device__ __forceinline__ float pos_inf() { return __int_as_float(0x7f800000); }

__device__ __forceinline__ float f16_bits_to_f32(unsigned short h) { return __half2float(__ushort_as_half(h)); }
// Element i of a row array of type dt, as fp32.
__device__ __forceinline__ float ld_elem(const void* base, int64_t i, int dt) {
    if (dt == DT_F32) return __ldg(static_cast<const float*>(base) + i);
    const unsigned short h = __ldg(static_cast<const unsigned short*>(base) + i);
    return dt == DT_BF16 ? __uint_as_float((uint32_t)h << 16) : f16_bits_to_f32(h);
}
// Elements i .. i+3 (the address must allow one load: see dt_vec_ok).
__device__ __forceinline__ float4 ld_elem4(const void* base, int64_t i, int dt) {
    if (dt == DT_F32) return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + i));
    const uint2 w = __ldg(reinterpret_cast<const uint2*>(static_cast<const unsigned short*>(base) + i));
    if (dt == DT_BF16)
        return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                           __uint_as_float(w.y & 0xffff0000u));
    return make_float4(f16_bits_to_f32((unsigned short)(w.x & 0xffffu)), f16_bits_to_f32((unsigned short)(w.x >> 16)),
                       f16_bits_to_f32((unsigned short)(w.y & 0xffffu)), f16_bits_to_f32((unsigned short)(w.y >> 16)));
}
// Four values as bf16 (round to nearest even), for one 8-byte store.
__device__ __forceinline__ uint2 bf16x4_bits(float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 w;
    w.x = *reinterpret_cast<const uint32_t*>(&a);
    w.y = *reinterpret_cast<const uint32_t*>(&b);
    return w;
}
// Elements c .. c + 3 of a row of d (zero beyond it); vec: the row allows one wide read and d is a multiple of 4.
__device__ __forceinline__ float4 ld_row4(const void* p, int c, int d, int vec, int dt) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c >= d) return v;
    if (vec) return ld_elem4(p, c, dt);
    v.x = ld_elem(p, c, dt);
    if (c + 1 < d) v.y = ld_elem(p, c + 1, dt);
    if (c + 2 < d) v.z = ld_elem(p, c + 2, dt);
    if (c + 3 < d) v.w = ld_elem(p, c + 3, dt);
    return v;
}
__device__ __forceinline__ int dt_size_dev(int dt) { return dt == DT_F32 ? 4 : 2; }
// Address of row r (ld in elements).
__host__ __device__ __forceinline__ const void* row_at(const void* base, int64_t r, int64_t ld, int dt) {
    return static_cast<const char*>(base) + r * ld * (dt == DT_F32 ? 4 : 2);
}

// Bitonic sorting network over NPL*32 (key, id) pairs held NPL per lane; the element at
// register r of lane l has position r*32 + l.  Sorts by DESCENDING key.  With TIEBREAK,
// equal keys are ordered by ascending id, which makes the order total and the result
// independent of where the elements started.
template <int NPL, bool TIEBREAK>
__device__ __forceinline__ void warp_sort_desc(float (&key)[NPL], uint32_t (&id)[NPL]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= NPL * 32; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                const int jr = j >> 5;
#pragma unroll
                for (int r = 0; r < NPL; ++r) {
                    const int pr = r ^ jr;
                    if (pr > r) {
                        const bool desc_block = (((r << 5) & k) == 0);
                        const float a = key[r], b = key[pr];
                        const uint32_t ia = id[r], ib = id[pr];
                        // "a should come after b" in a descending block
                        bool a_lt_b = a < b;
                        bool a_gt_b = a > b;
                        if (TIEBREAK) {
                            a_lt_b = a_lt_b || (a == b && ia > ib);
                            a_gt_b = a_gt_b || (a == b && ia < ib);
                        }
                        const bool sw = desc_block ? a_lt_b : a_gt_b;
                        if (sw) {
                            key[r] = b; key[pr] = a;
                            id[r] = ib; id[pr] = ia;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < NPL; ++r) {
                    const int p = (r << 5) | lane;
                    const float ok = __shfl_xor_sync(FULL_MASK, key[r], j);
                    const uint32_t oi = __shfl_xor_sync(FULL_MASK, id[r], j);
                    const bool lower = (lane & j) == 0;
                    const bool desc_block = ((p & k) == 0);
                    const bool take_max = (lower == desc_block);
                    bool o_gt = ok > key[r];
                    bool o_lt = ok < key[r];
                    if (TIEBREAK) {
                        o_gt = o_gt || (ok == key[r] && oi < id[r]);
                        o_lt = o_lt || (ok == key[r] && oi > id[r]);
                    }
                    const bool take = take_max ? o_gt : o_lt;
                    if (take) { key[r] = ok; id[r] = oi; }
                }
            }
        }
    }
}

// Merges two DESCENDING sequences of NPL*32 (key, id) pairs (same position layout as
// warp_sort_desc) and leaves the NPL*32 largest of their union in (ka, ia), descending.
// Position p of the result is first max(a[p], b[N-1-p]) -- that picks the N largest and
// forms a bitonic sequence -- which the final stages of the bitonic network then sort.
template <int NPL, bool TIEBREAK>
__device__ __forceinline__ void warp_merge_desc(float (&ka)[NPL], uint32_t (&ia)[NPL], const float (&kb)[NPL],
                                                const uint32_t (&ib)[NPL]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
        const float ok = __shfl_sync(FULL_MASK, kb[NPL - 1 - r], 31 - lane);
        const uint32_t oi = __shfl_sync(FULL_MASK, ib[NPL - 1 - r], 31 - lane);
        bool take = ok > ka[r];
        if (TIEBREAK) take = take || (ok == ka[r] && oi < ia[r]);
        if (take) { ka[r] = ok; ia[r] = oi; }
    }
    constexpr int k = NPL * 32;
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
        if (j >= 32) {
            const int jr = j >> 5;
#pragma unroll
            for (int r = 0; r < NPL; ++r) {
                const int pr = r ^ jr;
                if (pr > r) {
                    const float a = ka[r], b = ka[pr];
                    const uint32_t xa = ia[r], xb = ia[pr];
                    bool a_lt_b = a < b;
                    if (TIEBREAK) a_lt_b = a_lt_b || (a == b && xa > xb);
                    if (a_lt_b) { ka[r] = b; ka[pr] = a; ia[r] = xb; ia[pr] = xa; }
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < NPL; ++r) {
                const float ok = __shfl_xor_sync(FULL_MASK, ka[r], j);
                const uint32_t oi = __shfl_xor_sync(FULL_MASK, ia[r], j);
                const bool lower = (lane & j) == 0;       // the lower position keeps the larger key
                bool o_gt = ok > ka[r];
                bool o_lt = ok < ka[r];
                if (TIEBREAK) {
                    o_gt = o_gt || (ok == ka[r] && oi < ia[r]);
                    o_lt = o_lt || (ok == ka[r] && oi > ia[r]);
                }
                const bool take = lower ? o_gt : o_lt;
                if (take) { ka[r] = ok; ia[r] = oi; }
            }
        }
    }
}

// Compacts one row's candidate pool: reads `cnt` (score, id) entries from sc/idv (any
// address space), keeps the K1 best (largest score) at positions [0, K1) in descending
// order and returns the new threshold: the K1-th best score, or -inf while fewer than
// K1 entries exist.  NPL*32 must be >= the pool capacity.  All 32 lanes must call it.
template <int NPL>
__device__ __forceinline__ float warp_pool_compact(float* sc, uint32_t* idv, int cnt, int K1) {
    const int lane = threadIdx.x & 31;
    float key[NPL];
    uint32_t id[NPL];
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
        const int e = (r << 5) | lane;
        const bool ok = e < cnt;
        key[r] = ok ? sc[e] : neg_inf();
        id[r] = ok ? idv[e] : INVALID_ID;
    }
    warp_sort_desc<NPL, false>(key, id);
    float thr = neg_inf();
#pragma unroll
    for (int r = 0; r < NPL; ++r) {
        const int e = (r << 5) | lane;
        if (e < K1) { sc[e] = key[r]; idv[e] = id[r]; }
        if (((K1 - 1) >> 5) == r) thr = __shfl_sync(FULL_MASK, key[r], (K1 - 1) & 31);
    }
    __syncwarp();
    return thr;
}

// Bitonic sort of n (power of two) entries in shared memory: larger key first, smaller id first
// among equal keys.  All THREADS threads of the block must call it.
template <int THREADS>
__device__ __forceinline__ void block_sort_desc(float* key, uint32_t* id, int n) {
    for (int size = 2; size <= n; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < (n >> 1); i += THREADS) {
                const int a = 2 * i - (i & (stride - 1));
                const int b = a + stride;
                const float ka = key[a], kb = key[b];
                const uint32_t ia = id[a], ib = id[b];
                const bool a_first = ka > kb || (ka == kb && ia <= ib);
                const bool desc = (a & size) == 0;
                if (a_first != desc) { key[a] = kb; key[b] = ka; id[a] = ib; id[b] = ia; }
            }
        }
    }
    __syncthreads();
}

__device__ __forceinline__ int pow2_ceil_dev(int v) { return v <= 1 ? 1 : 1 << (32 - __clz(v - 1)); }

// Largest-value update of a float in global memory (compare-and-swap; a few writers at most).
__device__ __forceinline__ void atomic_max_f32(float* addr, float v) {
    int* ai = reinterpret_cast<int*>(addr);
    int old = *reinterpret_cast<volatile int*>(ai);
    while (__int_as_float(old) < v) {
        const int assumed = old;
        old = atomicCAS(ai, assumed, __float_as_int(v));
        if (old == assumed) break;
    }
}

// What rounding a value to bf16 takes from it (exact in fp32; NaN for infinities).
__device__ __forceinline__ float bf16_lost(float v) { return v - __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float sq4(float4 v) { return v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; }
__device__ __forceinline__ float4 bf16_lost4(float4 v) {
    return make_float4(bf16_lost(v.x), bf16_lost(v.y), bf16_lost(v.z), bf16_lost(v.w));
}
// The same from the rounded values (bf16x4_bits(v)).
__device__ __forceinline__ float4 bf16_lost4(float4 v, uint2 w) {
    return make_float4(v.x - __uint_as_float(w.x << 16), v.y - __uint_as_float(w.x & 0xffff0000u),
                       v.z - __uint_as_float(w.y << 16), v.w - __uint_as_float(w.y & 0xffff0000u));
}

// The same for operands in fp16 (saturating: what lies beyond 65 504 is lost and counted, NaN too).
__device__ __forceinline__ uint2 f16x4_bits(float4 v) {
    auto fit = [](float x) { return fminf(fmaxf(x, -65504.f), 65504.f); };
    const __half2 a = __floats2half2_rn(fit(v.x), fit(v.y)), b = __floats2half2_rn(fit(v.z), fit(v.w));
    uint2 w;
    w.x = *reinterpret_cast<const uint32_t*>(&a);
    w.y = *reinterpret_cast<const uint32_t*>(&b);
    return w;
}
__device__ __forceinline__ float4 f16_lost4(float4 v, uint2 w) {
    return make_float4(v.x - f16_bits_to_f32((unsigned short)(w.x & 0xffffu)), v.y - f16_bits_to_f32((unsigned short)(w.x >> 16)),
                       v.z - f16_bits_to_f32((unsigned short)(w.y & 0xffffu)), v.w - f16_bits_to_f32((unsigned short)(w.y >> 16)));
}
// Operand format of a plane (FMT_*): the values to store, and what storing them takes away.
constexpr uint32_t FMT_BF16 = 0, FMT_F16 = 1;
__device__ __forceinline__ uint2 operand4_bits(float4 v, uint32_t fmt) { return fmt == FMT_F16 ? f16x4_bits(v) : bf16x4_bits(v); }
__device__ __forceinline__ float4 operand4_lost(float4 v, uint2 w, uint32_t fmt) { return fmt == FMT_F16 ? f16_lost4(v, w) : bf16_lost4(v, w); }

// Largest norms over the rows of a database, left by the passes that write its operand planes: of the rows x, of what
// one rounding to the operands' format takes from them (x - hi) and of what the second half of a split plane still misses
// (x - hi - lo).  The word after them holds the operand format of planes that choose it (kmeans_tc.cu, ivf_tc.cu).
enum { NORM_ROW = 0, NORM_LOST = 1, NORM_LOST2 = 2, NORM_FMT = 3, NORM_WORDS = 4 };
__device__ __forceinline__ uint32_t operand_format(const float* norms) { return __float_as_uint(__ldg(norms + NORM_FMT)); }

// Bound on |score - (<q,x> - ||x||^2/2)| over the rows behind `norms`, from the rounding that happened to this query
// (sums of squares: qsq of its values, lost of q - hi, lost2 of q - hi - lo) and to those rows.  With
// q' = q - dq, x' = x - dx the product errs by <dq, x> + <q', dx>; the split planes leave out <lo, lo> besides.
// Whatever the values, no constant is assumed: a bf16 rounding may move a value by 2^-8 of itself, and where
// all roundings go one way the product is off by nearly 2^-7 ||q|| ||x||; on ordinary data the norms give
// half of that.  Nothing is lost where the rows are stored as bf16.  `acc`: see score_acc().
// OPERANDS_BF16 stands for one rounding, to bf16 or fp16: `lost` and the norms are those of the one that happened.
constexpr int OPERANDS_F32 = 0, OPERANDS_BF16 = 1, OPERANDS_SPLIT = 2;
__device__ __forceinline__ float score_eps(int operands, float qsq, float lost, float lost2, const float* __restrict__ norms, float acc) {
    const float qn = sqrtf(qsq), xn = __ldg(norms + NORM_ROW);
    float eps = acc * qn * xn;
    if (operands == OPERANDS_BF16) {
        const float l = sqrtf(lost);
        eps += l * xn + (qn + l) * __ldg(norms + NORM_LOST);
    } else if (operands == OPERANDS_SPLIT) {
        const float l = sqrtf(lost), l2 = sqrtf(lost2), xl = __ldg(norms + NORM_LOST), xl2 = __ldg(norms + NORM_LOST2);
        eps += l2 * xn + (qn + l2) * xl2 + (l + l2) * (xl + xl2);
    }
    return eps;
}
// What the fp32 sums beside the product -- ||q||^2, ||x||^2, the exact distances, the norm columns -- may be off by
// together, in squared distance: chains of d / 32 + 10 roundings of 2^-24 at most.
__device__ __forceinline__ float proof_slack(float qsq, float xn, int d) {
    return fmaxf(1e-5f, 1e-8f * (float)d) * (qsq + xn * xn);
}

// The proof that a candidate list is complete: every row outside it has a score (half of qsq minus its distance) of at
// most bound + eps, so none of them comes closer than the k-th distance dk on it.  A bound of -inf says that no row
// was left out at all, which a score of NaN -- infinite or NaN operands, a norm that overflows -- does
// not obey: such a row passes no comparison and raises no threshold.  Where one can exist, `slack` (a
// multiple of ||q||^2 plus the square of the largest row norm) is not finite and nothing is proven.
__device__ __forceinline__ bool list_proven(float dk, float qsq, float bound, float eps, float slack) {
    if (bound == neg_inf()) return slack < pos_inf();
    return dk < qsq - 2.f * (bound + eps) - slack;
}

// The split -||x||^2 / 2 columns of a plane row (lanes below PLANE_AUG_COLS write them): three bf16 terms that sum to it.
__device__ __forceinline__ void write_norm_columns(__nv_bfloat16* o, float sq, int cols) {
    const int lane = threadIdx.x & 31;
    if (lane >= cols) return;
    const float nh = -0.5f * sq;
    const __nv_bfloat16 h1 = __float2bfloat16_rn(nh);
    const float r1 = nh - __bfloat162float(h1);
    const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(h2);
    const __nv_bfloat16 h3 = __float2bfloat16_rn(r2);
    o[lane] = lane == 0 ? h1 : lane == 1 ? h2 : lane == 2 ? h3 : __float2bfloat16_rn(0.f);
}

// Folds the squares that lane 0 of every warp holds (0 where its row is none) into the largest norms; all threads of
// a block call it.  A maximum per block in shared memory first: one read of the global words per warp and norm
// made the planes of 262 144 x 16 rows 200 us slower, so many reads of one address they are.
template <int N>
__device__ __forceinline__ void block_norms_update(unsigned int* norm_bits, const float (&sq)[N]) {
    __shared__ unsigned int s_norm[N];
    if (threadIdx.x < N) s_norm[threadIdx.x] = 0u;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int i = 0; i < N; ++i) atomicMax(s_norm + i, __float_as_uint(sqrtf(sq[i])));      // (NaN orders above infinity)
    }
    __syncthreads();
    if (threadIdx.x < N) {
        const unsigned int v = s_norm[threadIdx.x];
        if (*reinterpret_cast<volatile unsigned int*>(norm_bits + threadIdx.x) < v) atomicMax(norm_bits + threadIdx.x, v);
    }
}

// Folds sqrt(sq) into the largest row norm (its bits, zero-initialised: norms are >= 0, so bit patterns
// order like values).  A plain read first: all but a few dozen of a million rows find a larger norm
// already there, and a million atomics on one address take 0.7 ms.
__device__ __forceinline__ void max_norm_update(unsigned int* maxnorm_bits, float sq) {
    const unsigned int v = __float_as_uint(sqrtf(sq));           // (NaN orders above infinity)
    if (*reinterpret_cast<volatile unsigned int*>(maxnorm_bits) < v) atomicMax(maxnorm_bits, v);
}

#endif  // __CUDACC__

}  // namespace fl
