// Row norms and the database operand plane (bf16 rows + half squared norms) that the
// tensor-core kNN / assign kernels stream with TMA.
#include "common.cuh"
#include "knn_internal.h"
#include <cuda_bf16.h>

namespace fl {

// One warp per row; out[row] = sum of squares in fp32.
__global__ void rownorm_kernel(const float* __restrict__ x, int64_t n, int d, int64_t ld,
                               float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n) return;
    const float* p = x + row * ld;
    float s = 0.f;
    const bool vec = ((ld & 3) == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    if (vec) {
        const int d4 = d >> 2;
        const float4* p4 = reinterpret_cast<const float4*>(p);
        for (int c = lane; c < d4; c += 32) {
            const float4 v = __ldg(p4 + c);
            s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        for (int c = (d4 << 2) + lane; c < d; c += 32) { const float v = p[c]; s += v * v; }
    } else {
        for (int c = lane; c < d; c += 32) { const float v = p[c]; s += v * v; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL_MASK, s, o);
    if (lane == 0) out[row] = s;
}

// One warp per plane row: converts the fp32 row to bf16 (round to nearest even), zero
// pads columns [d, d_pad), writes ||x||^2/2 (+inf for padding rows) and folds the row's
// norm into the plane-wide maximum (non-negative floats order like their bit patterns).
// Columns [d_pad, d_pad+3) carry -||x||^2/2 split into three bf16 terms (their sum is exact
// to 2^-24 relative); multiplied by the ones the query plane holds in the same columns they
// make the tensor-core product come out as <q,x> - ||x||^2/2.  Padding rows carry a huge
// negative value there so they can never rank.
// Rows of 16-bit storage (dt): bf16 values enter the plane as they are, fp16 values are rounded to
// bf16 like fp32 ones; the norms are those of the stored values.  m_pad is a multiple of the block's rows.  Four columns a lane: 16-byte reads where the
// rows allow them (vec) and 8-byte writes.
__global__ void plane_build_kernel(const void* __restrict__ db, int64_t m, int d, int64_t ld,
                                   __nv_bfloat16* __restrict__ rows, float* __restrict__ hnorm,
                                   unsigned int* __restrict__ norm_bits, int64_t m_pad, int d_pad, int dt, int vec,
                                   const uint32_t* __restrict__ fmt_word) {
    const uint32_t fmt = fmt_word != nullptr ? __ldg(fmt_word) : FMT_BF16;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int pitch = d_pad + PLANE_AUG_COLS;
    __nv_bfloat16* o = rows + row * pitch;
    float sq[2] = {0.f, 0.f};                   // NORM_ROW, NORM_LOST
    if (row >= m) {
        for (int c = lane; c < pitch; c += 32) o[c] = __float2bfloat16_rn(c == d_pad ? -3.0e38f : 0.f);
        if (lane == 0) hnorm[row] = pos_inf();
    } else {
        const void* p = row_at(db, row, ld, dt);
        for (int c = lane * 4; c < d_pad; c += 128) {
            const float4 v = ld_row4(p, c, d, vec, dt);
            const uint2 w = operand4_bits(v, fmt);
            sq[0] += sq4(v);
            sq[1] += sq4(operand4_lost(v, w, fmt));
            *reinterpret_cast<uint2*>(o + c) = w;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            sq[0] += __shfl_xor_sync(FULL_MASK, sq[0], off);
            sq[1] += __shfl_xor_sync(FULL_MASK, sq[1], off);
        }
        if (lane == 0) hnorm[row] = 0.5f * sq[0];
        write_norm_columns(o + d_pad, sq[0], PLANE_AUG_COLS);
    }
    block_norms_update(norm_bits, sq);
}

// Operand format of a set of fp32 rows, from FMT_SAMPLE of them spread over the set: fp16 where it loses less than half
// as much as bf16 (eight times less on values between 2^-14 and 65 504, which rows mostly are), bf16 where values lie beyond
// fp16's range, or NaN or infinities make the comparison fail.  Only speed hangs on the choice: what rounding
// takes from each row is measured by the pass that does it, in either format, and the proofs build on that.
constexpr int FMT_SAMPLE = 128;
__global__ void __launch_bounds__(1024) operand_format_kernel(const float* __restrict__ x, int64_t n, int64_t ld, int d,
                                                              uint32_t* __restrict__ fmt) {
    __shared__ float s_b[32], s_h[32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t count = n < FMT_SAMPLE ? n : FMT_SAMPLE;
    float lb = 0.f, lh = 0.f;
    for (int64_t i = warp; i < count; i += 32) {
        const float* p = x + (i * n / count) * ld;
        for (int c = lane; c < d; c += 32) {
            const float v = __ldg(p + c);
            const float4 v4 = make_float4(v, 0.f, 0.f, 0.f);
            const float b = bf16_lost(v), h = f16_lost4(v4, f16x4_bits(v4)).x;
            lb += b * b;
            lh += h * h;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lb += __shfl_xor_sync(FULL_MASK, lb, o);
        lh += __shfl_xor_sync(FULL_MASK, lh, o);
    }
    if (lane == 0) { s_b[warp] = lb; s_h[warp] = lh; }
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = 0.f, h = 0.f;
        for (int w = 0; w < 32; ++w) { b += s_b[w]; h += s_h[w]; }
        *fmt = h < 0.25f * b ? FMT_F16 : FMT_BF16;
    }
}
int launch_operand_format(const float* x, int64_t n, int64_t ld, int d, uint32_t* fmt, cudaStream_t st) {
    operand_format_kernel<<<1, 1024, 0, st>>>(x, n, ld, d, fmt);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

PlaneLayout plane_layout(int64_t m, int d) {
    PlaneLayout L;
    L.m_pad = round_up(m, 256);
    L.d_pad = (int)round_up(d, 64);
    L.pitch = L.d_pad + PLANE_AUG_COLS;
    L.off_rows = 0;
    L.off_hnorm = round_up(L.m_pad * (int64_t)L.pitch * 2, 1024);
    L.off_meta = L.off_hnorm + round_up(L.m_pad * 4, 1024);
    L.bytes = L.off_meta + 1024;
    return L;
}

// Fills `plane` (layout plane_layout(m, d)) for the fp32 rows of db.
int launch_plane_build(const void* db, int64_t m, int d, int64_t ld, void* plane, cudaStream_t st, int dt, const uint32_t* fmt) {
    const PlaneLayout L = plane_layout(m, d);
    char* base = static_cast<char*>(plane);
    FL_CHECK_CUDA(cudaMemsetAsync(base + L.off_meta, 0, 1024, st));
    const int wpb = 8;
    plane_build_kernel<<<(unsigned)ceil_div(L.m_pad, wpb), wpb * 32, 0, st>>>(
        db, m, d, ld, reinterpret_cast<__nv_bfloat16*>(base + L.off_rows),
        reinterpret_cast<float*>(base + L.off_hnorm), reinterpret_cast<unsigned int*>(base + L.off_meta),
        L.m_pad, L.d_pad, dt, dt_vec_ok(db, ld, dt) && d % 4 == 0, fmt);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

}  // namespace fl

using namespace fl;

extern "C" int fl_rownorm_f32(const float* x, int64_t n, int d, int64_t ld, float* out, void* stream) {
    FL_CHECK_ARG(n >= 0 && d >= 1 && ld >= d, "fl_rownorm_f32: bad shape n=%lld d=%d ld=%lld",
                 (long long)n, d, (long long)ld);
    if (n == 0) return FL_OK;
    FL_CHECK_ARG(x && out, "fl_rownorm_f32: null pointer");
    const int wpb = 8;
    rownorm_kernel<<<(unsigned)ceil_div(n, wpb), wpb * 32, 0, (cudaStream_t)stream>>>(x, n, d, ld, out);
    FL_CHECK_LAUNCH();
    return FL_OK;
}

extern "C" int64_t fl_knn_plane_bytes(int64_t m, int d) {
    if (m < 1 || d < 1) return 0;
    return plane_layout(m, d).bytes;
}

extern "C" int fl_knn_prepare_db_rows(const void* db, int dtype, int64_t m, int d, int64_t ld, void* plane,
                                      int64_t plane_bytes, void* stream) {
    FL_CHECK_ARG(m >= 1 && d >= 1 && ld >= d, "fl_knn_prepare_db: bad shape m=%lld d=%d ld=%lld",
                 (long long)m, d, (long long)ld);
    FL_CHECK_ARG(dtype == DT_F32 || dtype == DT_BF16 || dtype == DT_F16, "fl_knn_prepare_db: unknown dtype %d", dtype);
    FL_CHECK_ARG(db && plane, "fl_knn_prepare_db: null pointer");
    FL_CHECK_ARG((reinterpret_cast<uintptr_t>(plane) & 255) == 0,
                 "fl_knn_prepare_db: plane must be 256-byte aligned");
    const PlaneLayout L = plane_layout(m, d);
    if (plane_bytes < L.bytes) {
        set_error("fl_knn_prepare_db: plane buffer %lld < %lld bytes", (long long)plane_bytes,
                  (long long)L.bytes);
        return FL_EWORKSPACE;
    }
    return launch_plane_build(db, m, d, ld, plane, (cudaStream_t)stream, dtype);
}

extern "C" int fl_knn_prepare_db_f32(const float* db, int64_t m, int d, int64_t ld, void* plane,
                                     int64_t plane_bytes, void* stream) {
    return fl_knn_prepare_db_rows(db, DT_F32, m, d, ld, plane, plane_bytes, stream);
}
