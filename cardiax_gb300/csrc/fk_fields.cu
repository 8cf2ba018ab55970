// Classification of stimulus fields: the bounding box of a field's non-zero cells, their number and
// the range of their values, which tell a constant rectangle (a descriptor in the kernels, no
// memory traffic) from a dense field and from an empty one.
//
// Set-up work of every tissue.  As a chain of library reductions with a synchronisation after each
// it took 0.3 ms per field, 5 of the 11 ms of a gradient of 16 experiments; here all fields of a
// call are read once by one launch and the host waits once: 20 us for a call, whatever its fields.
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "../../include/cardiax_gb300.h"

namespace fk {

namespace {

constexpr int kFieldsPerLaunch = 64;

struct FieldPtrs {
    const float *p[kFieldsPerLaunch];
};

// Floats as unsigned integers of the same order.
__host__ __device__ inline uint32_t order_key(uint32_t b) { return b & 0x80000000u ? ~b : b | 0x80000000u; }
inline uint32_t from_key(uint32_t k) { return k & 0x80000000u ? k & 0x7fffffffu : ~k; }

// Maxima over the non-zero cells (minima as maxima of the complement, so that zeroed memory is the
// neutral element of all).
struct FieldStats {
    uint32_t r_hi, c_hi, r_lo, c_lo;  // r + 1, c + 1, and ~r, ~c
    uint32_t v_hi, v_lo;              // order_key and its complement
    uint32_t nan, pad;
    unsigned long long count;
};

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads)
    fk_field_stats_kernel(FieldPtrs f, int H, int W, int64_t pitch, FieldStats *out) {
    const float *p = f.p[blockIdx.y];
    uint32_t m[7] = {0, 0, 0, 0, 0, 0, 0};
    unsigned count = 0;
    for (int r = blockIdx.x; r < H; r += gridDim.x) {
        const float *row = p + (int64_t)r * pitch;
        for (int c = threadIdx.x; c < W; c += kThreads) {
            const float v = __ldg(row + c);
            if (v != 0.0f) {  // true for NaN
                const uint32_t k = order_key(__float_as_uint(v));
                m[0] = max(m[0], (uint32_t)r + 1u);
                m[1] = max(m[1], (uint32_t)c + 1u);
                m[2] = max(m[2], ~(uint32_t)r);
                m[3] = max(m[3], ~(uint32_t)c);
                m[4] = max(m[4], k);
                m[5] = max(m[5], ~k);
                m[6] |= v != v ? 1u : 0u;
                ++count;
            }
        }
    }
    __shared__ uint32_t s[7];
    __shared__ unsigned s_count;
    if (threadIdx.x < 7) s[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        const uint32_t x = __reduce_max_sync(0xffffffffu, m[k]);
        if ((threadIdx.x & 31) == 0 && x) atomicMax(&s[k], x);
    }
    const unsigned n = __reduce_add_sync(0xffffffffu, count);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&s_count, n);
    __syncthreads();
    if (s_count == 0) return;
    uint32_t *o = reinterpret_cast<uint32_t *>(out + blockIdx.y);
    if (threadIdx.x < 7 && s[threadIdx.x]) atomicMax(o + threadIdx.x, s[threadIdx.x]);
    if (threadIdx.x == 0) atomicAdd(&out[blockIdx.y].count, (unsigned long long)s_count);
}

}  // namespace

}  // namespace fk

extern "C" size_t fk_analyse_workspace_bytes(int n) {
    return n > 0 ? sizeof(fk::FieldStats) * (size_t)n : 0;
}

extern "C" int fk_analyse_fields(const float *const *fields, int n, int64_t H, int64_t W, int64_t pitch,
                                 void *workspace, size_t workspace_bytes, fk_field_kind *out,
                                 void *stream) {
    if (n == 0) return FK_OK;
    if (!fields || !workspace || !out) return FK_ERR_NULL;
    if (n < 0 || H < 1 || W < 1 || pitch < W || H > (1 << 24) || W > (1 << 24)) return FK_ERR_SHAPE;
    if (workspace_bytes < fk_analyse_workspace_bytes(n)) return FK_ERR_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(workspace) & 7u) return FK_ERR_ALIGN;
    for (int k = 0; k < n; ++k)
        if (!fields[k]) return FK_ERR_NULL;
    cudaStream_t s = (cudaStream_t)stream;
    fk::FieldStats *stats = static_cast<fk::FieldStats *>(workspace);
    if (cudaMemsetAsync(stats, 0, sizeof(fk::FieldStats) * n, s) != cudaSuccess) return FK_ERR_CUDA;
    for (int k0 = 0; k0 < n; k0 += fk::kFieldsPerLaunch) {
        const int m = n - k0 < fk::kFieldsPerLaunch ? n - k0 : fk::kFieldsPerLaunch;
        fk::FieldPtrs f{};
        for (int k = 0; k < m; ++k) f.p[k] = fields[k0 + k];
        const unsigned rows = (unsigned)(H < 608 ? H : 608);
        fk::fk_field_stats_kernel<<<dim3(rows, (unsigned)m), fk::kThreads, 0, s>>>(f, (int)H, (int)W, pitch,
                                                                                  stats + k0);
        if (cudaGetLastError() != cudaSuccess) return FK_ERR_CUDA;
    }
    std::vector<fk::FieldStats> h((size_t)n);
    if (cudaMemcpyAsync(h.data(), stats, sizeof(fk::FieldStats) * n, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return FK_ERR_CUDA;
    for (int k = 0; k < n; ++k) {
        const fk::FieldStats &x = h[k];
        fk_field_kind &o = out[k];
        o = fk_field_kind{};
        if (x.count == 0) continue;  // kind 0: empty
        o.r0 = (int32_t)~x.r_lo;
        o.r1 = (int32_t)x.r_hi;
        o.c0 = (int32_t)~x.c_lo;
        o.c1 = (int32_t)x.c_hi;
        const uint32_t lo = fk::from_key(~x.v_lo), hi = fk::from_key(x.v_hi);
        const unsigned long long area = (unsigned long long)(o.r1 - o.r0) * (unsigned long long)(o.c1 - o.c0);
        o.kind = !x.nan && lo == hi && x.count == area ? 1 : 2;
        static_assert(sizeof(float) == sizeof(uint32_t), "");
        __builtin_memcpy(&o.amplitude, &hi, sizeof hi);
    }
    return FK_OK;
}
