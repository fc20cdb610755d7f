// Counts over the device arithmetic that the field kernels call exact: built
// and called by test_device_math.py.
#include "rf_kernel.cuh"

namespace {

__device__ uint64_t mix(uint64_t x) {   // splitmix64
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}
__device__ double unit(uint64_t r) { return (double)(r >> 11) * 0x1p-53; }
__device__ float mantissa(uint32_t bits, int exponent) {
    return __uint_as_float((bits & 0x807fffffu) | (uint32_t)(exponent + 127) << 23);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

typedef unsigned long long Count;

// every float of [2^-120, 2^120)
__global__ void k_recip(Count *bad) {
    const uint32_t first = (127u - 120u) << 23, last = (127u + 120u) << 23;
    Count n = 0;
    for (uint64_t i = first + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < last; i += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)i);
        n += !same(recip_rn(x), 1.f / x) + !same(recip_rn(-x), 1.f / -x);
    }
    if (n) atomicAdd(bad, n);
}
// random pairs with exponents within +-60
__global__ void k_quot(Count pairs, Count *bad) {
    Count n = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < pairs; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = mix(2 * i), e = mix(2 * i + 1);
        const float a = mantissa((uint32_t)r, (int)(e % 121) - 60), b = mantissa((uint32_t)(r >> 32), (int)((e >> 32) % 121) - 60);
        n += !same(quot_rn(a, b), a / b);
    }
    if (n) atomicAdd(bad, n);
}
// nodes inside and on the unit sphere, directions of unit length up to rounding
// (kind 0, 1) or of any length (2)
__global__ void k_exit(Count rays, Count *bad) {
    Count n = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < rays; i += (uint64_t)gridDim.x * blockDim.x) {
        double v[6];
        for (int k = 0; k < 6; k++) v[k] = 2.0 * unit(mix(8 * i + k)) - 1.0;
        const int kind = (int)(i % 3);
        const double lp = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]), ld = sqrt(v[3] * v[3] + v[4] * v[4] + v[5] * v[5]);
        if (!(lp > 0.0) || !(ld > 0.0)) continue;
        const double rp = (kind == 1 ? 1.0 : unit(mix(8 * i + 6))) / lp, rd = (kind == 2 ? 1.0 : 1.0 / ld);
        const double p[3] = {v[0] * rp, v[1] * rp, v[2] * rp}, d[3] = {v[3] * rd, v[4] * rd, v[5] * rd};
        const double np = __dsqrt_rn(dsum3sq(p[0], p[1], p[2])), c = __dsub_rn(__dmul_rn(np, np), 1.0);
        const double a = sphere_exit_unit(p[0], p[1], p[2], c, d[0], d[1], d[2]), b = sphere_exit(p[0], p[1], p[2], d[0], d[1], d[2]);
        n += __double_as_longlong(a) != __double_as_longlong(b);
    }
    if (n) atomicAdd(bad, n);
}
// 2^x over every float of [-1/16, 0]: none above 1
__global__ void k_ex2(Count *bad) {
    const uint32_t first = 0x80000000u, last = __float_as_uint(-0.0625f);
    Count n = 0;
    for (uint64_t i = first + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= last; i += (uint64_t)gridDim.x * blockDim.x)
        n += !(ex2(__uint_as_float((uint32_t)i)) <= 1.f);
    if (n) atomicAdd(bad, n);
}
// a dust cell's update with and without the division's slow path, over cells
// inside the range of the fast one (dust_in_range)
__global__ void k_dust(Count cells, Count *bad) {
    Count n = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cells; i += (uint64_t)gridDim.x * blockDim.x) {
        float v[8], g[2], I[2];
        for (int k = 0; k < 8; k++) {   // A A' E E' Ad Ad' Jd Jd': opacities to 2^88, emissivities to 2^-36
            const uint64_t r = mix(16 * i + k);
            const int top = (k / 2) % 2 ? -36 : (r >> 60) ? 8 : 88, span = (k / 2) % 2 ? 80 : 100;
            v[k] = mantissa((uint32_t)r & (k / 2 == 0 ? 0xffffffffu : 0x7fffffffu), top - (int)((r >> 32) % span));
            if ((r >> 56) % 16 == 0) v[k] = 0.f;
        }
        for (int k = 0; k < 2; k++) {
            g[k] = ex2(-(float)(unit(mix(16 * i + 8 + k)) * 40.0));
            I[k] = mantissa((uint32_t)mix(16 * i + 10 + k) & 0x7fffffffu, -30 - (int)(mix(16 * i + 12 + k) % 60));
        }
        if (!dust_in_range(make_float4(v[0], v[2], v[4], v[6])) || !dust_in_range(make_float4(v[1], v[3], v[5], v[7]))) {
            n++;
            continue;
        }
        const DustPack c{make_float2(v[0], v[1]), make_float2(v[2], v[3]), make_float2(v[4], v[5]), make_float2(v[6], v[7])};
        float2 a = make_float2(I[0], I[1]), b = a;
        transfer2_dust(false, true, a, c, make_float2(g[0], g[1]));
        transfer2_dust(false, false, b, c, make_float2(g[0], g[1]));
        n += !same(a.x, b.x) + !same(a.y, b.y);
    }
    if (n) atomicAdd(bad, n);
}

}  // namespace

// number of exceptions (-1: the device failed)
extern "C" long long device_math(int which, long long count) {
    Count *d = nullptr, h = 0;
    if (cudaMalloc(&d, sizeof h) || cudaMemset(d, 0, sizeof h)) return -1;
    const int grid = 4 * 152, block = 256;
    if (which == 0) k_recip<<<grid, block>>>(d);
    if (which == 1) k_quot<<<grid, block>>>((Count)count, d);
    if (which == 2) k_exit<<<grid, block>>>((Count)count, d);
    if (which == 3) k_ex2<<<grid, block>>>(d);
    if (which == 4) k_dust<<<grid, block>>>((Count)count, d);
    const bool ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(d);
    return ok ? (long long)h : -1;
}
