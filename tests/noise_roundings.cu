// The quotient and the square root of the noise's radius for every one of the
// 2^23 values of u1, in both lanes, against the IEEE operations: the number of
// values that differ, quotients and roots.
#include "lbm_noise.cuh"

namespace {

__global__ void compare(unsigned long long *wrong)
{
    const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x, w = v ^ 0x2aaaaau;  // the other lane: another value
    if (v >= 1u << 23) return;
    const float2 u1 = make_float2(((float)v + 0.5f) / 8388608.0f, ((float)w + 0.5f) / 8388608.0f);  // exact
    float2 m, fe;
    lbm::log_split(u1.x, m.x, fe.x);
    lbm::log_split(u1.y, m.y, fe.y);
    const float2 num = make_float2(m.x - 1.0f, m.y - 1.0f), den = make_float2(m.x + 1.0f, m.y + 1.0f);
    const float2 q = lbm::nz_div(num, den);
    if (__float_as_uint(q.x) != __float_as_uint(__fdiv_rn(num.x, den.x)) ||
        __float_as_uint(q.y) != __float_as_uint(__fdiv_rn(num.y, den.y)))
        atomicAdd(wrong, 1ull);
    const float2 l2 = lbm::nz_mul(lbm::nz_f2(-2.0f), lbm::series_logf2(u1));
    const float2 r = lbm::nz_sqrt(l2);
    if (__float_as_uint(r.x) != __float_as_uint(__fsqrt_rn(l2.x)) ||
        __float_as_uint(r.y) != __float_as_uint(__fsqrt_rn(l2.y)))
        atomicAdd(wrong + 1, 1ull);
    atomicAdd(wrong + 2, 1ull);
}

}  // namespace

// out: wrong quotients, wrong roots, values compared
extern "C" int noise_roundings(unsigned long long *out)
{
    unsigned long long *d = nullptr;
    cudaError_t e = cudaMalloc(&d, 3 * sizeof *d);
    if (e == cudaSuccess) e = cudaMemset(d, 0, 3 * sizeof *d);
    if (e == cudaSuccess) {
        compare<<<(1u << 23) / 256, 256>>>(d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 3 * sizeof *d, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
