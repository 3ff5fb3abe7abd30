// An eighth of eight_over_density for every float dr, alone and in pairs, against
// __frcp_rn of the floored density. Prints "wrong subnormal", exit status 1 when one differs
// (subnormal reciprocals, densities above 2^126: by more than 2^-149), 2 on a
// CUDA error.
#include <cstdio>

#include "shifted_math.cuh"

using namespace lbm;

__global__ void sweep(unsigned long long *out) {
    unsigned long long wrong = 0, sub = 0;
    const unsigned long long n = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long q = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; q < 1ull << 32; q += n) {
        const float dr = __uint_as_float((unsigned int)q), other = __uint_as_float(~(unsigned int)q);
        const float rho = __fadd_rn(1.0f, dr), want = __frcp_rn(rho < 1e-16f ? 1e-16f : rho);
        const float2 p = eight_over_density(make_float2(dr, other)), r = eight_over_density(make_float2(other, dr));
        const float got[3] = {0.125f * eight_over_density(dr), 0.125f * p.x, 0.125f * r.y};
        const bool small = rho > 0x1p126f && rho < INFINITY;
        if (small) sub++;
        for (int k = 0; k < 3; k++) {
            if (isnan(want)) wrong += !isnan(got[k]);
            else if (small) wrong += !(fabsf(got[k] - want) <= 0x1p-149f);
            else wrong += !(got[k] == want);
        }
    }
    if (wrong) atomicAdd(out, wrong);
    if (sub) atomicAdd(out + 1, sub);
}

int main() {
    unsigned long long *d = nullptr, h[2] = {0, 0};
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return 2;
    sweep<<<1216, 256>>>(d);
    if (cudaGetLastError() != cudaSuccess || cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%llu %llu\n", h[0], h[1]);
    return h[0] ? 1 : 0;
}
