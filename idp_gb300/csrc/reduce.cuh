// Per-instance sums in one launch: every CTA reduces its chunk and leaves the
// partial sum; the last CTA of an instance to finish adds the instance's
// partials in chunk order (strided over its threads, then a fixed tree), so the
// result does not depend on the order in which the CTAs ran. (A second launch
// for the partials cost as much as the sums of a small mesh: 33 of the 312
// launches of a four-iteration step.)
#pragma once
#include "common.cuh"

namespace idp {

// sum over the CTA in a fixed order, on every thread (blockDim.x <= 1024, a
// multiple of 32)
__device__ inline double cta_sum_fixed(double v) {
    __shared__ double sw[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = sw[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r += sw[w];
    return r;
}

struct InstSum {
    const int* coff;        // chunk range of every instance (nI + 1)
    int per;                // CTAs per chunk
    int nI;
    double* part;           // one value per CTA
    unsigned int* counter;  // nI, zero between launches
    double* out;            // nI
    int accumulate;         // out += instead of =
};

// v: this thread's share; every thread of every CTA of the launch calls this
// (CTA b works on chunk b / per; instances without chunks get 0)
__device__ inline void inst_sum(const InstSum& r, int inst, double v) {
    __shared__ bool last;
    const double s = cta_sum_fixed(v);
    if (blockIdx.x == 0 && !r.accumulate)
        for (int i = threadIdx.x; i < r.nI; i += blockDim.x)
            if (r.coff[i + 1] == r.coff[i]) r.out[i] = 0.0;
    const int c0 = r.per * r.coff[inst], n = r.per * (r.coff[inst + 1] - r.coff[inst]);
    if (n <= 0) return;  // the placeholder chunk of an empty list
    if (threadIdx.x == 0) {
        r.part[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(r.counter + inst, 1u) == (unsigned int)n - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) a += __ldcg(r.part + c0 + k);
    a = cta_sum_fixed(a);
    if (threadIdx.x == 0) {
        r.out[inst] = r.accumulate ? r.out[inst] + a : a;
        r.counter[inst] = 0;
    }
}

}  // namespace idp
