// x(0) + x(1) + ... + x(n - 1) added left to right into one FP64 accumulator,
// bit for bit, by many threads. While the accumulator stays in one binade
// (unit in the last place u), an addition only adds x rounded to a multiple of
// u: an integer that does not depend on the accumulator, except for a tie,
// which goes by its parity. So an item, or a run of items, is a pair of
// integers (the growth from an even and from an odd accumulator), pairs join
// associatively, and a scan over the threads' runs finds every partial sum and
// the first item that leaves the binade. That item is added in FP64 and the
// next pass starts behind it. Negative, infinite or NaN items, and sums near
// the ends of the exponent range, are added one at a time.
//
// Bound by the integer work per item (about 40 instructions, against a chain of
// dependent FP64 additions of about 100 cycles each). The mean of the 43,000 edges
// of a stack of seven plates, eight chains: 293 -> 109 us.
#pragma once
#include "common.cuh"

namespace idp {

struct SumInc { unsigned long long a0, a1; };

constexpr unsigned long long kSumOne = 1ull << 52, kSumFull = 1ull << 53, kSumSat = 1ull << 54;

__device__ __forceinline__ SumInc sum_join(SumInc f, SumInc g) {
    return {min(f.a0 + ((f.a0 & 1) ? g.a1 : g.a0), kSumSat), min(f.a1 + ((f.a1 & 1) ? g.a0 : g.a1), kSumSat)};
}

// f followed by the item with these bits, for an accumulator of biased exponent e
__device__ __forceinline__ SumInc sum_item(SumInc f, unsigned long long bits, int e) {
    const int ex = (int)(bits >> 52), d = e - ex;
    if (ex == 0 || d > 53) return f;  // below half of the last place
    if (d < 0) return {kSumSat, kSumSat};
    const unsigned long long m = (bits & (kSumOne - 1)) | kSumOne, q = m >> d, r = m & ((1ull << d) - 1);
    const unsigned long long half = d ? 1ull << (d - 1) : 1ull;
    f.a0 += q;
    f.a1 += q;
    if (r > half) {
        ++f.a0;
        ++f.a1;
    } else if (r == half) {  // tie: to even
        f.a0 += f.a0 & 1;
        f.a1 += (f.a1 & 1) ^ 1;
    }
    return {min(f.a0, kSumSat), min(f.a1, kSumSat)};
}

// WARPS = 1: by the calling warp; otherwise by the whole CTA of 32 * WARPS
// threads. Every thread of the group calls it and receives the sum.
template <int WARPS, class F>
__device__ double serial_sum(const F& x, long n) {
    constexpr int G = 32 * WARPS, kHead = 32, kRun = 64;
    __shared__ SumInc tot[WARPS];
    __shared__ double s_next;
    __shared__ long k_next;
    __shared__ int first_next;
    const int lane = threadIdx.x & 31, warp = WARPS > 1 ? threadIdx.x >> 5 : 0, tid = 32 * warp + lane;
    double s = 0.0;
    long k = 0;
    long head = min(n, (long)kHead);  // items before this one are added one at a time
    while (true) {
        for (; k < head; ++k) s += x(k);
        if (k >= n) return s;
        const unsigned long long sb = (unsigned long long)__double_as_longlong(s);
        const int e = (int)(sb >> 52);
        if (e < 64 || e > 2000) {
            head = min(n, k + kHead);
            continue;
        }
        const unsigned long long S = (sb & (kSumOne - 1)) | kSumOne;
        // the sum leaves its binade within about as many items as it holds
        const int run = (int)max(1L, min((long)kRun, (min(k, n - k) + G - 1) / G));
        const long base = k + (long)tid * run;
        const int cnt = (int)max(0L, min((long)run, n - base));
        SumInc own{0, 0};
        bool bad = false;
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            const unsigned long long b = (unsigned long long)__double_as_longlong(x(base + j));
            bad |= b >= 0x7ff0000000000000ull;
            own = sum_item(own, b, e);
        }
        SumInc inc = own;
        for (int o = 1; o < 32; o <<= 1) {
            const SumInc p = {__shfl_up_sync(0xffffffffu, inc.a0, o), __shfl_up_sync(0xffffffffu, inc.a1, o)};
            if (lane >= o) inc = sum_join(p, inc);
        }
        SumInc before = {__shfl_up_sync(0xffffffffu, inc.a0, 1), __shfl_up_sync(0xffffffffu, inc.a1, 1)};
        if (lane == 0) before = {0, 0};
        if (WARPS > 1) {
            if (lane == 31) tot[warp] = inc;
            if (tid == 0) first_next = G;
            bad = __syncthreads_or(bad);
            SumInc w{0, 0};
            for (int i = 0; i < warp; ++i) w = sum_join(w, tot[i]);
            before = sum_join(w, before);
        } else {
            bad = __any_sync(0xffffffffu, bad);
        }
        if (bad) {
            head = n;
            continue;
        }
        unsigned long long P = S + ((S & 1) ? before.a1 : before.a0);
        const unsigned long long E = P + ((P & 1) ? own.a1 : own.a0);
        const bool leaves = E >= kSumFull;
        int first;
        if (WARPS > 1) {
            const unsigned int bal = __ballot_sync(0xffffffffu, leaves);
            if (bal && lane == 0) atomicMin(&first_next, 32 * warp + __ffs(bal) - 1);
            __syncthreads();
            first = first_next;
        } else {
            const unsigned int bal = __ballot_sync(0xffffffffu, leaves);
            first = bal ? __ffs(bal) - 1 : G;
        }
        auto value = [&](unsigned long long v) {  // of an accumulator of v units
            return __longlong_as_double((long long)(((unsigned long long)e << 52) + (v - kSumOne)));
        };
        double sn = value(E);
        long kn = min(n, k + (long)G * run);
        if (tid == first) {
            for (int j = 0;; ++j) {  // ends before cnt: the run's growth leaves the binade
                const double xj = x(base + j);
                const SumInc g = sum_item({0, 0}, (unsigned long long)__double_as_longlong(xj), e);
                const unsigned long long N = P + ((P & 1) ? g.a1 : g.a0);
                if (N >= kSumFull || j + 1 >= cnt) {
                    sn = value(P) + xj;
                    kn = base + j + 1;
                    break;
                }
                P = N;
            }
        }
        const int src = first < G ? first : G - 1;
        if (WARPS > 1) {
            if (tid == src) {
                s_next = sn;
                k_next = kn;
            }
            __syncthreads();
            s = s_next;
            k = k_next;
        } else {
            s = __shfl_sync(0xffffffffu, sn, src);
            k = __shfl_sync(0xffffffffu, kn, src);
        }
        head = k;
    }
}

}  // namespace idp
