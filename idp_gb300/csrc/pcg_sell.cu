// PCG for instances without contact blocks: persistent CTAs that hold their
// rows' matrix in shared memory and every vector in registers, exchanging
// nothing but two values per halo component and five partial sums per iteration.
//
// Partition. An instance of V vertices is cut into runs of consecutive vertices
// (rows), one CTA each; the cut depends on V (and the context's parameters)
// alone, so a result does not depend on what else is solved. Up to kSellSolo
// vertices take one CTA: no exchange at all. Above that at least kSellRows rows
// per CTA, and at most one CTA per SM.
//
// Layout. A warp works on a slice of 8 rows, 4 lanes per row; a CTA's rows are
// sorted by length and a slice stores its blocks as slot rows of 32 lanes, the
// nine values in nine arrays of 32 (shared-memory reads without bank
// conflicts). Blocks whose column lies in the CTA's own rows come first in a
// slice; the other columns are numbered in the CTA's halo list. Both lists depend
// on the pattern only and are laid out once per commit (k_sell_plan).
//
// Exchange. A value is stored as a 64-bit word of 32 payload bits and a 32-bit
// tag that no earlier exchange used (FP64: two words), and its readers poll the
// data itself: neither a fence nor a flag is waited for, and a halo value is
// usable one L2 round trip after it was written. The CTAs' partial sums travel
// the same way and every CTA adds them in the same order. Two slots by parity
// suffice: a CTA overwrites exchange e with e + 2 only after it has every CTA's
// sums of e + 1, which each wrote after it had read all of e.
//
// PCG with one exchange per iteration (predict and recompute, after Chen &
// Carson 2020): s = A p and q = M^{-1} s are formed, and the sums p.s, r.u, r.q,
// s.q and r.r travel together with q; they give alpha, and beta by predicting
// the next r.u, which the next iteration recomputes. The owner of a row sends u =
// M^{-1} r a phase ahead, so that a neighbour can form the next u = u - alpha q
// and p = u + beta p of its halo by itself: only the halo's p is carried on.
// No product with A and no residual but r is kept by recurrence, and on the
// matrices of bars with E = 1e4 to 1e11 (h = 0.1) the solves end at the residual
// of classical PCG, and up to 1e7 within 10 % of its iterations, in FP32 and FP64.
// (The pipelined recurrences of Ghysels & Vanroose, which hide the exchange behind
// half of the product, lose the residual on stiff bodies: E = 1e9, FP32 sweeps
// stall at 2e-3 to 2e-2, FP64 ends at 1e-8 for an asked 1e-12.)
//
// Bound by the shared-memory reads of the matrix (20 wavefronts per slot row, 10 of
// them bank conflicts of the gathers), the FP64 pipe, or, with few rows, the
// exchange. Microseconds per iteration, with the pipelined recurrences -> now: blob of
// 220,515 tets (49,863 vertices, 328 rows per SM) in FP32 5.7 -> 6.9 (k_pcg_grid: 12),
// blob of 18,210 vertices 2.9 -> 3.7, bar of 160 vertices on one CTA 2.3 (k_pcg_cluster:
// 10.5); blob of 5,838 vertices in FP64 14 (66 on 16 cluster CTAs). Tried on the
// exchange and taken back: copies of the sums for groups of CTAs, warps that poll the
// sums while others gather the halo (5.8 against 4.5 per iteration of that blob in
// FP32), waits before the first poll, 6 or 8 polls in flight.
#include <algorithm>
#include "engine.hpp"

namespace idp {

namespace {

constexpr int kST = 512;                 // threads per CTA
constexpr int kSW = kST / 32;
constexpr int kSliceRows = 8;
// Rows per CTA at least, where there are several, and the largest instance of one
// CTA, {FP32, FP64}. Microseconds per iteration on bars and blobs of 160 to
// 18,210 vertices: FP32 2.8-3.5 with 40 to 128 rows, 3.8-4.5 with 160 (a second slice
// per warp); 2.3 on one CTA of 160 rows, 3.5 of 320. FP64 is bound by its pipe:
// 12.3-14 with 40 rows, 13-17.5 with 128, 17 on one CTA of 160.
constexpr int kSellRows[2] = {64, 40}, kSellSolo[2] = {192, 40};
constexpr int kSellMaxRows = 3 * kSW * kSliceRows;  // rows per CTA: three slices per warp
constexpr int kHaloTable = 4096;         // hash slots of the halo search
constexpr int kHaloMax = 2600;           // halo vertices per CTA
constexpr int kSellSmem = 222 * 1024;    // dynamic shared memory limit
constexpr int kPollCtas = 5;             // CTAs whose sums a lane polls at a time (152 / 32)
constexpr unsigned int kSellSpin = 1u << 21;  // polls before giving up (about 1 s)

template <class T>
constexpr int words() { return sizeof(T) / 4; }

__device__ __forceinline__ void put_word(unsigned long long* p, unsigned int v, unsigned int tag) {
    const unsigned long long w = ((unsigned long long)tag << 32) | v;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long get_word(const unsigned long long* p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ void get_words2(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool tagged(unsigned long long w, unsigned int tag) { return (unsigned int)(w >> 32) == tag; }
__device__ __forceinline__ double join(unsigned long long lo, unsigned long long hi) {
    return __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
}
// a value at p (FP64: its halves `next` words apart)
__device__ __forceinline__ void put_value(unsigned long long* p, long, float v, unsigned int tag) {
    put_word(p, __float_as_uint(v), tag);
}
__device__ __forceinline__ void put_value(unsigned long long* p, long next, double v, unsigned int tag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    put_word(p, (unsigned int)b, tag);
    put_word(p + next, (unsigned int)(b >> 32), tag);
}
__device__ __forceinline__ bool get_value(const unsigned long long* p, long, float& v, unsigned int tag) {
    const unsigned long long w = get_word(p);
    v = __uint_as_float((unsigned int)w);
    return tagged(w, tag);
}
__device__ __forceinline__ bool get_value(const unsigned long long* p, long next, double& v, unsigned int tag) {
    const unsigned long long a = get_word(p), b = get_word(p + next);
    v = join(a, b);
    return tagged(a, tag) && tagged(b, tag);
}
// the pair (u, q) at p; without `both` only u has to have arrived
__device__ __forceinline__ bool get_pair(const unsigned long long* p, float& u, float& q, unsigned int tag, bool both) {
    unsigned long long a, b;
    get_words2(p, a, b);
    u = __uint_as_float((unsigned int)a);
    q = __uint_as_float((unsigned int)b);
    return tagged(a, tag) && (!both || tagged(b, tag));
}
__device__ __forceinline__ bool get_pair(const unsigned long long* p, double& u, double& q, unsigned int tag, bool both) {
    unsigned long long a, b, c, d;
    get_words2(p, a, b);
    get_words2(p + 2, c, d);
    u = join(a, b);
    q = join(c, d);
    return tagged(a, tag) && tagged(b, tag) && (!both || (tagged(c, tag) && tagged(d, tag)));
}

// The warp's sums of kSums values: value j ends on the lanes whose bits 4, 3, 2
// are those of j (sum_value). The lanes halve the values they carry at each of
// the first three steps: 9 additions, not 25.
constexpr int kSums = 5;
__device__ __forceinline__ int sum_value(int lane) { return (lane >> 4 & 1) << 2 | (lane >> 3 & 1) << 1 | (lane >> 2 & 1); }
template <class T>
__device__ __forceinline__ T warp_sums(const T (&v)[kSums], int lane) {
    const unsigned full = 0xffffffffu;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    // the upper half goes on with value 4 alone
    T a0 = b4 ? v[4] : v[0], a1 = b4 ? T(0) : v[1], a2 = b4 ? T(0) : v[2], a3 = b4 ? T(0) : v[3];
    a0 += __shfl_xor_sync(full, b4 ? v[0] : v[4], 16);
    a1 += __shfl_xor_sync(full, b4 ? v[1] : T(0), 16);
    a2 += __shfl_xor_sync(full, b4 ? v[2] : T(0), 16);
    a3 += __shfl_xor_sync(full, b4 ? v[3] : T(0), 16);
    T c0 = b3 ? a2 : a0, c1 = b3 ? a3 : a1;
    c0 += __shfl_xor_sync(full, b3 ? a0 : a2, 8);
    c1 += __shfl_xor_sync(full, b3 ? a1 : a3, 8);
    T r = b2 ? c1 : c0;
    r += __shfl_xor_sync(full, b2 ? c0 : c1, 4);
    r += __shfl_xor_sync(full, r, 2);
    r += __shfl_xor_sync(full, r, 1);
    return r;
}

// Layout of one CTA's rows: halo list (hash of the columns outside its rows),
// rows sorted by (halo slots, local slots), slices and their slot rows.
// total[0], total[1]: slot rows and halo entries given out; total[2]: something
// did not fit (the CTA's instance then keeps to the other kernels).
__global__ void k_sell_plan(SellCta* __restrict__ cta, const int* __restrict__ rowptr, const int* __restrict__ colidx,
                            int2* __restrict__ slice, int* __restrict__ src, unsigned short* __restrict__ col,
                            unsigned short* __restrict__ prow, int* __restrict__ halo, unsigned int slot_cap,
                            unsigned int halo_cap, unsigned int* __restrict__ total) {
    __shared__ int hkey[kHaloTable];
    __shared__ unsigned short hidx[kHaloTable];
    __shared__ unsigned int key[512];
    __shared__ int wl[kSellMaxRows / kSliceRows], wh[kSellMaxRows / kSliceRows], so[kSellMaxRows / kSliceRows + 1];
    __shared__ int cnt, s_halo0, s_slot0, s_bad;
    __shared__ int scan[256];
    SellCta me = cta[blockIdx.x];
    const int tid = threadIdx.x, nt = blockDim.x, v0 = me.v0, nv = me.nv;
    for (int i = tid; i < kHaloTable; i += nt) hkey[i] = -1;
    if (tid == 0) { cnt = 0; s_bad = 0; }
    __syncthreads();
    // halo: every column outside [v0, v0 + nv)
    for (int lv = tid; lv < nv; lv += nt)
        for (int k = rowptr[v0 + lv]; k < rowptr[v0 + lv + 1]; ++k) {
            const int c = colidx[k];
            if (c >= v0 && c < v0 + nv) continue;
            unsigned int h = ((unsigned int)c * 2654435761u) >> 20;
            for (int probe = 0; probe < kHaloTable; ++probe, h = (h + 1) & (kHaloTable - 1)) {
                if (*(volatile int*)&cnt > kHaloMax) break;
                const int old = atomicCAS(&hkey[h], -1, c);
                if (old == c) break;
                if (old == -1) { atomicAdd(&cnt, 1); break; }
            }
        }
    __syncthreads();
    if (cnt > kHaloMax) {
        if (tid == 0) { atomicOr(total + 2, 1u); cta[blockIdx.x].nsr = -1; }
        return;
    }
    // compact: thread t numbers the occupied slots of its 16
    const int per = kHaloTable / 256;
    int mine = 0;
    if (tid < 256)
        for (int i = 0; i < per; ++i) mine += hkey[tid * per + i] >= 0;
    if (tid < 256) scan[tid] = mine;
    __syncthreads();
    for (int o = 1; o < 256; o <<= 1) {
        int add = 0;
        if (tid < 256 && tid >= o) add = scan[tid - o];
        __syncthreads();
        if (tid < 256) scan[tid] += add;
        __syncthreads();
    }
    if (tid == 0) s_halo0 = (int)atomicAdd(total + 1, (unsigned int)cnt);
    __syncthreads();
    const bool hfit = (unsigned int)s_halo0 + (unsigned int)cnt <= halo_cap;
    if (tid < 256) {
        int id = scan[tid] - mine;
        for (int i = 0; i < per; ++i)
            if (hkey[tid * per + i] >= 0) {
                hidx[tid * per + i] = (unsigned short)id;
                if (hfit) halo[s_halo0 + id] = hkey[tid * per + i];
                ++id;
            }
    }
    // rows by (halo slots, local slots), longest first
    for (int p = tid; p < 512; p += nt) {
        unsigned int kk = 0;
        if (p < nv) {
            int nl = 0, nh = 0;
            for (int k = rowptr[v0 + p]; k < rowptr[v0 + p + 1]; ++k) {
                const int c = colidx[k];
                if (c >= v0 && c < v0 + nv) ++nl;
                else ++nh;
            }
            const unsigned int sl = min((nl + 3) / 4, 1023), sh = min((nh + 3) / 4, 1023);
            kk = 0x80000000u | (sh << 19) | (sl << 9) | (unsigned int)p;
            if ((nl + 3) / 4 > 1022 || (nh + 3) / 4 > 1022) s_bad = 1;
        }
        key[p] = kk;
    }
    __syncthreads();
    for (int size = 2; size <= 512; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < 256; i += nt) {
                const int a = 2 * i - (i & (stride - 1)), b = a + stride;
                const bool desc = (a & size) == 0;
                const unsigned int x = key[a], y = key[b];
                if (desc ? x < y : x > y) { key[a] = y; key[b] = x; }
            }
            __syncthreads();
        }
    const int ns = (nv + kSliceRows - 1) / kSliceRows;
    for (int s = tid; s < ns; s += nt) {
        int l = 0, h = 0;
        for (int r = 0; r < kSliceRows; ++r) {
            const unsigned int kk = key[s * kSliceRows + r];
            l = max(l, (int)((kk >> 9) & 1023u));
            h = max(h, (int)((kk >> 19) & 1023u));
        }
        wl[s] = l;
        wh[s] = h;
    }
    __syncthreads();
    if (tid == 0) {
        so[0] = 0;
        for (int s = 0; s < ns; ++s) so[s + 1] = so[s] + wl[s] + wh[s];
        s_slot0 = (int)atomicAdd(total, (unsigned int)so[ns]);
        if (!hfit || (unsigned int)s_slot0 + (unsigned int)so[ns] > slot_cap || s_bad) s_bad = 1;
        me.nh = cnt;
        me.halo0 = s_halo0;
        me.slot0 = s_slot0;
        me.nsr = s_bad ? -1 : so[ns];
        if (s_bad) atomicOr(total + 2, 1u);
        cta[blockIdx.x] = me;
    }
    __syncthreads();
    if (s_bad) return;
    for (int s = tid; s < ns; s += nt) slice[me.slice0 + s] = make_int2(so[s], wl[s] | (wh[s] << 16));
    for (int p = tid; p < nv; p += nt) prow[v0 + p] = (unsigned short)(key[p] & 511u);
    const long sb = 32L * s_slot0;
    for (int i = tid; i < 32 * so[ns]; i += nt) {
        src[sb + i] = -1;
        col[sb + i] = 0;
    }
    __syncthreads();
    // lane l4 of a row takes every 4th local block, then every 4th halo block
    for (int i = tid; i < 4 * nv; i += nt) {
        const int p = i >> 2, l4 = i & 3, s = p / kSliceRows, lane = (p % kSliceRows) * 4 + l4;
        const int lv = (int)(key[p] & 511u);
        int nl = 0, nh = 0;
        for (int k = rowptr[v0 + lv]; k < rowptr[v0 + lv + 1]; ++k) {
            const int c = colidx[k];
            const bool local = c >= v0 && c < v0 + nv;
            int& n = local ? nl : nh;
            if ((n & 3) == l4) {
                int id = c - v0;
                if (!local) {
                    unsigned int h = ((unsigned int)c * 2654435761u) >> 20;
                    for (int probe = 0; probe < kHaloTable && hkey[h] != c; ++probe) h = (h + 1) & (kHaloTable - 1);
                    id = hidx[h];
                }
                const long at = sb + 32L * (so[s] + (local ? 0 : wl[s]) + (n >> 2)) + lane;
                src[at] = k;
                col[at] = (unsigned short)id;
            }
            ++n;
        }
    }
}

// halo values whose u and q a thread keeps in registers, and those that go to
// shared memory
template <class T>
constexpr int kHeld = sizeof(T) == 4 ? 4 : 2;
template <class T>
__host__ __device__ inline int halo_rest(int nh) { return 3 * nh > kHeld<T> * kST ? 3 * nh - kHeld<T> * kST : 0; }

template <class T>
struct SellArgs {
    const SellCta* cta;
    const int* list;              // plan CTA of every launched CTA
    const int2* slice;
    const int* src;
    const unsigned short* col;
    const unsigned short* prow;
    const int* halo;
    const T* val;
    const T* dinv;
    const unsigned char* dbc;
    const double* b;
    T* x;
    unsigned long long* xu;       // [2][3 V] pairs of values (u, q)
    unsigned long long* xr;       // [2][kSums][words of a value][plan CTAs]
    long xu_half, xr_half;        // words per parity
    long xr_row;                  // plan CTAs
    unsigned int tag0;
    int nvmax, nhmax, cap;        // rows and halo entries of the largest CTA; slot rows held in shared memory
    const double* tol_inst;
    double rel_tol;
    int max_iters;
    int* iters_out;
    int* err;
};

template <class T, int STEPS>
__global__ void __launch_bounds__(kST, 1) k_pcg_sell(const SellArgs<T> A) {
    extern __shared__ __align__(16) unsigned char sell_smem[];
    T* sval = reinterpret_cast<T*>(sell_smem);                    // [cap][9][32]
    T* sp = sval + 288L * A.cap;                                  // p of the own rows
    T* sph = sp + 3L * A.nvmax;                                   // of the halo: p
    T* suq = sph + 3L * A.nhmax;                                  // and (u, q) past the threads' own
    unsigned short* scol = reinterpret_cast<unsigned short*>(suq + 2L * halo_rest<T>(A.nhmax));  // [cap][32]
    __shared__ T spart[kSW][kSums];   // partial sums by warp
    __shared__ T sred[kSums];         // the instance's
    __shared__ T sscal[2];
    __shared__ int sstop, sbad;
    const SellCta me = A.cta[A.list[blockIdx.x]];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l4 = lane & 3;
    const int nv = me.nv, v0 = me.v0, nc = me.nc, nh3 = 3 * me.nh;
    const int ns = (nv + kSliceRows - 1) / kSliceRows;
    constexpr int W = words<T>();
    if (tid == 0) sbad = 0;
    // ---- stage the slot rows
    const int held = min(me.nsr, A.cap);
    for (int t = warp; t < held; t += kSW) {
        const long at = 32L * (me.slot0 + t) + lane;
        const int k = A.src[at];
        scol[32 * t + lane] = A.col[at];
        const T* m = A.val + 9L * max(k, 0);
#pragma unroll
        for (int j = 0; j < 9; ++j) sval[(9 * t + j) * 32 + lane] = k >= 0 ? m[j] : T(0);
    }
    __syncthreads();
    // ---- this lane's rows (component l4 < 3 of row position p) and their state
    int lv[STEPS], off[STEPS], wl[STEPS], wt[STEPS];
    bool own[STEPS], fixed[STEPS];
    T D0[STEPS], D1[STEPS], D2[STEPS];
    T p[STEPS], x[STEPS], r[STEPS];
#pragma unroll
    for (int t = 0; t < STEPS; ++t) {
        const int sl = warp + kSW * t, pos = sl * kSliceRows + (lane >> 2);
        const bool act = pos < nv;
        off[t] = wl[t] = wt[t] = 0;
        if (sl < ns) {
            const int2 e = A.slice[me.slice0 + sl];
            off[t] = e.x;
            wl[t] = e.y & 0xffff;
            wt[t] = wl[t] + (e.y >> 16);
        }
        lv[t] = act ? A.prow[v0 + pos] : 0;
        const int v = v0 + lv[t];
        fixed[t] = act && A.dbc[v];
        own[t] = act && l4 < 3;
        D0[t] = D1[t] = D2[t] = p[t] = x[t] = r[t] = T(0);
        if (own[t] && !fixed[t]) {
            const T* D = A.dinv + 9L * v + 3 * l4;
            D0[t] = D[0]; D1[t] = D[1]; D2[t] = D[2];
            r[t] = (T)A.b[3L * v + l4];
        }
    }
    const int gb = lane & ~3;
    // M^{-1} applied to the row whose components sit on the group's lanes
    auto precond = [&](int t, T a) -> T {
        const T a0 = __shfl_sync(0xffffffffu, a, gb), a1 = __shfl_sync(0xffffffffu, a, gb + 1),
                a2 = __shfl_sync(0xffffffffu, a, gb + 2);
        return D0[t] * a0 + D1[t] * a1 + D2[t] * a2;
    };
    // slot rows [a, e) of this warp's slice against the vector at vin
    auto spmv = [&](int a, int e, const T* vin, T& y0, T& y1, T& y2) {
        const int eh = min(e, held);
#pragma unroll 2
        for (int t = a; t < eh; ++t) {
            const T* xv = vin + 3 * scol[32 * t + lane];
            const T* mv = sval + 288 * t + lane;
            const T x0 = xv[0], x1 = xv[1], x2 = xv[2];
            y0 += mv[0] * x0 + mv[32] * x1 + mv[64] * x2;
            y1 += mv[96] * x0 + mv[128] * x1 + mv[160] * x2;
            y2 += mv[192] * x0 + mv[224] * x1 + mv[256] * x2;
        }
        for (int t = max(a, held); t < e; ++t) {  // past the shared-memory image: through L2
            const long at = 32L * (me.slot0 + t) + lane;
            const int k = A.src[at];
            if (k < 0) continue;
            const T* xv = vin + 3 * A.col[at];
            const T* mv = A.val + 9L * k;
            const T x0 = xv[0], x1 = xv[1], x2 = xv[2];
            y0 += mv[0] * x0 + mv[1] * x1 + mv[2] * x2;
            y1 += mv[3] * x0 + mv[4] * x1 + mv[5] * x2;
            y2 += mv[6] * x0 + mv[7] * x1 + mv[8] * x2;
        }
    };
    // the row's sum over its four lanes, component l4 on lane l4
    auto row_sum = [&](T y0, T y1, T y2) -> T {
        for (int o = 2; o > 0; o >>= 1) {
            y0 += __shfl_xor_sync(0xffffffffu, y0, o);
            y1 += __shfl_xor_sync(0xffffffffu, y1, o);
            y2 += __shfl_xor_sync(0xffffffffu, y2, o);
        }
        return l4 == 0 ? y0 : (l4 == 1 ? y1 : y2);
    };
    // own u (which = 0) or q (1) of step t to the neighbours, as exchange e
    auto publish = [&](int t, int which, T a, unsigned int e) {
        if (nc > 1 && own[t])
            put_value(A.xu + (e & 1) * A.xu_half + (2 * (3L * (v0 + lv[t]) + l4) + which) * W, 1, a, A.tag0 + e);
    };
    // the halo's u and q of exchange e (before the first iteration: u alone, which
    // is its p): kHeld<T> values per thread stay in its registers, the rest goes to
    // shared memory; all of a thread's polls are in flight together
    constexpr int H = kHeld<T>;
    int ha[H];                    // word of the value in the pairs, -1: none
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const int i = tid + j * kST;
        ha[j] = i < nh3 ? 2 * W * (3 * A.halo[me.halo0 + i / 3] + i % 3) : -1;
    }
    T hu[H], hq[H];
    auto gather = [&](unsigned int e, bool both) {
        const unsigned long long* from = A.xu + (e & 1) * A.xu_half;
        bool need[H];
#pragma unroll
        for (int j = 0; j < H; ++j) need[j] = ha[j] >= 0;
        for (unsigned int k = 0;; ++k) {
            bool wait = false;
#pragma unroll
            for (int j = 0; j < H; ++j)
                if (need[j]) need[j] = !get_pair(from + ha[j], hu[j], hq[j], A.tag0 + e, both);
#pragma unroll
            for (int j = 0; j < H; ++j) wait |= need[j];
            if (!wait) break;
            if (k > kSellSpin) { sbad = 1; break; }
        }
        for (int i = H * kST + tid; i < nh3; i += kST) {
            const unsigned long long* a = from + 2L * W * (3 * A.halo[me.halo0 + i / 3] + i % 3);
            T u, q;
            for (unsigned int k = 0; !get_pair(a, u, q, A.tag0 + e, both); ++k)
                if (k > kSellSpin) { sbad = 1; break; }
            suq[2 * (i - H * kST)] = u;
            suq[2 * (i - H * kST) + 1] = q;
        }
    };
    // the halo's next p
    auto advance_halo = [&](T alpha, T beta) {
#pragma unroll
        for (int j = 0; j < H; ++j) {
            const int i = tid + j * kST;
            if (i < nh3) sph[i] = (hu[j] - alpha * hq[j]) + beta * sph[i];
        }
        for (int i = H * kST + tid; i < nh3; i += kST)
            sph[i] = (suq[2 * (i - H * kST)] - alpha * suq[2 * (i - H * kST) + 1]) + beta * sph[i];
    };
    // ---- u = M^{-1} r, p = u
    T nu_l = T(0), rr_l = T(0);
#pragma unroll
    for (int t = 0; t < STEPS; ++t) {
        p[t] = precond(t, r[t]);
        publish(t, 0, p[t], 0);
        if (own[t]) sp[3 * lv[t] + l4] = p[t];
        nu_l += r[t] * p[t];
        rr_l += r[t] * r[t];
    }
    if (nc > 1) {
        gather(0, false);
#pragma unroll
        for (int j = 0; j < H; ++j)
            if (tid + j * kST < nh3) sph[tid + j * kST] = hu[j];
        for (int i = H * kST + tid; i < nh3; i += kST) sph[i] = suq[2 * (i - H * kST)];
    }
    // ---- iterations; warp 0 carries the scalars
    int it = 0;
    T tol2 = 0;
    for (unsigned int e = 0;; ++e) {
        __syncthreads();
        // s = A p, q = M^{-1} s
        T s[STEPS], v[kSums] = {T(0), nu_l, T(0), T(0), rr_l};  // p.s, r.u, r.q, s.q, r.r
#pragma unroll
        for (int t = 0; t < STEPS; ++t) {
            T y0 = 0, y1 = 0, y2 = 0;
            spmv(off[t], off[t] + wl[t], sp, y0, y1, y2);
            spmv(off[t] + wl[t], off[t] + wt[t], sph, y0, y1, y2);
            const T y = row_sum(y0, y1, y2);
            s[t] = own[t] && !fixed[t] ? y : T(0);
            const T q = precond(t, s[t]);
            publish(t, 1, q, e);
            v[0] += p[t] * s[t];
            v[2] += r[t] * q;
            v[3] += s[t] * q;
        }
        {
            const T a = warp_sums(v, lane);
            const int j = sum_value(lane);
            if (l4 == 0 && j < kSums) spart[warp][j] = a;
        }
        __syncthreads();
        // the CTA's sums (warp 0), the halo, then the instance's sums: warp j < kSums
        // polls value j of every CTA
        if (warp == 0) {
#pragma unroll
            for (int j = 0; j < kSums; ++j) v[j] = lane < kSW ? spart[lane][j] : T(0);
            const T a = warp_sums(v, lane);
            const int j = sum_value(lane);
            if (nc == 1) {
                if (l4 == 0 && j < kSums) sred[j] = a;
                __syncwarp();
            } else if (l4 == 0 && j < kSums) {
                put_value(A.xr + (e & 1) * A.xr_half + (long)j * W * A.xr_row + me.c0 + me.rank, A.xr_row, a, A.tag0 + e);
            }
        }
        if (nc > 1) {
            gather(e, true);
            if (warp < kSums) {
                const unsigned long long* from = A.xr + (e & 1) * A.xr_half + (long)warp * W * A.xr_row + me.c0;
                T sum = T(0);
                // polls of sums that cannot be there yet hold up the stores of those that
                // come: not before this CTA's own are out (FP64: they take 1000 cycles
                // longer; in FP32 the halo's polls are wait enough)
                if constexpr (sizeof(T) == 8) asm volatile("bar.sync 1, %0;" ::"n"(32 * kSums) : "memory");
                for (int c0 = lane; c0 < nc; c0 += 32 * kPollCtas) {
                    T val[kPollCtas];
                    for (unsigned int k = 0;; ++k) {
                        bool wait = false;
#pragma unroll
                        for (int i = 0; i < kPollCtas; ++i) {
                            const int c = c0 + 32 * i;
                            val[i] = T(0);
                            if (c < nc) wait |= !get_value(from + c, A.xr_row, val[i], A.tag0 + e);
                        }
                        if (!wait) break;
                        if (k > kSellSpin) { sbad = 1; break; }
                    }
#pragma unroll
                    for (int i = 0; i < kPollCtas; ++i) sum += val[i];
                }
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane == 0) sred[warp] = sum;
                __syncwarp();
                asm volatile("bar.sync 1, %0;" ::"n"(32 * kSums) : "memory");
            }
        }
        if (warp == 0) {
            const T mu = sred[0], nu = sred[1], de = sred[2], ga = sred[3], rr = sred[4];
            if (it == 0) {
                const double tl = A.tol_inst ? fmax(A.tol_inst[me.inst], A.rel_tol) : A.rel_tol;
                tol2 = (T)(tl * tl) * rr;
            }
            const T alpha = nu / mu;
            // the next r.u as these sums predict it
            T beta = (nu - T(2) * alpha * de + alpha * alpha * ga) / nu;
            if (!(beta >= T(0)) || !(beta < T(INFINITY))) beta = T(0);
            if (lane == 0) {
                sscal[0] = alpha;
                sscal[1] = beta;
                // converged, out of iterations, or broken down (x is kept)
                sstop = !(rr > T(0)) || !(rr > tol2) || it >= A.max_iters || !(mu > T(0)) || !(alpha > T(0)) ||
                        !(alpha < T(INFINITY));
            }
        }
        __syncthreads();
        if (sbad) {
            if (tid == 0) atomicExch(A.err, 1);
            return;
        }
        if (sstop) break;
        const T alpha = sscal[0], beta = sscal[1];
        nu_l = rr_l = T(0);
#pragma unroll
        for (int t = 0; t < STEPS; ++t) {
            x[t] += alpha * p[t];
            r[t] -= alpha * s[t];
            const T u = precond(t, r[t]);
            publish(t, 0, u, e + 1);
            p[t] = u + beta * p[t];
            if (own[t]) sp[3 * lv[t] + l4] = p[t];
            nu_l += r[t] * u;
            rr_l += r[t] * r[t];
        }
        advance_halo(alpha, beta);
        ++it;
    }
#pragma unroll
    for (int t = 0; t < STEPS; ++t)
        if (own[t]) A.x[3L * (v0 + lv[t]) + l4] = x[t];
    if (me.rank == 0 && tid == 0) A.iters_out[me.inst] = it;
}

// dynamic shared memory besides the slot rows
template <class T>
size_t sell_fixed(int nvmax, int nhmax) { 
    return sizeof(T) * (3 * (size_t)nvmax + 3 * (size_t)nhmax + 2 * (size_t)halo_rest<T>(nhmax)) + 16;
}
template <class T>
size_t sell_row() { return 32 * (9 * sizeof(T) + 2); }

template <class T, int STEPS>
cudaError_t launch_steps(Work& W, const cudaLaunchConfig_t& cfg, const SellArgs<T>& a) {
    const cudaError_t e = W.attr.set(reinterpret_cast<const void*>(&k_pcg_sell<T, STEPS>),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, kSellSmem);
    if (e != cudaSuccess) return e;
    ::idp::count_launch();
    return cudaLaunchKernelEx(&cfg, k_pcg_sell<T, STEPS>, a);
}

}  // namespace

// rows per CTA of an instance of V vertices; 0: left to the other kernels
static int sell_rows(const Work& W, long V, int sms) {
    const int f64 = W.sell_f64 ? 1 : 0;
    const bool given = W.sell_vper > 0 && V > W.grid_min_v;
    if (!given && V <= kSellSolo[f64]) return (int)V;
    const long rows = std::max<long>(given ? W.sell_vper : kSellRows[f64], (V + sms - 1) / sms);
    return rows <= kSellMaxRows ? (int)rows : 0;
}

int sell_plan(Arena& A, Work& W, cudaStream_t s) {
    Work::Sell& P = W.sell;
    P.ready = false;  // until the layout is on the device: a plan that failed is made again
    P.first.assign(A.nI, -1);
    P.cta.clear();
    int dev = 0, sms = 0;
    IDP_CUDA_TRY(cudaGetDevice(&dev));
    IDP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    P.sms = sms;
    int slices = 0;
    for (int i = 0; i < A.nI; ++i) {
        const int iv0 = A.v_off[i], V = A.v_off[i + 1] - iv0;
        const int rows = V > 0 ? sell_rows(W, V, sms) : 0;
        if (rows <= 0) continue;
        const int nc = (V + rows - 1) / rows, per = (V + nc - 1) / nc;
        P.first[i] = (int)P.cta.size();
        for (int k = 0; k < nc; ++k) {
            SellCta c = {};
            c.inst = i;
            c.v0 = iv0 + std::min(V, k * per);
            c.nv = std::min(V, (k + 1) * per) - std::min(V, k * per);
            c.c0 = P.first[i];
            c.nc = nc;
            c.rank = k;
            c.slice0 = slices;
            slices += (c.nv + kSliceRows - 1) / kSliceRows;
            P.cta.push_back(c);
        }
    }
    if (P.cta.empty()) {
        P.ready = true;
        return IDP_OK;
    }
    const long nC = (long)P.cta.size();
    const unsigned int slot_cap = (unsigned int)std::min<long>(A.B / 12 + 4 * slices + 64, 0x7fffffffL / 32);
    const unsigned int halo_cap = (unsigned int)std::min<long>(A.B + 64, 0x7fffffffL);
    DBuf &bc = W[W_SELL_CTA], &bs = W[W_SELL_SLOT], &bh = W[W_SELL_HALO];
    const size_t o_slice = (sizeof(SellCta) * nC + 255) & ~size_t(255);
    const size_t o_prow = o_slice + ((sizeof(int2) * slices + 255) & ~size_t(255));
    const size_t o_total = o_prow + ((sizeof(unsigned short) * A.V + 255) & ~size_t(255));
    if (bc.ensure(o_total + 64) || bs.ensure((sizeof(int) + sizeof(unsigned short)) * 32 * (size_t)slot_cap) ||
        bh.ensure(sizeof(int) * (size_t)halo_cap))
        return IDP_ERR_CUDA;
    P.d_cta = bc.as<SellCta>();
    P.d_slice = reinterpret_cast<int2*>(bc.as<char>() + o_slice);
    P.d_prow = reinterpret_cast<unsigned short*>(bc.as<char>() + o_prow);
    unsigned int* d_total = reinterpret_cast<unsigned int*>(bc.as<char>() + o_total);
    P.d_src = bs.as<int>();
    P.d_col = reinterpret_cast<unsigned short*>(P.d_src + 32L * slot_cap);
    P.d_halo = bh.as<int>();
    IDP_CUDA_TRY(cudaMemcpyAsync(P.d_cta, P.cta.data(), sizeof(SellCta) * nC, cudaMemcpyHostToDevice, s));
    IDP_CUDA_TRY(cudaMemsetAsync(d_total, 0, 64, s));
    (::idp::count_launch(), k_sell_plan<<<(int)nC, 256, 0, s>>>(P.d_cta, A.rowptr, A.colidx, P.d_slice, P.d_src, P.d_col,
                                                               P.d_prow, P.d_halo, slot_cap, halo_cap, d_total));
    IDP_CUDA_TRY(cudaGetLastError());
    IDP_CUDA_TRY(cudaMemcpyAsync(P.cta.data(), P.d_cta, sizeof(SellCta) * nC, cudaMemcpyDeviceToHost, s));
    IDP_CUDA_TRY(cudaStreamSynchronize(s));
    for (const SellCta& c : P.cta)  // an instance with a CTA that did not fit keeps to the other kernels
        if (c.nsr < 0) P.first[c.inst] = -1;
    P.ready = true;
    return IDP_OK;
}

// the instances of `which` (each with a plan) on the right-hand side b; x, iters
// and the error flag are written on the device. Waves of at most one CTA per
// SM: the CTAs of one instance wait for one another and must be resident.
template <class T>
int sell_solve(Arena& A, Work& W, const std::vector<int>& which, const double* b, T* x, double rel_tol, int max_iters,
               int* d_iters, int* d_err, cudaStream_t s) {
    Work::Sell& P = W.sell;
    const long nC = (long)P.cta.size();
    DBuf& bx = W[W_SELL_XCH];
    const size_t xu_half = 6 * (size_t)A.V * words<T>(), xr_half = (size_t)kSums * nC * words<T>();
    const size_t need = 8 * 2 * (xu_half + xr_half) + 64;
    if (need > P.xch_bytes || P.tag > 0xe0000000u) {
        if (bx.ensure(need)) return IDP_ERR_CUDA;
        P.xch_bytes = bx.bytes;
        P.tag = 1;  // tags of earlier exchanges are cleared with the words
        IDP_CUDA_TRY(cudaMemsetAsync(bx.p, 0, bx.bytes, s));
    }
    if (W[W_SELL_LIST].ensure(sizeof(int) * (size_t)nC)) return IDP_ERR_CUDA;
    std::vector<int> list;
    std::vector<std::pair<int, int>> waves;  // ranges of the list
    int begin = 0;
    for (int i : which) {
        const int f = P.first[i], nc = P.cta[f].nc;
        // single CTAs wait for nobody: they only open a wave of their own kind
        if ((int)list.size() - begin + nc > P.sms) {
            waves.push_back({begin, (int)list.size()});
            begin = (int)list.size();
        }
        for (int k = 0; k < nc; ++k) list.push_back(f + k);
    }
    waves.push_back({begin, (int)list.size()});
    int* d_list = W[W_SELL_LIST].as<int>();
    IDP_CUDA_TRY(cudaMemcpyAsync(d_list, list.data(), sizeof(int) * list.size(), cudaMemcpyHostToDevice, s));
    for (auto& wv : waves) {
        int nvmax = 1, nhmax = 0, nsr = 0;
        for (int k = wv.first; k < wv.second; ++k) {
            const SellCta& c = P.cta[list[k]];
            nvmax = std::max(nvmax, c.nv);
            nhmax = std::max(nhmax, c.nh);
            nsr = std::max(nsr, c.nsr);
        }
        SellArgs<T> a;
        a.cta = P.d_cta;
        a.list = d_list + wv.first;
        a.slice = P.d_slice;
        a.src = P.d_src;
        a.col = P.d_col;
        a.prow = P.d_prow;
        a.halo = P.d_halo;
        a.val = W[W_BSR_VAL].as<T>();
        a.dinv = W[W_DIAG_INV].as<T>();
        a.dbc = A.dbc;
        a.b = b;
        a.x = x;
        a.xu = bx.as<unsigned long long>();
        a.xr = a.xu + 2 * xu_half;
        a.xu_half = (long)xu_half;
        a.xr_half = (long)xr_half;
        a.xr_row = nC;
        a.tag0 = P.tag;
        a.nvmax = nvmax;
        a.nhmax = nhmax;
        a.cap = (int)std::min<size_t>((size_t)nsr, (kSellSmem - sell_fixed<T>(nvmax, nhmax)) / sell_row<T>());
        a.tol_inst = W.tol_inst;
        a.rel_tol = rel_tol;
        a.max_iters = max_iters;
        a.iters_out = d_iters;
        a.err = d_err;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(wv.second - wv.first);
        cfg.blockDim = dim3(kST);
        cfg.dynamicSmemBytes = sell_fixed<T>(nvmax, nhmax) + sell_row<T>() * a.cap;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        const int steps = (nvmax + kSW * kSliceRows - 1) / (kSW * kSliceRows);
        IDP_CUDA_TRY(steps <= 1 ? (launch_steps<T, 1>(W, cfg, a))
                                : (steps == 2 ? (launch_steps<T, 2>(W, cfg, a)) : (launch_steps<T, 3>(W, cfg, a))));
        W.stats.pcg_launches += 1;
    }
    return IDP_OK;
}

template int sell_solve<float>(Arena&, Work&, const std::vector<int>&, const double*, float*, double, int, int*, int*,
                               cudaStream_t);
template int sell_solve<double>(Arena&, Work&, const std::vector<int>&, const double*, double*, double, int, int*, int*,
                                cudaStream_t);

}  // namespace idp
