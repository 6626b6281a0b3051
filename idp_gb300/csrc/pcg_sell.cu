// PCG for instances without contact blocks: persistent CTAs that hold their
// rows' matrix in shared memory and every vector in registers, exchanging
// nothing but the vector the SpMV gathers and three partial sums per iteration.
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
// slice, so that their part of A m runs while the neighbours' m is under way;
// the other columns are numbered in the CTA's halo list. Both lists depend on
// the pattern only and are laid out once per commit (k_sell_plan).
//
// Exchange. A value is stored as a 64-bit word of 32 payload bits and a 32-bit
// tag that no earlier exchange used (FP64: two words), and its readers poll the
// data itself: neither a fence nor a flag is waited for, and a halo value is
// usable one L2 round trip after it was written. The CTAs' partial sums travel
// the same way and every CTA adds them in the same order. Two slots by parity
// suffice: a CTA overwrites exchange e with e + 2 only after it has read every
// CTA's sums of e + 1, which each wrote after reading e.
//
// Pipelined PCG (Ghysels & Vanroose) as in k_pcg_grid, one reduction per
// iteration. On the 220,515-tet blob (49,863 vertices, FP32) k_pcg_grid took
// 12 us per iteration: vectors in global memory, the gathers from L2 and a
// counter, a release word and a reduction by the last CTA to arrive; here 5.7,
// most of it reading the matrix (328 rows per SM: 20 shared-memory wavefronts
// per slot row, 10 of them bank conflicts of the gathers). A bar of 160
// vertices: 10.5 us on one cluster CTA (k_pcg_cluster) -> 2.4 on one CTA here; a
// blob of 5,838 vertices in FP64: 66 us on 16 cluster CTAs -> 13.
#include <algorithm>
#include <atomic>
#include "engine.hpp"

namespace idp {

namespace {

constexpr int kST = 512;                 // threads per CTA
constexpr int kSW = kST / 32;
constexpr int kSliceRows = 8;
// Rows per CTA at least, where there are several, and the largest instance of one
// CTA, {FP32, FP64}. Microseconds per iteration on bars and blobs of 160 to
// 18,210 vertices: FP32 2.8-3.0 with 40 to 128 rows, 3.7 with 160 (a second slice
// per warp); 2.4 on one CTA of 160 rows, 3.4 of 320. FP64 is bound by its pipe:
// 13.3-14 with 40 rows, 17 with 128, 18 on one CTA of 160.
constexpr int kSellRows[2] = {64, 40}, kSellSolo[2] = {192, 40};
constexpr int kSellMaxRows = 3 * kSW * kSliceRows;  // rows per CTA: three slices per warp
constexpr int kHaloTable = 4096;         // hash slots of the halo search
constexpr int kHaloMax = 2600;           // halo vertices per CTA
constexpr int kSellSmem = 222 * 1024;    // dynamic shared memory limit
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
__device__ __forceinline__ void put_value(unsigned long long* p, float v, unsigned int tag) {
    put_word(p, __float_as_uint(v), tag);
}
__device__ __forceinline__ void put_value(unsigned long long* p, double v, unsigned int tag) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    put_word(p, (unsigned int)b, tag);
    put_word(p + 1, (unsigned int)(b >> 32), tag);
}
__device__ __forceinline__ bool get_value(const unsigned long long* p, float& v, unsigned int tag) {
    const unsigned long long w = get_word(p);
    v = __uint_as_float((unsigned int)w);
    return (unsigned int)(w >> 32) == tag;
}
__device__ __forceinline__ bool get_value(const unsigned long long* p, double& v, unsigned int tag) {
    const unsigned long long a = get_word(p), b = get_word(p + 1);
    v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return (unsigned int)(a >> 32) == tag && (unsigned int)(b >> 32) == tag;
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
    unsigned long long* xm;       // [2][3 V] values
    unsigned long long* xr;       // [2][3 plan CTAs] values
    long xm_half, xr_half;        // words per parity
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
    T* sm = sval + 288L * A.cap;                                  // m of the own rows, two parities
    T* smh = sm + 6L * A.nvmax;                                   // m of the halo
    unsigned short* scol = reinterpret_cast<unsigned short*>(smh + 3L * A.nhmax);  // [cap][32]
    __shared__ T spart[kSW][3];   // partial sums by warp
    __shared__ T sred[kSW][3];    // the CTAs' sums by polling warp
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
    // ---- this lane's rows (component l4 < 3 of row position p) and their state
    int lv[STEPS], off[STEPS], wl[STEPS], wt[STEPS];
    bool own[STEPS], fixed[STEPS];
    T D0[STEPS], D1[STEPS], D2[STEPS];
    T z[STEPS], q[STEPS], s[STEPS], p[STEPS], u[STEPS], w[STEPS], x[STEPS], r[STEPS], m[STEPS];
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
        D0[t] = D1[t] = D2[t] = z[t] = q[t] = s[t] = p[t] = u[t] = w[t] = x[t] = r[t] = m[t] = T(0);
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
    // own value a of step t: to shared memory and, as exchange e, to the neighbours
    auto publish = [&](int t, T a, unsigned int e) {
        if (!own[t]) return;
        sm[(e & 1) * 3 * A.nvmax + 3 * lv[t] + l4] = a;
        if (nc > 1) put_value(A.xm + (e & 1) * A.xm_half + (3L * (v0 + lv[t]) + l4) * W, a, A.tag0 + e);
    };
    // halo values of exchange e into shared memory, four polls in flight per thread
    auto gather = [&](unsigned int e) {
        const unsigned long long* from = A.xm + (e & 1) * A.xm_half;
        for (int i0 = tid; i0 < nh3; i0 += 4 * kST) {
            const unsigned long long* a[4];
            bool need[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + j * kST;
                need[j] = i < nh3;
                a[j] = need[j] ? from + (3L * A.halo[me.halo0 + i / 3] + i % 3) * W : from;
            }
            for (unsigned int n = 0;; ++n) {
                bool wait = false;
                T v[4];
                bool got[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) got[j] = need[j] && get_value(a[j], v[j], A.tag0 + e);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (got[j]) {
                        smh[i0 + j * kST] = v[j];
                        need[j] = false;
                    }
                    wait |= need[j];
                }
                if (!wait) break;
                if (n > kSellSpin) { sbad = 1; break; }
            }
        }
    };
    T gam_l, del_l, rho_l;
    // partial sums of this CTA: by warp, then (warp 0) in warp order; the others'
    // copies travel as exchange e
    auto reduce_out = [&](unsigned int e) {
        for (int o = 16; o > 0; o >>= 1) {
            gam_l += __shfl_xor_sync(0xffffffffu, gam_l, o);
            del_l += __shfl_xor_sync(0xffffffffu, del_l, o);
            rho_l += __shfl_xor_sync(0xffffffffu, rho_l, o);
        }
        if (lane == 0) { spart[warp][0] = gam_l; spart[warp][1] = del_l; spart[warp][2] = rho_l; }
        __syncthreads();
        if (warp == 0) {
            T a = lane < kSW ? spart[lane][0] : T(0), b = lane < kSW ? spart[lane][1] : T(0),
              c = lane < kSW ? spart[lane][2] : T(0);
            for (int o = 8; o > 0; o >>= 1) {
                a += __shfl_xor_sync(0xffffffffu, a, o);
                b += __shfl_xor_sync(0xffffffffu, b, o);
                c += __shfl_xor_sync(0xffffffffu, c, o);
            }
            if (nc == 1) {
                if (lane == 0) { sred[0][0] = a; sred[0][1] = b; sred[0][2] = c; }
            } else if (lane < 3) {
                put_value(A.xr + (e & 1) * A.xr_half + (3L * (me.c0 + me.rank) + lane) * W,
                          lane == 0 ? a : (lane == 1 ? b : c), A.tag0 + e);
            }
        }
    };
    // every CTA's sums of exchange e: a thread per CTA, added by warp
    auto reduce_in = [&](unsigned int e) {
        if (32 * warp >= nc) return;
        T v[3] = {T(0), T(0), T(0)};
        if (tid < nc) {
            const unsigned long long* a = A.xr + (e & 1) * A.xr_half + 3L * (me.c0 + tid) * W;
            for (unsigned int n = 0;; ++n) {
                const bool g0 = get_value(a, v[0], A.tag0 + e), g1 = get_value(a + W, v[1], A.tag0 + e),
                           g2 = get_value(a + 2 * W, v[2], A.tag0 + e);
                if (g0 && g1 && g2) break;
                if (n > kSellSpin) { sbad = 1; break; }
            }
        }
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < 3; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < 3; ++j) sred[warp][j] = v[j];
    };
    // ---- u = M^{-1} r, w = A u, m = M^{-1} w
#pragma unroll
    for (int t = 0; t < STEPS; ++t) {
        u[t] = precond(t, r[t]);
        publish(t, u[t], 0);
    }
    __syncthreads();
    if (nc > 1) gather(0);
    __syncthreads();
    if (sbad) {
        if (tid == 0) atomicExch(A.err, 1);
        return;
    }
    gam_l = del_l = rho_l = T(0);
#pragma unroll
    for (int t = 0; t < STEPS; ++t) {
        T y0 = 0, y1 = 0, y2 = 0;
        spmv(off[t], off[t] + wl[t], sm, y0, y1, y2);
        spmv(off[t] + wl[t], off[t] + wt[t], smh, y0, y1, y2);
        const T y = row_sum(y0, y1, y2);
        w[t] = own[t] && !fixed[t] ? y : T(0);
        m[t] = precond(t, w[t]);
        publish(t, m[t], 1);
        gam_l += r[t] * u[t];
        del_l += w[t] * u[t];
        rho_l += r[t] * r[t];
    }
    reduce_out(1);
    // ---- iterations; warp 0 carries the scalar recurrences
    int it = 0;
    T gam_prev = 1, inv_alpha = 0, tol2 = 0;  // gam and 1 / alpha of the previous iteration
    for (unsigned int e = 1;; ++e) {
        const T* mo = sm + (e & 1) * 3 * A.nvmax;
        T y0[STEPS], y1[STEPS], y2[STEPS];
#pragma unroll
        for (int t = 0; t < STEPS; ++t) {
            y0[t] = y1[t] = y2[t] = T(0);
            spmv(off[t], off[t] + wl[t], mo, y0[t], y1[t], y2[t]);
        }
        if (nc > 1) {
            gather(e);
            reduce_in(e);
        }
        __syncthreads();
        if (warp == 0) {
            T gam = 0, del = 0, rho = 0;
            for (int k = 0; 32 * k < nc; ++k) { gam += sred[k][0]; del += sred[k][1]; rho += sred[k][2]; }
            int stop = 0;
            if (it == 0) {
                const double tl = A.tol_inst ? fmax(A.tol_inst[me.inst], A.rel_tol) : A.rel_tol;
                tol2 = (T)(tl * tl) * rho;
                if (!(rho > T(0)) || !(rho > tol2)) stop = 1;
            } else if (rho <= tol2) {
                stop = 1;
            }
            if (it >= A.max_iters) stop = 1;
            const T beta = it == 0 ? T(0) : gam / gam_prev, alpha = gam / (del - beta * gam * inv_alpha);
            if (!(alpha > T(0)) || !(alpha < T(INFINITY)) || !(beta < T(INFINITY))) stop = 1;  // breakdown: keep x
            if (lane == 0) {
                sscal[0] = alpha;
                sscal[1] = beta;
                sstop = stop;
            }
            gam_prev = gam;
            inv_alpha = T(1) / alpha;
        }
#pragma unroll
        for (int t = 0; t < STEPS; ++t) spmv(off[t] + wl[t], off[t] + wt[t], smh, y0[t], y1[t], y2[t]);
        __syncthreads();
        if (sbad) {
            if (tid == 0) atomicExch(A.err, 1);
            return;
        }
        if (sstop) break;
        const T alpha = sscal[0], beta = sscal[1];
        gam_l = del_l = rho_l = T(0);
#pragma unroll
        for (int t = 0; t < STEPS; ++t) {
            const T y = row_sum(y0[t], y1[t], y2[t]);
            const T n = own[t] && !fixed[t] ? y : T(0);
            z[t] = n + beta * z[t];
            q[t] = m[t] + beta * q[t];
            s[t] = w[t] + beta * s[t];
            p[t] = u[t] + beta * p[t];
            x[t] += alpha * p[t];
            r[t] -= alpha * s[t];
            u[t] -= alpha * q[t];
            w[t] -= alpha * z[t];
            m[t] = precond(t, w[t]);
            publish(t, m[t], e + 1);
            gam_l += r[t] * u[t];
            del_l += w[t] * u[t];
            rho_l += r[t] * r[t];
        }
        ++it;
        reduce_out(e + 1);
    }
#pragma unroll
    for (int t = 0; t < STEPS; ++t)
        if (own[t]) A.x[3L * (v0 + lv[t]) + l4] = x[t];
    if (me.rank == 0 && tid == 0) A.iters_out[me.inst] = it;
}

// dynamic shared memory besides the slot rows
template <class T>
size_t sell_fixed(int nvmax, int nhmax) { return sizeof(T) * (6 * (size_t)nvmax + 3 * (size_t)nhmax) + 16; }
template <class T>
size_t sell_row() { return 32 * (9 * sizeof(T) + 2); }

template <class T, int STEPS>
cudaError_t launch_steps(const cudaLaunchConfig_t& cfg, const SellArgs<T>& a) {
    static std::atomic<bool> attr{false};  // one per instantiation
    if (!attr.load()) {
        const cudaError_t e = cudaFuncSetAttribute(k_pcg_sell<T, STEPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   kSellSmem);
        if (e != cudaSuccess) return e;
        attr.store(true);
    }
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
    P.ready = true;
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
    if (P.cta.empty()) return IDP_OK;
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
    const size_t xm_half = 3 * (size_t)A.V * words<T>(), xr_half = 3 * (size_t)nC * words<T>();
    const size_t need = 8 * 2 * (xm_half + xr_half) + 64;
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
        a.xm = bx.as<unsigned long long>();
        a.xr = a.xm + 2 * xm_half;
        a.xm_half = (long)xm_half;
        a.xr_half = (long)xr_half;
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
        IDP_CUDA_TRY(steps <= 1 ? (launch_steps<T, 1>(cfg, a))
                                : (steps == 2 ? (launch_steps<T, 2>(cfg, a)) : (launch_steps<T, 3>(cfg, a))));
        W.stats.pcg_launches += 1;
    }
    return IDP_OK;
}

template int sell_solve<float>(Arena&, Work&, const std::vector<int>&, const double*, float*, double, int, int*, int*,
                               cudaStream_t);
template int sell_solve<double>(Arena&, Work&, const std::vector<int>&, const double*, double*, double, int, int*, int*,
                                cudaStream_t);

}  // namespace idp
