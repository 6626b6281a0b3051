// Contact-cluster blocks of the PCG preconditioner.
//
// Barrier Hessians couple the 2-4 vertices of a constraint with stiffness
// many orders above the elastic and inertial terms, and 3x3 block-Jacobi
// cannot see those couplings. Vertices linked through constraints are grouped
// (union-find over the constraint stencils, groups larger than kClusterCap
// split in breadth-first order so coupled vertices stay together); every
// group's dense block of the system matrix is gathered and factored
// (Cholesky, then the inverse factor) on the device, one CTA per group, and
// the PCG applies the block inverse to the group's rows. All other vertices keep their 3x3
// block-Jacobi inverse. A block whose factorisation fails falls back to the
// 3x3 inverses of its vertices.
#include <algorithm>
#include <deque>
#include <numeric>
#include <vector>
#include <cooperative_groups.h>
#include "engine.hpp"

namespace cg = cooperative_groups;

namespace idp {

namespace {

// Row stride of a block's dense matrices: N = 3n rounded up to 4 values, so that
// rows start on a 16-byte boundary.
__host__ __device__ inline int block_ld(int N) { return (N + 3) & ~3; }

// dense block of the system matrix for every cluster (K zeroed before):
// a warp per row, lanes over the row's blocks (their columns differ), then over
// the contact tail's; blockIdx.y slices of the rows
template <class T>
__global__ void k_cl_gather(int ncl, const int* __restrict__ off, const int* __restrict__ vert,
                            const int* __restrict__ vcl, const int* __restrict__ vloc,
                            const long long* __restrict__ doff, const int* __restrict__ rowptr,
                            const int* __restrict__ colidx, const T* __restrict__ val, const int* __restrict__ trp,
                            const int* __restrict__ tcol, const T* __restrict__ tval,
                            const unsigned char* __restrict__ dbc, T* __restrict__ K) {
    const int c = blockIdx.x;
    const int n = off[c + 1] - off[c];
    const int ld = block_ld(3 * n);
    T* Kc = K + doff[c];
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int li = blockIdx.y * warps + (threadIdx.x >> 5); li < n; li += gridDim.y * warps) {
        const int v = vert[off[c] + li];
        T* row = Kc + 3L * li * ld;
        if (dbc[v]) {
            if (lane < 3) row[(long)lane * ld + 3 * li + lane] = T(1);
            continue;
        }
        for (int k = rowptr[v] + lane; k < rowptr[v + 1]; k += 32) {
            const int col = colidx[k];
            if (vcl[col] != c) continue;
            const int lj = 3 * vloc[col];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) row[(long)a * ld + lj + b] = val[9 * (long)k + 3 * a + b];
        }
        __syncwarp();
        for (int k = trp[v] + lane; k < trp[v + 1]; k += 32) {
            const int col = tcol[k];
            if (dbc[col] || vcl[col] != c) continue;
            const int lj = 3 * vloc[col];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) row[(long)a * ld + lj + b] += tval[9 * (long)k + 3 * a + b];
        }
    }
}

// Factor every block, one thread-block cluster per block (8 CTAs above 96
// rows, one CTA below), in 32-wide panels:
//  Cholesky K = L L^T, right-looking. Every CTA factors the 32x32 diagonal
//  tile and inverts the factor (one warp, rows in registers) and solves the
//  whole panel below it (a thread per row) while it sits in shared memory, so
//  the panel needs no exchange; the trailing lower triangle takes the rank-32
//  update in 64x64 tiles, 4x4 values per thread, shared out over the cluster;
//  one cluster barrier per panel. L's panels go to the upper triangle
//  (transposed), the inverted diagonal tiles to Y.
//  Y = L^{-1} by 32-wide columns, which do not depend on one another and are
//  shared out over the cluster: a column stays in shared memory and its row
//  tiles follow in order, Y_i = L_ii^{-1} (- sum_k L_ik Y_k), the sum's k split
//  over four groups of 64 threads of 4x4 values each.
// The PCG applies K^{-1} = Y^T Y as z = Y^T (Y r). ok[c] = 0 when a pivot is
// not positive (the block then falls back to 3x3 inverses).
// Bound by the chain of 18 panels (tile factor, panel, update, barrier) and the
// FP32 or FP64 pipe. (One CTA per block with one output per lane and a column
// of Y per thread took 3.4 ms a call on 20 pairs of bars of 200 to 6,000 tets,
// a third of their step; with this and the shared-out applies of solver.cu the
// step went from 175 to 93 ms.) Blocks of up to 96 rows, 3 panels, have too
// little work between the barriers to share.
constexpr int kInvThreads = 256;
constexpr int kTB = 32;
constexpr int kNMax = 3 * kClusterCap;
constexpr int kInvClusterRows = 96;              // blocks of more rows take a cluster
constexpr int kInvCluster = 8;
constexpr int kPanLd = kNMax + 4;                // panel: [k][row]
constexpr int kTileLd = kTB + 4;
constexpr int kInvBuf = kTB * kPanLd;            // panel, or a column of Y ([row][32])
constexpr int kInvStage = 128 * kTB;             // L rows of one pass, or the groups' partial sums

template <class T>
struct alignas(16) Vec4 {
    T x, y, z, w;
};
__device__ __forceinline__ Vec4<float> ldcg4(const float* p) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Vec4<double> ldcg4(const double* p) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p)), b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    return {a.x, a.y, b.x, b.y};
}
template <class T>
__device__ __forceinline__ Vec4<T> lds4(const T* p) {
    return *reinterpret_cast<const Vec4<T>*>(p);
}
template <class T>
__device__ __forceinline__ void st4(T* p, const Vec4<T>& v) {
    *reinterpret_cast<Vec4<T>*>(p) = v;
}
// acc (4x4) += a b^T
template <class T>
__device__ __forceinline__ void outer4(T (&acc)[4][4], const Vec4<T>& a, const Vec4<T>& b) {
    const T av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
}

template <class T>
size_t invert_smem_bytes() {
    return sizeof(T) * (kInvBuf + kInvStage + 3 * kTB * kTileLd);
}

// one warp: the kw x kw tile at A (row stride ld, lower triangle) into its
// Cholesky factor (tile) and that factor's inverse (inv), both 32 x 32 padded
// with the identity; false when a pivot is not positive
template <class T>
__device__ bool tile_factor(const T* A, int ld, int kw, T* tile, T* inv, int lane) {
    T a[kTB];
#pragma unroll
    for (int q = 0; q < kTB; q += 4) {
        Vec4<T> v = {T(0), T(0), T(0), T(0)};
        if (lane < kw && q < kw) v = ldcg4(A + (long)lane * ld + q);
        a[q] = v.x; a[q + 1] = v.y; a[q + 2] = v.z; a[q + 3] = v.w;
    }
#pragma unroll
    for (int q = 0; q < kTB; ++q)
        if (lane >= kw || q >= kw) a[q] = lane == q ? T(1) : T(0);
    bool good = true;
#pragma unroll
    for (int j = 0; j < kTB; ++j) {
        const T d = __shfl_sync(0xffffffffu, a[j], j);
        good = good && d > T(0);
        const T ljj = sqrt(d), r = T(1) / ljj;
        a[j] = lane == j ? ljj : (lane > j ? a[j] * r : T(0));
#pragma unroll
        for (int q = j + 1; q < kTB; ++q) a[q] -= a[j] * __shfl_sync(0xffffffffu, a[j], q);
    }
#pragma unroll
    for (int q = 0; q < kTB; ++q) tile[lane * kTileLd + q] = a[q];
    __syncwarp();
    // column `lane` of the inverse by forward substitution
    T x[kTB];
#pragma unroll
    for (int r = 0; r < kTB; ++r) {
        T s = r == lane ? T(1) : T(0);
#pragma unroll
        for (int t = 0; t < r; ++t) s -= tile[r * kTileLd + t] * x[t];
        x[r] = s / tile[r * kTileLd + r];
        inv[r * kTileLd + lane] = x[r];
    }
    __syncwarp();
    return good;
}

template <class T>
__global__ void __launch_bounds__(kInvThreads) k_cl_invert(const int* __restrict__ list, const int* __restrict__ off,
                                                           const long long* __restrict__ doff, T* __restrict__ K,
                                                           T* __restrict__ Ybuf, int* __restrict__ ok) {
    extern __shared__ __align__(16) unsigned char inv_smem[];
    T* buf = reinterpret_cast<T*>(inv_smem);
    T* stage = buf + kInvBuf;
    T* tile = stage + kInvStage;
    T* inv = tile + kTB * kTileLd;
    T* R = inv + kTB * kTileLd;
    __shared__ int fail;
    cg::cluster_group cl = cg::this_cluster();
    const int csize = (int)cl.num_blocks(), crank = (int)cl.block_rank();
    const int c = list[blockIdx.x / csize];
    const int N = 3 * (off[c + 1] - off[c]), ld = block_ld(N);
    T* L = K + doff[c];
    T* Y = Ybuf + doff[c];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // ---- Cholesky
    for (int k0 = 0; k0 < N; k0 += kTB) {
        const int kw = min(kTB, N - k0), m0 = k0 + kw, m = N - m0, mt = (m + 63) / 64;
        if (warp == 0) {
            const bool good = tile_factor(L + (long)k0 * ld + k0, ld, kw, tile, inv, lane);
            if (lane == 0) fail = good ? 0 : 1;
        } else {
            // the panel below, [column][row], rows padded with zeros to the 64-row tiles
            for (int ri = tid - 32; ri < mt * 64; ri += kInvThreads - 32)
#pragma unroll
                for (int q = 0; q < kTB; q += 4) {
                    Vec4<T> v = {T(0), T(0), T(0), T(0)};
                    if (ri < m && q < kw) v = ldcg4(L + (long)(m0 + ri) * ld + k0 + q);
                    buf[q * kPanLd + ri] = v.x;
                    buf[(q + 1) * kPanLd + ri] = v.y;
                    buf[(q + 2) * kPanLd + ri] = v.z;
                    buf[(q + 3) * kPanLd + ri] = v.w;
                }
        }
        __syncthreads();
        if (fail) {  // the same in every CTA of the cluster: they factor the same tile
            if (crank == 0 && tid == 0) ok[c] = 0;
            return;
        }
        if (crank == 0)
            for (int e = tid; e < kw * kw; e += kInvThreads) {
                const int r = e / kw, q = e % kw;
                Y[(long)(k0 + r) * ld + k0 + q] = inv[r * kTileLd + q];
            }
        // panel rows x = a L_kk^{-T}, in place; this CTA's rows to L^T
        for (int ri = tid; ri < m; ri += kInvThreads) {
            T a[kTB];
#pragma unroll
            for (int q = 0; q < kTB; ++q) a[q] = buf[q * kPanLd + ri];
            const bool mine = (ri >> 5) % csize == crank;
#pragma unroll
            for (int q = 0; q < kTB; ++q) {
                T x = 0;
#pragma unroll
                for (int t = 0; t <= q; t += 4) {  // the inverse is zero right of its diagonal
                    const Vec4<T> w = lds4(inv + q * kTileLd + t);
                    x += a[t] * w.x + a[t + 1] * w.y + a[t + 2] * w.z + a[t + 3] * w.w;
                }
                buf[q * kPanLd + ri] = x;
                if (mine && q < kw) L[(long)(k0 + q) * ld + m0 + ri] = x;
            }
        }
        __syncthreads();
        // trailing lower triangle, 64x64 tiles: A[i][j] -= panel_i . panel_j
        const int tx = tid & 15, ty = tid >> 4;
        for (int e = crank; e < mt * (mt + 1) / 2; e += csize) {
            int ti = 0;
            while ((ti + 1) * (ti + 2) / 2 <= e) ++ti;
            const int tj = e - ti * (ti + 1) / 2;
            const int ri = 64 * ti + 4 * ty, rj = 64 * tj + 4 * tx;
            T acc[4][4] = {};
#pragma unroll 8
            for (int q = 0; q < kTB; ++q) outer4(acc, lds4(buf + q * kPanLd + ri), lds4(buf + q * kPanLd + rj));
            if (rj < m)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (ri + i >= m) continue;
                    T* p = L + (long)(m0 + ri + i) * ld + m0 + rj;
                    Vec4<T> v = ldcg4(p);
                    v.x -= acc[i][0]; v.y -= acc[i][1]; v.z -= acc[i][2]; v.w -= acc[i][3];
                    st4(p, v);
                }
        }
        cl.sync();
    }
    // ---- Y = L^{-1}, a 32-wide column of tiles at a time; the columns with the
    // most rows go round first, then back (the cluster's shares even out)
    const int nb = (N + kTB - 1) / kTB;
    const int gq = tid >> 6, rx = tid & 7, ry = (tid >> 3) & 7;
    for (int turn = 0; turn * csize < nb; ++turn) {
        const int jb = turn * csize + ((turn & 1) ? csize - 1 - crank : crank);
        if (jb >= nb) continue;
        const int j0 = jb * kTB, jw = min(kTB, N - j0);
        __syncthreads();
        for (int e = tid; e < kTB * kTB; e += kInvThreads) {
            const int r = e / kTB, q = e % kTB;
            buf[e] = r < jw && q < jw ? __ldcg(Y + (long)(j0 + r) * ld + j0 + q) : T(0);
        }
        for (int i0 = j0 + kTB; i0 < N; i0 += kTB) {
            const int iw = min(kTB, N - i0);
            T acc[4][4] = {};
            for (int k0 = j0; k0 < i0; k0 += 128) {
                const int kn = min(128, i0 - k0);
                __syncthreads();
                for (int e = tid; e < kn * (kTB / 4); e += kInvThreads) {
                    const int k = e / (kTB / 4), q = 4 * (e % (kTB / 4));
                    Vec4<T> v = {T(0), T(0), T(0), T(0)};
                    if (q < iw) v = ldcg4(L + (long)(k0 + k) * ld + i0 + q);
                    if (q + 1 >= iw) v.y = T(0);
                    if (q + 2 >= iw) v.z = T(0);
                    if (q + 3 >= iw) v.w = T(0);
                    st4(stage + k * kTB + q, v);
                }
                if (k0 == j0)
                    for (int e = tid; e < kTB * kTB; e += kInvThreads) {
                        const int r = e / kTB, q = e % kTB;
                        inv[r * kTileLd + q] = r < iw && q < iw ? __ldcg(Y + (long)(i0 + r) * ld + i0 + q) : T(0);
                    }
                __syncthreads();
#pragma unroll 4
                for (int k = gq; k < kn; k += 4)
                    outer4(acc, lds4(stage + k * kTB + 4 * ry), lds4(buf + (k0 - j0 + k) * kTB + 4 * rx));
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i)
                st4(stage + gq * kTB * kTB + (4 * ry + i) * kTB + 4 * rx, Vec4<T>{acc[i][0], acc[i][1], acc[i][2], acc[i][3]});
            __syncthreads();
            for (int e = tid; e < kTB * kTB; e += kInvThreads)
                R[(e / kTB) * kTileLd + e % kTB] =
                    -((stage[e] + stage[kTB * kTB + e]) + (stage[2 * kTB * kTB + e] + stage[3 * kTB * kTB + e]));
            __syncthreads();
            const int r = tid >> 3, q = 4 * (tid & 7);
            Vec4<T> y = {T(0), T(0), T(0), T(0)};
            for (int t = 0; t <= r; ++t) {
                const T w = inv[r * kTileLd + t];
                const Vec4<T> v = lds4(R + t * kTileLd + q);
                y.x += w * v.x; y.y += w * v.y; y.z += w * v.z; y.w += w * v.w;
            }
            st4(buf + (i0 - j0 + r) * kTB + q, y);
            if (r < iw) st4(Y + (long)(i0 + r) * ld + j0 + q, y);  // jw = 32 here
        }
    }
    if (crank == 0 && tid == 0) ok[c] = 1;
}

struct DSU {
    std::vector<int> p;
    explicit DSU(int n) : p(n) { std::iota(p.begin(), p.end(), 0); }
    int find(int a) {
        while (p[a] != a) a = p[a] = p[p[a]];
        return a;
    }
    void unite(int a, int b) {
        a = find(a);
        b = find(b);
        if (a != b) p[a < b ? b : a] = a < b ? a : b;
    }
};

template <class T>
int factor_blocks(Arena& A, Work& W, const int* list, int nbig, int nfew, cudaStream_t s) {
    Work::Clusters& cl = W.cl;
    T* K = W[W_CL_DENSE].as<T>();
    T* Y = K + cl.dense;
    IDP_CUDA_TRY(cudaMemsetAsync(K, 0, sizeof(T) * (size_t)cl.dense, s));
    (::idp::count_launch(), k_cl_gather<T><<<dim3(cl.n, 4), 256, 0, s>>>(
                                cl.n, cl.off, cl.vert, cl.vcl, cl.vloc, cl.doff, A.rowptr, A.colidx,
                                W[W_BSR_VAL].as<T>(), W[W_TAIL_ROWPTR].as<int>(), W[W_TAIL_COL].as<int>(),
                                W[W_TAIL_VAL].as<T>(), A.dbc, K));
    IDP_CUDA_TRY(W.attr.set(reinterpret_cast<const void*>(&k_cl_invert<T>),
                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)invert_smem_bytes<T>()));
    for (int part = 0; part < 2; ++part) {
        const int n = part ? nfew : nbig, cs = part ? 1 : kInvCluster;
        if (!n) continue;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(n * cs);
        cfg.blockDim = dim3(kInvThreads);
        cfg.dynamicSmemBytes = invert_smem_bytes<T>();
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        ::idp::count_launch();
        IDP_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_cl_invert<T>, list + (part ? nbig : 0), (const int*)cl.off,
                                        (const long long*)cl.doff, K, Y, (int*)cl.ok));
    }
    return cudaGetLastError() == cudaSuccess ? IDP_OK : IDP_ERR_CUDA;
}

}  // namespace

int build_contact_clusters(Arena& A, Work& W, const ContactSet& cs, bool fp64, cudaStream_t s) {
    Work::Clusters& cl = W.cl;
    cl.n = 0;
    cl.nvert = 0;
    const long C = cs.C;
    const int nI = A.nI;
    cl.ioff_h.assign(nI + 1, 0);
    if (W[W_CL_INT].ensure(sizeof(int) * (2 * A.V + 8 * (nI + 1) + 64))) return IDP_ERR_CUDA;
    int* base = W[W_CL_INT].as<int>();
    if (C <= 0) {
        cl.vcl = base;
        IDP_CUDA_TRY(cudaMemsetAsync(cl.vcl, 0xff, sizeof(int) * A.V, s));
        cl.ioff = base + A.V;
        IDP_CUDA_TRY(cudaMemsetAsync(cl.ioff, 0, sizeof(int) * (nI + 1), s));
        return IDP_OK;
    }
    // constraints to the host (C x 20 bytes)
    std::vector<int4> hc(C);
    std::vector<int> hi(C);
    IDP_CUDA_TRY(cudaMemcpyAsync(hc.data(), W[W_CONS].p, sizeof(int4) * C, cudaMemcpyDeviceToHost, s));
    IDP_CUDA_TRY(cudaMemcpyAsync(hi.data(), W[W_CONS_INST].p, sizeof(int) * C, cudaMemcpyDeviceToHost, s));
    IDP_CUDA_TRY(cudaStreamSynchronize(s));
    // stencil vertices of each constraint (sign encoding of FEM/IPC.h:202-250)
    auto stencil = [](int4 c, int* v) {
        if (c.x >= 0) {
            v[0] = c.x;
            v[1] = c.y;
            v[2] = c.z >= 0 ? c.z : -c.z - 1;
            v[3] = c.w >= 0 ? c.w : -c.w - 1;
            return 4;
        }
        v[0] = -c.x - 1;
        v[1] = c.y;
        if (c.w >= 0) { v[2] = c.z; v[3] = c.w; return 4; }
        if (c.z >= 0) { v[2] = c.z; return 3; }
        return 2;
    };
    // compact the vertices that appear in constraints
    std::vector<int> gid;
    gid.reserve(4 * C);
    for (long k = 0; k < C; ++k) {
        int v[4];
        int nv = stencil(hc[k], v);
        for (int a = 0; a < nv; ++a) gid.push_back(v[a]);
    }
    std::sort(gid.begin(), gid.end());
    gid.erase(std::unique(gid.begin(), gid.end()), gid.end());
    const int m = (int)gid.size();
    auto lid = [&](int v) { return (int)(std::lower_bound(gid.begin(), gid.end(), v) - gid.begin()); };
    DSU dsu(m);
    std::vector<std::vector<int>> adj(m);
    for (long k = 0; k < C; ++k) {
        int v[4];
        int nv = stencil(hc[k], v);
        int l[4];
        for (int a = 0; a < nv; ++a) l[a] = lid(v[a]);
        for (int a = 1; a < nv; ++a) dsu.unite(l[0], l[a]);
        for (int a = 0; a < nv; ++a)
            for (int b = 0; b < nv; ++b)
                if (a != b) adj[l[a]].push_back(l[b]);
    }
    for (auto& a : adj) {
        std::sort(a.begin(), a.end());
        a.erase(std::unique(a.begin(), a.end()), a.end());
    }
    // components in order of their smallest vertex, split breadth-first
    std::vector<std::vector<int>> comps;
    {
        std::vector<int> rootc(m, -1);
        for (int i = 0; i < m; ++i) {
            int r = dsu.find(i);
            if (rootc[r] < 0) {
                rootc[r] = (int)comps.size();
                comps.emplace_back();
            }
            comps[rootc[r]].push_back(i);
        }
    }
    std::vector<std::vector<int>> blocks;
    std::vector<char> taken(m, 0);
    for (auto& comp : comps) {
        if ((int)comp.size() < 2) continue;
        if ((int)comp.size() <= W.cl_cap) {
            blocks.push_back(comp);
            continue;
        }
        for (int st : comp) {
            if (taken[st]) continue;
            std::vector<int> blk;
            std::deque<int> q{st};
            taken[st] = 1;
            while (!q.empty() && (int)blk.size() < W.cl_cap) {
                int u = q.front();
                q.pop_front();
                blk.push_back(u);
                for (int w : adj[u])
                    if (!taken[w] && (int)(blk.size() + q.size()) < W.cl_cap) {
                        taken[w] = 1;
                        q.push_back(w);
                    }
            }
            for (int u : q) taken[u] = 0;  // not placed: left for the next block
            if (blk.size() >= 2) blocks.push_back(blk);
        }
    }
    // sort blocks by instance; device arrays
    std::vector<int> vinst_h(blocks.size());
    {
        // instance of a global vertex from the arena offsets
        for (size_t b = 0; b < blocks.size(); ++b) {
            int v = gid[blocks[b][0]];
            vinst_h[b] = (int)(std::upper_bound(A.v_off.begin(), A.v_off.end(), v) - A.v_off.begin()) - 1;
        }
    }
    std::vector<int> order(blocks.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return vinst_h[a] < vinst_h[b]; });
    std::vector<int> off(1, 0), vert, ioff(nI + 1, 0), vcl(A.V, -1), vloc(A.V, 0);
    std::vector<long long> doff(1, 0);
    std::vector<int> big, few;  // blocks factored by a cluster, by one CTA
    int maxn = 0;
    for (int bi = 0; bi < (int)order.size(); ++bi) {
        auto& blk = blocks[order[bi]];
        std::vector<int> vs;
        for (int l : blk) vs.push_back(gid[l]);
        std::sort(vs.begin(), vs.end());
        for (size_t k = 0; k < vs.size(); ++k) {
            vcl[vs[k]] = bi;
            vloc[vs[k]] = (int)k;
        }
        vert.insert(vert.end(), vs.begin(), vs.end());
        off.push_back((int)vert.size());
        const int N = 3 * (int)vs.size();
        doff.push_back(doff.back() + (long long)N * block_ld(N));
        (N > kInvClusterRows ? big : few).push_back(bi);
        ioff[vinst_h[order[bi]] + 1]++;
        maxn = std::max(maxn, (int)vs.size());
    }
    for (int i = 0; i < nI; ++i) ioff[i + 1] += ioff[i];
    cl.ioff_h = ioff;
    const int ncl = (int)order.size();
    cl.n = ncl;
    cl.nvert = (long)vert.size();
    cl.dense = doff.back();
    cl.max_n = maxn;
    // int buffer layout: vcl[V] vloc[V] ioff[nI+1] off[ncl+1] vert[nvert] ok[ncl] list[ncl] | doff (8-byte aligned)
    size_t ints = 2 * (size_t)A.V + (nI + 1) + (ncl + 1) + vert.size() + 2 * ncl + 8;
    size_t bytes = sizeof(int) * ints + sizeof(long long) * (ncl + 2) + 64;
    if (W[W_CL_INT].ensure(bytes)) return IDP_ERR_CUDA;
    base = W[W_CL_INT].as<int>();
    cl.vcl = base;
    cl.vloc = cl.vcl + A.V;
    cl.ioff = cl.vloc + A.V;
    cl.off = cl.ioff + (nI + 1);
    cl.vert = cl.off + (ncl + 1);
    int* okp = cl.vert + vert.size();
    cl.ok = okp;
    int* list = okp + ncl;  // the cluster-factored blocks, then the others
    size_t used = (size_t)(list + ncl - base);
    used = (used + 1) / 2 * 2;
    cl.doff = reinterpret_cast<long long*>(base + used);
    IDP_CUDA_TRY(cudaMemcpyAsync(cl.vcl, vcl.data(), sizeof(int) * A.V, cudaMemcpyHostToDevice, s));
    IDP_CUDA_TRY(cudaMemcpyAsync(cl.vloc, vloc.data(), sizeof(int) * A.V, cudaMemcpyHostToDevice, s));
    IDP_CUDA_TRY(cudaMemcpyAsync(cl.ioff, ioff.data(), sizeof(int) * (nI + 1), cudaMemcpyHostToDevice, s));
    IDP_CUDA_TRY(cudaMemcpyAsync(cl.off, off.data(), sizeof(int) * (ncl + 1), cudaMemcpyHostToDevice, s));
    if (!vert.empty())
        IDP_CUDA_TRY(cudaMemcpyAsync(cl.vert, vert.data(), sizeof(int) * vert.size(), cudaMemcpyHostToDevice, s));
    IDP_CUDA_TRY(cudaMemcpyAsync(cl.doff, doff.data(), sizeof(long long) * (ncl + 1), cudaMemcpyHostToDevice, s));
    if (ncl == 0) {
        IDP_CUDA_TRY(cudaStreamSynchronize(s));
        return IDP_OK;
    }
    std::vector<int> order_l(big);
    order_l.insert(order_l.end(), few.begin(), few.end());
    IDP_CUDA_TRY(cudaMemcpyAsync(list, order_l.data(), sizeof(int) * ncl, cudaMemcpyHostToDevice, s));
    // K | Y | t = Y r of the PCG's block applies
    size_t el = fp64 ? sizeof(double) : sizeof(float);
    if (W[W_CL_DENSE].ensure(el * (2 * (size_t)cl.dense + 3 * (size_t)cl.nvert + 16))) return IDP_ERR_CUDA;
    return fp64 ? factor_blocks<double>(A, W, list, (int)big.size(), (int)few.size(), s)
                : factor_blocks<float>(A, W, list, (int)big.size(), (int)few.size(), s);
}

}  // namespace idp
