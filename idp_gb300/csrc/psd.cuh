// PSD projection of a small symmetric matrix (n <= 12), following the
// reference's makePD (Math/UTILS.h:10-27: eigen-decompose, clamp negative
// eigenvalues to zero, recompose): a per-thread Cholesky test first (a
// positive definite matrix is left unchanged, chol_pd), else Jacobi rotations
// by 16 lanes (psd_group_project).
#pragma once
#include "common.cuh"

namespace idp {
namespace {

template <class T>
__device__ bool chol_pd(const T* A, int n) {
    T L[78];
    for (int j = 0; j < n; ++j) {
        T s = A[j * n + j];
        for (int k = 0; k < j; ++k) s -= L[j * (j + 1) / 2 + k] * L[j * (j + 1) / 2 + k];
        if (!(s > T(0))) return false;
        T ljj = sqrt(s);
        L[j * (j + 1) / 2 + j] = ljj;
        for (int i = j + 1; i < n; ++i) {
            T t = A[i * n + j];
            for (int k = 0; k < j; ++k) t -= L[i * (i + 1) / 2 + k] * L[j * (j + 1) / 2 + k];
            L[i * (i + 1) / 2 + j] = t / ljj;
        }
    }
    return true;
}

// Projection by 16 lanes per matrix (two matrices per warp): one-sided
// Jacobi. The matrix is scaled by a power of two to a row-sum norm below 1 and
// shifted, B = A / 2^e + I, so that every eigenvalue of B is positive and its
// singular vectors are A's eigenvectors. Lane j of the group keeps column j of
// B in registers; a round pairs the lanes round-robin (tournament order, a
// dummy player for odd n), each fetches its partner's column by shuffle, both
// form the same inner product and the rotation that makes the two columns
// orthogonal: zeta = (|g_q|^2 - |g_p|^2) / (2 g_p.g_q), t = sign(zeta) /
// (|zeta| + sqrt(zeta^2 + 1)), c = 1 / sqrt(t^2 + 1), s = t c. Sweeps stop
// when every pair is orthogonal to 4 eps of its norms (20 at most). The
// eigenvalues are then the Rayleigh quotients of the normalised columns with A
// itself (FP32 sums compensated, so that a zero eigenvalue beside a large one
// does not come out as its rounding), and the projection is a sum of outer
// products that takes the off-diagonals the sweeps left into account: a sum of
// squares stays PSD to rounding, which A minus its negative part does not. (No
// floor under the eigenvalues: one of eps / 4 of the largest already leads mixed
// solves with stiff contact to other minima than FP64 takes in 5 of 14 runs.)
// Only columns move: no shared memory, no row updates and no separate
// eigenvector matrix in the sweeps, which are bound by instruction issue
// (FP32) or the FP64 pipe. 22,000 random 12x12 matrices: FP32 0.17 ms (3.4 ms
// for two-sided sweeps over A and V in shared memory, one warp per matrix,
// whose FP32 runs never met their stopping test and took 20 sweeps), FP64
// 4.3 to 4.6 ms (7.1 ms).
constexpr int kPsdDim = 12;                 // row stride of the matrices in shared memory
constexpr int kPsdGroup = 16;               // lanes per matrix
constexpr int kPsdThreads = 128;
constexpr int kPsdPerCta = kPsdThreads / kPsdGroup;
template <class T>
struct PsdScratch {
    T A[kPsdDim * kPsdDim];                 // the matrix, zero-padded
    T V[kPsdDim * kPsdDim];                 // row j = v_j, then h_j: the projection is sum_j h_j h_j^T
};

// acc += a * b with the rounding errors of the product and the sum kept in
// err (two-product, two-sum); FP64 adds plainly
__device__ __forceinline__ void acc_product(float& acc, float& err, float a, float b) {
    const float p = __fmul_rn(a, b), t = __fadd_rn(acc, p), z = __fsub_rn(t, acc);
    err += __fmaf_rn(a, b, -p) + (__fsub_rn(acc, __fsub_rn(t, z)) + __fsub_rn(p, z));
    acc = t;
}
__device__ __forceinline__ void acc_product(double& acc, double&, double a, double b) { acc += a * b; }

// n x n matrices (n = N: 6, 9 or 12) of the groups with `mine`; every lane of
// the warp calls this. A group's result does not depend on its neighbour.
template <class T, int N>
__device__ void psd_jacobi(PsdScratch<T>& sc, int j, bool mine) {
    const unsigned full = 0xffffffffu;
    constexpr int M = N + (N & 1);          // players
    const int base = threadIdx.x & 16;
    const bool act = mine && j < N;
    T g[N];
    T rs = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        g[i] = act ? sc.A[j * kPsdDim + i] : T(0);
        rs += fabs(g[i]);
    }
    for (int o = 8; o > 0; o >>= 1) rs = fmax(rs, __shfl_xor_sync(full, rs, o));
    int e = 0;
    if (rs > T(0)) frexp(rs, &e);
    e = max(e, sizeof(T) == 4 ? -120 : -1000);  // the scale stays finite
    const T scale = scalbn(T(1), -e);
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] = g[i] * scale + (i == j ? T(1) : T(0));
    constexpr T eps4 = sizeof(T) == 4 ? T(4 * 1.1920929e-7) : T(4 * 2.220446049250313e-16);
    bool done = !mine;
    for (int sweep = 0; sweep < 20; ++sweep) {
        T a2 = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) a2 += g[i] * g[i];
        bool rotated = false;
        for (int r = 0; r < M - 1; ++r) {
            int q = 2 * r - j + (j > 2 * r ? M - 1 : 0);
            if (q >= M - 1) q -= M - 1;
            if (j == r) q = M - 1;
            if (j == M - 1) q = r;
            if (j >= M) q = j;
            T y[N], gam = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                y[i] = __shfl_sync(full, g[i], base | q);
                gam += g[i] * y[i];
            }
            const T b2 = __shfl_sync(full, a2, base | q);
            if (act && !done && q < N && gam * gam > eps4 * eps4 * (a2 * b2)) {
                const bool first = j < q;
                const T zeta = (first ? b2 - a2 : a2 - b2) / (T(2) * gam);
                const T t = (zeta >= T(0) ? T(1) : T(-1)) / (fabs(zeta) + sqrt(zeta * zeta + T(1)));
                const T c = T(1) / sqrt(t * t + T(1));
                const T s = first ? -t * c : t * c;
#pragma unroll
                for (int i = 0; i < N; ++i) g[i] = c * g[i] + s * y[i];
                a2 += first ? -t * gam : t * gam;
                rotated = true;
            }
        }
        // a group that made no rotation in a sweep is finished for good
        const unsigned rot = __ballot_sync(full, rotated);
        done = done || ((rot >> base) & 0xffffu) == 0;
        if (!rot) break;
    }
    T nn = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) nn += g[i] * g[i];
    const T inv = nn > T(0) ? T(1) / sqrt(nn) : T(0);
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] *= inv;
    // y = A v_j, the eigenvalue v_j . y, and the off-diagonals m_ij = v_i . y
    T y[N], lam = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        T av = 0, ae = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) acc_product(av, ae, sc.A[i * kPsdDim + k], g[k]);
        y[i] = act ? av + ae : T(0);
        lam += g[i] * y[i];
    }
    const T sl = act && lam > T(0) ? sqrt(lam) : T(0);  // 0: not among the kept ones
    if (act)
#pragma unroll
        for (int i = 0; i < N; ++i) sc.V[j * kPsdDim + i] = g[i];
    __syncwarp();
    // h_j = sqrt(lam_j) v_j + sum_i E_ij v_i with E, to first order in the
    // off-diagonals m, what makes V^T (sum_j h_j h_j^T) V the projection of
    // lam + m (bounded by sqrt |m|, so that its square stays below m)
#pragma unroll
    for (int i = 0; i < N; ++i) g[i] *= sl;
    for (int i = 0; i < N; ++i) {
        const T li = __shfl_sync(full, lam, base | i), sli = __shfl_sync(full, sl, base | i);
        T m = 0, v[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            v[k] = sc.V[i * kPsdDim + k];
            m += v[k] * y[k];
        }
        if (i == j || !(sl > T(0))) continue;
        const T most = sqrt(fabs(m));
        T E = sli > T(0) ? m / (sli + sl) : m * sl / (lam - li);
        E = fmin(fmax(E, -most), most);
#pragma unroll
        for (int k = 0; k < N; ++k) g[k] += E * v[k];
    }
    __syncwarp();
    if (act)
#pragma unroll
        for (int i = 0; i < N; ++i) sc.V[j * kPsdDim + i] = g[i];
    __syncwarp();
}

// projection of the group's n x n matrix in sc.A (n = 0: nothing to do); all
// lanes of a warp call this together, then psd_entry gives the result
template <class T>
__device__ void psd_group_project(PsdScratch<T>& sc, int n, int j) {
    const unsigned full = 0xffffffffu;
    if (__any_sync(full, n == 12)) psd_jacobi<T, 12>(sc, j, n == 12);
    if (__any_sync(full, n == 9)) psd_jacobi<T, 9>(sc, j, n == 9);
    if (__any_sync(full, n == 6)) psd_jacobi<T, 6>(sc, j, n == 6);
}

// entry (r, c) of the projected n x n matrix
template <class T>
__device__ __forceinline__ T psd_entry(const PsdScratch<T>& sc, int n, int r, int c) {
    T acc = 0;
    for (int k = 0; k < n; ++k) acc += sc.V[k * kPsdDim + r] * sc.V[k * kPsdDim + c];
    return acc;
}

}  // namespace
}  // namespace idp
