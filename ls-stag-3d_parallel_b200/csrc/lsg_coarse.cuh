// The smallest multigrid levels in one kernel.
//
// On levels of a few hundred cells every V-cycle operation (restriction,
// 27-point residual update, line solve, prolongation) is a kernel launch of a
// few microseconds for almost no data.  k_vcycle_tail runs the lower part of
// the cycle (MultiGridSolver::solve, multigrid_solver.h:48-75, from level l0
// down to the coarsest solve and back up through the smoothing of level l0) in
// one CTA, one thread per cell.  Everything it touches more than once is
// brought to the SM at the start: the vectors, the line factors and the rows of
// the lower levels in shared memory, the first level's rows in registers.  A
// direction step is then two barriers apart: the residual from the iterate's
// box (stored with a zero margin, so no neighbour needs a bounds test), and the
// line recurrences, one thread per line.  The steps are latency chains: with
// the level data in L1 only, they took 72 (FP32) and 104 us (FP64) per cycle on
// levels of 8^3 and below; 18 direction steps and the coarsest solve.
//
// Each phase performs the same arithmetic, in the same order, as the
// stand-alone kernel it replaces (k_restrict, k_prolong, k_apply27z,
// k_tdma_strided); the coarsest solve's sums are taken by columns.
#pragma once

#include "lsg_kernels.cuh"

namespace lsg {

constexpr int kTailThreads = 512;       // one per cell of the first level
constexpr int kTailMaxCells = 512;      // levels fused into the tail kernel hold at most this many cells
constexpr int kTailMaxLevels = 12;
constexpr int kTailMaxSmem = 200 * 1024;
constexpr int kTailDense = 32;          // coarsest systems up to this size are solved by one warp

template <typename T>
struct TailLevel {
    int N, M, K;
    const int* cls;
    const T* dict28;                    // 27-point rows, stride 28 (z, y, x box order)
    const T* lo[3];
    const T* dinv[3];
    const T* up[3];
    const T* r;                         // level l0: its right-hand side
    T* ch;                              // level l0: its correction
    // transfer tables between this level (fine side) and the next coarser one
    PTab px, py, pz;
    RTab rx, ry, rz;
    int agg;
    // shared memory, in values from the start: right-hand side (n), box of the
    // iterate (with margin), line right-hand sides (n), factors (9 n; not for
    // the coarsest), rows (27 n; levels after the first, without the coarsest)
    int s_r, s_c, s_w, s_f, s_a;
};

template <typename T>
struct TailArgs {
    TailLevel<T> lev[kTailMaxLevels];   // levels l0 .. L (index 0 = level l0)
    int nlev;                           // number of levels including the coarsest
    // coarsest dense LU (LUDecompositionSparseMatrix)
    int nc;
    int s_lu;                           // shared memory of its factors (doubles from the start), n <= kTailDense
    const double* L;
    const double* U;
    const double* scale;
    const int* perm;
    double* work;
    int n_post;
    int zquirk;
    T omega;
};

__host__ __device__ inline int tail_box(int N, int M, int K) { return (N + 2) * (M + 2) * (K + 2); }

// Lays out the shared memory of the levels; returns the number of values.
template <typename T>
inline size_t tail_layout(TailArgs<T>& A)
{
    size_t at = 0;
    auto take = [&](size_t n) {
        const size_t p = at;
        at += n;
        return (int)p;
    };
    A.s_lu = 0;
    if (A.nc <= kTailDense) take(2 * (size_t)kTailDense * (kTailDense + 1) * (sizeof(double) / sizeof(T)));
    for (int l = 0; l < A.nlev; l++) {
        TailLevel<T>& v = A.lev[l];
        const size_t n = (size_t)v.N * v.M * v.K;
        const bool last = l == A.nlev - 1;
        v.s_r = take(n);
        v.s_c = take((size_t)tail_box(v.N, v.M, v.K));
        v.s_w = take(last ? 0 : n);
        v.s_f = take(last ? 0 : 9 * n);
        v.s_a = take(last || l == 0 ? 0 : 27 * n);
    }
    return at;
}

// Position of a cell in the iterate's box.
template <typename T>
__device__ __forceinline__ int tail_at(const TailLevel<T>& v, int x, int y, int z)
{
    return ((z + 1) * (v.M + 2) + y + 1) * (v.N + 2) + x + 1;
}

// coarse = R fine (k_restrict)
template <typename T>
__device__ __forceinline__ void tail_restrict(const TailLevel<T>& f, const TailLevel<T>& c, T* sm)
{
    const int nc = c.N * c.M * c.K, NMc = c.N * c.M, NM = f.N * f.M;
    const T* fr = sm + f.s_r;
    for (int I = threadIdx.x; I < nc; I += kTailThreads) {
        const int Z = I / NMc, rem = I - Z * NMc, Y = rem / c.N, X = rem - Y * c.N;
        T acc = 0;
        if (f.agg) {
            const int f0 = (2 * Z) * NM + (2 * Y) * f.N + 2 * X;
            const T w = (T)0.125;
            acc += w * fr[f0];
            acc += w * fr[f0 + 1];
            acc += w * fr[f0 + f.N];
            acc += w * fr[f0 + f.N + 1];
            acc += w * fr[f0 + NM];
            acc += w * fr[f0 + NM + 1];
            acc += w * fr[f0 + NM + f.N];
            acc += w * fr[f0 + NM + f.N + 1];
        } else {
            for (int a = 0; a < 4; a++) {
                const int fz = f.rz.f[4 * Z + a];
                if (fz < 0) continue;
                const float wz = f.rz.w[4 * Z + a];
                for (int b = 0; b < 4; b++) {
                    const int fy = f.ry.f[4 * Y + b];
                    if (fy < 0) continue;
                    const float wy = f.ry.w[4 * Y + b];
                    for (int q = 0; q < 4; q++) {
                        const int fx = f.rx.f[4 * X + q];
                        if (fx < 0) continue;
                        acc += (T)(wz * wy * f.rx.w[4 * X + q]) * fr[fz * NM + fy * f.N + fx];
                    }
                }
            }
        }
        sm[c.s_r + I] = acc;
    }
}

// This thread's cell of P coarse (k_prolong)
template <typename T>
__device__ __forceinline__ T tail_prolong(const TailLevel<T>& f, const TailLevel<T>& c, const T* sm, int x, int y,
                                          int z)
{
    T acc = 0;
#pragma unroll
    for (int q = 0; q < 8; q++) {                   // z, y, x ascending; unused slots hold index 0, weight 0
        const int a = q >> 2, b = (q >> 1) & 1, e = q & 1;
        const float w = f.pz.w[2 * z + a] * f.py.w[2 * y + b] * f.px.w[2 * x + e];
        if (w != 0.f)
            acc += (T)w * sm[c.s_c + tail_at(c, f.px.c[2 * x + e], f.py.c[2 * y + b], f.pz.c[2 * z + a])];
    }
    return acc;
}

// n_post sweeps of z, y, x direction steps on one level, from the iterate in
// its box; leaves the accumulated correction in the box.  row: this thread's
// 27 coefficients (registers, or shared memory).
template <typename T, typename Row>
__device__ __forceinline__ void tail_smooth(const TailArgs<T>& A, const TailLevel<T>& v, T* sm, const Row& row, T r,
                                            T ch, bool in, int at, int w0)
{
    const int n = v.N * v.M * v.K, RS = v.N + 2, PS = RS * (v.M + 2);
    T* c = sm + v.s_c;
    T* w = sm + v.s_w;
    for (int it = 0; it < A.n_post; it++)
        for (int d = 2; d >= 0; d--) {
            if (in) {                               // r -= A c
                T acc = 0;
#pragma unroll
                for (int q = 0; q < 27; q++) {
                    const int dz = q / 9 - 1, dy = (q / 3) % 3 - 1, dx = q % 3 - 1;
                    acc += row[q] * c[at + dz * PS + dy * RS + dx];
                }
                r = r - acc;
                w[w0] = r;
            }
            __syncthreads();
            const int L = d == 0 ? v.N : (d == 1 ? v.M : v.K);
            const int nl = d == 0 ? v.M * v.K : (d == 1 ? v.N * v.K : v.N * v.M);
            for (int l = threadIdx.x; l < nl; l += kTailThreads) {   // c = omega T_d^-1 r, one line a thread
                int i0, a0;                         // first cell of the line: flat, and in the box
                if (d == 0) {
                    const int z = l / v.M, y = l - z * v.M;
                    i0 = l * v.N;
                    a0 = tail_at(v, 0, y, z);
                } else {
                    const int q = l / v.N, x = l - q * v.N;
                    i0 = d == 1 ? q * v.N * v.M + x : l;
                    a0 = d == 1 ? tail_at(v, x, 0, q) : tail_at(v, x, q, 0);
                }
                const int st = d == 0 ? 1 : (d == 1 ? v.N : v.N * v.M), sb = d == 0 ? 1 : (d == 1 ? RS : PS);
                const T* lo = sm + v.s_f + 3 * d * n;
                const T* dinv = lo + n;
                const T* up = dinv + n;
                // the z-line's first right-hand side is read where the reference does
                const int first = d == 2 && A.zquirk ? (l / v.N) * v.N * v.K + l % v.N : i0;
                T y = 0;
                for (int t0 = 0; t0 < L; t0 += 8) {
                    T rv[8], lv[8], dv[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const int i = i0 + min(t0 + u, L - 1) * st;
                        rv[u] = w[t0 + u == 0 ? first : i];
                        lv[u] = lo[i];
                        dv[u] = dinv[i];
                    }
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        y = t0 + u == 0 ? rv[u] * dv[u] : (rv[u] - lv[u] * y) * dv[u];
                        if (t0 + u < L) c[a0 + (t0 + u) * sb] = y;
                    }
                }
                T x = 0;
                for (int t1 = L - 1; t1 >= 0; t1 -= 8) {
                    T yv[8], uv[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const int t = max(t1 - u, 0);
                        yv[u] = c[a0 + t * sb];
                        uv[u] = up[i0 + t * st];
                    }
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        x = t1 - u == L - 1 ? yv[u] : yv[u] - uv[u] * x;
                        if (t1 - u >= 0) c[a0 + (t1 - u) * sb] = A.omega * x;
                    }
                }
            }
            __syncthreads();
            if (in) ch += c[at];
        }
    __syncthreads();                                // every thread has read its last correction
    if (in) c[at] = ch;
}

// The coarsest dense system.  Up to kTailDense rows: one warp, lane i keeping
// row i's sum and taking the columns in turn, n dependent steps per triangle
// instead of n (n - 1) / 2.  Larger systems: the loop of k_coarse_solve.
template <typename T>
__device__ __forceinline__ void tail_coarsest(const TailArgs<T>& A, const TailLevel<T>& c, T* sm, const double* lu)
{
    const int n = A.nc, lane = threadIdx.x, NM = c.N * c.M;
    constexpr int LD = kTailDense + 1;
    const T* r = sm + c.s_r;
    auto put = [&](int i, double v) {
        const int z = i / NM, y = (i - z * NM) / c.N, x = i - z * NM - y * c.N;
        sm[c.s_c + tail_at(c, x, y, z)] = (T)v;
    };
    if (n <= kTailDense) {
        if (lane >= 32) return;
        const bool in = lane < n;
        const double* sL = lu;                      // [column][row]
        const double* sU = lu + kTailDense * LD;
        double aux = 0.0, sc = 0.0, piv = 1.0;
        if (in) {
            sc = A.scale[lane];
            piv = sU[lane * LD + lane];
            aux = A.scale[A.perm[lane]] * (double)r[A.perm[lane]];
        }
        for (int j = 0; j < n; j++) {
            const double y = __shfl_sync(0xffffffffu, aux, j);
            if (in && lane > j) aux -= sL[j * LD + lane] * y;
        }
        double z = 0.0;
        for (int j = n - 1; j >= 0; j--) {
            if (lane == j) z = aux / piv;
            const double zj = __shfl_sync(0xffffffffu, z, j);
            if (lane < j) aux -= sU[j * LD + lane] * zj;
        }
        if (in) put(lane, sc * z);
        return;
    }
    if (lane != 0) return;
    double* y = A.work;
    double* z = A.work + n;
    for (int i = 0; i < n; i++) {
        double aux = A.scale[A.perm[i]] * (double)r[A.perm[i]];
        for (int j = 0; j < i; j++) aux -= A.L[i * n + j] * y[j];
        y[i] = aux;
    }
    for (int i = n - 1; i >= 0; i--) {
        double aux = y[i];
        for (int j = i + 1; j < n; j++) aux -= A.U[i * n + j] * z[j];
        z[i] = aux / A.U[i * n + i];
    }
    for (int i = 0; i < n; i++) put(i, A.scale[i] * z[i]);
}

template <typename T>
__global__ void __launch_bounds__(kTailThreads, 1) k_vcycle_tail(const TailArgs<T>* __restrict__ argp)
{
    extern __shared__ __align__(16) unsigned char tail_smem[];
    T* sm = reinterpret_cast<T*>(tail_smem);
    double* lu = reinterpret_cast<double*>(tail_smem);
    const TailArgs<T>& A = *argp;
    const int last = A.nlev - 1, tid = threadIdx.x;
    // everything in: the first level's rows, the right-hand side, factors,
    // the lower levels' rows, the coarsest factors; empty boxes
    const TailLevel<T>& v0 = A.lev[0];
    const int n0 = v0.N * v0.M * v0.K;
    T a[28];
    if (tid < n0) load_row28(v0.dict28 + (size_t)v0.cls[tid] * 28, a);
    for (int l = 0; l <= last; l++) {
        const TailLevel<T>& v = A.lev[l];
        const int n = v.N * v.M * v.K, nb = tail_box(v.N, v.M, v.K);
        for (int i = tid; i < nb; i += kTailThreads) sm[v.s_c + i] = 0;
        if (l == last) break;
        for (int d = 0; d < 3; d++)
            for (int i = tid; i < n; i += kTailThreads) {
                sm[v.s_f + 3 * d * n + i] = v.lo[d][i];
                sm[v.s_f + (3 * d + 1) * n + i] = v.dinv[d][i];
                sm[v.s_f + (3 * d + 2) * n + i] = v.up[d][i];
            }
        if (l > 0)
            for (int e = tid; e < 27 * n; e += kTailThreads) {
                const int q = e / n, i = e - q * n;             // [coefficient][cell]
                sm[v.s_a + e] = v.dict28[(size_t)v.cls[i] * 28 + q];
            }
    }
    if (A.nc <= kTailDense)
        for (int e = tid; e < A.nc * A.nc; e += kTailThreads) {
            const int i = e / A.nc, j = e - i * A.nc;
            lu[j * (kTailDense + 1) + i] = A.L[e];
            lu[(kTailDense + j) * (kTailDense + 1) + i] = A.U[e];
        }
    dep_begin();                                    // all of the above is the operator's
    for (int i = tid; i < n0; i += kTailThreads) sm[v0.s_r + i] = v0.r[i];
    __syncthreads();
    for (int l = 0; l < last; l++) {
        tail_restrict<T>(A.lev[l], A.lev[l + 1], sm);
        __syncthreads();
    }
    tail_coarsest<T>(A, A.lev[last], sm, lu);
    __syncthreads();
    for (int l = last - 1; l >= 0; l--) {
        const TailLevel<T>& v = A.lev[l];
        const int n = v.N * v.M * v.K, NM = v.N * v.M;
        const bool in = tid < n;
        const int i = in ? tid : 0;
        const int z = i / NM, y = (i - z * NM) / v.N, x = i - z * NM - y * v.N;
        const int at = tail_at(v, x, y, z);
        const T p = tail_prolong<T>(v, A.lev[l + 1], sm, x, y, z);
        if (in) sm[v.s_c + at] = p;
        __syncthreads();
        const T r = sm[v.s_r + i];
        if (l == 0) {
            tail_smooth<T>(A, v, sm, a, r, p, in, at, i);
        } else {
            struct Strided {                        // [coefficient][cell]
                const T* p;
                int n;
                __device__ T operator[](int q) const { return p[q * n]; }
            };
            tail_smooth<T>(A, v, sm, Strided{sm + v.s_a + i, n}, r, p, in, at, i);
        }
        if (l == 0) {
            if (in) v.ch[i] = sm[v.s_c + at];
        } else {
            __syncthreads();
        }
    }
}

}  // namespace lsg
