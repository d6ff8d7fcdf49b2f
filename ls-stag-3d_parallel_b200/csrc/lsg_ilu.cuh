// ILU(0) of the 7-point operator and its level-scheduled triangular solves.
//
// For a 7-point pattern in natural order (with N, M >= 3) the reference's
// general row-by-row ILU(0) (ilu_decomposition_sparse_matrix.h:63-119)
// reduces to
//     L_kj = A_kj / U_jj            j in {b, s, w}  (|U_jj| clamped at 1e-12)
//     U_kk = A_kk - (L_kb A_bk + L_ks A_sk + L_kw A_wk)   (clamped at 1e-16)
//     U_kj = A_kj                   j in {e, n, t}
// so only the pivots U_kk need computing; they depend on the three upstream
// neighbours, i.e. on the previous hyperplane x + y + z = const.  The
// triangular solves (ILUDecomposition7pStencilMatrix::DirectGauss/InverseGauss,
// ilu_decomposition_7p_stencil_matrix.h:90-134) have the same dependencies;
// they run as a pipeline of tiles of x-lines (k_ilu_tile_sweep).
#pragma once

#include "lsg_kernels.cuh"

namespace lsg {

// cell of hyperplane `level` handled by thread t: (x, y) enumerate the plane
// rows, z = level - x - y.
__device__ __forceinline__ bool plane_cell(int level, long long t, int N, int M, int K, long long& i)
{
    const int x = (int)(t % N);
    const int y = (int)(t / N);
    if (y >= M) return false;
    const int z = level - x - y;
    if (z < 0 || z >= K) return false;
    i = (long long)z * N * M + (long long)y * N + x;
    return true;
}

// the divisor U_jj of a lower coefficient, kept away from 0
__device__ __forceinline__ double ilu_clamp(double u)
{
    return fabs(u) < 1e-12 ? ((u < 0.0) ? -1e-12 : 1e-12) : u;
}

// Pivots of one hyperplane.  A: 7 planes b s w p e n t; U: pivot array.
__global__ void k_ilu_pivots(int level, int N, int M, int K, const double* __restrict__ A, double* __restrict__ U)
{
    const long long n = (long long)N * M * K;
    const int NM = N * M;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)N * M;
         t += (long long)gridDim.x * blockDim.x) {
        long long i;
        if (!plane_cell(level, t, N, M, K, i)) continue;
        const int x = (int)(t % N), y = (int)(t / N), z = level - x - y;
        double aux = 0.0;
        // lower entries in column order b (i-NM), s (i-N), w (i-1)
        if (z > 0) {
            double u = U[i - NM];
            if (fabs(u) < 1e-12) u = (u < 0.0) ? -1e-12 : 1e-12;
            aux += (A[i] / u) * A[6 * n + i - NM];
        }
        if (y > 0) {
            double u = U[i - N];
            if (fabs(u) < 1e-12) u = (u < 0.0) ? -1e-12 : 1e-12;
            aux += (A[n + i] / u) * A[5 * n + i - N];
        }
        if (x > 0) {
            double u = U[i - 1];
            if (fabs(u) < 1e-12) u = (u < 0.0) ? -1e-12 : 1e-12;
            aux += (A[2 * n + i] / u) * A[4 * n + i - 1];
        }
        double cur = A[3 * n + i] - aux;
        if (fabs(cur) < 1e-16) cur = (cur < 0.0) ? -1e-16 : 1e-16;
        U[i] = cur;
    }
}

// L planes (b, s, w) from the pivots: L_kj = A_kj / clamp(U_jj).
__global__ void k_ilu_lower(int N, int M, int K, const double* __restrict__ A, const double* __restrict__ U,
                            double* __restrict__ Lp)
{
    const long long n = (long long)N * M * K;
    const int NM = N * M;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        int x, y, z;
        cell_xyz(i, N, NM, x, y, z);
        double lb = 0, ls = 0, lw = 0;
        if (z > 0) {
            double u = U[i - NM];
            if (fabs(u) < 1e-12) u = (u < 0.0) ? -1e-12 : 1e-12;
            lb = A[i] / u;
        }
        if (y > 0) {
            double u = U[i - N];
            if (fabs(u) < 1e-12) u = (u < 0.0) ? -1e-12 : 1e-12;
            ls = A[n + i] / u;
        }
        if (x > 0) {
            double u = U[i - 1];
            if (fabs(u) < 1e-12) u = (u < 0.0) ? -1e-12 : 1e-12;
            lw = A[2 * n + i] / u;
        }
        Lp[i] = lb;
        Lp[n + i] = ls;
        Lp[2 * n + i] = lw;
    }
}

// forward sweep of one hyperplane: y = b - (L_b y_b + L_s y_s + L_w y_w)
__global__ void k_ilu_fwd(int level, int N, int M, int K, const double* __restrict__ Lp, const double* __restrict__ b,
                          double* __restrict__ y)
{
    const long long n = (long long)N * M * K;
    const int NM = N * M;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)N * M;
         t += (long long)gridDim.x * blockDim.x) {
        long long i;
        if (!plane_cell(level, t, N, M, K, i)) continue;
        const int x = (int)(t % N), yy = (int)(t / N), z = level - x - yy;
        double aux = b[i];
        if (z > 0) aux -= Lp[i] * y[i - NM];
        if (yy > 0) aux -= Lp[n + i] * y[i - N];
        if (x > 0) aux -= Lp[2 * n + i] * y[i - 1];
        y[i] = aux;
    }
}

// backward sweep of one hyperplane: x = (y - (U_e x_e + U_n x_n + U_t x_t)) / U_p
__global__ void k_ilu_bwd(int level, int N, int M, int K, const double* __restrict__ A, const double* __restrict__ U,
                          const double* __restrict__ y, double* __restrict__ xo)
{
    const long long n = (long long)N * M * K;
    const int NM = N * M;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < (long long)N * M;
         t += (long long)gridDim.x * blockDim.x) {
        long long i;
        if (!plane_cell(level, t, N, M, K, i)) continue;
        const int x = (int)(t % N), yy = (int)(t / N), z = level - x - yy;
        double aux = y[i];
        if (x < N - 1) aux -= A[4 * n + i] * xo[i + 1];
        if (yy < M - 1) aux -= A[5 * n + i] * xo[i + N];
        if (z < K - 1) aux -= A[6 * n + i] * xo[i + NM];
        xo[i] = aux / U[i];
    }
}

// ---------------------------------------------------------------------------
// The triangular solves as a pipeline of tiles.
//
// The grid's x-lines are cut into tiles of 16 x 16 lines in (y, z), one CTA
// per tile, one thread per line.  At step s the thread of line (ty, tz) works
// on cell x = s - ty - tz, so the cells of one step lie on one hyperplane, the
// values of a line's lower neighbours were computed one step earlier by this
// thread (x - 1) and by the threads next to it (y - 1, z - 1, through shared
// memory), and a step costs one barrier of one CTA.  Only the tile's two
// faces are exchanged between CTAs.
//
// Bound by the chain of dependent steps, N + M + K - 2 of them and the hand-over
// at each tile border, until a grid has enough tiles to fill the memory pipe.
// 16 x 16 lines keep the border crossings few (M/16 + K/16) with a barrier over
// only eight warps.  Measured on a B200, a momentum solve of 127 x 64 x 64 (two
// iterations): 0.48 ms against 2.25 ms with one cooperative launch and a grid
// barrier per hyperplane; an ILU-BiCGStab solve of 64 x 48 x 40: 29 against
// 143 ms.  The same bits for finite values (see the quotient below).
//
// Storage follows the steps: position (tile, step, thread), so that every
// stream is contiguous in the order in which it is used.  A tile has
// S = N + 30 steps, rounded up to whole chunks of kIluC; positions outside
// the grid hold zeros.
// ---------------------------------------------------------------------------
constexpr int kIluTY = 16, kIluTZ = 16, kIluT = kIluTY * kIluTZ;
constexpr int kIluC = 4;                  // steps per chunk
constexpr int kIluSlots = 3;              // chunks of factors and right-hand side in flight
constexpr int kIluFaceSlots = 4;          // chunks of face values in flight
constexpr int kIluThreads = kIluT + 96;   // line threads, the loading, face-in and face-out warps

struct IluTiles {
    int N, M, K;
    int nty, ntz;                         // tiles in y and z
    int nc;                               // chunks per tile
    long long steps() const { return (long long)nc * kIluC; }
    long long positions() const { return (long long)nty * ntz * steps() * kIluT; }
};

inline IluTiles ilu_tiles(int N, int M, int K)
{
    IluTiles g;
    g.N = N;
    g.M = M;
    g.K = K;
    g.nty = (M + kIluTY - 1) / kIluTY;
    g.ntz = (K + kIluTZ - 1) / kIluTZ;
    g.nc = (N + kIluTY + kIluTZ - 2 + kIluC - 1) / kIluC;
    return g;
}

// Coefficients per position: L_b, L_s, L_w of the forward sweep; U_e, U_n,
// U_t, U_p and 1 / U_p of the backward sweep, stored as [tile][chunk][kind]
// [step of the chunk][thread].
constexpr int kIluFwd = 3, kIluBwd = 5;

// Fills both coefficient arrays from the operator's planes and the pivots
// (L_kj = A_kj / clamp(U_jj), U_kj = A_kj); one thread per position.
__global__ void k_ilu_tile_factors(IluTiles g, const double* __restrict__ A, const double* __restrict__ U,
                                   double* __restrict__ facL, double* __restrict__ facU)
{
    const long long n = (long long)g.N * g.M * g.K;
    const long long NM = (long long)g.N * g.M;
    const long long S = (long long)g.nc * kIluC, total = (long long)g.nty * g.ntz * S * kIluT;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(q % kIluT);
        const long long ts = q / kIluT;                   // tile * S + step
        const int step = (int)(ts % S), tile = (int)(ts / S);
        const int ty = t % kIluTY, tz = t / kIluTY;
        const int x = step - ty - tz, y = (tile % g.nty) * kIluTY + ty, z = (tile / g.nty) * kIluTZ + tz;
        double l[kIluFwd] = {0, 0, 0}, u[kIluBwd] = {0, 0, 0, 0, 0};
        if (x >= 0 && x < g.N && y < g.M && z < g.K) {
            const long long i = x + g.N * ((long long)y + (long long)g.M * z);
            if (z > 0) l[0] = A[i] / ilu_clamp(U[i - NM]);
            if (y > 0) l[1] = A[n + i] / ilu_clamp(U[i - g.N]);
            if (x > 0) l[2] = A[2 * n + i] / ilu_clamp(U[i - 1]);
            if (x < g.N - 1) u[0] = A[4 * n + i];
            if (y < g.M - 1) u[1] = A[5 * n + i];
            if (z < g.K - 1) u[2] = A[6 * n + i];
            u[3] = U[i];
            u[4] = 1.0 / U[i];
        }
        const long long chunk = (long long)tile * g.nc + step / kIluC;
        const int in = (step % kIluC) * kIluT + t;
        for (int k = 0; k < kIluFwd; k++) facL[(chunk * kIluFwd + k) * kIluC * kIluT + in] = l[k];
        for (int k = 0; k < kIluBwd; k++) facU[(chunk * kIluBwd + k) * kIluC * kIluT + in] = u[k];
    }
}

// A vector of the grid into the tiles' step order (IN) or back: a CTA takes 32
// steps of 64 of a tile's lines through shared memory, so that both sides move
// whole 256-byte rows.  Positions outside the grid are set to 0.
template <bool IN>
__global__ void __launch_bounds__(256) k_ilu_tile_vector(IluTiles g, const double* __restrict__ src,
                                                          double* __restrict__ dst)
{
    __shared__ double sm[64][33];
    const int S = g.nc * kIluC, ns = (S + 31) / 32;
    const int tile = blockIdx.x / ns, s0 = (blockIdx.x - tile * ns) * 32, zg = blockIdx.y;
    const int y0 = (tile % g.nty) * kIluTY, z0 = (tile / g.nty) * kIluTZ + zg * 4;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int l0 = threadIdx.x & 63, u0 = threadIdx.x >> 6;
    const long long base = ((long long)tile * S + s0) * kIluT + zg * 64;
    auto rows = [&](auto&& body) {                        // the CTA's lines along x: one warp a line
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int l = wid + 8 * k, ty = l & 15, tz = zg * 4 + (l >> 4);
            const int x = s0 + lane - ty - tz, y = y0 + ty, z = z0 + (l >> 4);
            const bool in = x >= 0 && x < g.N && y < g.M && z < g.K;
            body(l, in, x + g.N * ((long long)y + (long long)g.M * z));
        }
    };
    if (IN) {
        rows([&](int l, bool in, long long i) { sm[l][lane] = in ? src[i] : 0.0; });
        __syncthreads();
#pragma unroll
        for (int u = u0; u < 32; u += 4)
            if (s0 + u < S) dst[base + (long long)u * kIluT + l0] = sm[l0][u];
    } else {
#pragma unroll
        for (int u = u0; u < 32; u += 4)
            sm[l0][u] = s0 + u < S ? src[base + (long long)u * kIluT + l0] : 0.0;
        __syncthreads();
        rows([&](int l, bool in, long long i) {
            if (in) dst[i] = sm[l][lane];
        });
    }
}

__device__ __forceinline__ unsigned long long ilu_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned ilu_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ilu_mbar_arrive(unsigned long long* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ilu_smem(bar)) : "memory");
}

// Waits for the phase of `bar` with this parity, for four seconds at most (the
// face warps' polls, which these waits depend on, end after one), or, with
// heed, until another wait of the launch has given up.  Then the error flag is
// set and the kernel runs on without waiting (wrong values, reported by the
// solve), so no thread is left behind at a barrier.  Waits for the kernel's own
// copies do not heed the flag: a copy must not outlive its CTA.
__device__ __forceinline__ void ilu_mbar_wait(unsigned long long* bar, unsigned parity, int* err, bool& gave_up,
                                              bool heed = true)
{
    unsigned long long t0 = 0;
    for (unsigned it = 0; !gave_up; it++) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(ilu_smem(bar)), "r"(parity)
            : "memory");
        if (ok) break;
        if ((it & 7) == 0) {
            const unsigned long long now = ilu_now();
            if (it == 0) t0 = now;
            else if (now - t0 > 4000000000ull || (heed && *(volatile int*)err != 0)) {
                atomicExch(err, 1);
                gave_up = true;
            }
        }
    }
}

__device__ __forceinline__ void ilu_bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     ilu_smem(dst)),
                 "l"(src), "r"(bytes), "r"(ilu_smem(bar))
                 : "memory");
}

// A face value in global memory: the two halves of the double, each beside the
// sweep's tag, so the reader knows from the words themselves that the value is
// there (8-byte words are written whole) and neither side needs a fence.
__device__ __forceinline__ void ilu_face_store(uint4* p, double v, unsigned tag)
{
    const unsigned lo = (unsigned)__double2loint(v), hi = (unsigned)__double2hiint(v);
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p),
                 "l"(((unsigned long long)tag << 32) | lo), "l"(((unsigned long long)tag << 32) | hi)
                 : "memory");
}

__device__ __forceinline__ bool ilu_face_load(const uint4* p, double& v, unsigned tag)
{
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    v = __hiloint2double((int)(unsigned)b, (int)(unsigned)a);
    return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
}

template <bool FWD>
constexpr size_t ilu_sweep_smem()
{
    return sizeof(double) * ((size_t)kIluSlots * ((FWD ? kIluFwd : kIluBwd) + 1) * kIluC * kIluT +
                             (size_t)kIluFaceSlots * kIluC * 32 + 2 * kIluT) +
           8 * (2 * kIluSlots + 2 * kIluFaceSlots);
}

// One triangular sweep, in place on the tile-ordered vector v: forward
// y = b - (L_b y_b + L_s y_s + L_w y_w), or backward
// x = (y - (U_e x_e + U_n x_n + U_t x_t)) / U_p, the terms in that order.
//
// A CTA takes its tile from a ticket, in the order of the tiles' diagonals, so
// every tile it depends on is held by a CTA that started before it and no CTA
// waits for one that has not.  The loading warp brings chunks of coefficients
// and right-hand sides (contiguous) into a ring in shared memory with bulk
// copies; the face warp polls the two upstream tiles' face values of a chunk
// and puts them into a ring of their own, one lane per face line; the face-out
// warp sends the tile's own face values on after each step; the line threads
// take kIluC steps per chunk.  Each step also asks for the same
// step's operands of the next chunk, in the shadow of its barrier, so a step
// does not wait for them (0.52 against 0.56 ms for the momentum solve, 31.3
// against 34.9 ms for BiCGStab).  A poll for a face value gives up after a
// second; then the other waits of the launch end too (ilu_mbar_wait), and CTAs
// that start later leave at once, in this sweep and in those after it until
// the flag is read; withhold >= 0 (the wait-limit self-test only): the CTA
// with that ticket leaves at once and writes no face.
//
// The quotient by U_p comes from the rounded reciprocal r = 1 / U_p and one
// remainder step, q0 = a r, q = q0 + (a - q0 U_p) r, which rounds as the
// division does (Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), in three
// dependent operations instead of a division in the recurrence.  That holds
// where a, q and the remainder are normal numbers.  A quotient that overflows
// or an infinite a gives NaN instead of an infinity, a zero loses its sign, and
// below 1e-290 or so the last bit may differ.  The padding multiplies by stored
// zeros, so an infinity at a line's end also becomes NaN there, and in the
// backward sweep of that line.  Either way the solve reports a breakdown.
template <bool FWD>
__global__ void __launch_bounds__(kIluThreads) k_ilu_tile_sweep(IluTiles g, const int* __restrict__ order,
                                                                 const double* __restrict__ fac, double* v,
                                                                 uint4* faces, unsigned tag, unsigned* ticket,
                                                                 unsigned base, int* err, int withhold)
{
    constexpr int NK = FWD ? kIluFwd : kIluBwd;
    constexpr int CT = kIluC * kIluT;
    extern __shared__ __align__(128) unsigned char ilu_sm_raw[];
    double* ilu_sm = reinterpret_cast<double*>(ilu_sm_raw);
    double* ring = ilu_sm;                                        // [slot][kind, then v][step][thread]
    double* fring = ring + (size_t)kIluSlots * (NK + 1) * CT;     // [slot][step][32 face lines]
    double* sh = fring + kIluFaceSlots * kIluC * 32;              // [2][thread]
    unsigned long long* full = reinterpret_cast<unsigned long long*>(sh + 2 * kIluT);
    unsigned long long* empty = full + kIluSlots;
    unsigned long long* ffull = empty + kIluSlots;
    unsigned long long* fempty = ffull + kIluFaceSlots;
    __shared__ unsigned my;
    __shared__ int dead;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        const int failed = *(volatile int*)err;                   // read first: both round trips at once
        my = atomicAdd(ticket, 1u) - base;                        // base: the tickets of the earlier launches
        dead = failed;                                            // a wait has given up: no more of them
        for (int k = 0; k < kIluSlots; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ilu_smem(full + k)), "r"(1) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ilu_smem(empty + k)), "r"(kIluT / 32)
                         : "memory");
        }
        for (int k = 0; k < kIluFaceSlots; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ilu_smem(ffull + k)), "r"(1) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(ilu_smem(fempty + k)), "r"(kIluT / 32)
                         : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < kIluT) sh[tid] = sh[kIluT + tid] = 0.0;
    __syncthreads();
    if (dead || (int)my == withhold) return;
    const int ntile = g.nty * g.ntz;
    const int tile = order[FWD ? (int)my : ntile - 1 - (int)my];
    const int ta = tile % g.nty, tb = tile / g.nty;
    const int nc = g.nc, S = nc * kIluC;
    bool gave_up = false;

    if (warp == kIluT / 32) {                                     // the loading warp
        if (lane != 0) return;
        // A slot's barrier is armed again only when its copies have landed,
        // whoever has given up: line threads that no longer wait free slots
        // whose copies are still in flight, and a second arrival in that
        // phase would break the barrier.
        int issued = 0;
        for (; issued < nc; issued++) {
            const int c = issued, slot = c % kIluSlots, cf = FWD ? c : nc - 1 - c;
            if (c >= kIluSlots) {
                bool late = false;
                ilu_mbar_wait(full + slot, (unsigned)(c / kIluSlots - 1) & 1u, err, late, false);
                ilu_mbar_wait(empty + slot, (unsigned)(c / kIluSlots - 1) & 1u, err, gave_up);
                if (late || gave_up) break;
            }
            double* dst = ring + (size_t)slot * (NK + 1) * CT;
            const long long chunk = (long long)tile * nc + cf;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(ilu_smem(full + slot)),
                         "r"((unsigned)((NK + 1) * CT * sizeof(double)))
                         : "memory");
            ilu_bulk_load(dst, fac + chunk * NK * CT, NK * CT * sizeof(double), full + slot);
            ilu_bulk_load(dst + NK * CT, v + chunk * CT, CT * sizeof(double), full + slot);
        }
        for (int c = max(0, issued - kIluSlots); c < issued; c++) {   // no copy outlives the CTA
            bool late = false;
            ilu_mbar_wait(full + c % kIluSlots, (unsigned)(c / kIluSlots) & 1u, err, late, false);
        }
        return;
    }
    if (warp == kIluT / 32 + 1) {                                 // the face warp
        // lanes 0..15: the y-face line tz = lane of the tile before (FWD) or
        // after in y; lanes 16..31: the z-face line ty = lane - 16
        const bool yf = lane < 16;
        const bool has = FWD ? (yf ? ta > 0 : tb > 0) : (yf ? ta + 1 < g.nty : tb + 1 < g.ntz);
        const int up = tile + (FWD ? -1 : 1) * (yf ? 1 : g.nty);
        const uint4* src = faces + (long long)(has ? up : tile) * S * 32 + lane;
        for (int c = 0; c < nc; c++) {
            const int slot = c % kIluFaceSlots, s0 = (FWD ? c : nc - 1 - c) * kIluC;
            if (c >= kIluFaceSlots)
                ilu_mbar_wait(fempty + slot, (unsigned)(c / kIluFaceSlots - 1) & 1u, err, gave_up);
            gave_up = __any_sync(0xffffffffu, gave_up);
            double val[kIluC];
            unsigned long long t0 = 0;
            for (unsigned it = 0;; it++) {
                bool ok = true;
#pragma unroll
                for (int u = 0; u < kIluC; u++) {
                    const int st = s0 + u + (FWD ? 15 : -15);     // the upstream tile's step of the same cell column
                    val[u] = 0.0;
                    if (has && st >= 0 && st < S) ok = ilu_face_load(src + (long long)st * 32, val[u], tag) && ok;
                }
                if (__all_sync(0xffffffffu, ok) || gave_up) break;
                if ((it & 63) == 0) {
                    const unsigned long long now = ilu_now();
                    if (it == 0) t0 = now;
                    else if (now - t0 > 1000000000ull || *(volatile int*)err != 0) gave_up = true;
                    gave_up = __any_sync(0xffffffffu, gave_up);
                    if (gave_up && lane == 0) atomicExch(err, 1);
                }
            }
#pragma unroll
            for (int u = 0; u < kIluC; u++) fring[(slot * kIluC + u) * 32 + lane] = val[u];
            __syncwarp();
            if (lane == 0) ilu_mbar_arrive(ffull + slot);
        }
        return;
    }

    if (warp == kIluT / 32 + 2) {                                 // the face-out warp
        // after each step's barrier the tile's own two faces, for the tiles
        // downstream: lanes 0..15 the y-face line tz = lane, lanes 16..31 the
        // z-face line ty = lane - 16
        const int q = lane & 15, e = FWD ? 15 : 0;
        const double* src = sh + (lane < 16 ? e + kIluTY * q : q + kIluTY * e);
        uint4* face = faces + ((long long)tile * S + (FWD ? 0 : S - 1)) * 32 + lane;
        for (int st = 0; st < S; st++) {
            asm volatile("bar.sync 1, %0;" ::"n"(kIluT + 32) : "memory");
            ilu_face_store(face, src[((st + 1) & 1) * kIluT], tag);
            face += FWD ? 32 : -32;
        }
        return;
    }

    // the line threads
    const int ty = tid % kIluTY, tz = tid / kIluTY;
    const bool edge_y = FWD ? ty == 0 : ty == kIluTY - 1, edge_z = FWD ? tz == 0 : tz == kIluTZ - 1;
    double* vp = v + ((long long)tile * S + (FWD ? 0 : S - 1)) * kIluT + tid;   // this step's value
    constexpr int DIR = FWD ? 1 : -1;
    const double* ring_t = ring + tid;
    double a[kIluC][NK], r[kIluC], an[kIluC][NK], rn[kIluC];
    // one step's operands of the chunk in `slot`; the steps of a chunk are
    // taken in the sweep's direction
    auto operands = [&](int slot, int q, double (&ca)[NK], double& cr) {
        const double* in = ring_t + (size_t)slot * (NK + 1) * CT + (FWD ? q : kIluC - 1 - q) * kIluT;
#pragma unroll
        for (int k = 0; k < NK; k++) ca[k] = in[k * CT];
        cr = in[NK * CT];
    };
    ilu_mbar_wait(full, 0, err, gave_up);
#pragma unroll
    for (int q = 0; q < kIluC; q++) operands(0, q, a[q], r[q]);
    double own = 0.0;                                             // the line's previous value
    int p = 0, held = 0;                                          // held: the slot of this chunk's operands
    int slot = 0, phase = 0;                                      // of the next chunk's
    for (int c = 0; c < nc; c++) {
        const int fslot = c % kIluFaceSlots;
        const bool more = c + 1 < nc;
        if (++slot == kIluSlots) {
            slot = 0;
            phase ^= 1;
        }
        if (more) ilu_mbar_wait(full + slot, (unsigned)phase, err, gave_up);
        ilu_mbar_wait(ffull + fslot, (unsigned)(c / kIluFaceSlots) & 1u, err, gave_up);
        const double* fr = fring + (size_t)fslot * kIluC * 32;
#pragma unroll
        for (int q = 0; q < kIluC; q++) {
            const int u = FWD ? q : kIluC - 1 - q;
            const double ny = *(edge_y ? fr + u * 32 + tz : sh + p * kIluT + tid - DIR);
            const double nz = *(edge_z ? fr + u * 32 + 16 + ty : sh + p * kIluT + tid - DIR * kIluTY);
            double aux = r[q];
            if constexpr (FWD) {
                aux -= a[q][0] * nz;
                aux -= a[q][1] * ny;
                aux -= a[q][2] * own;
                own = aux;
            } else {
                aux -= a[q][0] * own;
                aux -= a[q][1] * ny;
                aux -= a[q][2] * nz;
                const double q0 = aux * a[q][NK - 1];
                own = fma(fma(-q0, a[q][NK - 2], aux), a[q][NK - 1], q0);
            }
            p ^= 1;
            sh[p * kIluT + tid] = own;
            // the next chunk's operands of this step, in the shadow of the barrier
            if (more) operands(slot, q, an[q], rn[q]);
            *vp = own;
            vp += DIR * kIluT;
            asm volatile("bar.sync 1, %0;" ::"n"(kIluT + 32) : "memory");
        }
        // this chunk's slots are free: its operands have been used, not only
        // asked for (an arrival may overtake shared loads in flight, and the
        // next copy into the slot would reach them)
        if (lane == 0) {
            ilu_mbar_arrive(fempty + fslot);
            ilu_mbar_arrive(empty + held);
        }
        held = slot;
#pragma unroll
        for (int q = 0; q < kIluC; q++) {
#pragma unroll
            for (int k = 0; k < NK; k++) a[q][k] = an[q][k];
            r[q] = rn[q];
        }
    }
}

}  // namespace lsg
