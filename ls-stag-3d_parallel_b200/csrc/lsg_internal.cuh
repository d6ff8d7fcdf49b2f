// Internal declarations of the B200 pressure-Poisson solver library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>
#include <vector>

#include "../../include/lsstag_b200.h"

namespace lsg {

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
struct Error {
    int code;
    std::string msg;
};

#define LSG_CUDA(call)                                                                    \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            throw ::lsg::Error{LSG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    } while (0)

// every kernel launch of the library is followed by this check, which also
// counts launches (reported per solve in lsg_stats.kernel_launches)
extern thread_local long long g_launches;
#define LSG_CHECK_LAUNCH()              \
    do {                                \
        ::lsg::g_launches++;            \
        LSG_CUDA(cudaGetLastError());   \
    } while (0)

#define LSG_REQUIRE(cond, code, text)                  \
    do {                                               \
        if (!(cond)) throw ::lsg::Error{(code), (text)}; \
    } while (0)

// ---------------------------------------------------------------------------
// per-call temporaries: stream-ordered allocations from a context's own memory
// pool, released on the context's stream when they go out of scope.  The
// pool keeps freed memory (release threshold: never), so a call that repeats
// every time step reuses its blocks instead of a cudaMalloc / cudaFree pair
// (cudaFree synchronises the device).
// ---------------------------------------------------------------------------
template <typename T>
struct TmpBuf {
    T* p = nullptr;
    size_t n = 0;
    cudaStream_t s = nullptr;
    cudaMemPool_t pool = nullptr;
    TmpBuf(cudaStream_t stream, cudaMemPool_t mp) : s(stream), pool(mp) {}
    TmpBuf(const TmpBuf&) = delete;
    TmpBuf& operator=(const TmpBuf&) = delete;
    ~TmpBuf() { release(); }
    void alloc(size_t count)
    {
        if (count == n && p) return;
        release();
        if (count == 0) return;
        cudaError_t e = cudaMallocFromPoolAsync((void**)&p, count * sizeof(T), pool, s);
        if (e != cudaSuccess) {
            p = nullptr;
            throw Error{LSG_ERR_NOMEM, std::string("stream-ordered allocation of ") +
                                           std::to_string(count * sizeof(T)) + " bytes: " + cudaGetErrorString(e)};
        }
        n = count;
    }
    void release()
    {
        if (p) cudaFreeAsync(p, s);
        p = nullptr;
        n = 0;
    }
    size_t bytes() const { return n * sizeof(T); }
};

// ---------------------------------------------------------------------------
// device buffers
// ---------------------------------------------------------------------------
template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }
    DevBuf& operator=(DevBuf&& o) noexcept
    {
        if (this != &o) { release(); p = o.p; n = o.n; o.p = nullptr; o.n = 0; }
        return *this;
    }
    ~DevBuf() { release(); }
    void alloc(size_t count)
    {
        if (count == n && p) return;
        release();
        if (count == 0) return;
        cudaError_t e = cudaMalloc(&p, count * sizeof(T));
        if (e != cudaSuccess) {
            p = nullptr;
            throw Error{LSG_ERR_NOMEM, std::string("cudaMalloc of ") + std::to_string(count * sizeof(T)) +
                                           " bytes: " + cudaGetErrorString(e)};
        }
        n = count;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    size_t bytes() const { return n * sizeof(T); }
};

// ---------------------------------------------------------------------------
// grids and stencils
// ---------------------------------------------------------------------------
struct Dims {
    int N = 0, M = 0, K = 0;
    long long n() const { return (long long)N * M * K; }
};

// Offsets of the fine-level 7-point operator, in the reference's CSR column
// order (b, s, w, p, e, n, t).
constexpr int kFineOffsets = 7;

// A box stencil operator on one grid level: coef[o * n + cell] multiplies the
// neighbour (x+ox, y+oy, z+oz).  Offsets outside the grid carry 0.
template <typename T>
struct Stencil {
    Dims d;
    int rx = 0, ry = 0, rz = 0;   // radius per dimension
    int noff = 0;                 // number of offsets
    std::vector<int> off;         // 3 * noff host copy (ox, oy, oz)
    DevBuf<int> d_off;            // 3 * noff on the device
    int center = -1;              // index of (0,0,0)
    DevBuf<T> coef;               // noff * n
};

// Line tridiagonal of one direction, stored per natural cell index:
//   lo[i] couples cell i to the previous cell of its line (0 at line start)
//   dinv[i] inverse pivot, up[i] (scaled) coupling to the next cell.
template <typename T>
struct LineFactor {
    DevBuf<T> lo, dinv, up;
};

// Multigrid level (precision T).
template <typename T>
struct Level {
    Dims d;
    Stencil<T> A;
    LineFactor<T> line[3];        // x, y, z
    bool oddN = false, oddM = false, oddK = false;   // parity of THIS level (fine side of the transfer)
    bool agglomerate = false;     // restriction to the next level is the 1/8 agglomeration
    DevBuf<T> r, c, ch;           // residual / right-hand side, correction, accumulated solution
};

struct CoarseLU {
    int n = 0;
    std::vector<double> L, U, scale;  // row-major n x n
    std::vector<int> perm;
    DevBuf<double> dL, dU, dscale;
    DevBuf<int> dperm;
};

template <typename T>
struct Hierarchy {
    std::vector<Level<T>> lev;    // lev[0] fine ... lev[L] coarsest
    CoarseLU lu;
    DevBuf<double> coarse_rhs, coarse_sol;
};

// ---------------------------------------------------------------------------
// reductions: deterministic two-stage (block partials + last-block sum)
// ---------------------------------------------------------------------------
struct Reducer {
    static constexpr int kMaxBlocks = 2048;   // default grid cap of the one-thread-per-cell kernels
    static constexpr int kCapBlocks = 8192;   // most blocks any reducing launch may use
    static constexpr int kSlots = 4;
    DevBuf<double> partial;       // kCapBlocks * kSlots
    DevBuf<unsigned int> counter; // one per concurrent reduction site
    void init()
    {
        partial.alloc((size_t)kCapBlocks * kSlots);
        counter.alloc(64);
        LSG_CUDA(cudaMemset(counter.p, 0, counter.bytes()));
    }
};

// FGMRES device-side scalars (one struct, device memory).
struct KrylovScalars {
    double H[64 * 65];      // column-major Hessenberg entries h[i + j*65]
    double cs[64], sn[64], y[64];
    double normW2;          // ||w||^2 of the latest Arnoldi vector
    double invNormW;        // 1 / ||w||
    // what the host reads when a cycle ends
    struct State {
        double norm_r;      // running |gamma|
        int it;
        int breakdown;
    } st;
    int done;               // 1 converged / capped
    int pad;
};

// The host's side of a solve in pinned memory: the flag that the kernels
// write each step, and the targets of the copies at a solve's end.
struct HostScalars {
    int flag;               // mapped: 2 finished, 1 not
    int ilu_err;
    double r2;              // ||b - A x||^2
    KrylovScalars::State st;
};

// ---------------------------------------------------------------------------
// dependent launches
//
// The V-cycle is a chain of kernels of a few microseconds on its lower levels,
// each waiting for the last block of the one before and then for its own
// start.  Its kernels are launched with programmatic stream serialization:
// the next one may be set up once every block of this one has started
// (dep_begin's first half) and waits in dep_begin's second half until this
// one's writes are visible.  Grids of up to 2048 threads per SM only: behind
// larger ones, several waves at these kernels' 64 to 255 registers, there is
// nothing to hide, and the waiting blocks take slots (256^3 FP32 solve 26.7
// against 26.3 ms; 64^3 2.86 against 2.94, 32 x 24 x 20 2.76 against 2.92,
// 150 x 90 x 70 6.89 against 7.36 ms with it).  Every kernel launched this way
// calls dep_begin<DEP>(pointers) before it reads or writes a vector; the
// pointers pass through it so that no load of them is moved ahead of the wait.
//
// That also splits the kernel's loads into those before and those after, and
// costs registers, launched dependently or not: the fused FP32 steps at 256^3
// took 76, 111 and 131 us with it (x, y, z) and 72, 100 and 125 without, the
// FP64 x and y steps 186 and 180 against 179 and 164.  The kernels that lose by
// it have a second instance, DEP false, which larger grids get.
// ---------------------------------------------------------------------------
template <bool DEP = true, typename... P>
__device__ __forceinline__ void dep_begin(P&... ptr)
{
    if constexpr (DEP) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        (([&] { asm volatile("" : "+l"(ptr)::"memory"); }()), ...);
    }
}

inline bool dep_grid(dim3 grid, dim3 block)
{
    return 1ull * grid.x * grid.y * grid.z * block.x * block.y * block.z <= 148ull * 2048;
}

template <typename... P, typename... A>
inline void launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = dep_grid(grid, block) ? 1 : 0;
    LSG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// The instance with dep_begin on grids that are launched dependently, the one
// without on larger ones.
template <typename... P, typename... A>
inline void launch_dep(void (*dep)(P...), void (*plain)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                       A... args)
{
    if (dep_grid(grid, block)) launch_dep(dep, grid, block, smem, s, args...);
    else plain<<<grid, block, smem, s>>>(static_cast<P>(args)...);
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
inline int grid_for(long long n, int block, int max_blocks = 148 * 16)
{
    long long g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > max_blocks) g = max_blocks;
    return (int)g;
}

}  // namespace lsg
