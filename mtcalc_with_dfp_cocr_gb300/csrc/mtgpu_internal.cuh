// Internal declarations shared by the libmtgpu translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <utility>
#include <vector>

#include "../../include/mtgpu.h"

namespace mtgpu {

// --------------------------------------------------------------- errors
#define MTGPU_TRY(expr)                                                        \
    do {                                                                       \
        cudaError_t e_ = (expr);                                               \
        if (e_ != cudaSuccess) {                                               \
            ::mtgpu::set_last_error(e_, #expr, __FILE__, __LINE__);           \
            return MTGPU_ERR_CUDA;                                             \
        }                                                                      \
    } while (0)

#define MTGPU_CHECK_ARG(cond, msg)                                             \
    do {                                                                       \
        if (!(cond)) {                                                         \
            ::mtgpu::set_last_message(msg);                                    \
            return MTGPU_ERR_ARG;                                              \
        }                                                                      \
    } while (0)

void set_last_error(cudaError_t e, const char *what, const char *file, int line);
void set_last_message(const char *msg);

constexpr int kSlice = 32;          // SELL slice height = one warp of rows
constexpr int kThreads = 256;       // default block size for row/edge kernels

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// ------------------------------------------------ device matrix (SELL-32)
// Full (both triangles) complex-symmetric matrix in sliced ELL with slice
// height 32.  Every row is split into complex slots (diagonal and parallel
// edge pairs: 16-byte values) and real slots (perpendicular pairs: 8-byte
// values).  Slot k of row (32*s + l) lives at sptr[s] + 32*k + l, so a warp
// reading one slot of its 32 rows touches one contiguous segment.
struct SellMatrix {
    int nb = 0;                 // rows (edges)
    int nslices = 0;
    long long nnz_c = 0, nnz_r = 0;          // stored entries without padding
    long long len_c = 0, len_r = 0;          // stored slots with padding
    int *d_wc = nullptr, *d_wr = nullptr;    // slice widths [nslices]
    long long *d_pc = nullptr, *d_pr = nullptr;  // slice offsets [nslices+1]
    int *d_col_c = nullptr, *d_col_r = nullptr;
    double2 *d_val_c = nullptr;
    double *d_val_r = nullptr;
    int *d_diag_slot = nullptr;   // complex slot index of the diagonal, per row
    int *d_nc = nullptr, *d_nr = nullptr;   // complex / real entries per row
    void release();
};

// Builds the SELL matrix from the reference lower 2x2-block storage that is
// already resident on the device (0-based arrays).
int sell_from_block2x2_device(int nb, const int *d_ig, const int *d_jg, const int *d_idi,
                              const int *d_ijg, const double *d_di, const double *d_gg,
                              int nnz_lower, SellMatrix &A, cudaStream_t st);

// y = A x  (x, y complex interleaved, device)
void sell_spmv(const SellMatrix &A, const double2 *x, double2 *y, cudaStream_t st);
// y = b - A x
void sell_residual(const SellMatrix &A, const double2 *b, const double2 *x, double2 *y,
                   cudaStream_t st);

// ------------------------------------------------ folded preconditioner
struct Folded {
    int n = 0, m = 0;                  // edges, interior conductive nodes
    int *d_gp = nullptr, *d_gj = nullptr;   double *d_gv = nullptr;   // G   (CSR, m rows)
    int *d_tp = nullptr, *d_tj = nullptr;   double *d_tv = nullptr;   // G^T (CSR, n rows)
    // G^T of a conforming mesh in compact form: per edge the G rows of its
    // first (-1/2) and second (+1/2) node, -1 where the node has no row;
    // null on meshes with T-matrix nodes
    int2 *d_tn = nullptr;
    double2 *d_da = nullptr;           // 1/diag(A)
    double2 *d_ds = nullptr;           // 1/diag(G A G^T)
    double2 *d_h = nullptr;            // node work vector
    void release();
};

// Host construction of G and G^T (FoldedPreconditioner.cpp:68-259 semantics),
// uploaded to the device.
int folded_build_g(const mtgpu_mesh_desc &mesh, Folded &P, cudaStream_t st);

// Device copies of the mesh tables that the set-up stages read (0-based)
struct DevMesh {
    int kpar = 0, nb = 0, nn = 0, nver_stride = 8, nmat = 0;
    const double *xyz = nullptr;            // [nn][3]; null where not needed
    const int *nver = nullptr;              // [kpar][nver_stride]
    const int *nvkat = nullptr;             // [kpar]
    const int *edges = nullptr;             // [nb][2]
    const double *sigflag = nullptr;        // [nmat]: > 0 for conductive materials
    const unsigned char *bnode = nullptr;   // [nn]: Dirichlet nodes
};
// A DevMesh over uploads of a host mesh description (or over tables
// already on the device plus the uploaded material flags); the uploads are
// freed with the object
struct DevMeshUpload {
    DevMesh view;
    int *nver = nullptr, *nvkat = nullptr, *edges = nullptr;
    double *xyz = nullptr, *sigflag = nullptr;
    unsigned char *bnode = nullptr;
    int upload(const mtgpu_mesh_desc &m, const double *xyz_host, cudaStream_t st);
    int over_device(int kpar, int nb, int nn, int nver_stride, const double *d_xyz,
                    const int *d_nver, const int *d_nvkat, const int *d_edges,
                    const unsigned char *d_bnode, const double *sigflag_host, int nmat,
                    cudaStream_t st);
    void release();
    ~DevMeshUpload() { release(); }
};
// G and G^T built on the device (same rows, entries and order as
// folded_build_g); *conforming = false, and nothing built, when an edge
// has a node beyond nn (T-matrix meshes: folded_build_g handles them)
int folded_build_g_device(const DevMesh &dm, Folded &P, cudaStream_t st, bool *conforming);
// G and G^T for a solver set-up: on the device from dm (or from an upload of
// the host mesh description when dm is null) where the mesh is conforming,
// else by the host construction
int folded_build_g_auto(const mtgpu_mesh_desc &mesh, const DevMesh *dm, Folded &P, cudaStream_t st);
// exclusive prefix sum: out[0..n] (out[n] = total), *total on the host
int dev_exclusive_scan(const int *d_in, long long n, int *d_out, long long *total, cudaStream_t st);
// D_A and D_S from the device matrix.
int folded_build_diag(const SellMatrix &A, Folded &P, cudaStream_t st);
// y = D_A x + G^T D_S G x
void folded_apply(const Folded &P, const double2 *x, double2 *y, cudaStream_t st);

// ------------------------------------------------ COCR solver state
struct Ctl;   // device control block (cocr.cu)
struct CocrSolver {
    SellMatrix A;
    Folded P;
    cudaStream_t st = nullptr;
    int nb = 0;
    int grid = 0;                 // blocks of the reduction kernels
    // one-kernel iterations (k_small64): blocks (0: not used), threads and rows per thread
    int g_small = 0, small_threads = 0, small_items = 0;
    double2 *r = nullptr, *p = nullptr, *s = nullptr, *z = nullptr, *a = nullptr,
            *w = nullptr, *sm = nullptr;
    double *partials = nullptr;
    Ctl *ctl = nullptr;           // device
    Ctl *hctl = nullptr;          // pinned host mirror
    cudaGraphExec_t graph = nullptr;
    int graph_iters = 0;
    void release();
};
int cocr_alloc(CocrSolver &S);
int cocr_solve(CocrSolver &S, const double2 *b, double2 *x, double eps, int maxiter,
               int stop_true, int iters_per_launch, mtgpu_solve_stats *stats);
void note_launches(unsigned long long k);

// ------------------------------------------------ small device helpers
__host__ __device__ inline double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ inline double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ inline double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a / b with scaling against overflow (Smith's algorithm)
__host__ __device__ inline double2 cdiv(double2 a, double2 b)
{
    if (fabs(b.x) >= fabs(b.y)) {
        const double r = b.y / b.x, d = b.x + b.y * r;
        return make_double2((a.x + a.y * r) / d, (a.y - a.x * r) / d);
    }
    const double r = b.x / b.y, d = b.x * r + b.y;
    return make_double2((a.x * r + a.y) / d, (a.y * r - a.x) / d);
}

// Programmatic dependent launch: the iteration's kernels are launched with
// the programmatic-serialization attribute, so the next grid is scheduled
// while the one before it drains; each of them waits here, before its first
// access to memory, until the grid before it has completed and its writes
// are visible (a no-op for a kernel launched without the attribute).  No
// kernel lets the next one's blocks be placed before its own have exited:
// placed early they share the SMs unevenly (launch_dependents at a kernel's
// start: FP64 solver on 45,000 edges 20.3 against 15.5 ms a solve, survey
// solver 3 % slower; before its grid sum: 16.7 ms, survey solver 1 %).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... K, typename... A>
void pdl(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// One component of a / b (c = 0 real, 1 imaginary): one divide (500 cycles here)
// deep, where cdiv's scaling by a quotient takes two.  |b|^2 as it stands where
// a and b are far inside FP64's range; else b is scaled by the power of two
// that brings its larger component to [1, 2), which changes no bit of a
// quotient that needs none (a zero, infinite or NaN b stays one).
__device__ __forceinline__ double cquot_part(double2 a, double2 b, int c)
{
    const int ea = max(__double2hiint(a.x) & 0x7ff00000, __double2hiint(a.y) & 0x7ff00000),
              eb = max(__double2hiint(b.x) & 0x7ff00000, __double2hiint(b.y) & 0x7ff00000);
    double s = 1.0;
    if (ea > (1023 + 500) << 20 || abs(eb - (1023 << 20)) > 400 << 20) {
        s = __hiloint2double(max(0x7fe00000 - eb, 0x00100000), 0);
        b = make_double2(b.x * s, b.y * s);
    }
    const double d = b.x * b.x + b.y * b.y;
    const double q = (c == 0 ? a.x * b.x + a.y * b.y : a.y * b.x - a.x * b.y) / d;
    return s == 1.0 ? q : q * s;
}
// both components, their divides side by side (two lanes with one each take
// 500 cycles, one lane with both 1000)
__device__ __forceinline__ double2 cquot(double2 a, double2 b)
{
    return make_double2(cquot_part(a, b, 0), cquot_part(a, b, 1));
}

// Barrier of all blocks of a cooperative launch on a counter that starts at 0.
// Everything a block stored before arrive() is visible to all blocks after
// wait() (to loads other than of the read-only path).  The wait is bounded:
// the blocks of a cooperative launch are resident together, so it ends; if it
// did not, the block marks the solve as failed and leaves instead of hanging.
// The other blocks may still pass that barrier (the late block had arrived at
// it) and end the launch as if nothing had happened, so the mark is a word that
// kernels only ever set: the launches after it end at their start, and the
// host, which alone clears it (with the counters) when a solve begins, fails
// the solve whatever its state says.
constexpr int kBarPolls = 1 << 22;     // about 2 s
struct GridBarrier {
    unsigned int *ctr;
    unsigned int target = 0;
    __device__ __forceinline__ void arrive()
    {
        __syncthreads();
        target += gridDim.x;
        if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    }
    // false: the other blocks did not arrive in `polls` polls, and *failed, the
    // mark in device memory, is set
    __device__ __forceinline__ bool wait(int *late, int *failed, int polls)
    {
        if (threadIdx.x == 0) {
            unsigned int v = 0;
            int q = 0;
            for (; q < polls; q++) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
                if ((int)(v - target) >= 0) break;
            }
            if (q == polls) {
                *late = 1;
                *(volatile int *)failed = 1;
            }
        }
        __syncthreads();
        return *late == 0;
    }
};
// MTGPU_BARRIER_POLLS (environment) makes a wait run out in a test: it lowers
// the bound of the FP64 solver's waits, and leaves a survey's counter one short
// (there the bound is a constant: the loop without one costs up to 2 % of an
// iteration)
inline int barrier_polls()
{
    const char *e = getenv("MTGPU_BARRIER_POLLS");
    const int n = e ? atoi(e) : 0;
    return n > 0 ? n : kBarPolls;
}
// A one-kernel launch needs its blocks resident together, so small solves from
// several threads follow one another where the separate kernels' overlap:
// MTGPU_ONE_KERNEL=0 (environment, read when a solver is set up) is for programs
// that run many.  Milliseconds a solve from 1, 2, 4, 8 threads, in one kernel and in
// separate ones: 45,000 edges x 2 systems 7.3 6.9 6.8 6.7 and 8.9 5.5 3.6 3.5; 26,500 x 1 4.1
// 3.6 3.6 3.6 and 6.3 3.3 1.9 1.3; FP64 on 45,000 8.9 8.8 8.7 8.7 and 14.2 8.5 6.1 4.8.
inline bool one_kernel_wanted()
{
    const char *e = getenv("MTGPU_ONE_KERNEL");
    return !(e && *e == '0');
}
// the total of output o of the blocks' partials part[output][block], from G
// lanes of a warp (j: the lane among them), in all of them; 8 loads in flight
template <int G>
__device__ __forceinline__ double grid_total(const double *part, int o, int j)
{
    constexpr int U = 8;
    const int B = gridDim.x;
    double s = 0.0;
    for (int q0 = j; q0 < B; q0 += U * G) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = q0 + u * G < B ? __ldcg(part + (size_t)o * B + q0 + u * G) : 0.0;
#pragma unroll
        for (int h = 1; h < U; h <<= 1)
#pragma unroll
            for (int u = 0; u + h < U; u += 2 * h) v[u] += v[u + h];
        s += v[0];
    }
#pragma unroll
    for (int d = G / 2; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    return s;
}

// Counts this block on a ticket; the blocks that arrived before.  Called by
// one thread after a barrier: release of the block's stores, which the barrier
// ordered before it, acquire of those of the blocks counted before.
__device__ __forceinline__ unsigned int count_arrival(unsigned int *ticket)
{
    unsigned int seen;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(seen) : "l"(ticket) : "memory");
    return seen;
}

// device allocation helpers (record the failing call)
template <class T>
int dev_alloc(T **p, size_t count)
{
    *p = nullptr;
    if (count == 0) count = 1;
    MTGPU_TRY(cudaMalloc((void **)p, count * sizeof(T)));
    return MTGPU_OK;
}
template <class T>
void dev_free(T *&p)
{
    if (p) cudaFree((void *)p);
    p = nullptr;
}

}  // namespace mtgpu

// opaque handle of the C ABI
struct mtgpu_cocr_s {
    mtgpu::CocrSolver S;
    bool own_stream = false;
};

namespace mtgpu {
int make_stream(mtgpu_cocr_s *c, void *stream);
double now_seconds();

// MTGPU_TRACE=1 (environment): the phases of a set-up on stderr, each
// after a synchronisation of its stream so that device work is charged to
// the phase that launched it; MTGPU_TRACE=2: host time only, no
// synchronisation (where the host itself waits)
struct PhaseTrace {
    bool on = false, sync = true;
    cudaStream_t st;
    const char *what;
    double t0 = 0.0, last = 0.0;
    PhaseTrace(cudaStream_t s, const char *w) : st(s), what(w)
    {
        const char *e = getenv("MTGPU_TRACE");
        on = e && (*e == '1' || *e == '2');
        sync = !(e && *e == '2');
        t0 = last = now_seconds();
    }
    void mark(const char *phase)
    {
        if (!on) return;
        if (sync) cudaStreamSynchronize(st);
        const double now = now_seconds();
        fprintf(stderr, "[mtgpu] %s %-22s %8.2f ms (total %8.2f)\n", what, phase, 1e3 * (now - last),
                1e3 * (now - t0));
        last = now;
    }
};
}  // namespace mtgpu
