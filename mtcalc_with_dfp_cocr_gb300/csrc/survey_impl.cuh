// The batched survey solver's kernels and their launches for one lane count
// (systems padded to SP = 1, 2, ..., 32).  Every SP is a translation unit of
// its own (survey_sp.cu), so that they compile side by side; survey.cu holds
// the host side and calls Impl<SP>.
#pragma once
#include "survey.cuh"
#include "dfloat.cuh"

#include <algorithm>
#include <climits>

namespace mtgpu {
namespace sv {

using namespace dfl;

constexpr int kB = 256;   // threads per block of every survey kernel
enum : int { kRun = 1 };

__device__ __forceinline__ long long slot(const long long *p, int row, int k)
{
    return p[row / kSlice] + (long long)k * kSlice + (row % kSlice);
}
__device__ __forceinline__ df d2f(float2 v) { return df{v.x, v.y}; }
__device__ __forceinline__ dfc from_d2(double2 v) { return dfc{from_double(v.x), from_double(v.y)}; }

// ---- per-system sums over the grid
// Thread t carries N partial sums of system t % SP (SP <= 32 divides the
// warp); the outputs are numbered n SP + k, W = N SP of them.  Every order
// below is fixed, so the totals are run-to-run identical.
//
// Measured on 45,000 edges x 2 systems, where nothing else takes long: with
// FP64 shuffle trees k_update took 22 us, 13k of its 21k active cycles in the
// FP64 pipe and another 25k cycles in the last block alone.
template <int SP, int N, int NT>
struct GridSum {
    static constexpr int W = N * SP;
    static constexpr int SLOTS = NT / 32 * W;      // shared float4 slots
    // every thread has float4 partials of output t % W (W <= NT): the total
    // in threads t < W
    static __device__ __forceinline__ float4 block_rows(float4 v, float4 *sm)
    {
        const int t = threadIdx.x;
        if constexpr (W < 32) {
#pragma unroll
            for (int o = 16; o >= W; o >>= 1) {
                float4 u;
                u.x = __shfl_xor_sync(0xffffffffu, v.x, o);
                u.y = __shfl_xor_sync(0xffffffffu, v.y, o);
                u.z = __shfl_xor_sync(0xffffffffu, v.z, o);
                u.w = __shfl_xor_sync(0xffffffffu, v.w, o);
                v = tf4_add(v, u);
            }
            if ((t & 31) < W) sm[(t >> 5) * W + (t & 31)] = v;
            return columns<NT / 32>(sm);
        } else {
            sm[t] = v;
            return columns<NT / W>(sm);
        }
    }
    // the sum of R rows of W slots, pairwise
    template <int R>
    static __device__ __forceinline__ float4 columns(const float4 *sm)
    {
        __syncthreads();
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (threadIdx.x < W) {
            float4 v[R];
#pragma unroll
            for (int q = 0; q < R; q++) v[q] = sm[q * W + threadIdx.x];
#pragma unroll
            for (int h = 1; h < R; h <<= 1)
#pragma unroll
                for (int q = 0; q + h < R; q += 2 * h) v[q] = tf4_add(v[q], v[q + h]);
            s = v[0];
        }
        return s;
    }
    // the block's totals in threads t < W: a warp halves the number of values
    // per lane while it halves the lanes per value (N + log2 adds instead of
    // N log2), then thread t < W adds the warps' sums
    static __device__ __forceinline__ float4 block(const tf (&v)[N], float4 *sm)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        bool big = false;
#pragma unroll
        for (int n = 0; n < N; n++) big |= fabsf(v[n].a) >= kTfBig;
        big = __any_sync(0xffffffffu, big);
        tf u[N];
#pragma unroll
        for (int n = 0; n < N; n++) u[n] = big ? tf_scale(v[n], kTfDown) : v[n];
        int cnt = N, first = 0, dup = 0;
#pragma unroll
        for (int o = 16; o >= SP; o >>= 1) {
            if (cnt > 1) {
                const int h = cnt / 2;
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < (N + 1) / 2; i++)
                    if (i < h) {
                        const tf mine = up ? u[i + h] : u[i], give = up ? u[i] : u[i + h];
                        u[i] = tf_add(mine, shfl(give, o));
                    }
                first += up ? h : 0;
                cnt = h;
            } else {
                u[0] = tf_add(u[0], shfl(u[0], o));
                dup |= o;
            }
        }
        if (!(lane & dup)) {
#pragma unroll
            for (int i = 0; i < N; i++)
                if (i < cnt) sm[warp * W + (first + i) * SP + lane % SP] = tf_pack(u[i], big ? 1.f : 0.f);
        }
        return columns<NT / 32>(sm);
    }
    static __device__ __forceinline__ tf shfl(tf x, int o)
    {
        return tf{__shfl_xor_sync(0xffffffffu, x.a, o), __shfl_xor_sync(0xffffffffu, x.b, o),
                  __shfl_xor_sync(0xffffffffu, x.c, o)};
    }
    // the totals of `rows` partials in threads t < W
    static __device__ __forceinline__ float4 rows(const float4 *part, int rows, float4 *sm)
    {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int i = threadIdx.x; i < rows * W; i += NT) s = tf4_add(s, __ldcg(part + i));
        __syncthreads();
        return block_rows(s, sm);
    }
};

// Blocks per first-level group of a grid sum.  With few systems the block
// that finishes last adds all block partials (456 blocks x 2 systems: seven
// loads a thread); with 8 lanes and more that would be thousands of partials
// on one SM (456 x 32 x 4: 14 us in FP64), so the last block of every group of
// 24 adds the group's, and the last group's adds the groups'.
constexpr int kGroupBlocks = 24;
constexpr int kTicketSlots = 256;     // float4 slots before the partials: up to 1023 groups
template <int SP>
constexpr int group_blocks()
{
    return SP >= 8 ? kGroupBlocks : INT_MAX;
}
inline size_t partial_slots(int blocks, int SP)
{
    return kTicketSlots + ((size_t)blocks + ceil_div(blocks, kGroupBlocks)) * 4 * SP;
}

// Per-system sums over the grid: true in the block that finishes last, with
// the totals in tot[n][k].
template <int SP, int N, int NT = kB>
__device__ bool sys_grid_sum(const tf (&v)[N], float4 *partials, double (*tot)[32])
{
    using S = GridSum<SP, N, NT>;
    constexpr int W = S::W;
    __shared__ float4 sm[S::SLOTS];
    __shared__ bool last;
    unsigned int *tickets = reinterpret_cast<unsigned int *>(partials);
    float4 *part = partials + kTicketSlots;
    float4 s = S::block(v, sm);
    // one level: this block's sums to dst; whether it is the last of n blocks
    auto arrive = [&](float4 *dst, unsigned int *ticket, unsigned int n) {
        if (threadIdx.x < W) __stcg(dst + threadIdx.x, s);
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();      // the block's stores, ordered by the barrier
            last = atomicAdd(ticket, 1u) == n - 1;
            if (last) {
                *ticket = 0u;
                __threadfence();
            }
        }
        __syncthreads();
        return last;
    };
    if constexpr (group_blocks<SP>() == INT_MAX) {
        if (!arrive(part + (size_t)blockIdx.x * W, tickets, gridDim.x)) return false;
        s = S::rows(part, gridDim.x, sm);
    } else {
        const int G = kGroupBlocks, g = blockIdx.x / G, ng = (gridDim.x + G - 1) / G;
        const int nin = min(G, (int)gridDim.x - g * G);
        float4 *gpart = part + (size_t)gridDim.x * W;
        if (!arrive(part + (size_t)blockIdx.x * W, tickets + 1 + g, nin)) return false;
        s = S::rows(part + (size_t)g * G * W, nin, sm);
        if (!arrive(gpart + (size_t)g * W, tickets, ng)) return false;
        s = S::rows(gpart, ng, sm);
    }
    if (threadIdx.x < W) tot[threadIdx.x / SP][threadIdx.x % SP] = tf4_double(s);
    __syncthreads();
    return true;
}

// The same sums of FP64 values, in FP64 (the true residual): block partials
// in block order, shuffle trees, the last block's threads strided over them.
template <int SP, int N>
__device__ __forceinline__ void block_sum64(double (&v)[N], double (*smem)[kB / 32][SP])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int n = 0; n < N; n++) {
#pragma unroll
        for (int o = 16; o >= SP; o >>= 1) v[n] += __shfl_down_sync(0xffffffffu, v[n], o);
        if (lane < SP) smem[n][warp][lane] = v[n];
    }
    __syncthreads();
    if (threadIdx.x < SP) {
#pragma unroll
        for (int n = 0; n < N; n++) {
            double acc = 0.0;
            for (int q = 0; q < kB / 32; q++) acc += smem[n][q][threadIdx.x];
            v[n] = acc;
        }
    }
}
template <int SP, int N>
__device__ bool sys_grid_sum64(double (&v)[N], float4 *scratch, unsigned int *ticket,
                               double (*tot)[32])
{
    __shared__ double smem[N][kB / 32][SP];
    __shared__ bool last;
    double *partials = reinterpret_cast<double *>(scratch + kTicketSlots);
    block_sum64<SP, N>(v, smem);
    if (threadIdx.x < SP) {
#pragma unroll
        for (int n = 0; n < N; n++)
            partials[((size_t)n * gridDim.x + blockIdx.x) * SP + threadIdx.x] = v[n];
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    constexpr int G = kB / SP;
    const int k = threadIdx.x % SP, j = threadIdx.x / SP;
    double f[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
        double acc = 0.0;
#pragma unroll 4
        for (int q = j; q < (int)gridDim.x; q += G)
            acc += __ldcg(&partials[((size_t)n * gridDim.x + q) * SP + k]);
        f[n] = acc;
    }
    block_sum64<SP, N>(f, smem);
    if (threadIdx.x < SP) {
#pragma unroll
        for (int n = 0; n < N; n++) tot[n][threadIdx.x] = f[n];
    }
    if (threadIdx.x == 0) *ticket = 0u;
    __syncthreads();
    return true;
}

// Programmatic dependent launch: the iteration's kernels are launched with
// the programmatic-serialization attribute, so the next grid is scheduled
// while the one before it drains; each of them waits here, before its first
// access to memory, until the grid before it has completed and its writes
// are visible (a no-op for a kernel launched without the attribute).  Once
// its own blocks run, the grid lets the next one be scheduled behind it:
// launch latency then overlaps this grid's work (no grid has more blocks
// than fit at once, so waiting blocks never keep running ones out).
__device__ __forceinline__ void pdl_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Element i of a grid-stride sweep over n elements, forwards or backwards.
// Consecutive kernels of the iteration sweep in opposite directions, so
// that each starts on the end of what the previous one streamed, which is
// still in L2 (a 58 MB vector of two systems against ~126 MB of L2); only
// the order of the partial sums changes, and it is fixed.
__device__ __forceinline__ int sweep(int i, int n, int rev) { return rev ? n - 1 - i : i; }

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

struct Mat {
    const int *wc, *wr;
    const long long *pc, *pr;
    const int *col_c, *col_r;
    const float2 *kc, *mc, *kr;
};

// y = (K + i omega M) x for one (row, system): K x and M x accumulated
// separately, then combined.  Slots are processed in batches of CH: the
// batch's column indices and matrix values are loaded first, then all its x
// gathers are issued together, so CH gathers are in flight per thread.
// Offsets stay 32-bit inside a row; full batches carry no predicates.
__device__ __forceinline__ dfc from4(float4 v) { return dfc{df{v.x, v.y}, df{v.z, v.w}}; }
__device__ __forceinline__ float4 to4(dfc v) { return make_float4(v.re.h, v.re.l, v.im.h, v.im.l); }

template <int SP, int CH>
__device__ __forceinline__ dfc spmv_row(const Mat &A, int row, int k, df om,
                                        const float4 *__restrict__ x)
{
    const int sl = row >> 5, l = row & 31;
    const float4 *__restrict__ xk = x + k;
    acc kr_, ki_, mr_, mi_;
    {
        const long long b0 = A.pc[sl] + l;
        const int *__restrict__ cc = A.col_c + b0;
        const float2 *__restrict__ kk = A.kc + b0;
        const float2 *__restrict__ mm = A.mc + b0;
        const int n = A.wc[sl];
        int q = 0;
        for (; q + CH <= n; q += CH) {
            int c[CH];
            float2 kv[CH], mv[CH];
            float4 xv[CH];
#pragma unroll
            for (int j = 0; j < CH; j++) {
                c[j] = __ldg(cc + kSlice * (q + j));
                kv[j] = __ldg(kk + kSlice * (q + j));
                mv[j] = __ldg(mm + kSlice * (q + j));
            }
#pragma unroll
            for (int j = 0; j < CH; j++) xv[j] = __ldg(xk + c[j] * SP);
#pragma unroll
            for (int j = 0; j < CH; j++) {
                const df kd = d2f(kv[j]), md = d2f(mv[j]);
                const df xr{xv[j].x, xv[j].y}, xi{xv[j].z, xv[j].w};
                kr_.mac(kd, xr);
                ki_.mac(kd, xi);
                mr_.mac(md, xr);
                mi_.mac(md, xi);
            }
        }
        for (; q < n; q++) {
            const int c = __ldg(cc + kSlice * q);
            const df kd = d2f(__ldg(kk + kSlice * q)), md = d2f(__ldg(mm + kSlice * q));
            const float4 xv = __ldg(xk + c * SP);
            const df xr{xv.x, xv.y}, xi{xv.z, xv.w};
            kr_.mac(kd, xr);
            ki_.mac(kd, xi);
            mr_.mac(md, xr);
            mi_.mac(md, xi);
        }
    }
    {
        const long long b0 = A.pr[sl] + l;
        const int *__restrict__ cc = A.col_r + b0;
        const float2 *__restrict__ kk = A.kr + b0;
        const int n = A.wr[sl];
        int q = 0;
        for (; q + 2 * CH <= n; q += 2 * CH) {
            int c[2 * CH];
            float2 kv[2 * CH];
            float4 xv[2 * CH];
#pragma unroll
            for (int j = 0; j < 2 * CH; j++) {
                c[j] = __ldg(cc + kSlice * (q + j));
                kv[j] = __ldg(kk + kSlice * (q + j));
            }
#pragma unroll
            for (int j = 0; j < 2 * CH; j++) xv[j] = __ldg(xk + c[j] * SP);
#pragma unroll
            for (int j = 0; j < 2 * CH; j++) {
                const df kd = d2f(kv[j]);
                kr_.mac(kd, df{xv[j].x, xv[j].y});
                ki_.mac(kd, df{xv[j].z, xv[j].w});
            }
        }
        for (; q < n; q++) {
            const int c = __ldg(cc + kSlice * q);
            const df kd = d2f(__ldg(kk + kSlice * q));
            const float4 xv = __ldg(xk + c * SP);
            kr_.mac(kd, df{xv.x, xv.y});
            ki_.mac(kd, df{xv.z, xv.w});
        }
    }
    // y = Kx + i omega Mx
    const df mxr = mr_.get(), mxi = mi_.get();
    kr_.mac(neg(om), mxi);
    ki_.mac(om, mxr);
    return dfc{kr_.get(), ki_.get()};
}

__device__ __forceinline__ dfc csubd(dfc a, dfc b)
{
    return dfc{add(a.re, neg(b.re)), add(a.im, neg(b.im))};
}

// ------------------------------------------------------------ set-up
// the scalars that the row kernels read, in both forms
__device__ __forceinline__ void set_alpha(SysState &q, double2 v) { q.alpha = v; q.alpha_f = to4(from_d2(v)); }
__device__ __forceinline__ void set_beta(SysState &q, double2 v) { q.beta = v; q.beta_f = to4(from_d2(v)); }
__device__ __forceinline__ void set_mrs_w(SysState &q, double v)
{
    const df w = from_double(v);
    q.mrs_w = v;
    q.mrs_wf = make_float2(w.h, w.l);
}
// ... and on the host, for the states the set-up checks and timings start from
inline float4 host_c4(double2 v)
{
    const df r = from_double(v.x), i = from_double(v.y);
    return make_float4(r.h, r.l, i.h, i.l);
}
inline void host_scalars(SysState &q)
{
    const df w = from_double(q.mrs_w);
    q.alpha_f = host_c4(q.alpha);
    q.beta_f = host_c4(q.beta);
    q.mrs_wf = make_float2(w.h, w.l);
}

// s_m = r and ||r|| of the inner system A d = r (d = 0 initially, so its
// right-hand side is its residual): stage 2 and the x0 test
template <int SP>
__global__ void __launch_bounds__(kB)
k_init(int nb, const float4 *__restrict__ r, float4 *__restrict__ sm, SysState *sys, float4 *partials)
{
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    acc nr2;
    const int rpb = kB / SP;
    for (int row = blockIdx.x * rpb + threadIdx.x / SP; row < nb; row += gridDim.x * rpb) {
        if (!on) continue;
        const long long i = (long long)row * SP + k;
        const float4 v = r[i];
        const dfc rv = from4(v);
        sm[i] = v;
        nr2.mac(rv.re, rv.re); nr2.mac(rv.im, rv.im);
    }
    const tf v[1] = {tf_of(nr2)};
    __shared__ double tot[1][32];
    if (sys_grid_sum<SP, 1>(v, partials, tot) && threadIdx.x < SP) {
        SysState &q = sys[threadIdx.x];
        if (q.status == kRun) {
            const double rr = tot[0][threadIdx.x];
            q.residual = rr > 0.0 ? sqrt(rr) : 0.0;
            q.r_old = q.residual;
            q.residual_rel = 1.0;
            q.beta = make_double2(0.0, 0.0);
            q.beta_f = make_float4(0.f, 0.f, 0.f, 0.f);
            q.mrs_mode = 0;
            q.iter = 1;
            if (q.residual < 1e-30) {
                q.status = MTGPU_X0_NULL;
                q.iter = 0;
            } else if (q.maxiter < 1) {
                q.status = MTGPU_MAXITER;
            }
        }
    }
}

// h = D_S G (z + beta a); use_beta = 0: h = D_S G z
template <int SP>
__global__ void __launch_bounds__(kB)
k_node(int m, const int *__restrict__ gp, const int *__restrict__ gj, const float *__restrict__ gv,
       const float4 *__restrict__ ds, const float4 *__restrict__ z, const float4 *__restrict__ a,
       float4 *__restrict__ h, const SysState *sys, int use_beta, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    if (sys[k].status != kRun) return;
    const dfc be = from4(sys[k].beta_f);
    const int rpb = kB / SP;
    for (int vi = blockIdx.x * rpb + threadIdx.x / SP; vi < m; vi += gridDim.x * rpb) {
        const int v = sweep(vi, m, rev);
        const int j0 = __ldg(gp + v), j1 = __ldg(gp + v + 1);
        const float4 dsv = __ldg(ds + (long long)v * SP + k);
        acc hr, hi;
        for (int j = j0; j < j1; j++) {
            const long long idx = (long long)__ldg(gj + j) * SP + k;
            const float g = __ldg(gv + j);
            const float4 zv = __ldg(z + idx);
            dfc an = from4(zv);
            if (use_beta) an = caxpy(an, be, from4(__ldg(a + idx)));
            hr.macf(an.re, g);
            hi.macf(an.im, g);
        }
        h[(long long)v * SP + k] = to4(cmul(dfc{hr.get(), hi.get()}, from4(dsv)));
    }
}

// mode 1: a = z + beta a, w = D_A a + G^T h, (a, w) -> alpha; first: the
// iteration is the first of its group
// mode 0: w = D_A z + G^T h (preconditioner application, no reduction)
// Every input of an element is loaded before anything is stored.  p = s +
// beta p and x += alpha p are k_group's: reading s and p and x here and
// writing p and x were 5 of this kernel's 11 vector passes.
template <int SP>
__global__ void __launch_bounds__(kB)
k_edge(int n, const int *__restrict__ tp, const int *__restrict__ tj, const float *__restrict__ tv,
       const int2 *__restrict__ tn, const float4 *__restrict__ da, const float4 *__restrict__ h,
       const float4 *__restrict__ z, float4 *__restrict__ a, float4 *__restrict__ w, SysState *sys,
       float4 *partials, int mode, int first, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const dfc be = from4(sys[k].beta_f);
    acc awr, awi;
    const int rpb = kB / SP, stride = gridDim.x * rpb;
    // the compact G^T row of the next element is loaded one element ahead,
    // so that this element's h gathers issue with its other loads
    const int e_first = blockIdx.x * rpb + threadIdx.x / SP;
    int2 r2n = make_int2(-1, -1);
    if (tn && on && e_first < n) r2n = __ldg(tn + sweep(e_first, n, rev));
    for (int ei = e_first; ei < n; ei += stride) {
        if (!on) break;
        const int e = sweep(ei, n, rev);
        const long long idx = (long long)e * SP + k;
        // G^T row: compact (the rows of the edge's two nodes, -1/2 and +1/2
        // in that order) or the CSR of T-matrix meshes
        int j0, j1;
        int2 r2 = make_int2(-1, -1);
        if (tn) {
            r2 = r2n;
            if (ei + stride < n) r2n = __ldg(tn + sweep(ei + stride, n, rev));
            j0 = 0;
            j1 = (r2.x >= 0) + (r2.y >= 0);
        } else {
            j0 = __ldg(tp + e);
            j1 = __ldg(tp + e + 1);
        }
        const float4 zv = __ldg(z + idx), dav = __ldg(da + idx);
        float4 av = make_float4(0.f, 0.f, 0.f, 0.f);
        if (mode != 0) av = a[idx];
        float4 hv0 = make_float4(0.f, 0.f, 0.f, 0.f), hv1 = hv0;
        float t0 = 0.f, t1 = 0.f;
        if (tn) {
            // entries in the CSR's order: the first node's (if any), then the second's
            const int ra = r2.x >= 0 ? r2.x : r2.y, rb = r2.y;
            if (j1 > 0) {
                hv0 = __ldg(h + (long long)ra * SP + k);
                t0 = r2.x >= 0 ? -0.5f : 0.5f;
            }
            if (j1 > 1) {
                hv1 = __ldg(h + (long long)rb * SP + k);
                t1 = 0.5f;
            }
        } else {
            if (j1 > j0) {
                hv0 = __ldg(h + (long long)__ldg(tj + j0) * SP + k);
                t0 = __ldg(tv + j0);
            }
            if (j1 > j0 + 1) {
                hv1 = __ldg(h + (long long)__ldg(tj + j0 + 1) * SP + k);
                t1 = __ldg(tv + j0 + 1);
            }
        }
        dfc an;
        if (mode == 0) {
            an = from4(zv);
        } else {
            an = caxpy(from4(zv), be, from4(av));
            a[idx] = to4(an);
        }
        const dfc dv = cmul(an, from4(dav));
        acc wr, wi;
        wr.h = dv.re.h; wr.l = dv.re.l;
        wi.h = dv.im.h; wi.l = dv.im.l;
        if (j1 > j0) {
            wr.macf(df{hv0.x, hv0.y}, t0);
            wi.macf(df{hv0.z, hv0.w}, t0);
        }
        if (j1 > j0 + 1) {
            wr.macf(df{hv1.x, hv1.y}, t1);
            wi.macf(df{hv1.z, hv1.w}, t1);
        }
        for (int j = j0 + 2; j < j1 && !tn; j++) {       // T-matrix rows only
            const float4 hv = __ldg(h + (long long)__ldg(tj + j) * SP + k);
            const float t = __ldg(tv + j);
            wr.macf(df{hv.x, hv.y}, t);
            wi.macf(df{hv.z, hv.w}, t);
        }
        const dfc wn{wr.get(), wi.get()};
        w[idx] = to4(wn);
        awr.mac(an.re, wn.re);
        awr.mac(neg(an.im), wn.im);
        awi.mac(an.re, wn.im);
        awi.mac(an.im, wn.re);
    }
    if (mode == 0) return;
    const tf v[2] = {tf_of(awr), tf_of(awi)};
    __shared__ double tot[2][32];
    if (sys_grid_sum<SP, 2>(v, partials, tot) && threadIdx.x < SP) {
        SysState &q = sys[threadIdx.x];
        if (first) q.cnt = 0;
        if (q.status == kRun) {
            const double2 aw = make_double2(tot[0][threadIdx.x], tot[1][threadIdx.x]);
            if (fabs(aw.x) < 1e-40 && fabs(aw.y) < 1e-40) q.status = MTGPU_DIV_BY_ZERO;
            else set_alpha(q, cdiv(q.zs, aw));
        }
    }
}

// r -= alpha a, s -= alpha w, and the MRS smoothing of the residual
// (MRS.cpp:85-153): first the previous iteration's step of s_m, deferred to
// here where r and s_m are read anyway (mode 1: s_m = r, 2: s_m += w (r -
// s_m), on the r of that iteration), then the sums for this iteration's
// weight w = -(s_m, u) / ||u||^2, u = r - s_m, and for ||s_m|| after this
// iteration's step: ||s_m + w u||^2 = ||s_m||^2 + 2 w (s_m, u) + w^2 ||u||^2,
// or ||r||^2 (mode 1).  The new s goes to the group's next slot and alpha and
// beta into its record (k_group).  Every input of an element is loaded
// before anything is stored.
template <int SP>
__global__ void __launch_bounds__(kB)
k_update(int n, const float4 *__restrict__ a, const float4 *__restrict__ w, float4 *__restrict__ sm,
         float4 *__restrict__ r, const float4 *__restrict__ s_in, float4 *__restrict__ s_out,
         SysState *sys, float4 *hist, float4 *partials, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const dfc al = from4(sys[k].alpha_f);
    const dfc nal{neg(al.re), neg(al.im)};
    const int pm = sys[k].mrs_mode;
    const df pw = d2f(sys[k].mrs_wf);
    acc su, uu, nn, rr;
    const int rpb = kB / SP;
    const int stride = gridDim.x * rpb;
    // two elements per pass, all 10 loads issued before any store
    for (int e = blockIdx.x * rpb + threadIdx.x / SP; e < n; e += 2 * stride) {
        if (!on) break;
        const bool two = e + stride < n;
        float4 v[2][5];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (u == 1 && !two) break;
            const long long idx = (long long)sweep(e + u * stride, n, rev) * SP + k;
            v[u][0] = __ldg(a + idx); v[u][1] = __ldg(w + idx);
            v[u][2] = sm[idx]; v[u][3] = r[idx]; v[u][4] = __ldg(s_in + idx);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (u == 1 && !two) break;
            const long long idx = (long long)sweep(e + u * stride, n, rev) * SP + k;
            const dfc ro = from4(v[u][3]);
            dfc smv = from4(v[u][2]);
            if (pm == 1) {
                smv = ro;
            } else if (pm == 2) {
                acc tr, ti;
                tr.h = smv.re.h; tr.l = smv.re.l;
                ti.h = smv.im.h; ti.l = smv.im.l;
                tr.mac(pw, add(ro.re, neg(smv.re)));
                ti.mac(pw, add(ro.im, neg(smv.im)));
                smv = dfc{tr.get(), ti.get()};
            }
            const dfc rn = caxpy(ro, nal, from4(v[u][0]));
            r[idx] = to4(rn);
            s_out[idx] = to4(caxpy(from4(v[u][4]), nal, from4(v[u][1])));
            if (pm != 0) sm[idx] = to4(smv);
            const df ur = add(rn.re, neg(smv.re)), ui = add(rn.im, neg(smv.im));
            su.mac(smv.re, ur); su.mac(smv.im, ui);
            uu.mac(ur, ur); uu.mac(ui, ui);
            nn.mac(smv.re, smv.re); nn.mac(smv.im, smv.im);
            rr.mac(rn.re, rn.re); rr.mac(rn.im, rn.im);
        }
    }
    const tf v[4] = {tf_of(su), tf_of(uu), tf_of(nn), tf_of(rr)};
    __shared__ double tot[4][32];
    if (sys_grid_sum<SP, 4>(v, partials, tot) && threadIdx.x < SP) {
        SysState &q = sys[threadIdx.x];
        if (q.status == kRun) {
            const double s_u = tot[0][threadIdx.x], u_u = tot[1][threadIdx.x];
            const double n_n = tot[2][threadIdx.x], r_r = tot[3][threadIdx.x];
            const double wm = fabs(u_u) < 1e-100 ? 0.0 : -s_u / u_u;
            if (wm < 0.0) {
                q.mrs_mode = 0;
                q.res_next = q.residual;
            } else if (wm > 1.0) {
                q.mrs_mode = 1;
                q.res_next = r_r > 0.0 ? sqrt(r_r) : 0.0;
            } else {
                q.mrs_mode = 2;
                set_mrs_w(q, wm);
                const double m2 = n_n + 2.0 * wm * s_u + wm * wm * u_u;
                q.res_next = m2 > 0.0 ? sqrt(m2) : 0.0;
            }
            const int c = min(q.cnt, kGroupIters - 1);
            hist[2 * (threadIdx.x * kGroupIters + c)] = q.alpha_f;
            hist[2 * (threadIdx.x * kGroupIters + c) + 1] = q.beta_f;
            q.cnt = c + 1;
        }
    }
}

// Per-row tail of the SpMV kernels: store z = A s and accumulate (z, s).
// (The MRS smoothing of the residual runs in k_update.)
struct SpmvTail {
    acc zsr, zsi;
    __device__ __forceinline__ void row(long long i, dfc y, float4 sv4, float4 *__restrict__ z)
    {
        z[i] = to4(y);
        const dfc sv = from4(sv4);
        zsr.mac(y.re, sv.re); zsr.mac(neg(y.im), sv.im);
        zsi.mac(y.re, sv.im); zsi.mac(y.im, sv.re);
    }
    // grid totals -> stop test and beta (the last block only)
    template <int SP, int NT = kB>
    __device__ __forceinline__ void finish(SysState *sys, float4 *partials, int mode)
    {
        const tf v[2] = {tf_of(zsr), tf_of(zsi)};
        finish_v<SP, NT>(v, sys, partials, mode);
    }
    // the same from this thread's (z, s) re, im of system threadIdx.x % SP.
    // mode 1: the stop test on ||s_m|| of this iteration (k_update's
    // res_next), then beta; mode 0 (set-up): (z, s) only
    template <int SP, int NT = kB>
    static __device__ __forceinline__ void finish_v(const tf (&v)[2], SysState *sys,
                                                    float4 *partials, int mode)
    {
        __shared__ double tot[2][32];
        if (sys_grid_sum<SP, 2, NT>(v, partials, tot) && threadIdx.x < SP) {
            SysState &q = sys[threadIdx.x];
            if (q.status == kRun) {
                const double2 zs_new = make_double2(tot[0][threadIdx.x], tot[1][threadIdx.x]);
                if (mode == 0) {
                    q.zs = zs_new;
                } else {
                    q.residual = q.res_next;
                    q.residual_rel = q.residual / q.r_old;
                    set_beta(q, cdiv(zs_new, q.zs));
                    q.zs = zs_new;
                    if (q.residual_rel < q.eps_k) {
                        q.status = MTGPU_OK;
                    } else {
                        q.iter += 1;
                        if (q.iter > q.maxiter) q.status = MTGPU_MAXITER;
                    }
                }
            }
        }
    }
};

// z = A s, (z, s) -> stop test and beta.
// mode 0 (set-up): z = A s and (z, s) only.  x gathers straight from global
// memory, CH slots in flight per thread.
template <int SP, int CH>
__global__ void __launch_bounds__(kB, 3)
k_spmv(int nb, Mat A, const float2 *__restrict__ omega, const float4 *__restrict__ s,
       float4 *__restrict__ z,
       SysState *sys, float4 *partials, int mode)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const df om = d2f(omega[k]);
    SpmvTail tail;
    const int rpb = kB / SP;
    for (int row = blockIdx.x * rpb + threadIdx.x / SP; row < nb; row += gridDim.x * rpb) {
        if (!on) continue;
        const long long i = (long long)row * SP + k;
        const float4 sv4 = __ldg(s + i);
        tail.row(i, spmv_row<SP, CH>(A, row, k, om, s), sv4, z);
    }
    tail.finish<SP>(sys, partials, mode);
}

// y_k = (K + i omega_k M) x_k of one row for all SP systems in one thread:
// the row's column indices and matrix values are loaded once and serve
// every system (SP = 2: the x values of a column for both systems are one
// contiguous 32-byte pair).  Per system the products are summed in the same
// slot order as spmv_row.
template <int SP, int CH>
__device__ __forceinline__ void spmv_row_all(const Mat &A, int row, const df (&om)[SP],
                                             const float4 *__restrict__ x, dfc (&y)[SP])
{
    const int sl = row >> 5, l = row & 31;
    acc kr_[SP], ki_[SP], mr_[SP], mi_[SP];
    {
        const long long b0 = A.pc[sl] + l;
        const int *__restrict__ cc = A.col_c + b0;
        const float2 *__restrict__ kk = A.kc + b0;
        const float2 *__restrict__ mm = A.mc + b0;
        const int n = A.wc[sl];
        for (int q = 0; q < n; q += CH) {
            int c[CH];
            float2 kv[CH], mv[CH];
            float4 xv[CH][SP];
#pragma unroll
            for (int j = 0; j < CH; j++) {
                const bool in = q + j < n;
                c[j] = in ? __ldg(cc + kSlice * (q + j)) : -1;
                kv[j] = in ? __ldg(kk + kSlice * (q + j)) : make_float2(0.f, 0.f);
                mv[j] = in ? __ldg(mm + kSlice * (q + j)) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < CH; j++)
#pragma unroll
                for (int k = 0; k < SP; k++)
                    xv[j][k] = c[j] >= 0 ? __ldg(x + (long long)c[j] * SP + k)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < CH; j++) {
                if (c[j] < 0) break;
                const df kd = d2f(kv[j]), md = d2f(mv[j]);
#pragma unroll
                for (int k = 0; k < SP; k++) {
                    const df xr{xv[j][k].x, xv[j][k].y}, xi{xv[j][k].z, xv[j][k].w};
                    kr_[k].mac(kd, xr);
                    ki_[k].mac(kd, xi);
                    mr_[k].mac(md, xr);
                    mi_[k].mac(md, xi);
                }
            }
        }
    }
    {
        const long long b0 = A.pr[sl] + l;
        const int *__restrict__ cc = A.col_r + b0;
        const float2 *__restrict__ kk = A.kr + b0;
        const int n = A.wr[sl];
        for (int q = 0; q < n; q += 2 * CH) {
            int c[2 * CH];
            float2 kv[2 * CH];
            float4 xv[2 * CH][SP];
#pragma unroll
            for (int j = 0; j < 2 * CH; j++) {
                const bool in = q + j < n;
                c[j] = in ? __ldg(cc + kSlice * (q + j)) : -1;
                kv[j] = in ? __ldg(kk + kSlice * (q + j)) : make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int j = 0; j < 2 * CH; j++)
#pragma unroll
                for (int k = 0; k < SP; k++)
                    xv[j][k] = c[j] >= 0 ? __ldg(x + (long long)c[j] * SP + k)
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 2 * CH; j++) {
                if (c[j] < 0) break;
                const df kd = d2f(kv[j]);
#pragma unroll
                for (int k = 0; k < SP; k++) {
                    kr_[k].mac(kd, df{xv[j][k].x, xv[j][k].y});
                    ki_[k].mac(kd, df{xv[j][k].z, xv[j][k].w});
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < SP; k++) {
        const df mxr = mr_[k].get(), mxi = mi_[k].get();
        kr_[k].mac(neg(om[k]), mxi);
        ki_[k].mac(om[k], mxr);
        y[k] = dfc{kr_[k].get(), ki_[k].get()};
    }
}

// The SpMV with one thread per row serving both systems of a two-system
// batch (variants 16 + CH): half the matrix-slot loads of k_spmv, twice the
// independent work per thread.  Before the grid reduction every lane pair
// swaps partial sums so that lane l carries system l % 2, the layout
// sys_grid_sum expects.
template <int CH>
__global__ void __launch_bounds__(kB, 2)
k_spmv_r2(int nb, Mat A, const float2 *__restrict__ omega, const float4 *__restrict__ s,
          float4 *__restrict__ z,
          SysState *sys, float4 *partials, int mode)
{
    pdl_wait();
    constexpr int SP = 2;
    bool on[SP];
    df om[SP];
    SpmvTail tail[SP];
#pragma unroll
    for (int k = 0; k < SP; k++) {
        on[k] = sys[k].status == kRun;
        om[k] = d2f(omega[k]);
    }
    if (on[0] || on[1]) {
        for (int row = blockIdx.x * kB + threadIdx.x; row < nb; row += gridDim.x * kB) {
            dfc y[SP];
            spmv_row_all<SP, CH>(A, row, om, s, y);
#pragma unroll
            for (int k = 0; k < SP; k++) {
                if (!on[k]) continue;
                const long long i = (long long)row * SP + k;
                tail[k].row(i, y[k], __ldg(s + i), z);
            }
        }
    }
    const bool odd = threadIdx.x & 1;
    const acc z0[2] = {tail[0].zsr, tail[0].zsi}, z1[2] = {tail[1].zsr, tail[1].zsi};
    tf v[2];
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const tf mine = tf_of(odd ? z1[n] : z0[n]), give = tf_of(odd ? z0[n] : z1[n]);
        v[n] = tf_add(mine, GridSum<SP, 2, kB>::shfl(give, 1));
    }
    SpmvTail::finish_v<SP>(v, sys, partials, mode);
}

// ------------------------------------------------ matrix-free SpMV (tensor meshes)
// On a tensor mesh with RegularMeshBuilder's numbering the brick matrices
// factor: the curl-curl matrix B = D^T F D with D the 6 x 12 edge -> face
// circulation operator (entries +-1) and F block diagonal, per direction d
// (2 h_d / (h_t1 h_t2)) m, m = [[2/3, 1/3], [1/3, 2/3]] coupling the two
// faces of normal d; the edge mass matrix C is, per direction,
// (h_t1 h_t2 / h_d) m (x) m over the 4 parallel edges (both from the brick
// matrices of T_Brick.cpp:1361-1395 as oracle/mtcalc_oracle.c restates
// them).  So A s = D^T F_g D s + i omega M s with F_g, M regenerated from
// six weights per cell (wF / 3 and sigma wM / 9, double-float; the 1/3 and
// 1/9 make the remaining multipliers 1, 2, 4, exact) instead of 33 stored
// slots per row.  Variants 32 and 33 make two passes: the circulation of
// every face (k_mf_faces), then per edge the 4 faces through it, their
// neighbours along the normal and the 3 x 3 parallel edges of the 4 cells
// around it (k_mf_edges / k_mf_edges2: z and (z, s)).  Variant 35 forms
// g = F f per face straight from s (k_mf_gmarch) and sums the 4 g of each
// edge (k_mf_edges_g); variant 34 is one tiled kernel (mf_tile.cuh).
// Dirichlet edges (both nodes on the boundary) read as 0 and map to
// themselves, as in the assembled matrix.
struct MF {
    int nx, ny, nz;
    long long nfx, nfy, nfz, ncell;
    int plane, l3, l2;         // edges per node plane below the top one; per node line below / in it
    // strides of the index grids along x, y, z: faces of normal n (fs[n]),
    // cells (cs), and the edges of one direction away from the surface
    // (es = 3, l3, plane: every node before them has its +x, +y, +z edge)
    int fs[3][3], cs[3], es[3];
    int fb[3];                 // first face of each normal
    const unsigned *pos;       // row -> i | j << 10 | k << 20 | direction << 30 (plane by plane)
    const float2 *w;
    float4 *f;
    float4 *g;                 // F f (variant 35)
};

// the edge counts and index strides of M from its node lines nx, ny, nz
inline void mf_strides(MF &M)
{
    const int nx = M.nx, ny = M.ny;
    M.plane = (ny - 1) * (3 * nx - 1) + (2 * nx - 1);
    M.l3 = 3 * nx - 1;
    M.l2 = 2 * nx - 1;
    const int fsv[3][3] = {{1, nx, nx * (ny - 1)}, {1, nx - 1, (nx - 1) * ny},
                           {1, nx - 1, (nx - 1) * (ny - 1)}};
    for (int n = 0; n < 3; n++)
        for (int a = 0; a < 3; a++) M.fs[n][a] = fsv[n][a];
    M.cs[0] = 1;
    M.cs[1] = nx - 1;
    M.cs[2] = (nx - 1) * (ny - 1);
    M.es[0] = 3;
    M.es[1] = M.l3;
    M.es[2] = M.plane;
    M.fb[0] = 0;
    M.fb[1] = (int)M.nfx;
    M.fb[2] = (int)(M.nfx + M.nfy);
}

// first edge of node line (j, k): the node planes below, then the lines
// before it in its plane (edges are numbered node by node, each node's +x,
// +y, +z edge where present; the set-up verified this numbering)
__device__ __forceinline__ int mf_line(const MF &M, int j, int k)
{
    return k * M.plane + j * (k < M.nz - 1 ? M.l3 : M.l2);
}

// edge of direction d leaving node (i, j, k): the node's first edge
// mf_line + i (1 + [j < ny-1] + [k < nz-1]), then +x, +y, +z as present
// (32-bit: the set-up keeps edges x systems and faces x systems below 2^31)
__device__ __forceinline__ int mf_edge(const MF &M, int d, int i, int j, int k)
{
    const int ey = j < M.ny - 1, ex = i < M.nx - 1;
    int e = mf_line(M, j, k) + i * (1 + ey + (k < M.nz - 1));
    if (d >= 1) e += ex;
    if (d == 2) e += ey;
    return e;
}

// The matrix-free operator runs on lattice meshes only: every node of the
// outer surface, and no other, is a Dirichlet node, so the +d edge of node
// (i, j, k) is Dirichlet iff one of its two transverse node lines lies on
// the surface.  Every other edge has its two transverse coordinates inside,
// so its node and all nodes before it on its line have three edges: its
// number is k plane + j l3 + 3 i + d, and moving it by one node along an
// axis adds es[axis].
__device__ __forceinline__ bool mf_dirichlet(const MF &M, int d, int i, int j, int k)
{
    const bool bi = i == 0 || i == M.nx - 1, bj = j == 0 || j == M.ny - 1, bk = k == 0 || k == M.nz - 1;
    return d == 0 ? (bj || bk) : (d == 1 ? (bi || bk) : (bi || bj));
}
__device__ __forceinline__ int mf_edge_in(const MF &M, int d, int i, int j, int k)
{
    return k * M.plane + j * M.l3 + 3 * i + d;
}

// x of the +d edge of node (i, j, kk) for system k, 0 on Dirichlet edges
template <int SP>
__device__ __forceinline__ dfc mf_x(const MF &M, const float4 *__restrict__ x, int d, int i, int j,
                                    int kk, int k)
{
    if (mf_dirichlet(M, d, i, j, kk)) return dfc{df{0.f, 0.f}, df{0.f, 0.f}};
    return from4(__ldg(x + mf_edge_in(M, d, i, j, kk) * SP + k));
}

// k_node on a lattice mesh whose G rows are its interior nodes in node
// order (checked at set-up by k_g_lattice_check): row v is node (i, j, k)
// = v's position in the (nx-2) x (ny-2) x (nz-2) interior, and its entries
// are the node's six edges by increasing number, -z, -y, -x (+1/2), +x,
// +y, +z (-1/2), computed instead of read: the same products in the same
// order as k_node, without the CSR's dependent loads.
template <int SP>
__global__ void __launch_bounds__(kB)
k_node_lat(MF M, int m, const float4 *__restrict__ ds, const float4 *__restrict__ z,
           const float4 *__restrict__ a, float4 *__restrict__ h, const SysState *sys, int use_beta,
           int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    if (sys[k].status != kRun) return;
    const dfc be = from4(sys[k].beta_f);
    const int ix = M.nx - 2, iy = M.ny - 2;
    const int rpb = kB / SP;
    for (int vi = blockIdx.x * rpb + threadIdx.x / SP; vi < m; vi += gridDim.x * rpb) {
        const int v = sweep(vi, m, rev);
        const int i = v % ix + 1, t = v / ix, j = t % iy + 1, kk = t / iy + 1;
        const int e0 = mf_edge_in(M, 0, i, j, kk);
        const int es[6] = {e0 + 2 - M.plane, e0 + 1 - M.l3, e0 - 3, e0, e0 + 1, e0 + 2};
        float4 zv[6], av[6];
#pragma unroll
        for (int q = 0; q < 6; q++) {
            zv[q] = __ldg(z + (long long)es[q] * SP + k);
            av[q] = use_beta ? __ldg(a + (long long)es[q] * SP + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float4 dsv = __ldg(ds + (long long)v * SP + k);
        acc hr, hi;
#pragma unroll
        for (int q = 0; q < 6; q++) {
            dfc an = from4(zv[q]);
            if (use_beta) an = caxpy(an, be, from4(av[q]));
            const float g = q < 3 ? 0.5f : -0.5f;
            hr.macf(an.re, g);
            hi.macf(an.im, g);
        }
        h[(long long)v * SP + k] = to4(cmul(dfc{hr.get(), hi.get()}, from4(dsv)));
    }
}

// face t (faces numbered by normal, then z, y, x) -> normal n and position;
// 32-bit (the set-up keeps faces x systems below 2^31)
__device__ __forceinline__ void mf_face_pos(const MF &M, int t, int &n, int &i, int &j, int &kk)
{
    const int fx = (int)M.nfx, fy = (int)M.nfy;
    int q = t, a, b;
    if (q < fx) {
        n = 0;
        a = M.nx;
        b = M.ny - 1;
    } else if ((q -= fx) < fy) {
        n = 1;
        a = M.nx - 1;
        b = M.ny;
    } else {
        q -= fy;
        n = 2;
        a = M.nx - 1;
        b = M.ny - 1;
    }
    const int r = q / a;
    i = q - r * a;
    kk = r / b;
    j = r - kk * b;
}

// the circulation of system k's x around face (n, i, j, kk)
template <int SP>
__device__ __forceinline__ dfc mf_face_f(const MF &M, const float4 *__restrict__ x, int n, int i,
                                         int j, int kk, int k)
{
    dfc a, b, c, d;
    if (n == 0) {
        a = mf_x<SP>(M, x, 1, i, j, kk, k);
        b = mf_x<SP>(M, x, 2, i, j + 1, kk, k);
        c = mf_x<SP>(M, x, 1, i, j, kk + 1, k);
        d = mf_x<SP>(M, x, 2, i, j, kk, k);
    } else if (n == 1) {
        a = mf_x<SP>(M, x, 2, i, j, kk, k);
        b = mf_x<SP>(M, x, 0, i, j, kk + 1, k);
        c = mf_x<SP>(M, x, 2, i + 1, j, kk, k);
        d = mf_x<SP>(M, x, 0, i, j, kk, k);
    } else {
        a = mf_x<SP>(M, x, 0, i, j, kk, k);
        b = mf_x<SP>(M, x, 1, i + 1, j, kk, k);
        c = mf_x<SP>(M, x, 0, i, j + 1, kk, k);
        d = mf_x<SP>(M, x, 1, i, j, kk, k);
    }
    acc fr, fi;
    fr.add(a.re); fr.add(b.re); fr.add(neg(c.re)); fr.add(neg(d.re));
    fi.add(a.im); fi.add(b.im); fi.add(neg(c.im)); fi.add(neg(d.im));
    return dfc{fr.get(), fi.get()};
}

// the circulation a + b - c - d in mf_face_f's order
__device__ __forceinline__ dfc mf_circ(dfc a, dfc b, dfc c, dfc d)
{
    acc fr, fi;
    fr.add(a.re); fr.add(b.re); fr.add(neg(c.re)); fr.add(neg(d.re));
    fi.add(a.im); fi.add(b.im); fi.add(neg(c.im)); fi.add(neg(d.im));
    return dfc{fr.get(), fi.get()};
}

// f = D s: x(e0) + x(e1) - x(e2) - x(e3) around every face (counterclockwise
// seen from +n: y then z for n = x, z then x for n = y, x then y for n = z).
// One thread per node and system forms the x-, y- and z-normal faces at the
// node (those that exist): 9 edge values instead of 12 (the node's own
// three edges are shared), one position decode instead of three; each sum
// is mf_face_f's, so f is the same to the last bit.
template <int SP>
__global__ void __launch_bounds__(kB)
k_mf_faces(MF M, const float4 *__restrict__ x, const SysState *sys, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    if (sys[k].status != kRun) return;
    const int nx = M.nx, ny = M.ny, nz = M.nz;
    const int nn = nx * ny * nz;
    const int rpb = kB / SP;
    const dfc zero{df{0.f, 0.f}, df{0.f, 0.f}};
    for (int ti = blockIdx.x * rpb + threadIdx.x / SP; ti < nn; ti += gridDim.x * rpb) {
        const int v = sweep(ti, nn, rev);
        const int r = v / nx, i = v - r * nx;
        const int kk = r / ny, j = r - kk * ny;
        // the node's +x, +y, +z edges exist below the last line of their axis
        const bool hx = i < nx - 1, hy = j < ny - 1, hz = kk < nz - 1;
        const dfc ex = hx ? mf_x<SP>(M, x, 0, i, j, kk, k) : zero;
        const dfc ey = hy ? mf_x<SP>(M, x, 1, i, j, kk, k) : zero;
        const dfc ez = hz ? mf_x<SP>(M, x, 2, i, j, kk, k) : zero;
        if (hy && hz)
            M.f[(M.fb[0] + (kk * (ny - 1) + j) * nx + i) * SP + k] =
                to4(mf_circ(ey, mf_x<SP>(M, x, 2, i, j + 1, kk, k), mf_x<SP>(M, x, 1, i, j, kk + 1, k), ez));
        if (hx && hz)
            M.f[(M.fb[1] + (kk * ny + j) * (nx - 1) + i) * SP + k] =
                to4(mf_circ(ez, mf_x<SP>(M, x, 0, i, j, kk + 1, k), mf_x<SP>(M, x, 2, i + 1, j, kk, k), ex));
        if (hx && hy)
            M.f[(M.fb[2] + (kk * (ny - 1) + j) * (nx - 1) + i) * SP + k] =
                to4(mf_circ(ex, mf_x<SP>(M, x, 1, i + 1, j, kk, k), mf_x<SP>(M, x, 0, i, j + 1, kk, k), ey));
    }
}

__device__ __forceinline__ df scale(df a, float s) { return df{a.h * s, a.l * s}; }   // s = +-1, 2, 4

// lattice position of an edge: along its direction the cell index, across
// it node indices
struct Pos {
    int x, y, z;
};
// Index context of a non-Dirichlet edge of direction D at lattice position
// p (p along D a cell index, along T1 = D+1 and T2 = D+2 (mod 3) node
// indices): the cell, T1-normal face and T2-normal face at p, the edge, and
// whether the node lines one below / above along T1 (T2) lie on the
// surface.  Every neighbour the row reads is one of these plus strides.
template <int D>
struct MfRow {
    static constexpr int T1 = (D + 1) % 3, T2 = (D + 2) % 3;
    int cell, f1, f2, e;
    bool lo1, hi1, lo2, hi2;
};
template <int A>
__device__ __forceinline__ int coord(Pos p) { return A == 0 ? p.x : (A == 1 ? p.y : p.z); }
template <int A>
__device__ __forceinline__ int extent(const MF &M) { return A == 0 ? M.nx : (A == 1 ? M.ny : M.nz); }
template <int D>
__device__ __forceinline__ MfRow<D> mf_rowctx(const MF &M, Pos p)
{
    constexpr int T1 = MfRow<D>::T1, T2 = MfRow<D>::T2;
    MfRow<D> r;
    r.cell = p.x * M.cs[0] + p.y * M.cs[1] + p.z * M.cs[2];
    r.f1 = M.fb[T1] + p.x * M.fs[T1][0] + p.y * M.fs[T1][1] + p.z * M.fs[T1][2];
    r.f2 = M.fb[T2] + p.x * M.fs[T2][0] + p.y * M.fs[T2][1] + p.z * M.fs[T2][2];
    r.e = mf_edge_in(M, D, p.x, p.y, p.z);
    const int t1 = coord<T1>(p), t2 = coord<T2>(p);
    r.lo1 = t1 == 1;
    r.hi1 = t1 == extent<T1>(M) - 2;
    r.lo2 = t2 == 1;
    r.hi2 = t2 == extent<T2>(M) - 2;
    return r;
}
// the 3 x 3 parallel edges around the row (grid position (a, b) along
// (T1, T2), the row at (1, 1)): Dirichlet, and the edge number otherwise
template <int D>
__device__ __forceinline__ bool mf_mass_dir(const MfRow<D> &r, int a, int b)
{
    return (a == 0 && r.lo1) || (a == 2 && r.hi1) || (b == 0 && r.lo2) || (b == 2 && r.hi2);
}
template <int D>
__device__ __forceinline__ int mf_mass_edge(const MF &M, const MfRow<D> &r, int a, int b)
{
    return r.e + (a - 1) * M.es[MfRow<D>::T1] + (b - 1) * M.es[MfRow<D>::T2];
}

// one non-Dirichlet edge of direction D at lattice position p:
// (K + i omega M) s.  D, and with it the two transverse axes T1 = D+1,
// T2 = D+2 (mod 3), are compile-time constants: the rows run direction by
// direction, so warps are uniform.
template <int SP, int D>
__device__ __forceinline__ dfc mf_row(const MF &M, Pos p, int k, df om, const float4 *__restrict__ x)
{
    constexpr int T1 = (D + 1) % 3, T2 = (D + 2) % 3;
    const int nc = (int)M.ncell;
    const MfRow<D> r = mf_rowctx<D>(M, p);
    // weights of the 4 cells around the edge, offsets (a - 1, b - 1) along (T1, T2)
    df w1[2][2], w2[2][2], wm[2][2];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int cc = r.cell + (a - 1) * M.cs[T1] + (b - 1) * M.cs[T2];
            w1[a][b] = d2f(__ldg(M.w + T1 * nc + cc));
            w2[a][b] = d2f(__ldg(M.w + T2 * nc + cc));
            wm[a][b] = d2f(__ldg(M.w + (3 + D) * nc + cc));
        }
    acc kr, ki, mr, mi;
    // D^T F D: faces of normal T1 through the edge (T2 cells b - 1 = -1: +1,
    // 0: -1), then faces of normal T2 (T1 cells -1: -1, 0: +1); each face's
    // F row: wa (f_-1 + 2 f_0) + wb (2 f_0 + f_+1) over the cells before and
    // after it along the normal
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const int q = r.f1 + (b - 1) * M.fs[T1][T2];
        const float sg = b == 0 ? 1.f : -1.f;
        const df wa = w1[0][b], wb = w1[1][b];
        const dfc fm = from4(__ldg(M.f + (q - M.fs[T1][T1]) * SP + k));
        const dfc f0 = from4(__ldg(M.f + q * SP + k));
        const dfc fp = from4(__ldg(M.f + (q + M.fs[T1][T1]) * SP + k));
        const df ca = scale(wa, sg), cb = scale(wb, sg), c0 = scale(add(wa, wb), 2.f * sg);
        kr.mac(ca, fm.re); kr.mac(c0, f0.re); kr.mac(cb, fp.re);
        ki.mac(ca, fm.im); ki.mac(c0, f0.im); ki.mac(cb, fp.im);
    }
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const int q = r.f2 + (a - 1) * M.fs[T2][T1];
        const float sg = a == 0 ? -1.f : 1.f;
        const df wa = w2[a][0], wb = w2[a][1];
        const dfc fm = from4(__ldg(M.f + (q - M.fs[T2][T2]) * SP + k));
        const dfc f0 = from4(__ldg(M.f + q * SP + k));
        const dfc fp = from4(__ldg(M.f + (q + M.fs[T2][T2]) * SP + k));
        const df ca = scale(wa, sg), cb = scale(wb, sg), c0 = scale(add(wa, wb), 2.f * sg);
        kr.mac(ca, fm.re); kr.mac(c0, f0.re); kr.mac(cb, fp.re);
        ki.mac(ca, fm.im); ki.mac(c0, f0.im); ki.mac(cb, fp.im);
    }
    // M: the 3 x 3 parallel edges around (grid position (A, B), this edge at
    // (1, 1)); edge (A, B) lies in the cells (a, b) with a in {A-1, A},
    // b in {B-1, B}, each contributing its weight times 2 per axis on which
    // A (B) is the edge's own position: coefficients 4 (w00+w01+w10+w11),
    // 2 (pair sums) and 1 (corner cells)
    const df s0_ = add(wm[0][0], wm[0][1]), s1_ = add(wm[1][0], wm[1][1]);
    const df r0_ = add(wm[0][0], wm[1][0]), r1_ = add(wm[0][1], wm[1][1]);
    const df cm[3][3] = {{wm[0][0], scale(s0_, 2.f), wm[0][1]},
                         {scale(r0_, 2.f), scale(add(s0_, s1_), 4.f), scale(r1_, 2.f)},
                         {wm[1][0], scale(s1_, 2.f), wm[1][1]}};
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            dfc xe{df{0.f, 0.f}, df{0.f, 0.f}};
            if (!mf_mass_dir(r, a, b)) xe = from4(__ldg(x + mf_mass_edge(M, r, a, b) * SP + k));
            mr.mac(cm[a][b], xe.re);
            mi.mac(cm[a][b], xe.im);
        }
    const df mxr = mr.get(), mxi = mi.get();
    kr.mac(neg(om), mxi);
    ki.mac(om, mxr);
    return dfc{kr.get(), ki.get()};
}

// The same row for two systems (k0, k0 + 1) at once: the index arithmetic,
// the weights and their combinations are shared; the adjacent systems'
// values are one contiguous 32-byte pair.
template <int SP, int D>
__device__ __forceinline__ void mf_row2(const MF &M, Pos p, int k0, const df (&om)[2],
                                        const float4 *__restrict__ x, dfc (&y)[2])
{
    constexpr int T1 = (D + 1) % 3, T2 = (D + 2) % 3;
    const int nc = (int)M.ncell;
    const MfRow<D> r = mf_rowctx<D>(M, p);
    df w1[2][2], w2[2][2], wm[2][2];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int cc = r.cell + (a - 1) * M.cs[T1] + (b - 1) * M.cs[T2];
            w1[a][b] = d2f(__ldg(M.w + T1 * nc + cc));
            w2[a][b] = d2f(__ldg(M.w + T2 * nc + cc));
            wm[a][b] = d2f(__ldg(M.w + (3 + D) * nc + cc));
        }
    acc kr[2], ki[2], mr[2], mi[2];
#pragma unroll
    for (int nn = 0; nn < 2; nn++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            df wa, wb;
            float sg;
            int im, i0, ip;
            if (nn == 0) {
                sg = b == 0 ? 1.f : -1.f;
                wa = w1[0][b];
                wb = w1[1][b];
                i0 = r.f1 + (b - 1) * M.fs[T1][T2];
                im = i0 - M.fs[T1][T1];
                ip = i0 + M.fs[T1][T1];
            } else {
                sg = b == 0 ? -1.f : 1.f;
                wa = w2[b][0];
                wb = w2[b][1];
                i0 = r.f2 + (b - 1) * M.fs[T2][T1];
                im = i0 - M.fs[T2][T2];
                ip = i0 + M.fs[T2][T2];
            }
            const df ca = scale(wa, sg), cb = scale(wb, sg), c0 = scale(add(wa, wb), 2.f * sg);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const dfc fm = from4(__ldg(M.f + im * SP + k0 + u));
                const dfc f0 = from4(__ldg(M.f + i0 * SP + k0 + u));
                const dfc fp = from4(__ldg(M.f + ip * SP + k0 + u));
                kr[u].mac(ca, fm.re); kr[u].mac(c0, f0.re); kr[u].mac(cb, fp.re);
                ki[u].mac(ca, fm.im); ki[u].mac(c0, f0.im); ki[u].mac(cb, fp.im);
            }
        }
    const df s0_ = add(wm[0][0], wm[0][1]), s1_ = add(wm[1][0], wm[1][1]);
    const df r0_ = add(wm[0][0], wm[1][0]), r1_ = add(wm[0][1], wm[1][1]);
    const df cm[3][3] = {{wm[0][0], scale(s0_, 2.f), wm[0][1]},
                         {scale(r0_, 2.f), scale(add(s0_, s1_), 4.f), scale(r1_, 2.f)},
                         {wm[1][0], scale(s1_, 2.f), wm[1][1]}};
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            if (mf_mass_dir(r, a, b)) continue;
            const int e = mf_mass_edge(M, r, a, b);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const dfc xe = from4(__ldg(x + e * SP + k0 + u));
                mr[u].mac(cm[a][b], xe.re);
                mi[u].mac(cm[a][b], xe.im);
            }
        }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const df mxr = mr[u].get(), mxi = mi[u].get();
        kr[u].mac(neg(om[u]), mxi);
        ki[u].mac(om[u], mxr);
        y[u] = dfc{kr[u].get(), ki[u].get()};
    }
}

// The matrix-free SpMV with two systems per thread (variant 33, SP >= 2):
// SP / 2 threads per edge.  Partial sums are staged per system in shared
// memory so that the grid reduction sees lane l carrying system l % SP.
template <int SP>
__global__ void __launch_bounds__(kB, 2)
k_mf_edges2(int nb, MF M, const float2 *__restrict__ omega, const float4 *__restrict__ s,
            float4 *__restrict__ z,
            SysState *sys, float4 *partials, int mode, int rev)
{
    pdl_wait();
    constexpr int H = SP / 2;
    const int k0 = 2 * (threadIdx.x % H);
    bool on[2];
    df om[2];
    SpmvTail tail[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
        on[u] = sys[k0 + u].status == kRun;
        om[u] = d2f(omega[k0 + u]);
    }
    const int rpb = kB / H, stride = gridDim.x * rpb;
    if (on[0] || on[1]) {
        // the next row's position is loaded one row ahead
        const int r0 = blockIdx.x * rpb + threadIdx.x / H;
        unsigned cn = r0 < nb ? __ldg(M.pos + sweep(r0, nb, rev)) : 0u;
        for (int ri = r0; ri < nb; ri += stride) {
            const unsigned c = cn;
            if (ri + stride < nb) cn = __ldg(M.pos + sweep(ri + stride, nb, rev));
            const int d = (int)(c >> 30);
            const Pos p{(int)(c & 1023u), (int)((c >> 10) & 1023u), (int)((c >> 20) & 1023u)};
            const int e = mf_edge(M, d, p.x, p.y, p.z);
            const long long i = (long long)e * SP + k0;
            const float4 sv[2] = {__ldg(s + i), __ldg(s + i + 1)};
            dfc y[2];
            if (mf_dirichlet(M, d, p.x, p.y, p.z)) {
                y[0] = from4(sv[0]);
                y[1] = from4(sv[1]);
            } else if (d == 0) {
                mf_row2<SP, 0>(M, p, k0, om, s, y);
            } else if (d == 1) {
                mf_row2<SP, 1>(M, p, k0, om, s, y);
            } else {
                mf_row2<SP, 2>(M, p, k0, om, s, y);
            }
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (on[u]) tail[u].row(i + u, y[u], sv[u], z);
        }
    }
    // lanes t and t + H hold the same two systems: thread t keeps system
    // 2 (t % H) + [t & H] of both; moved to lane 2 (t % H) + [t & H] of each
    // group of SP lanes, lane l carries system l % SP
    const int lane = threadIdx.x & 31;
    const bool up = lane & H;
    const int from = (lane & ~(SP - 1)) | ((lane & 1) ? H : 0) | ((lane % SP) >> 1);
    const acc z0[2] = {tail[0].zsr, tail[0].zsi}, z1[2] = {tail[1].zsr, tail[1].zsi};
    tf v[2];
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const tf mine = tf_of(up ? z1[n] : z0[n]), give = tf_of(up ? z0[n] : z1[n]);
        const tf q = tf_add(mine, GridSum<SP, 2, kB>::shfl(give, H));
        v[n] = tf{__shfl_sync(0xffffffffu, q.a, from), __shfl_sync(0xffffffffu, q.b, from),
                  __shfl_sync(0xffffffffu, q.c, from)};
    }
    SpmvTail::finish_v<SP>(v, sys, partials, mode);
}

// z = A s by the matrix-free operator, with the SpMV tail of k_spmv
template <int SP>
__global__ void __launch_bounds__(kB, 2)
k_mf_edges(int nb, MF M, const float2 *__restrict__ omega, const float4 *__restrict__ s,
           float4 *__restrict__ z,
           SysState *sys, float4 *partials, int mode, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const df om = d2f(omega[k]);
    SpmvTail tail;
    const int rpb = kB / SP, stride = gridDim.x * rpb;
    // the next row's position is loaded one row ahead
    const int r0 = blockIdx.x * rpb + threadIdx.x / SP;
    unsigned cn = on && r0 < nb ? __ldg(M.pos + sweep(r0, nb, rev)) : 0u;
    for (int ri = r0; ri < nb; ri += stride) {
        if (!on) break;
        const unsigned c = cn;
        if (ri + stride < nb) cn = __ldg(M.pos + sweep(ri + stride, nb, rev));
        const int d = (int)(c >> 30);
        const Pos p{(int)(c & 1023u), (int)((c >> 10) & 1023u), (int)((c >> 20) & 1023u)};
        const int e = mf_edge(M, d, p.x, p.y, p.z);
        const long long i = (long long)e * SP + k;
        const float4 sv4 = __ldg(s + i);
        dfc y;
        if (mf_dirichlet(M, d, p.x, p.y, p.z))
            y = from4(sv4);
        else if (d == 0)
            y = mf_row<SP, 0>(M, p, k, om, s);
        else if (d == 1)
            y = mf_row<SP, 1>(M, p, k, om, s);
        else
            y = mf_row<SP, 2>(M, p, k, om, s);
        tail.row(i, y, sv4, z);
    }
    tail.finish<SP>(sys, partials, mode);
}

// ---- the curl-curl part as D^T (F f) (variant 35)
// The face mass matrix F couples each face only with its two neighbours
// along its normal (the faces of the two cells it separates), so g = F f is
// computed once per face: g = wa f_-1 + 2 (wa + wb) f_0 + wb f_+1 with wa, wb
// the normal-direction weights of the cells before and after it.  Every
// edge's curl-curl row is then the signed sum of g over its 4 faces, 8 adds
// instead of the 24 multiply-adds of mf_row.  g is needed only on faces
// whose position along the normal is interior (the faces of non-Dirichlet
// edges); the others get 0.

// g = F f straight from x, each circulation formed once (variant 35):
// y- and z-normal faces by columns along the normal — a thread owns a
// column (its transverse position; neighbouring threads, neighbouring
// columns) and a chunk of kMarch positions, computes the circulations of
// the chunk and of its two neighbours and keeps the last two in registers
// while it marches; x-normal faces, whose neighbours along the normal are
// the adjacent faces of the same row, one per thread with the two
// neighbours' circulations formed from the same cached loads.  Every
// circulation is k_mf_faces' sum and every g the same three multiply-adds
// in the same order whichever thread forms it, so g does not depend on the
// decomposition; no face array is written.
constexpr int kMarch = 16;

struct GMarch {
    int xitems, yitems;    // x-normal faces; y-normal column chunks (z-normal after)
    int ycols, zcols;      // columns per chunk row: (nx-1) for both
    int ych, zch;          // chunks per column
};

template <int SP>
__device__ __forceinline__ dfc mf_g(const MF &M, int n, int cb, int ca, dfc fm, dfc f0, dfc fp)
{
    const int nc = (int)M.ncell;
    const df wa = d2f(__ldg(M.w + n * nc + cb)), wb = d2f(__ldg(M.w + n * nc + ca));
    const df c0 = scale(add(wa, wb), 2.f);
    acc gr, gi;
    gr.mac(wa, fm.re); gr.mac(c0, f0.re); gr.mac(wb, fp.re);
    gi.mac(wa, fm.im); gi.mac(c0, f0.im); gi.mac(wb, fp.im);
    return dfc{gr.get(), gi.get()};
}

template <int SP>
__global__ void __launch_bounds__(kB)
k_mf_gmarch(MF M, GMarch G, const float4 *__restrict__ x, const SysState *sys, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    if (sys[k].status != kRun) return;
    const dfc zero{df{0.f, 0.f}, df{0.f, 0.f}};
    const int nx = M.nx, ny = M.ny, nz = M.nz;
    auto cell = [&](int a, int b, int c) { return (c * (ny - 1) + b) * (nx - 1) + a; };
    const int zitems = G.zcols * (ny - 1) * G.zch;
    const int nitems = G.xitems + G.yitems + zitems;
    const int rpb = kB / SP;
    for (int qi = blockIdx.x * rpb + threadIdx.x / SP; qi < nitems; qi += gridDim.x * rpb) {
        const int q = sweep(qi, nitems, rev);
        if (q < G.xitems) {
            // x-normal face t = (kk (ny-1) + j) nx + i: neighbours i -+ 1
            int n, i, j, kk;
            mf_face_pos(M, q, n, i, j, kk);
            dfc out = zero;
            if (i >= 1 && i < nx - 1) {
                const dfc fm = mf_face_f<SP>(M, x, 0, i - 1, j, kk, k);
                const dfc f0 = mf_face_f<SP>(M, x, 0, i, j, kk, k);
                const dfc fp = mf_face_f<SP>(M, x, 0, i + 1, j, kk, k);
                out = mf_g<SP>(M, 0, cell(i - 1, j, kk), cell(i, j, kk), fm, f0, fp);
            }
            M.g[(long long)q * SP + k] = to4(out);
            continue;
        }
        // a column chunk: y-normal (column (i, kk), positions j) or z-normal
        // (column (i, j), positions kk)
        int n, i, c2, p0, L;
        if (q < G.xitems + G.yitems) {
            const int r = q - G.xitems;
            n = 1;
            i = r % G.ycols;
            const int t = r / G.ycols;
            c2 = t % (nz - 1);              // kk
            p0 = (t / (nz - 1)) * kMarch;   // j
            L = ny - 1;
        } else {
            const int r = q - G.xitems - G.yitems;
            n = 2;
            i = r % G.zcols;
            const int t = r / G.zcols;
            c2 = t % (ny - 1);              // j
            p0 = (t / (ny - 1)) * kMarch;   // kk
            L = nz - 1;
        }
        const int p1 = min(p0 + kMarch, L + 1);
        auto fat = [&](int p) {
            return n == 1 ? mf_face_f<SP>(M, x, 1, i, p, c2, k) : mf_face_f<SP>(M, x, 2, i, c2, p, k);
        };
        auto face = [&](int p) -> long long {
            return n == 1 ? M.nfx + ((long long)c2 * ny + p) * (nx - 1) + i
                          : M.nfx + M.nfy + ((long long)p * (ny - 1) + c2) * (nx - 1) + i;
        };
        dfc fm = p0 >= 1 ? fat(p0 - 1) : zero;
        dfc f0 = fat(p0);
        for (int p = p0; p < p1; p++) {
            const dfc fp = p + 1 <= L ? fat(p + 1) : zero;
            dfc out = zero;
            if (p >= 1 && p < L) {
                const int cb = n == 1 ? cell(i, p - 1, c2) : cell(i, c2, p - 1);
                const int ca = n == 1 ? cell(i, p, c2) : cell(i, c2, p);
                out = mf_g<SP>(M, n, cb, ca, fm, f0, fp);
            }
            M.g[face(p) * SP + k] = to4(out);
            fm = f0;
            f0 = fp;
        }
    }
}

// one non-Dirichlet edge of direction D at lattice position p: the signed
// sum of g over its 4 faces (the signs of mf_row's groups) plus the mass
// part of mf_row
template <int SP, int D>
__device__ __forceinline__ dfc mf_row_g(const MF &M, Pos p, int k, df om, const float4 *__restrict__ x)
{
    constexpr int T1 = (D + 1) % 3, T2 = (D + 2) % 3;
    const int nc = (int)M.ncell;
    const MfRow<D> r = mf_rowctx<D>(M, p);
    df wm[2][2];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++)
            wm[a][b] = d2f(__ldg(M.w + (3 + D) * nc + r.cell + (a - 1) * M.cs[T1] + (b - 1) * M.cs[T2]));
    const dfc g1a = from4(__ldg(M.g + (r.f1 - M.fs[T1][T2]) * SP + k));
    const dfc g1b = from4(__ldg(M.g + r.f1 * SP + k));
    const dfc g2a = from4(__ldg(M.g + (r.f2 - M.fs[T2][T1]) * SP + k));
    const dfc g2b = from4(__ldg(M.g + r.f2 * SP + k));
    acc kr, ki;
    kr.add(g1a.re); kr.add(neg(g1b.re)); kr.add(neg(g2a.re)); kr.add(g2b.re);
    ki.add(g1a.im); ki.add(neg(g1b.im)); ki.add(neg(g2a.im)); ki.add(g2b.im);
    acc mr, mi;
    const df s0_ = add(wm[0][0], wm[0][1]), s1_ = add(wm[1][0], wm[1][1]);
    const df r0_ = add(wm[0][0], wm[1][0]), r1_ = add(wm[0][1], wm[1][1]);
    const df cm[3][3] = {{wm[0][0], scale(s0_, 2.f), wm[0][1]},
                         {scale(r0_, 2.f), scale(add(s0_, s1_), 4.f), scale(r1_, 2.f)},
                         {wm[1][0], scale(s1_, 2.f), wm[1][1]}};
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            dfc xe{df{0.f, 0.f}, df{0.f, 0.f}};
            if (!mf_mass_dir(r, a, b)) xe = from4(__ldg(x + mf_mass_edge(M, r, a, b) * SP + k));
            mr.mac(cm[a][b], xe.re);
            mi.mac(cm[a][b], xe.im);
        }
    const df mxr = mr.get(), mxi = mi.get();
    kr.mac(neg(om), mxi);
    ki.mac(om, mxr);
    return dfc{kr.get(), ki.get()};
}

// z = A s in the D^T (F f) form, with the SpMV tail of k_spmv
template <int SP>
__global__ void __launch_bounds__(kB)
k_mf_edges_g(int nb, MF M, const float2 *__restrict__ omega, const float4 *__restrict__ s,
             float4 *__restrict__ z,
             SysState *sys, float4 *partials, int mode, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const df om = d2f(omega[k]);
    SpmvTail tail;
    const int rpb = kB / SP, stride = gridDim.x * rpb;
    // the next row's position is loaded one row ahead
    const int r0 = blockIdx.x * rpb + threadIdx.x / SP;
    unsigned cn = on && r0 < nb ? __ldg(M.pos + sweep(r0, nb, rev)) : 0u;
    for (int ri = r0; ri < nb; ri += stride) {
        if (!on) break;
        const unsigned c = cn;
        if (ri + stride < nb) cn = __ldg(M.pos + sweep(ri + stride, nb, rev));
        const int d = (int)(c >> 30);
        const Pos p{(int)(c & 1023u), (int)((c >> 10) & 1023u), (int)((c >> 20) & 1023u)};
        const int e = mf_edge(M, d, p.x, p.y, p.z);
        const long long i = (long long)e * SP + k;
        const float4 sv4 = __ldg(s + i);
        dfc y;
        if (mf_dirichlet(M, d, p.x, p.y, p.z))
            y = from4(sv4);
        else if (d == 0)
            y = mf_row_g<SP, 0>(M, p, k, om, s);
        else if (d == 1)
            y = mf_row_g<SP, 1>(M, p, k, om, s);
        else
            y = mf_row_g<SP, 2>(M, p, k, om, s);
        tail.row(i, y, sv4, z);
    }
    tail.finish<SP>(sys, partials, mode);
}

#include "mf_tile.cuh"
#include "prec_tile.cuh"

// ------------------------------------------------ tiled SpMV (x staged)
// A tile is T consecutive SELL slices (32 T rows).  Its distinct columns
// (about 260 per 32-row slice on these meshes, against 1,030 slot reads) are
// listed once, and every slot carries its column's 16-bit index in that
// list.  The kernel copies the tile's x segments (SP lanes each) and the
// tile's matrix slots into shared memory with asynchronous copies, then
// every (row, system) thread runs its row from shared memory: each x
// segment crosses L2 once per tile instead of once per use, and no
// dependent global load is left in the row loop.
struct TileMat {
    const int *wc, *wr;
    const long long *pc, *pr;
    const float2 *kc, *mc, *kr;
    const unsigned short *lc, *lr;
    const int *uoff, *ucol;
    int T, ntiles, nslices;
};

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// shared-memory bytes of a tile: x segments, then K, M, K_real, local indices
__host__ __device__ __forceinline__ long long tile_bytes(int nu, int SP, long long nc, long long nr)
{
    return (long long)nu * SP * 16 + nc * 8 * 2 + nr * 8 + nc * 2 + nr * 2;
}

// a value from shared memory (plain load) or from global memory (read-only path)
template <class T>
__device__ __forceinline__ T ldv(const T *p, bool shared)
{
    return shared ? *p : __ldg(p);
}

// threads of the x-staged SpMV block: a tile of T slices in whole passes
template <int SP>
struct TileCfg {
    static constexpr int NT = SP >= 32 ? 1024 : (SP == 1 ? 256 : 512);
    // slices per tile
    static constexpr int T = SP >= 16 ? 1 : (SP == 1 ? 8 : (16 / SP < 8 ? 16 / SP : 8));
};

// MAT: also stage the tile's matrix slots (else they stream from global
// memory, each used once)
template <int SP, bool MAT>
__global__ void __launch_bounds__(TileCfg<SP>::NT)
k_spmv_t(int nb, TileMat A, const float2 *__restrict__ omega, const float4 *__restrict__ s,
         float4 *__restrict__ z,
         SysState *sys, float4 *partials, int mode)
{
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const df om = d2f(omega[k]);
    SpmvTail tail;
    for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
        const int s0 = t * A.T, s1 = min(s0 + A.T, A.nslices);
        const long long c0 = A.pc[s0], nc = A.pc[s1] - c0, q0 = A.pr[s0], nr = A.pr[s1] - q0;
        const int u0 = A.uoff[t], nu = A.uoff[t + 1] - u0;
        float4 *xs = reinterpret_cast<float4 *>(smem);
        // matrix slots: shared memory after x, or global memory from the tile's start
        const float2 *skc, *smc, *skr;
        const unsigned short *slc, *slr;
        __syncthreads();   // the previous tile's readers are done
        constexpr int NT = TileCfg<SP>::NT;
        for (int i = threadIdx.x; i < nu * SP; i += NT)
            cp_async16(xs + i, s + (long long)__ldg(A.ucol + u0 + i / SP) * SP + i % SP);
        if (MAT) {
            float2 *kc2 = reinterpret_cast<float2 *>(xs + (long long)nu * SP);
            float2 *mc2 = kc2 + nc;
            float2 *kr2 = mc2 + nc;
            unsigned short *lc2 = reinterpret_cast<unsigned short *>(kr2 + nr);
            unsigned short *lr2 = lc2 + nc;
            // slot counts are multiples of 32: whole 16-byte chunks, 16-byte aligned
            for (long long i = threadIdx.x; i < nc / 2; i += NT) {
                cp_async16(reinterpret_cast<float4 *>(kc2) + i, reinterpret_cast<const float4 *>(A.kc + c0) + i);
                cp_async16(reinterpret_cast<float4 *>(mc2) + i, reinterpret_cast<const float4 *>(A.mc + c0) + i);
            }
            for (long long i = threadIdx.x; i < nr / 2; i += NT)
                cp_async16(reinterpret_cast<float4 *>(kr2) + i, reinterpret_cast<const float4 *>(A.kr + q0) + i);
            for (long long i = threadIdx.x; i < nc / 8; i += NT)
                cp_async16(reinterpret_cast<float4 *>(lc2) + i, reinterpret_cast<const float4 *>(A.lc + c0) + i);
            for (long long i = threadIdx.x; i < nr / 8; i += NT)
                cp_async16(reinterpret_cast<float4 *>(lr2) + i, reinterpret_cast<const float4 *>(A.lr + q0) + i);
            skc = kc2; smc = mc2; skr = kr2; slc = lc2; slr = lr2;
        } else {
            skc = A.kc + c0; smc = A.mc + c0; skr = A.kr + q0; slc = A.lc + c0; slr = A.lr + q0;
        }
        cp_async_wait_all();
        __syncthreads();
        if (!on) continue;
        for (int rr = threadIdx.x / SP; rr < (s1 - s0) * 32; rr += NT / SP) {
            const int row = s0 * 32 + rr;
            if (row >= nb) break;
            const int sl = s0 + (rr >> 5), l = rr & 31;
            acc kr_, ki_, mr_, mi_;
            {
                const int b = (int)(A.pc[sl] - c0) + l, n = A.wc[sl];
#pragma unroll 4
                for (int q = 0; q < n; q++) {
                    const int t2 = b + 32 * q;
                    const float4 xv = xs[ldv(slc + t2, MAT) * SP + k];
                    const df kd = d2f(ldv(skc + t2, MAT)), md = d2f(ldv(smc + t2, MAT));
                    const df xr{xv.x, xv.y}, xi{xv.z, xv.w};
                    kr_.mac(kd, xr);
                    ki_.mac(kd, xi);
                    mr_.mac(md, xr);
                    mi_.mac(md, xi);
                }
            }
            {
                const int b = (int)(A.pr[sl] - q0) + l, n = A.wr[sl];
#pragma unroll 4
                for (int q = 0; q < n; q++) {
                    const int t2 = b + 32 * q;
                    const float4 xv = xs[ldv(slr + t2, MAT) * SP + k];
                    const df kd = d2f(ldv(skr + t2, MAT));
                    kr_.mac(kd, df{xv.x, xv.y});
                    ki_.mac(kd, df{xv.z, xv.w});
                }
            }
            const df mxr = mr_.get(), mxi = mi_.get();
            kr_.mac(neg(om), mxi);
            ki_.mac(om, mxr);
            const long long i = (long long)row * SP + k;
            tail.row(i, dfc{kr_.get(), ki_.get()}, __ldg(s + i), z);
        }
    }
    tail.finish<SP, TileCfg<SP>::NT>(sys, partials, mode);
}

// ---- tile set-up: sorted distinct columns of every tile, local indices
constexpr int kTileThreads = 1024;
constexpr int kTileMaxKeys = 16384;

// ---------------------------------------------- FP64 iterative refinement
// The double-float recurrences reach about 2^-48 |A| |x| / |b| of the true
// residual; at low frequencies (1e-3 Hz: the air regularised by
// omega sigma ~ 6e-11) that gap is above 1e-8.  The solution is therefore
// accumulated in FP64 and every true residual is evaluated in FP64 from the
// FP64 matrix; where the double-float iteration stalls above eps, it restarts
// on the FP64 residual (mixed-precision iterative refinement).
struct Mat64 {
    const int *wc, *wr;
    const long long *pc, *pr;
    const int *col_c, *col_r;
    const double *kc, *mc, *kr;
};

// r = b - A(omega) x in FP64 for the systems flagged in check;
// ||b||, ||r||, true_rel into the system state; write != 0: r also becomes
// the double-float residual rdf that the inner solve starts from.
template <int SP>
__global__ void __launch_bounds__(kB)
k_res64(int nb, Mat64 A, const double *__restrict__ omega64, const double2 *__restrict__ b64,
        const double2 *__restrict__ x, float4 *__restrict__ rdf,
        SysState *sys, const int *__restrict__ check, int write, float4 *partials)
{
    const int k = threadIdx.x % SP;
    const bool on = check[k] != 0;
    const double om = omega64[k];
    double nb2 = 0.0, nr2 = 0.0;
    const int rpb = kB / SP;
    for (int row = blockIdx.x * rpb + threadIdx.x / SP; row < nb; row += gridDim.x * rpb) {
        if (!on) continue;
        const int sl = row >> 5, l = row & 31;
        double kx = 0.0, ky = 0.0, mx = 0.0, my = 0.0;
        {
            const long long b0 = A.pc[sl] + l;
            const int n = A.wc[sl];
            for (int q = 0; q < n; q++) {
                const long long t = b0 + (long long)kSlice * q;
                const int c = __ldg(A.col_c + t);
                const double kv = __ldg(A.kc + t), mv = __ldg(A.mc + t);
                const double2 xv = __ldg(x + (long long)c * SP + k);
                kx += kv * xv.x;
                ky += kv * xv.y;
                mx += mv * xv.x;
                my += mv * xv.y;
            }
        }
        {
            const long long b0 = A.pr[sl] + l;
            const int n = A.wr[sl];
            for (int q = 0; q < n; q++) {
                const long long t = b0 + (long long)kSlice * q;
                const int c = __ldg(A.col_r + t);
                const double kv = __ldg(A.kr + t);
                const double2 xv = __ldg(x + (long long)c * SP + k);
                kx += kv * xv.x;
                ky += kv * xv.y;
            }
        }
        const long long i = (long long)row * SP + k;
        const double2 bv = b64[i];
        const double2 rv = make_double2(bv.x - (kx - om * my), bv.y - (ky + om * mx));
        if (write) rdf[i] = to4(from_d2(rv));
        nb2 += bv.x * bv.x + bv.y * bv.y;
        nr2 += rv.x * rv.x + rv.y * rv.y;
    }
    double v[2] = {nb2, nr2};
    __shared__ double tot[2][32];
    if (sys_grid_sum64<SP, 2>(v, partials, &sys[0].ticket[1], tot) && threadIdx.x < SP &&
        check[threadIdx.x]) {
        SysState &q = sys[threadIdx.x];
        const double bb = sqrt(tot[0][threadIdx.x]), rr = sqrt(tot[1][threadIdx.x]);
        q.bnorm = bb;
        q.rnorm = rr;
        q.true_rel = bb > 0.0 ? rr / bb : 0.0;
        q.checks += 1;
    }
}

// p and x of a group of iterations: for each, p = s + beta p and d += alpha p
// in double-float (d from 0), then x += d in FP64, and the last s to slot 0.
// The same operations on the same values as one iteration at a time, so the
// same p and x to the last bit; per iteration 1 + 6 / 16 vector passes instead
// of the 5.4 of updating p and x in k_edge and folding x every 16 iterations
// (1.8M edges x 2 systems: k_edge 95 -> 57 us, this kernel 11 us an iteration).
// Four s values are in flight per thread.
template <int SP>
__global__ void __launch_bounds__(kB)
k_group(long long n, float4 *__restrict__ s, float4 *__restrict__ p, double2 *__restrict__ x,
        const float4 *__restrict__ hist, const SysState *sys, int rev)
{
    pdl_wait();
    __shared__ float4 ab[SP * kGroupIters * 2];
    for (int i = threadIdx.x; i < SP * kGroupIters * 2; i += kB) ab[i] = hist[i];
    __syncthreads();
    const int k = threadIdx.x % SP;
    const int cnt = sys[k].cnt;
    if (cnt == 0) return;
    const float4 *c = ab + 2 * kGroupIters * k;
    const long long stride = (long long)gridDim.x * kB;
    for (long long ii = (long long)blockIdx.x * kB + threadIdx.x; ii < n; ii += stride) {
        // n is a multiple of SP: a backward sweep by rows keeps the lane's system
        const long long i = rev ? n - SP - (ii - k) + k : ii;
        dfc pv = from4(p[i]), d{df{0.f, 0.f}, df{0.f, 0.f}};
        const double2 xv = x[i];
        int j = 0;
        for (; j + 4 <= cnt; j += 4) {
            float4 sv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) sv[u] = s[(j + u) * n + i];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                pv = caxpy(from4(sv[u]), from4(c[2 * (j + u) + 1]), pv);
                d = caxpy(d, from4(c[2 * (j + u)]), pv);
            }
        }
        for (; j < cnt; j++) {
            pv = caxpy(from4(s[j * n + i]), from4(c[2 * j + 1]), pv);
            d = caxpy(d, from4(c[2 * j]), pv);
        }
        const float4 last = s[cnt * n + i];
        x[i] = make_double2(xv.x + ((double)d.re.h + (double)d.re.l),
                            xv.y + ((double)d.im.h + (double)d.im.l));
        p[i] = to4(pv);
        s[i] = last;
    }
}

template <int SP>
struct Impl {
    static Mat mat(const Survey &V)
    {
        const ParamMatrix &P = *V.P;
        return Mat{P.d_wc, P.d_wr, P.d_pc, P.d_pr, P.d_col_c, P.d_col_r, V.kc, V.mc, V.kr};
    }
    static TileMat tmat(const Survey &V)
    {
        const ParamMatrix &P = *V.P;
        return TileMat{P.d_wc, P.d_wr, P.d_pc, P.d_pr, V.kc, V.mc, V.kr, V.lc, V.lr,
                       V.uoff, V.ucol, V.tile_T, V.ntiles, P.nslices};
    }
    static void mfd_into(const Survey &V, MF &M) { M = mfd(V); }
    // the work items of k_mf_gmarch
    static GMarch gmarch(const Survey &V)
    {
        const MatFree &F = V.mf;
        GMarch G;
        G.ycols = G.zcols = F.nx - 1;
        G.ych = ceil_div(F.ny, kMarch);
        G.zch = ceil_div(F.nz, kMarch);
        G.xitems = (int)F.nfx;
        G.yitems = G.ycols * (F.nz - 1) * G.ych;
        return G;
    }
    static MF mfd(const Survey &V)
    {
        const MatFree &F = V.mf;
        MF M{};
        M.nx = F.nx;
        M.ny = F.ny;
        M.nz = F.nz;
        M.nfx = F.nfx;
        M.nfy = F.nfy;
        M.nfz = F.nfz;
        M.ncell = (long long)(F.nx - 1) * (F.ny - 1) * (F.nz - 1);
        mf_strides(M);
        M.pos = F.pos;
        M.w = F.w;
        M.f = F.f;
        M.g = F.g;
        return M;
    }
    // h = D_S G (src + beta a): the lattice form where G is the lattice's
    // the sweep direction of the next launch: opposite to the previous one's
    static int flip(Survey &V) { return V.dir ^= 1; }
    static void node(Survey &V, const float4 *src, const float4 *a, int use_beta)
    {
        const int rv = flip(V);
        if (V.g_lat)
            pdl(k_node_lat<SP>, V.g_node_lat, kB, 0, V.st, mfd(V), V.G.m, V.ds, src, a, V.h, V.sys,
                use_beta, rv);
        else
            pdl(k_node<SP>, V.g_node, kB, 0, V.st, V.G.m, V.G.d_gp, V.G.d_gj, V.gv32, V.ds, src, a,
                V.h, V.sys, use_beta, rv);
    }
    static void spmv(Survey &V, int mode, const float4 *s)
    {
        const Mat A = mat(V);
        if (V.ch == kMatFree + 2) {
            const MfTileGrid G{V.mft[0], V.mft[1], V.mft[2], V.mft[3], V.mft[4], V.mft[5], V.mft[6]};
            k_mf_tile<SP><<<V.g_mft, MfTile<SP>::NT, MfTile<SP>::SMEM, V.st>>>(
                mfd(V), G, V.omega, s, V.z, V.sys, V.partials, mode);
            return;
        }
        if (V.ch == kMatFree + 3) {
            const MF M = mfd(V);
            pdl(k_mf_gmarch<SP>, V.g_mfg, kB, 0, V.st, M, gmarch(V), s, V.sys, flip(V));
            pdl(k_mf_edges_g<SP>, V.g_mfe3, kB, 0, V.st, V.nb, M, V.omega, s, V.z, V.sys,
                                                       V.partials, mode, flip(V));
            return;
        }
        if (V.ch == kMatFree || V.ch == kMatFree + 1) {
            const MF M = mfd(V);
            pdl(k_mf_faces<SP>, V.g_mff, kB, 0, V.st, M, s, V.sys, flip(V));
            if constexpr (SP >= 2) {
                if (V.ch == kMatFree + 1) {
                    pdl(k_mf_edges2<SP>, V.g_mfe, kB, 0, V.st, V.nb, M, V.omega, s, V.z, V.sys, V.partials, mode, flip(V));
                    return;
                }
            }
            pdl(k_mf_edges<SP>, V.g_mfe, kB, 0, V.st, V.nb, M, V.omega, s, V.z, V.sys,
                                                    V.partials, mode, flip(V));
            return;
        }
        if (V.ch == 0) {
            k_spmv_t<SP, true><<<V.g_spmv_t, TileCfg<SP>::NT, V.tile_smem, V.st>>>(
                V.nb, tmat(V), V.omega, s, V.z, V.sys, V.partials, mode);
            return;
        }
        if (V.ch == 1) {
            k_spmv_t<SP, false><<<V.g_spmv_tx, TileCfg<SP>::NT, V.tile_smem_x, V.st>>>(
                V.nb, tmat(V), V.omega, s, V.z, V.sys, V.partials, mode);
            return;
        }
        if constexpr (SP == 2) {
            if (V.ch == kRowVariant + 2) {
                pdl(k_spmv_r2<2>, V.g_spmv, kB, 0, V.st, V.nb, A, V.omega, s, V.z, V.sys, V.partials, mode);
                return;
            }
            if (V.ch == kRowVariant + 4) {
                pdl(k_spmv_r2<4>, V.g_spmv, kB, 0, V.st, V.nb, A, V.omega, s, V.z, V.sys, V.partials, mode);
                return;
            }
        }
        switch (V.ch) {
        case 2: pdl(k_spmv<SP, 2>, V.g_spmv, kB, 0, V.st, V.nb, A, V.omega, s, V.z, V.sys, V.partials, mode); break;
        case 8: pdl(k_spmv<SP, 8>, V.g_spmv, kB, 0, V.st, V.nb, A, V.omega, s, V.z, V.sys, V.partials, mode); break;
        default: pdl(k_spmv<SP, 4>, V.g_spmv, kB, 0, V.st, V.nb, A, V.omega, s, V.z, V.sys, V.partials, mode); break;
        }
    }
    // slot t of the group's s vectors
    static float4 *slot_s(const Survey &V, int t) { return V.s + (size_t)t * V.nb * SP; }
    static void precond(Survey &V, const float4 *src, float4 *w, int mode, int first)
    {
        if (V.G.m > 0) node(V, src, V.a, mode);
        pdl(k_edge<SP>, V.g_edge, kB, 0, V.st, V.nb, V.G.d_tp, V.G.d_tj, V.tv32, V.G.d_tn, V.da, V.h,
            src, V.a, w, V.sys, V.partials, mode, first, flip(V));
    }
    static void prec_tile(Survey &V, const float4 *ain, float4 *aout, int first)
    {
        const PrecGrid G{V.pt[0], V.pt[1], V.pt[2], V.pt[3], V.pt[4]};
        k_prec_tile<SP><<<V.g_pt, PrecTile<SP>::NT, PrecTile<SP>::SMEM, V.st>>>(
            mfd(V), G, V.ds, V.da, V.z, ain, aout, V.w, V.sys, V.partials, first);
    }
    // iteration t of a sequence of n: the fused preconditioner alternates a's
    // buffers (t even reads a, writes a2; t odd the reverse); p and x follow at
    // the end of a group of iterations and of the sequence
    static void iteration(Survey &V, int t, int n)
    {
        const int j = t % V.group;
        float4 *a = V.a;
        if (V.prec_tile) {
            a = (t & 1) ? V.a : V.a2;
            prec_tile(V, (t & 1) ? V.a2 : V.a, a, j == 0);
        } else {
            precond(V, V.z, V.w, 1, j == 0);
        }
        pdl(k_update<SP>, V.g_update, kB, 0, V.st, V.nb, a, V.w, V.sm, V.r, slot_s(V, j),
            slot_s(V, j + 1), V.sys, V.hist, V.partials, flip(V));
        spmv(V, 1, slot_s(V, j + 1));
        if (j == V.group - 1 || t == n - 1)
            pdl(k_group<SP>, V.g_group, kB, 0, V.st, (long long)V.nb * SP, V.s, V.p, V.xacc, V.hist,
                V.sys, flip(V));
    }
    // one preconditioner step of the iteration (mode 1), unfused or fused
    static void precond_step(Survey &V, bool fused, float4 *ain, float4 *aout)
    {
        if (fused) prec_tile(V, ain, aout, 1);
        else precond(V, V.z, V.w, 1, 1);
    }
    static void prec_grid(Survey &V, int nsm)
    {
        using T = PrecTile<SP>;
        int res = 0;
        if (cudaFuncSetAttribute((const void *)k_prec_tile<SP>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, (const void *)k_prec_tile<SP>, T::NT,
                                                          T::SMEM) != cudaSuccess ||
            res < 1) {
            cudaGetLastError();
            res = 1;
        }
        const int tx = ceil_div(V.mf.nx, T::TX), ty = ceil_div(V.mf.ny, T::TY), grp = SP / T::SB;
        const int bxy = tx * ty * grp;
        int zc = 1;
        long long best = -1;
        for (int c = 1; c <= std::max(1, V.mf.nz / 4); c++) {
            const long long waves = ceil_div(bxy * c, res * nsm);
            const long long cost = waves * (ceil_div(V.mf.nz, c) + 1);
            if (best < 0 || cost < best) {
                best = cost;
                zc = c;
            }
        }
        const int kz = ceil_div(V.mf.nz, zc);
        zc = ceil_div(V.mf.nz, kz);
        V.pt[0] = tx; V.pt[1] = ty; V.pt[2] = zc; V.pt[3] = grp; V.pt[4] = kz;
        V.g_pt = bxy * zc;
    }
    // stages 1-4 of PCOCR_RCI::Run: r = b - A x, x0 test, s = M^-1 r,
    // p = a = 0, z = A s, (z, s)
    static void start(Survey &V)
    {
        k_init<SP><<<V.g_init, kB, 0, V.st>>>(V.nb, V.r, V.sm, V.sys, V.partials);
        precond(V, V.r, V.s, 0, 1);
        cudaMemsetAsync(V.p, 0, sizeof(float4) * (size_t)V.nb * SP, V.st);
        cudaMemsetAsync(V.a, 0, sizeof(float4) * (size_t)V.nb * SP, V.st);
        spmv(V, 0, V.s);
        note_launches(V.G.m > 0 ? 4 : 3);
    }
    static void res64(Survey &V, const int *check, int write)
    {
        const ParamMatrix &P = *V.P;
        const Mat64 A{P.d_wc, P.d_wr, P.d_pc, P.d_pr, P.d_col_c, P.d_col_r, P.d_kc, P.d_mc, P.d_kr};
        k_res64<SP><<<V.g_true, kB, 0, V.st>>>(V.nb, A, V.omega64, V.b64, V.xacc, V.r,
                                               V.sys, check, write, V.partials);
        note_launches(1);
    }
    static void spmv_only(Survey &V, int mode) { spmv(V, mode, V.s); }

    // launch grids: as many blocks as fit on the device at once (grid-stride
    // loops do the rest), never more than there is work for
    static int occ(const void *f)
    {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kB, 0) != cudaSuccess || b < 1) b = 1;
        return b;
    }
    static void grids(Survey &V, int nsm)
    {
        auto g = [&](const void *f, int work) { return std::max(1, std::min(occ(f) * nsm, work)); };
        V.g_init = g((const void *)k_init<SP>, V.grid_rows);
        V.g_node = g((const void *)k_node<SP>, V.grid_nodes);
        V.g_node_lat = g((const void *)k_node_lat<SP>, V.grid_nodes);
        V.g_edge = g((const void *)k_edge<SP>, V.grid_rows);
        V.g_update = g((const void *)k_update<SP>, V.grid_rows);
        V.g_group = g((const void *)k_group<SP>, V.grid_rows);
        V.g_true = g((const void *)k_res64<SP>, V.grid_rows);
        const void *fs = V.ch == 2 ? (const void *)k_spmv<SP, 2>
                         : V.ch == 8 ? (const void *)k_spmv<SP, 8> : (const void *)k_spmv<SP, 4>;
        V.g_spmv = g(fs, V.grid_rows);
        if (V.mf.on) {
            const long long nn = (long long)V.mf.nx * V.mf.ny * V.mf.nz;
            V.g_mff = g((const void *)k_mf_faces<SP>, (int)std::min<long long>(
                                                          (nn + kB / SP - 1) / (kB / SP), INT_MAX));
            V.g_mfe = g((const void *)k_mf_edges<SP>, V.grid_rows);
            {
                const GMarch G = gmarch(V);
                const long long items = (long long)G.xitems + G.yitems +
                                        (long long)G.zcols * (V.mf.ny - 1) * G.zch;
                V.g_mfg = g((const void *)k_mf_gmarch<SP>, (int)std::min<long long>(
                                                               (items + kB / SP - 1) / (kB / SP), INT_MAX));
            }
            V.g_mfe3 = g((const void *)k_mf_edges_g<SP>, V.grid_rows);
            if constexpr (SP >= 2) {
                if (V.ch == kMatFree + 1)
                    V.g_mfe = g((const void *)k_mf_edges2<SP>,
                                (V.nb + 2 * kB / SP - 1) / (2 * kB / SP));
            }
            // tiled variant: tiles x systems groups, the z range cut into
            // chunks so that about one wave of resident blocks is launched
            using T = MfTile<SP>;
            int res = 0;
            if (cudaFuncSetAttribute((const void *)k_mf_tile<SP>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, (const void *)k_mf_tile<SP>, T::NT,
                                                              T::SMEM) != cudaSuccess ||
                res < 1) {
                cudaGetLastError();
                res = 1;
            }
            // tile shape: the x columns split evenly in tiles of at most TX,
            // then as many rows as the threads and the halo frame allow
            const int ntx = ceil_div(V.mf.nx, T::TX);
            const int tw = ceil_div(V.mf.nx, ntx);
            int th = std::min(T::TX * T::TY / tw, T::NS / (tw + 2) - 2);
            th = std::max(1, std::min(th, V.mf.ny));
            const int tx = ntx, ty = ceil_div(V.mf.ny, th), grp = SP / T::SB;
            V.mft[5] = tw;
            V.mft[6] = th;
            const int bxy = tx * ty * grp;
            // z chunks: the fewest waves x (planes per chunk + 2 of prologue)
            int zc = 1;
            long long best = -1;
            for (int c = 1; c <= std::max(1, V.mf.nz / 4); c++) {
                const long long waves = ceil_div(bxy * c, res * nsm);
                const long long cost = waves * (ceil_div(V.mf.nz, c) + 2);
                if (best < 0 || cost < best) {
                    best = cost;
                    zc = c;
                }
            }
            const int kz = ceil_div(V.mf.nz, zc);
            zc = ceil_div(V.mf.nz, kz);
            V.mft[0] = tx; V.mft[1] = ty; V.mft[2] = zc; V.mft[3] = grp; V.mft[4] = kz;
            V.g_mft = bxy * zc;
        }
        if constexpr (SP == 2) {
            if (V.ch == kRowVariant + 2 || V.ch == kRowVariant + 4) {
                const void *fr = V.ch == kRowVariant + 2 ? (const void *)k_spmv_r2<2>
                                                         : (const void *)k_spmv_r2<4>;
                V.g_spmv = g(fr, (V.nb + kB - 1) / kB);
            }
        }
        if (V.ntiles > 0) {
            int b = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)k_spmv_t<SP, true>,
                                                              TileCfg<SP>::NT, V.tile_smem) !=
                    cudaSuccess || b < 1)
                b = 1;
            V.g_spmv_t = std::max(1, std::min(b * nsm, V.ntiles));
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)k_spmv_t<SP, false>,
                                                              TileCfg<SP>::NT, V.tile_smem_x) !=
                    cudaSuccess || b < 1)
                b = 1;
            V.g_spmv_tx = std::max(1, std::min(b * nsm, V.ntiles));
        }
    }
    static void tile_slices_of(int *T) { *T = TileCfg<SP>::T; }
    static void tile_attr(Survey &V, cudaError_t *e)
    {
        *e = cudaFuncSetAttribute((const void *)k_spmv_t<SP, true>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, V.tile_smem);
        if (*e == cudaSuccess)
            *e = cudaFuncSetAttribute((const void *)k_spmv_t<SP, false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, V.tile_smem_x);
    }
};

// Impl<SP> of one lane count as a table, so that survey.cu instantiates none of it
struct Ops {
    void (*mfd_into)(const Survey &V, MF &M);
    void (*iteration)(Survey &V, int t, int n);
    void (*precond_step)(Survey &V, bool fused, float4 *ain, float4 *aout);
    void (*prec_grid)(Survey &V, int nsm);
    void (*start)(Survey &V);
    void (*res64)(Survey &V, const int *check, int write);
    void (*spmv_only)(Survey &V, int mode);
    void (*grids)(Survey &V, int nsm);
    void (*tile_slices_of)(int *T);
    void (*tile_attr)(Survey &V, cudaError_t *e);
    void (*node)(Survey &V, const float4 *src, const float4 *a, int use_beta);
};
template <int SP>
Ops make_ops()
{
    using I = Impl<SP>;
    return Ops{I::mfd_into, I::iteration, I::precond_step, I::prec_grid, I::start, I::res64, I::spmv_only, I::grids, I::tile_slices_of, I::tile_attr, I::node};
}
const Ops &ops1();
const Ops &ops2();
const Ops &ops4();
const Ops &ops8();
const Ops &ops16();
const Ops &ops32();

}  // namespace sv
}  // namespace mtgpu
