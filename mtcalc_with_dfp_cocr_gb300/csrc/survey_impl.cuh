// The batched survey solver's kernels and their launches for one lane count
// (systems padded to SP = 1, 2, ..., 32).  Every SP is a translation unit of
// its own (survey_sp.cu), so that they compile side by side; survey.cu holds
// the host side and calls Impl<SP>.
#pragma once
#include "survey.cuh"
#include "dfloat.cuh"

#include <algorithm>
#include <climits>
#include <type_traits>

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
    // N log2), then thread t < W adds the warps' sums.  down: this thread's
    // values are scaled by 2^-64 already
    static __device__ __forceinline__ float4 block(const tf (&v)[N], float4 *sm, bool down)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        bool big = down;
#pragma unroll
        for (int n = 0; n < N; n++) big |= fabsf(v[n].a) >= kTfBig;
        big = __any_sync(0xffffffffu, big);
        tf u[N];
#pragma unroll
        for (int n = 0; n < N; n++) u[n] = big && !down ? tf_scale(v[n], kTfDown) : v[n];
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
    // the totals of `rows` partials in threads t < W: up to 12 loads a thread
    // in flight, added pairwise (one load latency for 456 blocks x 2 systems;
    // a loop of dependent adds took 4,300 cycles)
    static __device__ __forceinline__ float4 rows(const float4 *part, int rows, float4 *sm)
    {
        constexpr int U = 12;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 s = zero;
        for (int i0 = 0; i0 < rows * W; i0 += U * NT) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + u * NT + threadIdx.x;
                v[u] = i < rows * W ? __ldcg(part + i) : zero;
            }
#pragma unroll
            for (int h = 1; h < U; h <<= 1)
#pragma unroll
                for (int u = 0; u + h < U; u += 2 * h) v[u] = tf4_add(v[u], v[u + h]);
            s = i0 == 0 ? v[0] : tf4_add(s, v[0]);
        }
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
// float4 slots before the partials: the grid's ticket, the groups', and k_small's
// two counters (kBarSlot, kExitSlot)
constexpr int kTicketSlots = 256, kMaxGroups = 990;
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
__device__ bool sys_grid_sum(const tf (&v)[N], float4 *partials, double (*tot)[32], bool down = false)
{
    using S = GridSum<SP, N, NT>;
    constexpr int W = S::W;
    __shared__ float4 sm[S::SLOTS];
    __shared__ bool last;
    unsigned int *tickets = reinterpret_cast<unsigned int *>(partials);
    float4 *part = partials + kTicketSlots;
    float4 s = S::block(v, sm, down);
    // one level: this block's sums to dst; whether it is the last of n blocks
    auto arrive = [&](float4 *dst, unsigned int *ticket, unsigned int n) {
        if (threadIdx.x < W) __stcg(dst + threadIdx.x, s);
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned int seen = count_arrival(ticket);
            last = seen == n - 1;
            if (last) *ticket = 0u;
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

__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gsrc)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// asynchronous 16-byte copy global -> shared; valid = false writes zeros
// (source size 0: nothing is read)
__device__ __forceinline__ void cp_async16_zfill(void *smem_dst, const void *gsrc, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gsrc), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// the same, with a copy left in L1 for the neighbouring threads that read it too
__device__ __forceinline__ void cp_async16_l1(void *smem_dst, const void *gsrc, bool valid = true)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gsrc), "r"(n)
                 : "memory");
}
// 8 bytes
__device__ __forceinline__ void cp_async8(void *smem_dst, const void *gsrc)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gsrc) : "memory");
}

// Element i of a grid-stride sweep over n elements, forwards or backwards.
// Consecutive kernels of the iteration sweep in opposite directions, so
// that each starts on the end of what the previous one streamed, which is
// still in L2 (a 58 MB vector of two systems against ~126 MB of L2); only
// the order of the partial sums changes, and it is fixed.
__device__ __forceinline__ int sweep(int i, int n, int rev) { return rev ? n - 1 - i : i; }

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
                const df xr{xv[j].x, xv[j].z}, xi{xv[j].y, xv[j].w};
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
            const df xr{xv.x, xv.z}, xi{xv.y, xv.w};
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
                kr_.mac(kd, df{xv[j].x, xv[j].z});
                ki_.mac(kd, df{xv[j].y, xv[j].w});
            }
        }
        for (; q < n; q++) {
            const int c = __ldg(cc + kSlice * q);
            const df kd = d2f(__ldg(kk + kSlice * q));
            const float4 xv = __ldg(xk + c * SP);
            kr_.mac(kd, df{xv.x, xv.z});
            ki_.mac(kd, df{xv.y, xv.w});
        }
    }
    // y = Kx + i omega Mx
    const df mxr = mr_.get(), mxi = mi_.get();
    kr_.mac(neg(om), mxi);
    ki_.mac(om, mxr);
    return dfc{kr_.get(), ki_.get()};
}

// t x for t = +-1/2 (exact)
__device__ __forceinline__ cdf chalf(cdf x, float t) { return cdf{mul2(x.h, pk(t, t)), mul2(x.l, pk(t, t))}; }

// ------------------------------------------------------------ set-up
// the scalars that the row kernels read, in both forms
// (a / b of these sums: cquot_part without its look at the range, which sums of
// FP32 products, 2^-149 to 2^192 with their scaling, cannot leave; it took 0.5 us
// of a 17 us one-kernel iteration and 0.4 of the separate kernels' 30)
__device__ __forceinline__ double sum_quot_part(double2 a, double2 b, int c)
{
    const double d = b.x * b.x + b.y * b.y;
    return (c == 0 ? a.x * b.x + a.y * b.y : a.y * b.x - a.x * b.y) / d;
}
__device__ __forceinline__ double2 sum_quot(double2 a, double2 b)
{
    return make_double2(sum_quot_part(a, b, 0), sum_quot_part(a, b, 1));
}
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
    return to4(r, i);
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
    acc2 nr2;
    const int rpb = kB / SP;
    for (int row = blockIdx.x * rpb + threadIdx.x / SP; row < nb; row += gridDim.x * rpb) {
        if (!on) continue;
        const long long i = (long long)row * SP + k;
        const float4 v = r[i];
        sm[i] = v;
        nr2.mac(cdf_of(v), cdf_of(v));
    }
    const tf v[1] = {tf_sum(nr2)};
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

// (a, w) -> alpha, by the block that finishes last.  Here and in the other
// finishers the state is read before the sum, so that its latency passes
// behind the sum's, and independent FP64 chains (a divide or a square root is
// 500 cycles) run side by side.
template <int SP, int NT>
__device__ __forceinline__ void finish_alpha(const tf (&v)[2], SysState *sys, float4 *partials, int first,
                                             bool down = false)
{
    __shared__ double tot[2][32];
    SysState &q = sys[threadIdx.x % SP];
    const double2 zs = q.zs;
    const int status = q.status;
    if (sys_grid_sum<SP, 2, NT>(v, partials, tot, down) && threadIdx.x < SP) {
        if (first) q.cnt = 0;
        if (status == kRun) {
            const double2 aw = make_double2(tot[0][threadIdx.x], tot[1][threadIdx.x]);
            if (fabs(aw.x) < 1e-40 && fabs(aw.y) < 1e-40) q.status = MTGPU_DIV_BY_ZERO;
            else set_alpha(q, sum_quot(zs, aw));
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
    const cfac be = cfac_of(from4(sys[k].beta_f));
    const int rpb = kB / SP;
    for (int vi = blockIdx.x * rpb + threadIdx.x / SP; vi < m; vi += gridDim.x * rpb) {
        const int v = sweep(vi, m, rev);
        const int j0 = __ldg(gp + v), j1 = __ldg(gp + v + 1);
        const float4 dsv = __ldg(ds + (long long)v * SP + k);
        acc2 hv;
        for (int j = j0; j < j1; j++) {
            const long long idx = (long long)__ldg(gj + j) * SP + k;
            const float g = __ldg(gv + j);
            cdf an = cdf_of(__ldg(z + idx));
            if (use_beta) an = caxpy(an, be, cdf_of(__ldg(a + idx)));
            hv.mac(both(df{g, 0.f}), an);
        }
        h[(long long)v * SP + k] = to4(cmul(cfac_of(from4(dsv)), hv.get()));
    }
}

// mode 1: a = z + beta a, w = D_A a + G^T h, (a, w) -> alpha; first: the
// iteration is the first of its group
// mode 0: w = D_A z + G^T h (preconditioner application, no reduction)
// Every input of an element is loaded before anything is stored.  p = s +
// beta p and x += alpha p are k_group's: reading s and p and x here and
// writing p and x were 5 of this kernel's 11 vector passes.
template <int SP>
__global__ void __launch_bounds__(kB, 4)
k_edge(int n, const int *__restrict__ tp, const int *__restrict__ tj, const float *__restrict__ tv,
       const int2 *__restrict__ tn, const float4 *__restrict__ da, const float4 *__restrict__ h,
       const float4 *__restrict__ z, float4 *__restrict__ a, float4 *__restrict__ w, SysState *sys,
       float4 *partials, int mode, int first, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const cfac be = cfac_of(from4(sys[k].beta_f));
    acc2 aw1, aw2;     // a w component by component, and a with w's exchanged
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
        const cdf zv = ldn(z + idx), dav = ldn(da + idx);
        cdf av = czero(), h0 = czero(), h1 = czero();
        if (mode != 0) av = ldg(a + idx);
        acc2 wv;
        cdf an;
        // G^T row: compact (the rows of the edge's two nodes, -1/2 and +1/2
        // in that order) or the CSR of T-matrix meshes
        if (tn) {
            const int2 r2 = r2n;
            if (r2.x >= 0) h0 = ldn(h + (long long)r2.x * SP + k);
            if (r2.y >= 0) h1 = ldn(h + (long long)r2.y * SP + k);
            if (ei + stride < n) r2n = __ldg(tn + sweep(ei + stride, n, rev));
            an = mode != 0 ? caxpy(zv, be, av) : zv;
            wv.start(cmul(cfac_of(dav), an));
            // +-1/2 is exact: added instead of multiplied
            if (r2.x >= 0) wv.sub(chalf(h0, 0.5f));
            if (r2.y >= 0) wv.add(chalf(h1, 0.5f));
        } else {
            an = mode != 0 ? caxpy(zv, be, av) : zv;
            wv.start(cmul(cfac_of(dav), an));
            for (int j = __ldg(tp + e); j < __ldg(tp + e + 1); j++)
                wv.mac(both(df{__ldg(tv + j), 0.f}), ldn(h + (long long)__ldg(tj + j) * SP + k));
        }
        const cdf wn = wv.get();
        if (mode != 0) a[idx] = to4(an);
        w[idx] = to4(wn);
        aw1.mac(an, wn);
        aw2.mac(an, cswap(wn));
    }
    if (mode == 0) return;
    const tf v[2] = {tf_diff(aw1), tf_sum(aw2)};
    finish_alpha<SP, kB>(v, sys, partials, first);
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
    dfc al = from4(sys[k].alpha_f);
    al = dfc{neg(al.re), neg(al.im)};
    const cfac nal = cfac_of(al);
    const int pm = sys[k].mrs_mode;
    const cdf pw = both(d2f(sys[k].mrs_wf));
    acc2 su, uu, nn, rr;
    const int rpb = kB / SP;
    const int stride = gridDim.x * rpb;
    // two elements per pass, all 10 loads issued before any store
    for (int e = blockIdx.x * rpb + threadIdx.x / SP; e < n; e += 2 * stride) {
        if (!on) break;
        const bool two = e + stride < n;
        cdf v[2][5];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (u == 1 && !two) break;
            const long long idx = (long long)sweep(e + u * stride, n, rev) * SP + k;
            v[u][0] = ldn(a + idx); v[u][1] = ldn(w + idx);
            v[u][2] = ldg(sm + idx); v[u][3] = ldg(r + idx); v[u][4] = ldn(s_in + idx);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (u == 1 && !two) break;
            const long long idx = (long long)sweep(e + u * stride, n, rev) * SP + k;
            const cdf ro = v[u][3];
            cdf smv = v[u][2];
            if (pm == 1) {
                smv = ro;
            } else if (pm == 2) {
                acc2 t;
                t.start(smv);
                t.mac(pw, csub(ro, smv));
                smv = t.get();
            }
            const cdf rn = caxpy(ro, nal, v[u][0]);
            r[idx] = to4(rn);
            s_out[idx] = to4(caxpy(v[u][4], nal, v[u][1]));
            if (pm != 0) sm[idx] = to4(smv);
            const cdf ur = csub(rn, smv);
            su.mac(smv, ur);
            uu.mac(ur, ur);
            nn.mac(smv, smv);
            rr.mac(rn, rn);
        }
    }
    const tf v[4] = {tf_sum(su), tf_sum(uu), tf_sum(nn), tf_sum(rr)};
    __shared__ double tot[4][32];
    SysState &q = sys[threadIdx.x % SP];
    const int status = q.status, c = min(q.cnt, kGroupIters - 1);
    const float4 alpha_f = q.alpha_f, beta_f = q.beta_f;
    if (sys_grid_sum<SP, 4>(v, partials, tot) && threadIdx.x < SP && status == kRun) {
        const double s_u = tot[0][threadIdx.x], u_u = tot[1][threadIdx.x];
        const double n_n = tot[2][threadIdx.x], r_r = tot[3][threadIdx.x];
        hist[2 * (threadIdx.x * kGroupIters + c)] = alpha_f;
        hist[2 * (threadIdx.x * kGroupIters + c) + 1] = beta_f;
        q.cnt = c + 1;
        const double wm = fabs(u_u) < 1e-100 ? 0.0 : -s_u / u_u;
        if (wm < 0.0) {
            q.mrs_mode = 0;
        } else if (wm > 1.0) {
            q.mrs_mode = 1;
            q.res2_next = r_r;
        } else {
            q.mrs_mode = 2;
            set_mrs_w(q, wm);
            q.res2_next = n_n + 2.0 * wm * s_u + wm * wm * u_u;
        }
    }
}

// Per-row tail of the SpMV kernels: store z = A s and accumulate (z, s).
// (The MRS smoothing of the residual runs in k_update.)
struct SpmvTail {
    acc2 zs1, zs2;     // z s component by component, and z with s's exchanged
    __device__ __forceinline__ void row(long long i, cdf y, cdf s, float4 *__restrict__ z)
    {
        z[i] = to4(y);
        zs1.mac(y, s);
        zs2.mac(y, cswap(s));
    }
    __device__ __forceinline__ void row(long long i, dfc y, float4 sv4, float4 *__restrict__ z)
    {
        row(i, cdf_of(to4(y)), cdf_of(sv4), z);
    }
    __device__ __forceinline__ tf zsr() const { return tf_diff(zs1); }
    __device__ __forceinline__ tf zsi() const { return tf_sum(zs2); }
    // grid totals -> stop test and beta (the last block only)
    template <int SP, int NT = kB>
    __device__ __forceinline__ void finish(SysState *sys, float4 *partials, int mode)
    {
        const tf v[2] = {zsr(), zsi()};
        finish_v<SP, NT>(v, sys, partials, mode);
    }
    // the same from this thread's (z, s) re, im of system threadIdx.x % SP.
    // mode 1: the stop test on ||s_m|| of this iteration (k_update's
    // res2_next), then beta; mode 0 (set-up): (z, s) only
    template <int SP, int NT = kB>
    static __device__ __forceinline__ void finish_v(const tf (&v)[2], SysState *sys,
                                                    float4 *partials, int mode, bool down = false)
    {
        __shared__ double tot[2][32];
        SysState &q = sys[threadIdx.x % SP];
        const double2 zs = q.zs;
        const double r_old = q.r_old, eps_k = q.eps_k, res2 = q.res2_next, res = q.residual;
        const int status = q.status, mrs = q.mrs_mode, iter = q.iter, maxiter = q.maxiter;
        if (sys_grid_sum<SP, 2, NT>(v, partials, tot, down) && threadIdx.x < SP && status == kRun) {
            const double2 zs_new = make_double2(tot[0][threadIdx.x], tot[1][threadIdx.x]);
            q.zs = zs_new;
            if (mode == 0) return;
            const double2 beta = sum_quot(zs_new, zs);
            const double residual = mrs == 0 ? res : (res2 > 0.0 ? sqrt(res2) : 0.0);
            const double rel = residual / r_old;
            set_beta(q, beta);
            q.residual = residual;
            q.residual_rel = rel;
            if (rel < eps_k) {
                q.status = MTGPU_OK;
            } else {
                q.iter = iter + 1;
                if (iter + 1 > maxiter) q.status = MTGPU_MAXITER;
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
                    const df xr{xv[j][k].x, xv[j][k].z}, xi{xv[j][k].y, xv[j][k].w};
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
                    kr_[k].mac(kd, df{xv[j][k].x, xv[j][k].z});
                    ki_[k].mac(kd, df{xv[j][k].y, xv[j][k].w});
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
    const tf z0[2] = {tail[0].zsr(), tail[0].zsi()}, z1[2] = {tail[1].zsr(), tail[1].zsi()};
    tf v[2];
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const tf mine = odd ? z1[n] : z0[n], give = odd ? z0[n] : z1[n];
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
    const int *dir;            // the edges on the outer surface (variant 35)
    int ndir;
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
__device__ __forceinline__ cdf mf_x(const MF &M, const float4 *x, int d, int i, int j, int kk, int k)
{
    if (mf_dirichlet(M, d, i, j, kk)) return czero();
    return cdf_of(__ldg(x + mf_edge_in(M, d, i, j, kk) * SP + k));
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
    const cfac be = cfac_of(from4(sys[k].beta_f));
    const int ix = M.nx - 2, iy = M.ny - 2;
    const int rpb = kB / SP;
    for (int vi = blockIdx.x * rpb + threadIdx.x / SP; vi < m; vi += gridDim.x * rpb) {
        const int v = sweep(vi, m, rev);
        const int i = v % ix + 1, t = v / ix, j = t % iy + 1, kk = t / iy + 1;
        const int e0 = mf_edge_in(M, 0, i, j, kk);
        const int es[6] = {e0 + 2 - M.plane, e0 + 1 - M.l3, e0 - 3, e0, e0 + 1, e0 + 2};
        cdf zv[6], av[6];
#pragma unroll
        for (int q = 0; q < 6; q++) zv[q] = ldn(z + (long long)es[q] * SP + k);
#pragma unroll
        for (int q = 0; q < 6; q++) av[q] = use_beta ? ldn(a + (long long)es[q] * SP + k) : czero();
        const cdf dsv = ldn(ds + (long long)v * SP + k);
        // the entries are +-1/2: the sum is halved once (exact, as each product)
        acc2 hv;
#pragma unroll
        for (int q = 0; q < 6; q++) {
            cdf an = zv[q];
            if (use_beta) an = caxpy(an, be, av[q]);
            if (q == 0) hv.start(an);
            else if (q < 3) hv.add(an);
            else hv.sub(an);
        }
        h[(long long)v * SP + k] = to4(cmul(cfac_of(dsv), chalf(hv.get(), 0.5f)));
    }
}

// the circulation a + b - c - d
__device__ __forceinline__ cdf mf_circ(cdf a, cdf b, cdf c, cdf d)
{
    acc2 f;
    f.start(a);
    f.add(b);
    f.sub(c);
    f.sub(d);
    return f.get();
}

// f = D s: x(e0) + x(e1) - x(e2) - x(e3) around every face (counterclockwise
// seen from +n: y then z for n = x, z then x for n = y, x then y for n = z).
// One thread per node and system forms the x-, y- and z-normal faces at the
// node (those that exist): 9 edge values instead of 12 (the node's own
// three edges are shared), one position decode instead of three; each sum
// is mf_circ's, so f is the same to the last bit.
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
    const cdf zero = czero();
    for (int ti = blockIdx.x * rpb + threadIdx.x / SP; ti < nn; ti += gridDim.x * rpb) {
        const int v = sweep(ti, nn, rev);
        const int r = v / nx, i = v - r * nx;
        const int kk = r / ny, j = r - kk * ny;
        // the node's +x, +y, +z edges exist below the last line of their axis
        const bool hx = i < nx - 1, hy = j < ny - 1, hz = kk < nz - 1;
        const cdf ex = hx ? mf_x<SP>(M, x, 0, i, j, kk, k) : zero;
        const cdf ey = hy ? mf_x<SP>(M, x, 1, i, j, kk, k) : zero;
        const cdf ez = hz ? mf_x<SP>(M, x, 2, i, j, kk, k) : zero;
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
__device__ __forceinline__ int coord(int a, Pos p) { return a == 0 ? p.x : (a == 1 ? p.y : p.z); }
__device__ __forceinline__ int extent(int a, const MF &M) { return a == 0 ? M.nx : (a == 1 ? M.ny : M.nz); }
// Index context of a non-Dirichlet edge of direction d at lattice position
// p (p along d a cell index, along T1 = d+1 and T2 = d+2 (mod 3) node
// indices): the cell, T1-normal face and T2-normal face at p, the edge, their
// strides along the axes, and whether the node lines one below / above along
// T1 (T2) lie on the surface.  Every neighbour the row reads is one of these
// plus strides.
struct MfRow {
    int cell, c1, c2;          // cell, strides along T1, T2
    int f1, n1, t1;            // T1-normal face, strides along T1, T2
    int f2, n2, t2;            // T2-normal face, strides along T2, T1
    int e, e1, e2;             // edge, strides along T1, T2
    int w1, w2, wm;            // weights of the T1-, T2-normal faces and of the mass
    bool lo1, hi1, lo2, hi2;
};
__device__ __forceinline__ MfRow mf_rowctx(const MF &M, int d, Pos p)
{
    const int T1 = d == 2 ? 0 : d + 1, T2 = d == 0 ? 2 : d - 1;
    MfRow r;
    r.cell = p.x * M.cs[0] + p.y * M.cs[1] + p.z * M.cs[2];
    r.c1 = M.cs[T1];
    r.c2 = M.cs[T2];
    r.f1 = M.fb[T1] + p.x * M.fs[T1][0] + p.y * M.fs[T1][1] + p.z * M.fs[T1][2];
    r.n1 = M.fs[T1][T1];
    r.t1 = M.fs[T1][T2];
    r.f2 = M.fb[T2] + p.x * M.fs[T2][0] + p.y * M.fs[T2][1] + p.z * M.fs[T2][2];
    r.n2 = M.fs[T2][T2];
    r.t2 = M.fs[T2][T1];
    r.e = mf_edge_in(M, d, p.x, p.y, p.z);
    r.e1 = M.es[T1];
    r.e2 = M.es[T2];
    const int nc = (int)M.ncell;
    r.w1 = T1 * nc;
    r.w2 = T2 * nc;
    r.wm = (3 + d) * nc;
    const int q1 = coord(T1, p), q2 = coord(T2, p);
    r.lo1 = q1 == 1;
    r.hi1 = q1 == extent(T1, M) - 2;
    r.lo2 = q2 == 1;
    r.hi2 = q2 == extent(T2, M) - 2;
    return r;
}
// the 3 x 3 parallel edges around the row (grid position (a, b) along
// (T1, T2), the row at (1, 1)): Dirichlet, and the edge number otherwise
__device__ __forceinline__ bool mf_mass_dir(const MfRow &r, int a, int b)
{
    return (a == 0 && r.lo1) || (a == 2 && r.hi1) || (b == 0 && r.lo2) || (b == 2 && r.hi2);
}
__device__ __forceinline__ int mf_mass_edge(const MfRow &r, int a, int b)
{
    return r.e + (a - 1) * r.e1 + (b - 1) * r.e2;
}

// (a0 + b0, a1 + b1) of two double-float pairs, packed
__device__ __forceinline__ cdf pair_add(df a0, df a1, df b0, df b1)
{
    acc2 t;
    t.start(cdf{pk(a0.h, a1.h), pk(a0.l, a1.l)});
    t.add(cdf{pk(b0.h, b1.h), pk(b0.l, b1.l)});
    return t.get();
}

// the weights of table w at the 4 cells around a row, offsets (a - 1, b - 1) along (T1, T2)
__device__ __forceinline__ void mf_weights(const MF &M, const MfRow &r, int w, df (&out)[2][2])
{
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) out[a][b] = d2f(__ldg(M.w + w + r.cell + (a - 1) * r.c1 + (b - 1) * r.c2));
}

// The mass part of a row for U systems k0, k0 + 1, ...: the 3 x 3 parallel
// edges around (grid position (A, B), this edge at (1, 1)); edge (A, B) lies
// in the cells (a, b) with a in {A-1, A}, b in {B-1, B}, each contributing its
// weight times 2 per axis on which A (B) is the edge's own position:
// coefficients 4 (w00+w01+w10+w11), 2 (pair sums) and 1 (corner cells).
// Then y = kk + i omega (mass part).  sv: the row's own x.
template <int SP, int U>
__device__ __forceinline__ void mf_mass_row(const MF &M, const MfRow &r, int k0, const df (&om)[U],
                                            const float4 *x, const cdf (&sv)[U],
                                            acc2 (&kk)[U], cdf (&y)[U])
{
    df wm[2][2];
    mf_weights(M, r, r.wm, wm);
    const cdf s = pair_add(wm[0][0], wm[1][0], wm[0][1], wm[1][1]);      // sums over b
    const cdf q = pair_add(wm[0][0], wm[0][1], wm[1][0], wm[1][1]);      // sums over a
    const df s0 = lane0(s), s1 = lane1(s), r0 = lane0(q), r1 = lane1(q);
    const df cm[3][3] = {{wm[0][0], scale(s0, 2.f), wm[0][1]},
                         {scale(r0, 2.f), scale(add(s0, s1), 4.f), scale(r1, 2.f)},
                         {wm[1][0], scale(s1, 2.f), wm[1][1]}};
    acc2 mm[U];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const cdf c = both(cm[a][b]);
#pragma unroll
            for (int u = 0; u < U; u++) {
                cdf xe = czero();
                if (a == 1 && b == 1)
                    xe = sv[u];
                else if (!mf_mass_dir(r, a, b))
                    xe = cdf_of(__ldg(x + mf_mass_edge(r, a, b) * SP + k0 + u));
                if (a == 0 && b == 0) mm[u].first(c, xe);
                else mm[u].mac(c, xe);
            }
        }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const cdf f{pk(-om[u].h, om[u].h), pk(-om[u].l, om[u].l)};
        kk[u].mac(f, cswap(mm[u].get()));
        y[u] = kk[u].get();
    }
}

// one face group of a row: +- (wa f_-1 + 2 (wa + wb) f_0 + wb f_+1)
template <int SP, int U, bool PLUS, bool FIRST>
__device__ __forceinline__ void mf_face_group(const MF &M, int q, int step, int k0, df wa, df wb, df c2,
                                              acc2 (&kk)[U])
{
    const cdf ca = both(wa), c0 = both(scale(c2, 2.f)), cb = both(wb);
#pragma unroll
    for (int u = 0; u < U; u++) {
        const cdf fm = cdf_of(__ldg(M.f + (q - step) * SP + k0 + u));
        const cdf f0 = cdf_of(__ldg(M.f + q * SP + k0 + u));
        const cdf fp = cdf_of(__ldg(M.f + (q + step) * SP + k0 + u));
        if (PLUS) {
            if (FIRST) kk[u].first(ca, fm);
            else kk[u].mac(ca, fm);
            kk[u].mac(c0, f0);
            kk[u].mac(cb, fp);
        } else {
            kk[u].msub(ca, fm);
            kk[u].msub(c0, f0);
            kk[u].msub(cb, fp);
        }
    }
}

// one non-Dirichlet edge of direction d at lattice position p for U systems:
// (K + i omega M) s.  With d a constant of the call the two transverse axes
// and the strides are compile-time choices: the rows run direction by
// direction, so warps are uniform.  The adjacent systems' values are
// contiguous and share the index arithmetic, the weights and their
// combinations.
template <int SP, int U>
__device__ __forceinline__ void mf_row(const MF &M, int d, Pos p, int k0, const df (&om)[U],
                                       const float4 *x, const cdf (&sv)[U], cdf (&y)[U])
{
    const MfRow r = mf_rowctx(M, d, p);
    df w1[2][2], w2[2][2];
    mf_weights(M, r, r.w1, w1);
    mf_weights(M, r, r.w2, w2);
    // D^T F D: faces of normal T1 through the edge (T2 cells b - 1 = -1: +1,
    // 0: -1), then faces of normal T2 (T1 cells -1: -1, 0: +1); each face's
    // F row over the cells before and after it along the normal
    acc2 kk[U];
    const cdf c1 = pair_add(w1[0][0], w1[0][1], w1[1][0], w1[1][1]);
    mf_face_group<SP, U, true, true>(M, r.f1 - r.t1, r.n1, k0, w1[0][0], w1[1][0], lane0(c1), kk);
    mf_face_group<SP, U, false, false>(M, r.f1, r.n1, k0, w1[0][1], w1[1][1], lane1(c1), kk);
    const cdf c2 = pair_add(w2[0][0], w2[1][0], w2[0][1], w2[1][1]);
    mf_face_group<SP, U, false, false>(M, r.f2 - r.t2, r.n2, k0, w2[0][0], w2[0][1], lane0(c2), kk);
    mf_face_group<SP, U, true, false>(M, r.f2, r.n2, k0, w2[1][0], w2[1][1], lane1(c2), kk);
    mf_mass_row<SP, U>(M, r, k0, om, x, sv, kk, y);
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
            const cdf sv[2] = {cdf_of(__ldg(s + i)), cdf_of(__ldg(s + i + 1))};
            cdf y[2];
            if (mf_dirichlet(M, d, p.x, p.y, p.z)) {
                y[0] = sv[0];
                y[1] = sv[1];
            } else if (d == 0) {
                mf_row<SP, 2>(M, 0, p, k0, om, s, sv, y);
            } else if (d == 1) {
                mf_row<SP, 2>(M, 1, p, k0, om, s, sv, y);
            } else {
                mf_row<SP, 2>(M, 2, p, k0, om, s, sv, y);
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
    const tf z0[2] = {tail[0].zsr(), tail[0].zsi()}, z1[2] = {tail[1].zsr(), tail[1].zsi()};
    tf v[2];
#pragma unroll
    for (int n = 0; n < 2; n++) {
        const tf mine = up ? z1[n] : z0[n], give = up ? z0[n] : z1[n];
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
    const df om[1] = {d2f(omega[k])};
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
        const cdf sv[1] = {cdf_of(__ldg(s + i))};
        cdf y[1];
        if (mf_dirichlet(M, d, p.x, p.y, p.z))
            y[0] = sv[0];
        else if (d == 0)
            mf_row<SP, 1>(M, 0, p, k, om, s, sv, y);
        else if (d == 1)
            mf_row<SP, 1>(M, 1, p, k, om, s, sv, y);
        else
            mf_row<SP, 1>(M, 2, p, k, om, s, sv, y);
        tail.row(i, y[0], sv[0], z);
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
// edges); no row reads the others, and nothing forms them.

// g = F f straight from x, each circulation formed once (variant 35): a
// thread owns a column of faces along their normal and a chunk of len
// positions, computes the circulations of the chunk and of its two neighbours
// and keeps the last two in registers while it marches.  Every circulation
// is k_mf_faces' sum and every g the same three multiply-adds in the same
// order whichever thread forms it, so g does not depend on the
// decomposition; no face array is written.
//
// z = A s from g: a thread owns a line of parallel edges (direction D) along
// one transverse axis Q and marches a chunk of len of them; R is the other
// transverse axis.
// Curl-curl part: the signed sum of g over the row's 4 faces; the R-normal
// face shared with the row before stays in registers.
// Mass part: m (x) m with m = [2 1; 1 2] per cell is applied first along R,
// P_a(m) = 2 x(0, m) + x(+-1, m) for the cells a on either side, once per
// line position and kept for the three rows that use it; a row then is the sum
// over its 4 cells of w (2 P_a(m) + P_a(m +- 1)): 6 additions and 4
// multiply-adds instead of 9 multiply-adds whose coefficients (sums of the
// weights) have to be formed, and 8 loads a row (3 x, 3 g, 2 weights) instead
// of 17.
//
// The rows on the outer surface (the identity) come from a list of their own.
//
// The edge kernel's next positions are copied to shared memory
// asynchronously, kStages ahead, each thread into slots of its own: with
// loads straight to registers the march was bound by their latency (27 % of
// the issue slots used, 4 warps a scheduler for the registers).  The copies
// stay in L1, where the neighbouring lines' threads find them (71 -> 64 us on 1.8M
// edges x 2 systems, no change at 16).  Work is
// ordered in tiles of ly x lz lines and columns in y and z, all
// directions of a tile together, so that the vectors' cache lines, which hold
// the three edges of a node, are used while they are in L2 (300 -> 160 MB of
// DRAM traffic on 1.8M edges x 2 systems).
constexpr int kStages = 2;

// slots [stage][value][thread]
template <int V>
struct Ring {
    float4 *base;
    __device__ __forceinline__ float4 *at(int stage, int v) const
    {
        return base + (stage * V + v) * kB + threadIdx.x;
    }
};

__device__ __forceinline__ cdf mf_g(df wa, df wb, cdf fm, cdf f0, cdf fp)
{
    acc2 g;
    g.first(both(wa), fm);
    g.mac(both(scale(add(wa, wb), 2.f)), f0);
    g.mac(both(wb), fp);
    return g.get();
}

// the faces of normal N at c (c[N]: the chunk's first position) that are off
// the outer surface; no edge row reads those on it
template <int SP, int N>
__device__ __forceinline__ void mf_face_march(const MF &M, int len, const int (&c)[3],
                                              const float4 *__restrict__ x, int k)
{
    constexpr int A = (N + 1) % 3, B = (N + 2) % 3;        // transverse axes
    const int ext[3] = {M.nx, M.ny, M.nz};
    const int last = ext[N] - 1, p0 = max(c[N], 1), p1 = min(c[N] + len, last);
    if (p0 >= p1) return;
    // Dirichlet edges of the column's faces: a-edges at b = 0 and b + 1 on the
    // far side, b-edges at a = 0 and a + 1 on the far side
    const bool a0 = c[B] == 0, a1 = c[B] + 1 == ext[B] - 1, b0 = c[A] == 0, b1 = c[A] + 1 == ext[A] - 1;
    const int es = M.es[N] * SP, ea = M.es[A] * SP, eb = M.es[B] * SP;
    const float4 *__restrict__ xk = x + k;
    // the circulation at the position of edge index i; 0 on the surface
    auto fat = [&](int p, int i) {
        if (p <= 0 || p >= last) return czero();
        const cdf va = a0 ? czero() : ldn(xk + i + A * SP);
        const cdf vb = b1 ? czero() : ldn(xk + i + ea + B * SP);
        const cdf vc = a1 ? czero() : ldn(xk + i + eb + A * SP);
        const cdf vd = b0 ? czero() : ldn(xk + i + B * SP);
        return mf_circ(va, vb, vc, vd);
    };
    int e = (c[A] * M.es[A] + c[B] * M.es[B] + p0 * M.es[N]) * SP;
    int face = (M.fb[N] + c[A] * M.fs[N][A] + c[B] * M.fs[N][B] + p0 * M.fs[N][N]) * SP + k;
    int cell = N * (int)M.ncell + c[A] * M.cs[A] + c[B] * M.cs[B] + p0 * M.cs[N];
    cdf fm = fat(p0 - 1, e - es), f0 = fat(p0, e);
    df wa = d2f(__ldg(M.w + cell - M.cs[N]));
    for (int p = p0; p < p1; p++) {
        e += es;
        const df wb = d2f(__ldg(M.w + cell));
        const cdf fp = fat(p + 1, e);
        M.g[face] = to4(mf_g(wa, wb, fm, f0, fp));
        face += M.fs[N][N] * SP;
        cell += M.cs[N];
        wa = wb;
        fm = f0;
        f0 = fp;
    }
}

template <int SP>
__global__ void __launch_bounds__(kB, 4)
k_mf_gmarch(MF M, March G, const float4 *__restrict__ x, const SysState *sys, int rev)
{
    pdl_wait();
    const int k = threadIdx.x % SP;
    if (sys[k].status != kRun) return;
    const int rpb = kB / SP, nyz = G.ly * G.lz, cx = M.nx - 1;
    for (int qi = blockIdx.x * rpb + threadIdx.x / SP; qi < G.items; qi += gridDim.x * rpb) {
        const int q = sweep(qi, G.items, rev);
        const int tile = q / G.per_tile, r = q - tile * G.per_tile;
        const int tz = tile / G.ty, y0 = (tile - tz * G.ty) * G.ly, z0 = tz * G.lz;
        const int line = r / cx, i = r - line * cx;
        if (line < G.lz) {
            // y-normal columns (i, z)
            const int c[3] = {i, y0, z0 + line};
            if (c[2] < M.nz - 1) mf_face_march<SP, 1>(M, G.ly, c, x, k);
        } else if (line < G.lz + G.ly) {
            // z-normal columns (i, y)
            const int c[3] = {i, y0 + line - G.lz, z0};
            if (c[1] < M.ny - 1) mf_face_march<SP, 2>(M, G.lz, c, x, k);
        } else {
            // x-normal columns (y, z), chunks along x
            const int s = r - (G.lz + G.ly) * cx, ch = s / nyz, t = s - ch * nyz, jz = t / G.ly;
            const int c[3] = {ch * G.lx, y0 + t - jz * G.ly, z0 + jz};
            if (c[1] < M.ny - 1 && c[2] < M.nz - 1) mf_face_march<SP, 0>(M, G.lx, c, x, k);
        }
    }
}

constexpr int kEdgeValues = 7;    // x at R - 1, 0, R + 1; g of three faces; two weights
// the edges of direction D at c (c[Q]: the chunk's first position)
template <int SP, int D>
__device__ __forceinline__ void mf_edge_march(const MF &M, int len, const int (&c)[3], df om, int k,
                                              const float4 *__restrict__ x, float4 *__restrict__ z,
                                              SpmvTail &tail, Ring<kEdgeValues> ring)
{
    constexpr int Q = D == 2 ? 1 : 2, R = 3 - D - Q;
    constexpr bool FLIP = D == 1;                        // Q is D + 1 and not D + 2
    const int ext[3] = {M.nx, M.ny, M.nz};
    const int last = ext[Q] - 1, a = max(c[Q], 1), b = min(c[Q] + len, last);
    if (a >= b || c[R] == 0 || c[R] == ext[R] - 1) return;
    const float4 *__restrict__ xk = x + k;
    {
        const bool lo = c[R] == 1, hi = c[R] == ext[R] - 2;
        const int es = M.es[Q] * SP, er = M.es[R] * SP;
        // row m = a: its edge, the weight of the cell (R, a), the R-normal
        // face (R, a) and the Q-normal face (R, a)
        int e = (c[2] * M.plane + c[1] * M.l3 + 3 * c[0] + D) * SP + (a - c[Q]) * es;
        const int cell0 = (3 + D) * (int)M.ncell + c[R] * M.cs[R] + c[D] * M.cs[D];
        const int fr0 = (M.fb[R] + c[R] * M.fs[R][R] + c[D] * M.fs[R][D]) * SP + k, frq = M.fs[R][Q] * SP;
        const int fq0 = (M.fb[Q] + c[R] * M.fs[Q][R] + c[D] * M.fs[Q][D]) * SP + k, fqq = M.fs[Q][Q] * SP;
        const int fqr = M.fs[Q][R] * SP;
        // copies for row m (at edge i): line position m + 1, the faces and weights of row m
        auto copy = [&](int m, int i, int stage) {
            const bool in = m + 1 < last;
            const int j = in ? i + es : i;
            cp_async16_l1(ring.at(stage, 0), xk + (in && !lo ? j - er : j), in && !lo);
            cp_async16_l1(ring.at(stage, 1), xk + j, in);
            cp_async16_l1(ring.at(stage, 2), xk + (in && !hi ? j + er : j), in && !hi);
            cp_async16_l1(ring.at(stage, 3), M.g + fr0 + m * frq);
            cp_async16_l1(ring.at(stage, 4), M.g + fq0 + m * fqq - fqr);
            cp_async16_l1(ring.at(stage, 5), M.g + fq0 + m * fqq);
            float2 *w = reinterpret_cast<float2 *>(ring.at(stage, 6));
            cp_async8(w, M.w + cell0 + m * M.cs[Q] - M.cs[R]);
            cp_async8(w + 1, M.w + cell0 + m * M.cs[Q]);
        };
        int next = a, en = e, st_in = 0, st = 0;
#pragma unroll
        for (int s = 0; s < kStages - 1; s++) {
            if (next < b) copy(next, en, st_in);
            cp_async_commit();
            next++;
            en += es;
            st_in++;
        }
        // P_lo and P_hi of a line position (0 on the surface)
        auto sums = [&](cdf xc, cdf xl, cdf xh, acc2 &plo, acc2 &phi) {
            const cdf x2{add2(xc.h, xc.h), add2(xc.l, xc.l)};
            plo.start(x2);
            plo.add(xl);
            phi.start(x2);
            phi.add(xh);
        };
        auto line = [&](int i, acc2 &plo, acc2 &phi) {
            const cdf xc = cdf_of(__ldg(xk + i));
            sums(xc, lo ? czero() : cdf_of(__ldg(xk + i - er)), hi ? czero() : cdf_of(__ldg(xk + i + er)),
                 plo, phi);
            return xc;
        };
        acc2 pl0, ph0, pl1, ph1;
        if (a > 1) line(e - es, pl0, ph0);
        cdf x1 = line(e, pl1, ph1);
        df wl0 = d2f(__ldg(M.w + cell0 + (a - 1) * M.cs[Q] - M.cs[R])),
           wh0 = d2f(__ldg(M.w + cell0 + (a - 1) * M.cs[Q]));
        cdf gr = cdf_of(__ldg(M.g + fr0 + (a - 1) * frq));
        const cdf fom{pk(-om.h, om.h), pk(-om.l, om.l)};
        for (int m = a; m < b; m++) {
            if (next < b) copy(next, en, st_in);
            cp_async_commit();
            next++;
            en += es;
            st_in = st_in == kStages - 1 ? 0 : st_in + 1;
            cp_async_wait<kStages - 1>();
            auto value = [&](int v) { return cdf_of(*ring.at(st, v)); };
            const cdf x2 = value(1);
            acc2 pl2, ph2;
            sums(x2, value(0), value(2), pl2, ph2);
            const float4 w = *ring.at(st, 6);
            const df wl1{w.x, w.y}, wh1{w.z, w.w};
            // the mass part: 2 P(m) + P(m - 1) and 2 P(m) + P(m + 1)
            acc2 mm;
            auto cells = [&](const acc2 &p0, const acc2 &p1, const acc2 &p2, df w0, df w1, bool first) {
                const cdf d{add2(p1.h, p1.h), add2(p1.l, p1.l)};
                acc2 u, v;
                u.start(d);
                u.add(cdf{p0.h, p0.l});
                v.start(d);
                v.add(cdf{p2.h, p2.l});
                if (first) mm.first(both(w0), cdf{u.h, u.l});
                else mm.mac(both(w0), cdf{u.h, u.l});
                mm.mac(both(w1), cdf{v.h, v.l});
            };
            cells(pl0, pl1, pl2, wl0, wl1, true);
            cells(ph0, ph1, ph2, wh0, wh1, false);
            const cdf gn = value(3), ga = value(4), gb = value(5);
            acc2 kk;
            kk.start(FLIP ? gn : gr);
            kk.sub(FLIP ? gr : gn);
            kk.sub(FLIP ? gb : ga);
            kk.add(FLIP ? ga : gb);
            kk.mac(fom, cswap(mm.get()));
            tail.row(e + k, kk.get(), x1, z);
            st = st == kStages - 1 ? 0 : st + 1;
            e += es;
            gr = gn;
            pl0 = pl1; ph0 = ph1;
            pl1 = pl2; ph1 = ph2;
            wl0 = wl1; wh0 = wh1;
            x1 = x2;
        }
    }
}

template <int SP>
__global__ void __launch_bounds__(kB, 2)
k_mf_edges_g(MF M, March E, const float2 *__restrict__ omega, const float4 *__restrict__ s,
             float4 *__restrict__ z, SysState *sys, float4 *partials, int mode, int rev)
{
    pdl_wait();
    extern __shared__ __align__(16) float4 ring_smem[];
    const int k = threadIdx.x % SP;
    const bool on = sys[k].status == kRun;
    const df om = d2f(omega[k]);
    const Ring<kEdgeValues> ring{ring_smem};
    SpmvTail tail;
    const int rpb = kB / SP;
    for (int qi = blockIdx.x * rpb + threadIdx.x / SP; qi < E.items; qi += gridDim.x * rpb) {
        if (!on) break;
        const int q = sweep(qi, E.items, rev);
        const int tile = q / E.per_tile, r = q - tile * E.per_tile;
        const int tz = tile / E.ty;
        const int line = r / (M.nx - 1);
        int c[3] = {r - line * (M.nx - 1), (tile - tz * E.ty) * E.ly, tz * E.lz};
        // x- and y-edges: lines (x, y) along z; z-edges: lines (x, z) along y
        if (line < E.ly) {
            c[1] += line;
            if (c[1] < M.ny - 1) mf_edge_march<SP, 0>(M, E.lz, c, om, k, s, z, tail, ring);
        } else if (line < 2 * E.ly) {
            c[1] += line - E.ly;
            if (c[1] < M.ny - 1) mf_edge_march<SP, 1>(M, E.lz, c, om, k, s, z, tail, ring);
        } else {
            c[2] += line - 2 * E.ly;
            if (c[2] < M.nz - 1) mf_edge_march<SP, 2>(M, E.ly, c, om, k, s, z, tail, ring);
        }
    }
    // the rows on the outer surface are the identity
    for (int qi = blockIdx.x * rpb + threadIdx.x / SP; qi < M.ndir; qi += gridDim.x * rpb) {
        if (!on) break;
        const long long i = (long long)__ldg(M.dir + qi) * SP + k;
        const cdf sv = cdf_of(__ldg(s + i));
        tail.row(i, sv, sv, z);
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
                    const df xr{xv.x, xv.z}, xi{xv.y, xv.w};
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
                    kr_.mac(kd, df{xv.x, xv.z});
                    ki_.mac(kd, df{xv.y, xv.w});
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
// (1.8M edges x 2 systems: k_edge 95 -> 57 us, this kernel 16 us an iteration,
// two thirds of it arithmetic).  A whole group's s values are in flight per
// thread (1.8M x 2: 260 us a group with 4, 251 with 16); the lanes' coefficients
// lie side by side (512 bytes apart they met in one bank: 234,000 x 16 424 -> 258 us).
template <int SP>
__global__ void __launch_bounds__(kB, 3)
k_group(long long n, float4 *__restrict__ s, float4 *__restrict__ p, double2 *__restrict__ x,
        const float4 *__restrict__ hist, const SysState *sys, int rev)
{
    pdl_wait();
    __shared__ float4 ab[kGroupIters * 2][SP];
    for (int i = threadIdx.x; i < SP * kGroupIters * 2; i += kB) ab[i % (kGroupIters * 2)][i / (kGroupIters * 2)] = hist[i];
    __syncthreads();
    const int k = threadIdx.x % SP;
    const int cnt = sys[k].cnt;
    if (cnt == 0) return;
    const long long stride = (long long)gridDim.x * kB;
    for (long long ii = (long long)blockIdx.x * kB + threadIdx.x; ii < n; ii += stride) {
        // n is a multiple of SP: a backward sweep by rows keeps the lane's system
        const long long i = rev ? n - SP - (ii - k) + k : ii;
        cdf pv = ldg(p + i), d = czero();
        const double2 xv = x[i];
        const cdf last = ldg(s + cnt * n + i);
        int j = 0;
        // U of the group's iterations, their loads in flight together
        auto steps = [&](auto u_) {
            constexpr int U = decltype(u_)::value;
            for (; j + U <= cnt; j += U) {
                cdf sv[U];
#pragma unroll
                for (int u = 0; u < U; u++) sv[u] = ldg(s + (j + u) * n + i);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    pv = caxpy(sv[u], cfac_of(from4(ab[2 * (j + u) + 1][k])), pv);
                    d = caxpy(d, cfac_of(from4(ab[2 * (j + u)][k])), pv);
                }
            }
        };
        steps(std::integral_constant<int, 16>{});
        steps(std::integral_constant<int, 4>{});
        steps(std::integral_constant<int, 1>{});
        const double2 dv = to_d2(to4(d));
        x[i] = make_double2(xv.x + dv.x, xv.y + dv.y);
        p[i] = to4(pv);
        s[i] = to4(last);
    }
}

}  // namespace sv
}  // namespace mtgpu
#include "survey_small.cuh"
namespace mtgpu {
namespace sv {

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
    // The work of the marching kernels.  Chunk lengths: an item costs its
    // positions plus about 3 for its start (the neighbours' values, the first
    // loads' latency), so the length is the one with the least rounds of
    // resident threads times that cost: 16 on large problems, down to 1 where
    // longer ones would leave the chip idle.  Axes are cut evenly (41 cells
    // into 3 chunks of 14, not 2 of 16 and one of 9).
    static March march(const Survey &V, bool faces, long long threads)
    {
        const int cx = V.mf.nx - 1, cy = V.mf.ny - 1, cz = V.mf.nz - 1;
        March best;
        long long cost = -1;
        for (int len = 16; len >= 1; len--) {
            March G;
            G.ty = ceil_div(cy, len);
            G.tz = ceil_div(cz, len);
            G.ly = ceil_div(cy, G.ty);
            G.lz = ceil_div(cz, G.tz);
            G.lx = ceil_div(cx, ceil_div(cx, len));
            G.ty = ceil_div(cy, G.ly);
            G.tz = ceil_div(cz, G.lz);
            G.per_tile = faces ? (G.lz + G.ly) * cx + ceil_div(cx, G.lx) * G.ly * G.lz : (2 * G.ly + G.lz) * cx;
            G.items = G.ty * G.tz * G.per_tile;
            const long long c = ((long long)G.items * SP + threads - 1) / threads *
                                (std::max({G.ly, G.lz, faces ? G.lx : 1}) + 3);
            if (cost < 0 || c < cost) {
                cost = c;
                best = G;
            }
        }
        return best;
    }
    static constexpr int kEdgeSmem = kStages * kEdgeValues * kB * 16;
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
        M.dir = F.dir;
        M.ndir = F.ndir;
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
            pdl(k_mf_gmarch<SP>, V.g_mfg, kB, 0, V.st, M, V.mg, s, V.sys, flip(V));
            pdl(k_mf_edges_g<SP>, V.g_mfe3, kB, kEdgeSmem, V.st, M, V.me, V.omega, s, V.z, V.sys,
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
        if (small_used(V)) {
            if (j == 0) small(V, std::min(V.group, n - t));
            return;
        }
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
            // (the iteration's sweep directions, and with them its sums, do not
            // depend on the group's length)
            group(V);
    }
    static void group(Survey &V)
    {
        pdl(k_group<SP>, V.g_group, kB, 0, V.st, (long long)V.nb * SP, V.s, V.p, V.xacc, V.hist,
            V.sys, V.dir ^ 1);
    }
    // n iterations (a group, or what is left of the sequence) in one launch
    static void small(Survey &V, int n)
    {
        const SmallArgs A{V.nb, V.ds, V.da, V.G.d_tn, V.omega, V.r, V.a, V.w, V.sm,
                          V.z, V.s, V.sys, V.hist, V.partials};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = V.g_small;
        cfg.blockDim = V.small_threads + 32;
        cfg.dynamicSmemBytes = (size_t)V.small_items * kSmallItemBytes * V.small_threads;
        cfg.stream = V.st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, k_small<SP>, mfd(V), A, n, V.small_items);
        group(V);
    }
    // the grid of k_small and its rows x systems per thread; grid 0: not used.
    // Variant 35 on a lattice mesh, one block per SM; the batches of a survey
    // run side by side, which launches that need every SM would prevent
    static void small_grid(Survey &V, int nsm)
    {
        V.g_small = 0;
        const long long n = (long long)V.nb * SP;
        if (V.ch != kMatFree + 3 || !V.mf.on || !V.mf.gface || !V.g_lat || !V.G.d_tn) return;
        if (n > (long long)nsm * kSmallThreads * kSmallItems) return;
        if (SP > kSmallSystems || !V.alone || !one_kernel_wanted()) return;
        if ((size_t)nsm * 8 * SP > 2 * (partial_slots(V.pblocks, SP) - kTicketSlots)) return;
        // as few rows per thread as fit, the rows even over the SMs
        const int items = (int)((n + (long long)nsm * kSmallThreads - 1) / ((long long)nsm * kSmallThreads));
        const int per = (int)((n + (long long)nsm * items - 1) / ((long long)nsm * items));
        const int nt = std::max(kSmallMin, ceil_div(per, 32) * 32);
        const int grid = (int)std::min<long long>(nsm, (n + nt - 1) / nt);
        const int smem = items * kSmallItemBytes * nt;
        int dev = 0, coop = 0, b = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
            cudaFuncSetAttribute((const void *)k_small<SP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kSmallItems * kSmallItemBytes * kSmallThreads) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)k_small<SP>, nt + 32, smem) !=
                cudaSuccess || b < 1) {
            cudaGetLastError();
            return;
        }
        V.g_small = grid;
        V.small_items = items;
        V.small_threads = nt;
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
            auto gs = [&](const void *f, int smem, bool faces, March &G) {
                int b = 0;
                if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kB, smem) != cudaSuccess || b < 1) {
                    cudaGetLastError();
                    b = 1;
                }
                G = march(V, faces, (long long)b * nsm * kB);
                return std::max(1, std::min(b * nsm, ceil_div(G.items, kB / SP)));
            };
            V.g_mfg = gs((const void *)k_mf_gmarch<SP>, 0, true, V.mg);
            V.g_mfe3 = gs((const void *)k_mf_edges_g<SP>, kEdgeSmem, false, V.me);
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
        small_grid(V, nsm);
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
