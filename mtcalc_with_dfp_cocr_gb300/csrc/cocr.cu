// Preconditioned COCR for complex-symmetric systems, FP64, on the device.
//
// The recurrences are the reference's PCOCR_RCI::Run
// (Code/COCR_FP/pcocr_rci.cpp:52-181): unconjugated bilinear dots
// (base_solver.cpp:382-399), alpha = (z,s)/(a,w), beta = (z,s)_new/(z,s)_old,
// the stop test on the MRS-smoothed residual relative to ||b||
// (MRS.cpp:85-153, rci.cpp:66-75), REQ_DIV_BY_ZERO when (a,w) vanishes.
//
// One iteration is four kernels, captured into a CUDA graph several
// iterations at a time (up to 219,000 rows on 152 SMs: phases of one
// cooperative kernel, cocr_small.cuh); every decision (alpha, beta, the MRS weight, the
// stop test, the iteration limit) is taken on the device by the last block
// of the kernel that finishes the reduction, so the host only looks at the
// status word between graph launches.
//   k_it_node   h = D_S G (z + beta a)                      [node gather]
//   k_it_edge   p = s + beta p, a = z + beta a,
//               w = D_A a + G^T h, (a,w)  -> alpha            [edge gather]
//   k_it_update x += alpha p, r -= alpha a, s -= alpha w,
//               MRS weight from (s_m, r - s_m), |r - s_m|^2
//   k_it_spmv   z = A s, MRS smoothing of s_m, |s_m|, (z,s)
//               -> stop test, beta
// Reductions are two-level (fixed per-block partials, then the last block
// sums them in a fixed order), so results do not change run to run.
#include "mtgpu_internal.cuh"

namespace mtgpu {

enum : int { kRunning = 1 };

struct Ctl {
    int status;          // kRunning or a final MTGPU_* code
    int iter;            // number of the iteration in progress / at exit
    int maxiter;
    int mrs_mode;        // 0 keep s_m, 1 s_m = r, 2 s_m += w (r - s_m)
    double mrs_w;
    double eps;
    double r_old;        // ||b||
    double residual;     // ||s_m||
    double residual_rel;
    double2 alpha, beta, zs;
    double2 *x;          // the solution being updated (the graph does not depend on it)
    double sums[4];      // scratch results of one-off reductions
    unsigned int ticket[4];
    unsigned int bar, left;   // k_small64: barrier arrivals, blocks that left
    int failed, polls;        // ... a wait ran out (set by kernels, cleared by the host); its bound
};

namespace {

constexpr int kRedThreads = 256;   // threads of a reducing block

// ---------------------------------------------------------- reductions
// Sums of N <= 4 FP64 values over the block, totals in threads t < N: lanes
// exchange halves until each holds one value (6 adds a warp for 3 or 4 values
// instead of 15 or 20; GB300 issues an FP64 add of a warp once in 16 cycles),
// then thread t adds the warps' sums.
template <int N>
__device__ inline double block_sum(const double (&v)[N], double (*smem)[4] /* [32] */)
{
    constexpr int P = N <= 1 ? 1 : (N <= 2 ? 2 : 4);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double u[P];
#pragma unroll
    for (int k = 0; k < P; k++) u[k] = k < N ? v[k] : 0.0;
    int first = 0, o = 16;
#pragma unroll
    for (int h = P / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
        first += up ? h : 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const double mine = up ? u[i + h] : u[i], give = up ? u[i] : u[i + h];
            u[i] = mine + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    const int rest = 2 * o;
#pragma unroll
    for (; o >= 1; o >>= 1) u[0] += __shfl_xor_sync(0xffffffffu, u[0], o);
    if ((lane & (rest - 1)) == 0) smem[warp][first] = u[0];
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < N)
        for (int q = 0; q < nw; q++) s += smem[q][threadIdx.x];
    return s;
}

// Publish this block's partial sums; returns true in the one block that
// arrives last, which then holds the grid totals in v (thread 0).  Each of
// its threads adds whole partials, 12 loads in flight.
template <int N>
__device__ bool grid_sum(double (&v)[N], double *partials, unsigned int *ticket)
{
    __shared__ double smem[2][32][4];
    __shared__ double tot[4];
    __shared__ bool last;
    const double s = block_sum<N>(v, smem[0]);
    if (threadIdx.x < N) __stcg(partials + (size_t)blockIdx.x * 4 + threadIdx.x, s);
    __syncthreads();
    if (threadIdx.x == 0) {
        last = count_arrival(ticket) == gridDim.x - 1;
        if (last) *ticket = 0u;
    }
    __syncthreads();
    if (!last) return false;
    constexpr int U = 12;
    double acc[N] = {};
    for (int b0 = 0; b0 < (int)gridDim.x; b0 += U * blockDim.x) {
        double2 l[U], h[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int b = b0 + u * blockDim.x + threadIdx.x;
            const double2 *q = reinterpret_cast<const double2 *>(partials) + 2 * (size_t)b;
            const bool in = b < (int)gridDim.x;
            l[u] = in ? __ldcg(q) : make_double2(0.0, 0.0);
            if (N > 2) h[u] = in ? __ldcg(q + 1) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            acc[0] += l[u].x;
            if (N > 1) acc[N > 1 ? 1 : 0] += l[u].y;
            if (N > 2) acc[N > 2 ? 2 : 0] += h[u].x;
        }
    }
    const double r = block_sum<N>(acc, smem[1]);
    if (threadIdx.x < N) tot[threadIdx.x] = r;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = tot[k];
    return true;
}

__device__ inline bool running(const Ctl *c) { return *(volatile const int *)&c->status == kRunning; }

// ------------------------------------------------------------ set-up
// r = b - A x is computed by the SpMV kernel; this one finishes stage 2:
// ||b||, ||r||, the x0 test (rci.cpp:79-88) and MRS initialisation s_m = r.
__global__ void __launch_bounds__(kRedThreads)
k_init_norms(int nb, const double2 *__restrict__ b, const double2 *__restrict__ r,
             double2 *__restrict__ sm, Ctl *ctl, double *partials)
{
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
        const double2 bv = b[i], rv = r[i];
        v[0] += bv.x * bv.x + bv.y * bv.y;
        v[1] += rv.x * rv.x + rv.y * rv.y;
        sm[i] = rv;
    }
    if (grid_sum<2>(v, partials, &ctl->ticket[0]) && threadIdx.x == 0) {
        ctl->r_old = v[0] > 0.0 ? sqrt(v[0]) : 0.0;
        ctl->residual = v[1] > 0.0 ? sqrt(v[1]) : 0.0;
        ctl->residual_rel = ctl->r_old > 0.0 ? ctl->residual / ctl->r_old : 0.0;
        ctl->beta = make_double2(0.0, 0.0);
        ctl->iter = 1;
        if (ctl->residual < 1e-30) {
            ctl->status = MTGPU_X0_NULL;
            ctl->iter = 0;
            ctl->residual_rel = 1.0;   // the RCI's initial residualRel (rci.cpp:40)
        } else if (ctl->maxiter < 1) ctl->status = MTGPU_MAXITER;
        else ctl->status = kRunning;
    }
}

// zs = (z, s) for the first iteration (stage 4 -> 5)
__global__ void __launch_bounds__(kRedThreads)
k_init_zs(int nb, const double2 *__restrict__ z, const double2 *__restrict__ s, Ctl *ctl,
          double *partials)
{
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
        const double2 a = z[i], c = s[i];
        v[0] += a.x * c.x - a.y * c.y;
        v[1] += a.x * c.y + a.y * c.x;
    }
    if (grid_sum<2>(v, partials, &ctl->ticket[0]) && threadIdx.x == 0)
        ctl->zs = make_double2(v[0], v[1]);
}

// ||b - A x||^2 and ||b||^2 of a residual vector already formed
__global__ void __launch_bounds__(kRedThreads)
k_norm2(int nb, const double2 *__restrict__ r, const double2 *__restrict__ b, Ctl *ctl,
        double *partials)
{
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
        const double2 rv = r[i], bv = b[i];
        v[0] += rv.x * rv.x + rv.y * rv.y;
        v[1] += bv.x * bv.x + bv.y * bv.y;
    }
    if (grid_sum<2>(v, partials, &ctl->ticket[0]) && threadIdx.x == 0) {
        ctl->sums[0] = v[0];
        ctl->sums[1] = v[1];
    }
}

// ------------------------------------------------------- the iteration
__global__ void __launch_bounds__(kThreads, 2)
k_it_node(int m, const int *__restrict__ gp, const int *__restrict__ gj,
          const double *__restrict__ gv, const double2 *__restrict__ ds,
          const double2 *__restrict__ z, const double2 *__restrict__ a,
          double2 *__restrict__ h, const Ctl *ctl)
{
    pdl_wait();
    if (!running(ctl)) return;
    const double2 beta = ctl->beta;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x) {
        // up to six entries (all of a conforming mesh) with their loads in
        // flight together; one at a time each waits for two
        const int j0 = gp[v], n = gp[v + 1] - j0;
        const double2 dsv = ds[v];
        int e[6];
        double g[6];
        double2 zv[6], av[6];
#pragma unroll
        for (int q = 0; q < 6; q++) {
            e[q] = q < n ? gj[j0 + q] : 0;
            g[q] = q < n ? gv[j0 + q] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 6; q++)
            if (q < n) {
                zv[q] = z[e[q]];
                av[q] = a[e[q]];
            }
        double hr = 0.0, hi = 0.0;
#pragma unroll
        for (int q = 0; q < 6; q++)
            if (q < n) {
                const double2 an = cadd(zv[q], cmul(beta, av[q]));
                hr += g[q] * an.x;
                hi += g[q] * an.y;
            }
        for (int j = j0 + 6; j < j0 + n; j++) {          // T-matrix rows only
            const int k = gj[j];
            const double2 an = cadd(z[k], cmul(beta, a[k]));
            hr += gv[j] * an.x;
            hi += gv[j] * an.y;
        }
        h[v] = cmul(make_double2(hr, hi), dsv);
    }
}

__global__ void __launch_bounds__(kRedThreads, 3)
k_it_edge(int n, const int *__restrict__ tp, const int *__restrict__ tj,
          const double *__restrict__ tv, const int2 *__restrict__ tn, const double2 *__restrict__ da,
          const double2 *__restrict__ h, const double2 *__restrict__ s,
          const double2 *__restrict__ z, double2 *__restrict__ p, double2 *__restrict__ a,
          double2 *__restrict__ w, Ctl *ctl, double *partials)
{
    pdl_wait();
    if (!running(ctl)) return;
    const double2 zs = ctl->zs;
    const double2 beta = ctl->beta;
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        // G^T row of a conforming mesh: its two nodes' rows (one dependent
        // load), -1/2 and +1/2; else the CSR of T-matrix meshes
        const int2 row = tn ? tn[i] : make_int2(-1, -1);
        const double2 sv = s[i], po = p[i], zv = z[i], ao = a[i], dav = da[i];
        double2 h0 = make_double2(0.0, 0.0), h1 = h0;
        if (row.x >= 0) h0 = h[row.x];
        if (row.y >= 0) h1 = h[row.y];
        const double2 pn = cadd(sv, cmul(beta, po));
        const double2 an = cadd(zv, cmul(beta, ao));
        double2 wn = cmul(an, dav);
        if (tn) {
            if (row.x >= 0) {
                wn.x += -0.5 * h0.x;
                wn.y += -0.5 * h0.y;
            }
            if (row.y >= 0) {
                wn.x += 0.5 * h1.x;
                wn.y += 0.5 * h1.y;
            }
        } else {
            for (int j = tp[i]; j < tp[i + 1]; j++) {
                const double2 hv = h[tj[j]];
                wn.x += tv[j] * hv.x;
                wn.y += tv[j] * hv.y;
            }
        }
        p[i] = pn;
        a[i] = an;
        w[i] = wn;
        v[0] += an.x * wn.x - an.y * wn.y;
        v[1] += an.x * wn.y + an.y * wn.x;
    }
    if (grid_sum<2>(v, partials, &ctl->ticket[1]) && threadIdx.x == 0) {
        const double2 aw = make_double2(v[0], v[1]);
        if (fabs(aw.x) < 1e-40 && fabs(aw.y) < 1e-40) {
            ctl->status = MTGPU_DIV_BY_ZERO;
        } else {
            ctl->alpha = cquot(zs, aw);
        }
    }
}

__global__ void __launch_bounds__(kRedThreads, 3)
k_it_update(int n, const double2 *__restrict__ p, const double2 *__restrict__ a,
            const double2 *__restrict__ w, const double2 *__restrict__ sm,
            double2 *__restrict__ r, double2 *__restrict__ s, Ctl *ctl, double *partials)
{
    pdl_wait();
    if (!running(ctl)) return;
    double2 *const x = ctl->x;
    const double2 al = ctl->alpha;
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        x[i] = cadd(x[i], cmul(al, p[i]));
        const double2 rn = csub(r[i], cmul(al, a[i]));
        r[i] = rn;
        s[i] = csub(s[i], cmul(al, w[i]));
        const double2 sv = sm[i];
        const double ux = rn.x - sv.x, uy = rn.y - sv.y;
        v[0] += sv.x * ux + sv.y * uy;
        v[1] += ux * ux + uy * uy;
    }
    if (grid_sum<2>(v, partials, &ctl->ticket[2]) && threadIdx.x == 0) {
        const double su = v[0], uu = v[1];
        const double wm = fabs(uu) < 1e-100 ? 0.0 : -su / uu;
        if (wm < 0.0) {
            ctl->mrs_mode = 0;
        } else if (wm > 1.0) {
            ctl->mrs_mode = 1;
        } else {
            ctl->mrs_mode = 2;
            ctl->mrs_w = wm;
        }
    }
}

__global__ void __launch_bounds__(kRedThreads, 3)
k_it_spmv(int nb, const int *__restrict__ wc, const int *__restrict__ wr,
          const long long *__restrict__ pc, const long long *__restrict__ pr,
          const int *__restrict__ col_c, const double2 *__restrict__ val_c,
          const int *__restrict__ col_r, const double *__restrict__ val_r,
          const double2 *__restrict__ s, const double2 *__restrict__ r,
          double2 *__restrict__ z, double2 *__restrict__ sm, Ctl *ctl, double *partials)
{
    pdl_wait();
    if (!running(ctl)) return;
    const double2 zs = ctl->zs;
    const double residual = ctl->residual, r_old = ctl->r_old, eps = ctl->eps;
    const int iter = ctl->iter, maxiter = ctl->maxiter;
    const int mode = ctl->mrs_mode;
    const double wm = ctl->mrs_w;
    double v[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x) {
        const int sl = i / kSlice, l = i % kSlice;
        double ar = 0.0, ai = 0.0;
        {
            const long long base = pc[sl] + l;
            const int wdt = wc[sl];
#pragma unroll 4
            for (int k = 0; k < wdt; k++) {
                const double2 vv = val_c[base + (long long)k * kSlice];
                const double2 xv = s[col_c[base + (long long)k * kSlice]];
                ar += vv.x * xv.x - vv.y * xv.y;
                ai += vv.x * xv.y + vv.y * xv.x;
            }
        }
        {
            const long long base = pr[sl] + l;
            const int wdt = wr[sl];
#pragma unroll 8
            for (int k = 0; k < wdt; k++) {
                const double vv = val_r[base + (long long)k * kSlice];
                const double2 xv = s[col_r[base + (long long)k * kSlice]];
                ar += vv * xv.x;
                ai += vv * xv.y;
            }
        }
        z[i] = make_double2(ar, ai);
        const double2 si = s[i];
        v[0] += ar * si.x - ai * si.y;
        v[1] += ar * si.y + ai * si.x;
        if (mode != 0) {
            double2 smv = r[i];
            if (mode == 2) {
                const double2 old = sm[i];
                smv = make_double2(old.x + wm * (smv.x - old.x), old.y + wm * (smv.y - old.y));
            }
            sm[i] = smv;
            v[2] += smv.x * smv.x + smv.y * smv.y;
        }
    }
    if (grid_sum<3>(v, partials, &ctl->ticket[3]) && threadIdx.x == 0) {
        // (independent FP64 chains side by side)
        const double2 zs_new = make_double2(v[0], v[1]);
        const double2 beta = cquot(zs_new, zs);
        const double res = mode != 0 ? sqrt(v[2]) : residual;
        const double rel = res / r_old;
        ctl->residual = res;
        ctl->residual_rel = rel;
        ctl->beta = beta;
        ctl->zs = zs_new;
        if (rel < eps) {
            ctl->status = MTGPU_OK;
        } else {
            ctl->iter = iter + 1;
            if (iter + 1 > maxiter) ctl->status = MTGPU_MAXITER;
        }
    }
}

}  // namespace
}  // namespace mtgpu
#include "cocr_small.cuh"
namespace mtgpu {

// ---------------------------------------------------------------- solver
void CocrSolver::release()
{
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
    A.release();
    P.release();
    dev_free(r); dev_free(p); dev_free(s); dev_free(z); dev_free(a); dev_free(w); dev_free(sm);
    dev_free(partials);
    dev_free(ctl);
    if (hctl) cudaFreeHost(hctl);
    hctl = nullptr;
}

int cocr_alloc(CocrSolver &S)
{
    const int nb = S.nb;
    int dev = 0, nsm = 0;
    MTGPU_TRY(cudaGetDevice(&dev));
    MTGPU_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    // blocks of 256, as many as are resident (the loops are grid-stride)
    int occ = 64;
    const void *fs[] = {(const void *)k_it_edge, (const void *)k_it_update, (const void *)k_it_spmv,
                        (const void *)k_init_norms};
    for (const void *f : fs) {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, kRedThreads, 0) == cudaSuccess && b > 0)
            occ = std::min(occ, b);
    }
    S.grid = std::max(1, std::min(ceil_div(nb, kRedThreads), occ * nsm));
    small_grid(S, dev, nsm);
    int rc;
    if ((rc = dev_alloc(&S.r, nb)) || (rc = dev_alloc(&S.p, nb)) || (rc = dev_alloc(&S.s, nb)) ||
        (rc = dev_alloc(&S.z, nb)) || (rc = dev_alloc(&S.a, nb)) || (rc = dev_alloc(&S.w, nb)) ||
        (rc = dev_alloc(&S.sm, nb)) || (rc = dev_alloc(&S.partials, (size_t)std::max(4 * S.grid, 7 * nsm))) ||
        (rc = dev_alloc(&S.ctl, 1)))
        return rc;
    MTGPU_TRY(cudaMallocHost((void **)&S.hctl, sizeof(Ctl)));
    MTGPU_TRY(cudaMemsetAsync(S.ctl, 0, sizeof(Ctl), S.st));
    return MTGPU_OK;
}

static void launch_iteration(CocrSolver &S)
{
    const Folded &P = S.P;
    const SellMatrix &A = S.A;
    const int nb = S.nb, g = S.grid, th = kRedThreads;
    if (P.m > 0)
        pdl(k_it_node, std::max(1, std::min(ceil_div(P.m, th), g)), th, 0, S.st, P.m, P.d_gp, P.d_gj,
            P.d_gv, P.d_ds, S.z, S.a, P.d_h, S.ctl);
    pdl(k_it_edge, g, th, 0, S.st, nb, P.d_tp, P.d_tj, P.d_tv, P.d_tn, P.d_da, P.d_h, S.s, S.z, S.p, S.a, S.w,
        S.ctl, S.partials);
    pdl(k_it_update, g, th, 0, S.st, nb, S.p, S.a, S.w, S.sm, S.r, S.s, S.ctl, S.partials);
    pdl(k_it_spmv, g, th, 0, S.st, nb, A.d_wc, A.d_wr, A.d_pc, A.d_pr, A.d_col_c, A.d_val_c, A.d_col_r,
        A.d_val_r, S.s, S.r, S.z, S.sm, S.ctl, S.partials);
}

static int kernels_per_iteration(const CocrSolver &S) { return S.P.m > 0 ? 4 : 3; }

static int build_graph(CocrSolver &S, int iters)
{
    if (S.graph) cudaGraphExecDestroy(S.graph);
    S.graph = nullptr;
    cudaGraph_t g;
    MTGPU_TRY(cudaStreamBeginCapture(S.st, cudaStreamCaptureModeThreadLocal));
    if (S.g_small) launch_small(S, iters);
    else
        for (int k = 0; k < iters; k++) launch_iteration(S);
    MTGPU_TRY(cudaStreamEndCapture(S.st, &g));
    cudaError_t e = cudaGraphInstantiate(&S.graph, g, 0);
    cudaGraphDestroy(g);
    MTGPU_TRY(e);
    S.graph_iters = iters;
    return MTGPU_OK;
}

static int sync_ctl(CocrSolver &S)
{
    MTGPU_TRY(cudaMemcpyAsync(S.hctl, S.ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, S.st));
    MTGPU_TRY(cudaStreamSynchronize(S.st));
    return MTGPU_OK;
}

// true relative residual ||b - A x|| / ||b|| (FP64), via S.w as scratch
static int true_residual(CocrSolver &S, const double2 *b, const double2 *x, double *out)
{
    sell_residual(S.A, b, x, S.w, S.st);
    k_norm2<<<S.grid, kRedThreads, 0, S.st>>>(S.nb, S.w, b, S.ctl, S.partials);
    note_launches(2);
    MTGPU_TRY(cudaGetLastError());
    int rc = sync_ctl(S);
    if (rc) return rc;
    const double rr = S.hctl->sums[0], bb = S.hctl->sums[1];
    *out = bb > 0.0 ? sqrt(rr) / sqrt(bb) : 0.0;
    return MTGPU_OK;
}

int cocr_solve(CocrSolver &S, const double2 *b, double2 *x, double eps, int maxiter,
               int stop_true, int iters_per_launch, mtgpu_solve_stats *stats)
{
    const int nb = S.nb;
    if (iters_per_launch <= 0) iters_per_launch = S.g_small ? kSmallIters : 16;
    Ctl init{};
    init.status = kRunning;
    init.maxiter = maxiter;
    init.eps = eps;
    init.x = x;
    init.polls = barrier_polls();
    MTGPU_TRY(cudaMemcpyAsync(S.ctl, &init, sizeof(Ctl), cudaMemcpyHostToDevice, S.st));
    // stages 1-4 of PCOCR_RCI::Run
    sell_residual(S.A, b, x, S.r, S.st);                                    // r = b - A x
    k_init_norms<<<S.grid, kRedThreads, 0, S.st>>>(nb, b, S.r, S.sm, S.ctl, S.partials);
    folded_apply(S.P, S.r, S.s, S.st);                                      // s = M^-1 r
    MTGPU_TRY(cudaMemsetAsync(S.p, 0, sizeof(double2) * nb, S.st));
    MTGPU_TRY(cudaMemsetAsync(S.a, 0, sizeof(double2) * nb, S.st));
    MTGPU_TRY(cudaMemsetAsync(S.w, 0, sizeof(double2) * nb, S.st));
    sell_spmv(S.A, S.s, S.z, S.st);                                         // z = A s
    k_init_zs<<<S.grid, kRedThreads, 0, S.st>>>(nb, S.z, S.s, S.ctl, S.partials);
    note_launches(S.P.m > 0 ? 6 : 5);
    MTGPU_TRY(cudaGetLastError());
    int rc = sync_ctl(S);
    if (rc) return rc;

    if (S.graph == nullptr || S.graph_iters != iters_per_launch)
        if ((rc = build_graph(S, iters_per_launch))) return rc;

    const unsigned long long kpi = (unsigned long long)kernels_per_iteration(S);
    double true_rr = -1.0;
    // a launch runs at least one iteration and the device stops at maxiter, so
    // maxiter + 2 launches are enough; looking at a stop and going on is none
    for (long long left = (long long)maxiter + 2;;) {
        if (S.hctl->status != kRunning) {
            if (S.hctl->status == MTGPU_OK && stop_true) {
                if ((rc = true_residual(S, b, x, &true_rr))) return rc;
                if (true_rr >= eps) {
                    // keep iterating: the recurrences already hold the next
                    // iteration's z, s and beta
                    Ctl c = *S.hctl;
                    c.status = kRunning;
                    c.iter += 1;
                    if (c.iter > c.maxiter) c.status = MTGPU_MAXITER;
                    MTGPU_TRY(cudaMemcpyAsync(S.ctl, &c, sizeof(Ctl), cudaMemcpyHostToDevice, S.st));
                    if ((rc = sync_ctl(S))) return rc;
                    true_rr = -1.0;
                    continue;
                }
            }
            break;
        }
        if (left-- <= 0) {
            set_last_message("COCR loop ended without a final status");
            return MTGPU_ERR_TIMEOUT;
        }
        MTGPU_TRY(cudaGraphLaunch(S.graph, S.st));
        note_launches(S.g_small ? 1 : kpi * (unsigned long long)iters_per_launch);
        if ((rc = sync_ctl(S))) return rc;
        if (S.hctl->failed) {
            set_last_message("COCR: a grid barrier did not complete");
            return MTGPU_ERR_TIMEOUT;
        }
    }
    if (true_rr < 0.0 && (rc = true_residual(S, b, x, &true_rr))) return rc;
    if (stats) {
        stats->iterations = S.hctl->iter;
        stats->residual_rel = S.hctl->residual_rel;
        stats->true_residual_rel = true_rr;
        stats->status = S.hctl->status;
        stats->spmv_variant = -1;
        stats->matfree_check = -1.0;
    }
    return S.hctl->status;
}

}  // namespace mtgpu
