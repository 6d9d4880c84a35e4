// FP64 iterations of a small problem in one cooperative kernel (included by cocr.cu).
#pragma once

namespace mtgpu {
namespace {

// The iteration's four kernels as phases of one launch of n iterations, a grid
// barrier between them.  On 45,000 rows the kernels take 48 us an iteration, of
// which FP64 arithmetic (the pipe issues an operation of a warp once in 16
// cycles: 190 a row) is 15; the rest are launches, ramps, first loads and the
// last blocks' serial ends.  Here a block keeps its rows of the recurrences'
// vectors (x, p, a, w, r, s, s_m and the diagonal) in shared memory, so only z, a, h
// and s pass through L2; every block adds the blocks' partials itself, in
// the same order, and so takes the same decisions; the MRS weight is formed by a
// warp of its own beside the product.  Operations and their order within a
// row are the separate kernels'; the sums' grouping differs.
//
// Measured, per iteration with the solve's ends: 26,500 rows 46 -> 26 us, 45,000
// 48 -> 33, 104,500 79 -> 53, 217,000 (3 rows a thread) 135 -> 93 (all but the
// 48 against blocks of 256 threads).  Beyond 3 rows a thread shared memory ends.
constexpr int kSmallThreads = 480;     // threads with rows, at most; one warp more for the MRS weight
constexpr int kSmallMin = 128;         // ... at least
constexpr int kSmallItems = 3;         // rows per thread, at most
constexpr int kSmallItemBytes = 8 * sizeof(double2) + sizeof(int2);
constexpr int kSmallIters = 64;        // iterations a launch where the caller leaves it open

struct Small64 {
    int nb, m;
    const int *gp, *gj;
    const double *gv;
    const double2 *ds;
    const int *tp, *tj;
    const double *tv;
    const int2 *tn;
    const double2 *da;
    const int *wc, *wr;
    const long long *pc, *pr;
    const int *col_c, *col_r;
    const double2 *val_c;
    const double *val_r;
    double2 *r, *p, *s, *z, *a, *w, *sm, *h;
    Ctl *ctl;
    double *partials;
};

// a vector element written in this launch (never the read-only path)
__device__ __forceinline__ double2 ld2(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}

// (re, im) += a b, unconjugated: two multiply-adds each
__device__ __forceinline__ void dot_add(double &re, double &im, double2 a, double2 b)
{
    re = fma(-a.y, b.y, fma(a.x, b.x, re));
    im = fma(a.y, b.x, fma(a.x, b.y, im));
}

// the sums of N <= 4 values over the block's first nw warps to part[value][block]
template <int N>
__device__ __forceinline__ void small_block(const double (&v)[N], int nw, double (*sm)[4], double *part)
{
    constexpr int P = N <= 2 ? 2 : 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
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
    if (warp < nw && (lane & (rest - 1)) == 0) sm[warp][first] = u[0];
    __syncthreads();
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int q = lane / P; q < nw; q += 32 / P) s += sm[q][lane % P];
#pragma unroll
        for (int d = 16; d >= P; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane < N) __stcg(part + (size_t)lane * gridDim.x + blockIdx.x, s);
    }
}

__global__ void __launch_bounds__(kSmallThreads + 32, 1)
k_small64(const __grid_constant__ Small64 A, int n, int items)
{
    __shared__ Ctl c;
    __shared__ double sums[kSmallThreads / 32][4], tot[4];
    __shared__ int late;
    extern __shared__ double2 own64[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int NT = blockDim.x - 32, nw = NT / 32, B = gridDim.x;
    const bool work = tid < NT;        // the last warp has no rows
    const int stride = B * NT, row0 = work ? blockIdx.x * NT + tid : A.nb;
    double2 *ox = own64 + tid, *op = ox + items * NT, *oa = op + items * NT, *ow = oa + items * NT,
            *orr = ow + items * NT, *os = orr + items * NT, *osm = os + items * NT, *oda = osm + items * NT;
    int2 *otn = reinterpret_cast<int2 *>(own64 + 8 * items * NT) + tid;
    double *part_e = A.partials, *part_u = part_e + 2 * B, *part_r = part_u + 2 * B;

    if (tid == 0) {
        c = *A.ctl;
        late = 0;
    }
    __syncthreads();
    GridBarrier bar{&A.ctl->bar};
    double2 *const x = c.x;
    for (int u = 0; u < items; u++) {
        const int i = row0 + u * stride;
        if (i >= A.nb) break;
        ox[u * NT] = x[i];
        op[u * NT] = A.p[i];
        oa[u * NT] = A.a[i];
        orr[u * NT] = A.r[i];
        os[u * NT] = A.s[i];
        osm[u * NT] = A.sm[i];
        oda[u * NT] = A.da[i];
        otn[u * NT] = A.tn ? A.tn[i] : make_int2(-1, -1);
    }
    bool any = false;
    for (int t = 0; t < n && c.status == kRunning; t++) {
        any = true;
        const double2 beta = c.beta;
        // h = D_S G (z + beta a) (k_it_node)
        for (int v = row0; v < A.m; v += stride) {
            const int j0 = A.gp[v], k = A.gp[v + 1] - j0;
            const double2 dsv = A.ds[v];
            int e[6];
            double g[6];
            double2 zv[6], av[6];
#pragma unroll
            for (int q = 0; q < 6; q++) {
                e[q] = q < k ? A.gj[j0 + q] : 0;
                g[q] = q < k ? A.gv[j0 + q] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 6; q++)
                if (q < k) {
                    zv[q] = ld2(A.z + e[q]);
                    av[q] = ld2(A.a + e[q]);
                }
            double hr = 0.0, hi = 0.0;
#pragma unroll
            for (int q = 0; q < 6; q++)
                if (q < k) {
                    const double2 an = cadd(zv[q], cmul(beta, av[q]));
                    hr += g[q] * an.x;
                    hi += g[q] * an.y;
                }
            for (int j = j0 + 6; j < j0 + k; j++) {          // T-matrix rows only
                const double2 an = cadd(ld2(A.z + A.gj[j]), cmul(beta, ld2(A.a + A.gj[j])));
                hr += A.gv[j] * an.x;
                hi += A.gv[j] * an.y;
            }
            A.h[v] = cmul(make_double2(hr, hi), dsv);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.ctl->failed, c.polls)) break;

        // p = s + beta p, a = z + beta a, w = D_A a + G^T h, (a, w) (k_it_edge)
        {
            double v[2] = {0.0, 0.0};
#pragma unroll 1
            for (int u = 0; u < items; u++) {
                const int i = row0 + u * stride;
                if (i >= A.nb) break;
                const int2 row = otn[u * NT];
                const double2 zv = ld2(A.z + i);
                double2 h0 = make_double2(0.0, 0.0), h1 = h0;
                if (row.x >= 0) h0 = ld2(A.h + row.x);
                if (row.y >= 0) h1 = ld2(A.h + row.y);
                const double2 pn = cadd(os[u * NT], cmul(beta, op[u * NT]));
                const double2 an = cadd(zv, cmul(beta, oa[u * NT]));
                double2 wn = cmul(an, oda[u * NT]);
                if (A.tn) {
                    if (row.x >= 0) {
                        wn.x += -0.5 * h0.x;
                        wn.y += -0.5 * h0.y;
                    }
                    if (row.y >= 0) {
                        wn.x += 0.5 * h1.x;
                        wn.y += 0.5 * h1.y;
                    }
                } else {
                    for (int j = A.tp[i]; j < A.tp[i + 1]; j++) {
                        const double2 hv = ld2(A.h + A.tj[j]);
                        wn.x += A.tv[j] * hv.x;
                        wn.y += A.tv[j] * hv.y;
                    }
                }
                op[u * NT] = pn;
                oa[u * NT] = an;
                A.a[i] = an;
                ow[u * NT] = wn;
                dot_add(v[0], v[1], an, wn);
            }
            small_block<2>(v, nw, sums, part_e);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.ctl->failed, c.polls)) break;
        if (warp < 2) {
            const double q = grid_total<32>(part_e, warp, lane);
            if (lane == 0) tot[warp] = q;
        }
        __syncthreads();
        const double2 aw = make_double2(tot[0], tot[1]);
        if (fabs(aw.x) < 1e-40 && fabs(aw.y) < 1e-40) {
            if (tid == 0) c.status = MTGPU_DIV_BY_ZERO;
            break;                        // in every block: the totals are the same
        }
        if (tid < 2) (tid == 0 ? c.alpha.x : c.alpha.y) = cquot_part(c.zs, aw, tid);
        __syncthreads();

        // x += alpha p, r -= alpha a, s -= alpha w, sums of the MRS weight (k_it_update)
        {
            const double2 al = c.alpha;
            double v[2] = {0.0, 0.0};
#pragma unroll 1
            for (int u = 0; u < items; u++) {
                const int i = row0 + u * stride;
                if (i >= A.nb) break;
                const double2 sn = csub(os[u * NT], cmul(al, ow[u * NT]));
                os[u * NT] = sn;
                A.s[i] = sn;
                ox[u * NT] = cadd(ox[u * NT], cmul(al, op[u * NT]));
                const double2 rn = csub(orr[u * NT], cmul(al, oa[u * NT]));
                orr[u * NT] = rn;
                const double2 sv = osm[u * NT];
                const double ux = rn.x - sv.x, uy = rn.y - sv.y;
                v[0] = fma(sv.y, uy, fma(sv.x, ux, v[0]));
                v[1] = fma(uy, uy, fma(ux, ux, v[1]));
            }
            small_block<2>(v, nw, sums, part_u);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.ctl->failed, c.polls)) break;

        // z = A s, (z, s); beside it the MRS weight; then s_m and its norm (k_it_spmv)
        {
            double v[3] = {0.0, 0.0, 0.0};
            if (!work) {
                const double su = grid_total<32>(part_u, 0, lane), uu = grid_total<32>(part_u, 1, lane);
                if (lane == 0) {
                    const double wm = fabs(uu) < 1e-100 ? 0.0 : -su / uu;
                    if (wm < 0.0) {
                        c.mrs_mode = 0;
                    } else if (wm > 1.0) {
                        c.mrs_mode = 1;
                    } else {
                        c.mrs_mode = 2;
                        c.mrs_w = wm;
                    }
                }
            }
#pragma unroll 1
            for (int u = 0; u < items; u++) {
                const int i = row0 + u * stride;
                if (i >= A.nb) break;
                const int sl = i / kSlice, l = i % kSlice;
                double ar = 0.0, ai = 0.0;
                {
                    const long long base = A.pc[sl] + l;
                    const int wdt = A.wc[sl];
#pragma unroll 4
                    for (int k = 0; k < wdt; k++) {
                        const double2 vv = __ldg(A.val_c + base + (long long)k * kSlice);
                        const double2 xv = ld2(A.s + __ldg(A.col_c + base + (long long)k * kSlice));
                        ar += vv.x * xv.x - vv.y * xv.y;
                        ai += vv.x * xv.y + vv.y * xv.x;
                    }
                }
                {
                    const long long base = A.pr[sl] + l;
                    const int wdt = A.wr[sl];
#pragma unroll 8
                    for (int k = 0; k < wdt; k++) {
                        const double vv = __ldg(A.val_r + base + (long long)k * kSlice);
                        const double2 xv = ld2(A.s + __ldg(A.col_r + base + (long long)k * kSlice));
                        ar += vv * xv.x;
                        ai += vv * xv.y;
                    }
                }
                A.z[i] = make_double2(ar, ai);
                const double2 si = os[u * NT];
                dot_add(v[0], v[1], make_double2(ar, ai), si);
            }
            __syncthreads();
            const int mode = c.mrs_mode;
            const double wm = c.mrs_w;
            if (mode != 0) {
#pragma unroll 1
                for (int u = 0; u < items; u++) {
                    if (row0 + u * stride >= A.nb) break;
                    double2 smv = orr[u * NT];
                    if (mode == 2) {
                        const double2 old = osm[u * NT];
                        smv = make_double2(old.x + wm * (smv.x - old.x), old.y + wm * (smv.y - old.y));
                    }
                    osm[u * NT] = smv;
                    v[2] = fma(smv.y, smv.y, fma(smv.x, smv.x, v[2]));
                }
            }
            small_block<3>(v, nw, sums, part_r);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.ctl->failed, c.polls)) break;
        if (warp < 3) {
            const double q = grid_total<32>(part_r, warp, lane);
            if (lane == 0) tot[warp] = q;
        }
        __syncthreads();
        // beta and the stop test side by side, in two warps
        const double2 zs_new = make_double2(tot[0], tot[1]);
        if (tid < 2) (tid == 0 ? c.beta.x : c.beta.y) = cquot_part(zs_new, c.zs, tid);
        if (tid == 32) {
            if (c.mrs_mode != 0) c.residual = sqrt(tot[2]);
            c.residual_rel = c.residual / c.r_old;
            if (c.residual_rel < c.eps) {
                c.status = MTGPU_OK;
            } else {
                c.iter += 1;
                if (c.iter > c.maxiter) c.status = MTGPU_MAXITER;
            }
        }
        __syncthreads();
        if (tid == 0) c.zs = zs_new;
    }
    __syncthreads();
    if (late) return;
    if (any) {
        for (int u = 0; u < items; u++) {
            const int i = row0 + u * stride;
            if (i >= A.nb) break;
            x[i] = ox[u * NT];
            A.p[i] = op[u * NT];
            A.r[i] = orr[u * NT];
            A.sm[i] = osm[u * NT];
        }
        if (blockIdx.x == 0 && tid == 0) {
            Ctl *q = A.ctl;               // all but the barrier's words
            q->status = c.status;
            q->iter = c.iter;
            q->mrs_mode = c.mrs_mode;
            q->mrs_w = c.mrs_w;
            q->residual = c.residual;
            q->residual_rel = c.residual_rel;
            q->alpha = c.alpha;
            q->beta = c.beta;
            q->zs = c.zs;
        }
    }
    // the last block to leave sets the counters back for the next launch
    if (tid == 0 && count_arrival(&A.ctl->left) == (unsigned)B - 1) {
        A.ctl->bar = 0u;
        A.ctl->left = 0u;
    }
}

// the grid of k_small64 where the rows fit one block per SM
void small_grid(CocrSolver &S, int dev, int nsm)
{
    S.g_small = 0;
    if (S.nb < 1 || S.nb > (long long)nsm * kSmallThreads * kSmallItems || !one_kernel_wanted()) return;
    const int items = ceil_div(S.nb, nsm * kSmallThreads);
    const int nt = std::max(kSmallMin, ceil_div(ceil_div(S.nb, nsm * items), 32) * 32);
    const int smem = items * kSmallItemBytes * nt;
    int coop = 0, b = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaFuncSetAttribute((const void *)k_small64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kSmallItems * kSmallItemBytes * kSmallThreads) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)k_small64, nt + 32, smem) !=
            cudaSuccess || b < 1) {
        cudaGetLastError();
        return;
    }
    S.g_small = std::min(nsm, ceil_div(S.nb, nt));
    S.small_threads = nt;
    S.small_items = items;
}

void launch_small(CocrSolver &S, int n)
{
    const Folded &P = S.P;
    const SellMatrix &M = S.A;
    const Small64 A{S.nb, P.m, P.d_gp, P.d_gj, P.d_gv, P.d_ds, P.d_tp, P.d_tj, P.d_tv, P.d_tn, P.d_da,
                    M.d_wc, M.d_wr, M.d_pc, M.d_pr, M.d_col_c, M.d_col_r, M.d_val_c, M.d_val_r,
                    S.r, S.p, S.s, S.z, S.a, S.w, S.sm, P.d_h, S.ctl, S.partials};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = S.g_small;
    cfg.blockDim = S.small_threads + 32;
    cfg.dynamicSmemBytes = (size_t)S.small_items * kSmallItemBytes * S.small_threads;
    cfg.stream = S.st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_small64, A, n, S.small_items);
}

}  // namespace
}  // namespace mtgpu
