// Iterations of a small problem in one cooperative kernel (included by
// survey_impl.cuh).
#pragma once

namespace mtgpu {
namespace sv {

// The iteration of variant 35 (nodes, edges, update, faces, rows) as phases of
// one kernel, n iterations a launch, with a grid barrier where the separate
// kernels end.
//
// What bounds a small problem is not its work but the ends of its kernels: on
// 45,000 edges x 2 systems the five kernels of an iteration take 33 us, of
// which their bytes and operations are 4; each has a launch, a ramp, a last
// block that adds the partials alone, and the next kernel's first loads start
// after all that.  Here an iteration has three barriers:
//   - nodes and edges in one phase: h at the edge's two nodes is formed by its
//     thread (24 values of z and a instead of 2 of h), so a alternates buffers;
//   - the update;
//   - faces and rows in one phase: 33 values of s and four g = F f a row
//     (small_row) instead of a pass over the faces.
// Every block adds the blocks' partials itself (in the same order, so with the
// same totals and decisions in every block); the systems' state and each
// thread's own rows of a, r, s_m and s stay in shared memory; the sums of the
// update and the stop test's FP64 chain are the work of one warp of their
// own beside the row phase.  A phase boundary costs 2.5k cycles (arrival 1.1k, the
// slowest block and the poll 1.4k), a sum's totals 1.8k, its quotient 1.7k; the
// row phase 8k a row per thread, the arithmetic's time.
//
// Measured, solve of 45,000 edges x 2 systems: 13.4 -> 10.9 ms (33 -> 25 us an
// iteration); 58,000 x 1: 17.0 -> 12.7; 13,900 x 2: 4.5 -> 2.9; 104,500 x 2 (3 rows a
// thread): 10.1 -> 9.3; 26,500 x 8: 9.3 -> 8.2.  With 16 lanes the row phase's
// redundant work shows: 9,450 x 16 8.0 -> 8.3, so up to 8 lanes only.
//
// Phases read what other blocks wrote in the same launch: those loads go
// through ldg (ld.global after the barrier's acquire), never the read-only path.
//
// Every wait is bounded; one that runs out fails the solve with
// MTGPU_ERR_TIMEOUT (GridBarrier; the mark is the state slot after the
// systems').  The launch is cooperative, so all blocks are resident
// and the waits end.
constexpr int kSmallThreads = 480;     // threads with rows, at most; one warp more for the stop test
constexpr int kSmallMin = 256;         // ... at least
constexpr int kSmallSystems = 8;       // systems, at most
constexpr int kSmallItems = 3;         // rows x systems per thread, at most
constexpr int kSmallItemBytes = 6 * sizeof(float4) + sizeof(int4) + sizeof(unsigned);
constexpr int kBarSlot = 992, kExitSlot = 1008;   // counters among the ticket slots
static_assert(kMaxGroups < kBarSlot && kExitSlot < 4 * kTicketSlots, "the counters lie behind the groups' tickets");

struct SmallArgs {
    int nb;
    const float4 *ds, *da;
    const int2 *tn;
    const float2 *omega;
    float4 *r, *a, *a2, *sm, *z;       // a2: a of the odd iterations
    float4 *s;                         // the group's slots, nb * SP apart
    SysState *sys;
    float4 *hist, *partials;
};

// Sums over the grid for k_small: thread t carries N partial sums of system
// t % SP.  Inside a warp in three FP32 (GridSum's halving exchange), from
// there on in FP64, which a few warps add in fewer instructions and steps
// than three FP32 take; every block adds the blocks' partials itself, all
// loads in flight (152 blocks: 1,800 cycles, 4,100 with two or three rounds of loads).
template <int SP, int N>
struct SmallSum {
    static constexpr int NW = kSmallThreads / 32, W = N * SP;
    // the sums of the block's first nw warps to part[output][block]; sm: nw * W doubles
    static __device__ __forceinline__ void block(const tf (&v)[N], int nw, double *sm, double *part)
    {
        const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
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
                        u[i] = tf_add(mine, GridSum<SP, N, kB>::shfl(give, o));
                    }
                first += up ? h : 0;
                cnt = h;
            } else {
                u[0] = tf_add(u[0], GridSum<SP, N, kB>::shfl(u[0], o));
                dup |= o;
            }
        }
        if (warp < nw && !(lane & dup)) {
#pragma unroll
            for (int i = 0; i < N; i++)
                if (i < cnt) sm[warp * W + (first + i) * SP + lane % SP] = tf4_double(tf_pack(u[i], big ? 1.f : 0.f));
        }
        __syncthreads();
        // the warps' sums: L lanes for each output
        constexpr int L = W < 32 ? 32 / W : 1, TH = W < 32 ? 32 : W;
        if (t < TH) {
            double s = 0.0;
            for (int q = t / W; q < nw; q += L) s += sm[q * W + t % W];
#pragma unroll
            for (int o = 16; o >= W; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (t < W) __stcg(part + (size_t)t * gridDim.x + blockIdx.x, s);
        }
    }
    // the grid's totals by the block's first kSmallMin threads
    static __device__ __forceinline__ void totals(const double *part, double (*tot)[32])
    {
        constexpr int G = kSmallMin / W < 32 ? kSmallMin / W : 32;
        const int o = threadIdx.x / G, j = threadIdx.x % G;
        if (o < W) {
            const double s = grid_total<G>(part, o, j);
            if (j == 0) tot[o / SP][o % SP] = s;
        }
        __syncthreads();
    }
    // ... by one warp
    static __device__ __forceinline__ void totals_warp(const double *part, double (*tot)[32])
    {
        constexpr int G = W < 32 ? 32 / W : 1;
        const int lane = threadIdx.x & 31;
        for (int o = lane / G; o < W; o += 32 / G) {
            const double s = grid_total<G>(part, o, lane % G);
            if (lane % G == 0) tot[o / SP][o % SP] = s;
        }
        __syncwarp();
    }
};

// z = A s of one row by variant 35's sums, with the face circulations and g = F f
// formed in the row: 33 values of s, and no pass and barrier for the faces.
// The four rows of a face form the same g to the last bit, so the curl-curl
// part still is D^T of one g (its rounding has no gradient part, which the
// small mass part of air cells would show).
template <int SP>
__device__ __forceinline__ cdf small_row(const MF &M, int d, Pos p, int k, df om, const float4 *x, cdf own)
{
    const MfRow r = mf_rowctx(M, d, p);
    const int T1 = d == 2 ? 0 : d + 1, T2 = d == 0 ? 2 : d - 1;
    const int es = M.es[d], c = coord(d, p);
    const bool end[2] = {c == 0, c == extent(d, M) - 2};   // the edge's ends on the surface
    const float4 *xk = x + k;
    // the parallel edges
    cdf xd[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            xd[a][b] = czero();
            if (a == 1 && b == 1) xd[a][b] = own;
            else if (!mf_mass_dir(r, a, b)) xd[a][b] = ldg(xk + mf_mass_edge(r, a, b) * SP);
        }
    acc2 kk;
    // D^T (F f): g = F f of the T1-normal faces, then of the T2-normal ones (b
    // = 0, 1 across the other transverse axis), from the circulations at
    // positions a = 0, 1, 2 along their normal
#pragma unroll
    for (int g = 0; g < 2; g++) {
        df w[2][2];
        mf_weights(M, r, g == 0 ? r.w1 : r.w2, w);
        // g = 0: the T2 edges at T1 offset a - 1; g = 1: the T1 edges at T2 offset a - 1
        const int et = mf_edge_in(M, g == 0 ? T2 : T1, p.x, p.y, p.z);
        const int en = g == 0 ? r.e1 : r.e2, ec = g == 0 ? r.e2 : r.e1;
        const bool lo = g == 0 ? r.lo1 : r.lo2, hi = g == 0 ? r.hi1 : r.hi2;
#pragma unroll
        for (int b = 0; b < 2; b++) {
            cdf f[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                cdf xt[2];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    xt[q] = czero();
                    if (!((a == 0 && lo) || (a == 2 && hi) || end[q]))
                        xt[q] = ldg(xk + (et + (a - 1) * en + (b - 1) * ec + q * es) * SP);
                }
                f[a] = g == 0 ? mf_circ(xt[0], xd[a][b + 1], xt[1], xd[a][b])
                              : mf_circ(xd[b][a], xt[1], xd[b + 1][a], xt[0]);
            }
            const cdf gv = g == 0 ? mf_g(w[0][b], w[1][b], f[0], f[1], f[2]) : mf_g(w[b][0], w[b][1], f[0], f[1], f[2]);
            if (g == 0 && b == 0) kk.start(gv);
            else if ((g == 0) == (b == 0)) kk.add(gv);
            else kk.sub(gv);
        }
    }
    // the mass part, the sum over the 4 cells of w (2 P_a(1) + P_a(0 or 2)),
    // P_a(b) = 2 x(1, b) + x(0 or 2, b)
    df w[2][2];
    mf_weights(M, r, r.wm, w);
    acc2 mm;
#pragma unroll
    for (int a = 0; a < 2; a++) {
        acc2 P[3];
#pragma unroll
        for (int b = 0; b < 3; b++) {
            P[b].start(cdf{add2(xd[1][b].h, xd[1][b].h), add2(xd[1][b].l, xd[1][b].l)});
            P[b].add(xd[2 * a][b]);
        }
#pragma unroll
        for (int b = 0; b < 2; b++) {
            acc2 u;
            u.start(cdf{add2(P[1].h, P[1].h), add2(P[1].l, P[1].l)});
            u.add(cdf{P[2 * b].h, P[2 * b].l});
            if (a == 0 && b == 0) mm.first(both(w[a][b]), cdf{u.h, u.l});
            else mm.mac(both(w[a][b]), cdf{u.h, u.l});
        }
    }
    kk.mac(cdf{pk(-om.h, om.h), pk(-om.l, om.l)}, cswap(mm.get()));
    return kk.get();
}

// a component of a / b into a state's double and double-float forms
__device__ __forceinline__ void small_quot(double2 a, double2 b, int c, double2 &q, float4 &qf)
{
    const double v = sum_quot_part(a, b, c);
    const df f = from_double(v);
    (c == 0 ? q.x : q.y) = v;
    (c == 0 ? qf.x : qf.y) = f.h;
    (c == 0 ? qf.z : qf.w) = f.l;
}

template <int SP>
__global__ void __launch_bounds__(kSmallThreads + 32, 1)
k_small(const __grid_constant__ MF M, const __grid_constant__ SmallArgs A, int n, int items)
{
    using S2 = SmallSum<SP, 2>;
    using S4 = SmallSum<SP, 4>;
    __shared__ SysState st[SP];
    __shared__ double sums[S4::NW * S4::W];
    __shared__ double tot[2][32], tot4[4][32];
    __shared__ int late, alive, brk[SP];
    // this thread's rows, kept for the launch: [item][thread]
    extern __shared__ float4 own[];
    const int tid = threadIdx.x, k = tid % SP, B = gridDim.x, NT = blockDim.x - 32, nw = NT / 32;
    const bool work = tid < NT;        // the last warp has no rows
    const int rows = NT / SP, stride = B * rows, row0 = work ? blockIdx.x * rows + tid / SP : A.nb;
    const int len = A.nb * SP;
    float4 *oa = own + tid, *ow = oa + items * NT, *orr = ow + items * NT, *osm = orr + items * NT,
           *os = osm + items * NT, *oda = os + items * NT;
    int4 *otn = reinterpret_cast<int4 *>(own + 6 * items * NT) + tid;
    unsigned *opos = reinterpret_cast<unsigned *>(own + 7 * items * NT) + tid;
    unsigned int *tickets = reinterpret_cast<unsigned int *>(A.partials);
    double *part_e = reinterpret_cast<double *>(A.partials + kTicketSlots), *part_u = part_e + (size_t)B * 2 * SP,
           *part_r = part_u + (size_t)B * 4 * SP;
    GridBarrier bar{tickets + kBarSlot};
    const df om = d2f(A.omega[k]);

    if (tid < SP) {
        st[tid] = A.sys[tid];
        st[tid].cnt = 0;
        brk[tid] = 0;
    }
    if (tid == 0) late = *(volatile const int *)&A.sys[kBarState].status != 0;
    __syncthreads();
    if (late) return;                  // an earlier launch failed
    for (int u = 0; u < items; u++) {
        const int e = row0 + u * stride, i = e * SP + k;
        if (e >= A.nb) break;
        oa[u * NT] = A.a[i];
        orr[u * NT] = A.r[i];
        osm[u * NT] = A.sm[i];
        os[u * NT] = A.s[i];
        oda[u * NT] = A.da[i];
        // the rows of G at the edge's nodes, and their +x edges
        const int2 v = A.tn[e];
        int4 q = make_int4(v.x, 0, v.y, 0);
        const int ix = M.nx - 2, iy = M.ny - 2;
        if (v.x >= 0) q.y = mf_edge_in(M, 0, v.x % ix + 1, v.x / ix % iy + 1, v.x / ix / iy + 1);
        if (v.y >= 0) q.w = mf_edge_in(M, 0, v.y % ix + 1, v.y / ix % iy + 1, v.y / ix / iy + 1);
        otn[u * NT] = q;
        opos[u * NT] = M.pos[e];
    }
    for (int t = 0; t < n; t++) {
        if (tid == 0) alive = 0;
        __syncthreads();
        if (tid < SP && st[tid].status == kRun) alive = 1;
        __syncthreads();
        if (!alive) break;
        bool on = st[k].status == kRun;
        float4 *s_out = A.s + (size_t)(t + 1) * len;
        const float4 *a_in = t & 1 ? A.a2 : A.a;
        float4 *a_out = t & 1 ? A.a : A.a2;

        // h = D_S G (z + beta a) at the edge's nodes (k_node_lat's sums), then
        // a = z + beta a, w = D_A a + G^T h, (a, w) (k_edge)
        {
            const cfac be = cfac_of(from4(st[k].beta_f));
            acc2 aw1, aw2;
            if (on) {
#pragma unroll 1
                for (int u = 0; u < items; u++) {
                    const int e = row0 + u * stride;
                    if (e >= A.nb) break;
                    const int4 tn = otn[u * NT];
                    const cdf zo = ldg(A.z + e * SP + k);
                    cdf h[2];
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                        const int v = q ? tn.z : tn.x, e0 = q ? tn.w : tn.y;
                        if (v < 0) continue;
                        const int es[6] = {e0 + 2 - M.plane, e0 + 1 - M.l3, e0 - 3, e0, e0 + 1, e0 + 2};
                        const cdf dsv = ldn(A.ds + v * SP + k);
                        cdf zv[6], av[6];
#pragma unroll
                        for (int i = 0; i < 6; i++) zv[i] = ldg(A.z + es[i] * SP + k);
#pragma unroll
                        for (int i = 0; i < 6; i++) av[i] = ldg(a_in + es[i] * SP + k);
                        acc2 hv;
#pragma unroll
                        for (int i = 0; i < 6; i++) {
                            const cdf an = caxpy(zv[i], be, av[i]);
                            if (i == 0) hv.start(an);
                            else if (i < 3) hv.add(an);
                            else hv.sub(an);
                        }
                        h[q] = cmul(cfac_of(dsv), chalf(hv.get(), 0.5f));
                        h[q] = cdf_of(to4(h[q]));
                    }
                    const cdf an = caxpy(zo, be, cdf_of(oa[u * NT]));
                    acc2 x;
                    x.start(cmul(cfac_of(cdf_of(oda[u * NT])), an));
                    if (tn.x >= 0) x.sub(chalf(h[0], 0.5f));
                    if (tn.z >= 0) x.add(chalf(h[1], 0.5f));
                    const cdf wn = x.get();
                    oa[u * NT] = to4(an);
                    a_out[e * SP + k] = to4(an);
                    ow[u * NT] = to4(wn);
                    aw1.mac(an, wn);
                    aw2.mac(an, cswap(wn));
                }
            }
            const tf v[2] = {tf_diff(aw1), tf_sum(aw2)};
            S2::block(v, nw, sums, part_e);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.sys[kBarState].status, kBarPolls)) break;
        S2::totals(part_e, tot);
        if (tid < 2 * SP && st[k].status == kRun) {
            const double2 aw = make_double2(tot[0][k], tot[1][k]);
            if (fabs(aw.x) < 1e-40 && fabs(aw.y) < 1e-40) brk[k] = 1;
            else small_quot(st[k].zs, aw, tid / SP, st[k].alpha, st[k].alpha_f);
        }
        __syncthreads();
        // (a, w) = 0: alpha stays, and the system stops here
        if (tid < SP && brk[tid] && st[tid].status == kRun) st[tid].status = MTGPU_DIV_BY_ZERO;

        // r -= alpha a, s -= alpha w, s_m and the sums of the smoothing (k_update)
        on = on && !brk[k];
        {
            acc2 su, uu, nn, rr;
            if (on) {
                dfc al = from4(st[k].alpha_f);
                al = dfc{neg(al.re), neg(al.im)};
                const cfac nal = cfac_of(al);
                const int pm = st[k].mrs_mode;
                const cdf pw = both(d2f(st[k].mrs_wf));
#pragma unroll 1
                for (int u = 0; u < items; u++) {
                    const int e = row0 + u * stride;
                    if (e >= A.nb) break;
                    const cdf sn = caxpy(cdf_of(os[u * NT]), nal, cdf_of(ow[u * NT]));
                    s_out[e * SP + k] = to4(sn);
                    os[u * NT] = to4(sn);
                    const cdf ro = cdf_of(orr[u * NT]);
                    cdf x = cdf_of(osm[u * NT]);
                    if (pm == 1) {
                        x = ro;
                    } else if (pm == 2) {
                        acc2 y;
                        y.start(x);
                        y.mac(pw, csub(ro, x));
                        x = y.get();
                    }
                    const cdf rn = caxpy(ro, nal, cdf_of(oa[u * NT]));
                    orr[u * NT] = to4(rn);
                    osm[u * NT] = to4(x);
                    const cdf ur = csub(rn, x);
                    su.mac(x, ur);
                    uu.mac(ur, ur);
                    nn.mac(x, x);
                    rr.mac(rn, rn);
                }
            }
            const tf v[4] = {tf_sum(su), tf_sum(uu), tf_sum(nn), tf_sum(rr)};
            S4::block(v, nw, sums, part_u);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.sys[kBarState].status, kBarPolls)) break;

        // z = A s, (z, s); meanwhile the last warp adds the update's
        // sums and prepares the stop test
        acc2 zs1, zs2;
        if (!work) {
            S4::totals_warp(part_u, tot4);
            const int l = tid - NT;
            if (l < SP && st[l].status == kRun) {
                SysState &q = st[l];
                const double s_u = tot4[0][l], u_u = tot4[1][l], n_n = tot4[2][l], r_r = tot4[3][l];
                const int c = min(q.cnt, kGroupIters - 1);
                if (blockIdx.x == 0) {
                    A.hist[2 * (l * kGroupIters + c)] = q.alpha_f;
                    A.hist[2 * (l * kGroupIters + c) + 1] = q.beta_f;
                }
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
                if (q.mrs_mode != 0) q.residual = q.res2_next > 0.0 ? sqrt(q.res2_next) : 0.0;
                q.residual_rel = q.residual / q.r_old;
            }
        } else if (on) {
#pragma unroll 1
            for (int u = 0; u < items; u++) {
                if (row0 + u * stride >= A.nb) break;
                const unsigned c = opos[u * NT];
                const int d = (int)(c >> 30);
                const Pos p{(int)(c & 1023u), (int)((c >> 10) & 1023u), (int)((c >> 20) & 1023u)};
                const int i = mf_edge(M, d, p.x, p.y, p.z) * SP + k;
                const cdf x = ldg(s_out + i);
                cdf y = x;
                if (!mf_dirichlet(M, d, p.x, p.y, p.z)) y = small_row<SP>(M, d, p, k, om, s_out, x);
                A.z[i] = to4(y);
                zs1.mac(y, x);
                zs2.mac(y, cswap(x));
            }
        }
        {
            const tf v[2] = {tf_diff(zs1), tf_sum(zs2)};
            S2::block(v, nw, sums, part_r);
        }
        bar.arrive();
        if (!bar.wait(&late, &A.sys[kBarState].status, kBarPolls)) break;
        S2::totals(part_r, tot);
        if (tid < 2 * SP && st[k].status == kRun)
            small_quot(make_double2(tot[0][k], tot[1][k]), st[k].zs, tid / SP, st[k].beta, st[k].beta_f);
        __syncthreads();
        if (tid < SP && st[tid].status == kRun) {
            SysState &q = st[tid];
            q.zs = make_double2(tot[0][tid], tot[1][tid]);
            if (q.residual_rel < q.eps_k) {
                q.status = MTGPU_OK;
            } else {
                q.iter += 1;
                if (q.iter > q.maxiter) q.status = MTGPU_MAXITER;
            }
        }
    }
    __syncthreads();
    if (late) return;
    for (int u = 0; u < items; u++) {
        const int e = row0 + u * stride, i = e * SP + k;
        if (e >= A.nb) break;
        A.a[i] = oa[u * NT];
        A.r[i] = orr[u * NT];
        A.sm[i] = osm[u * NT];
    }
    if (blockIdx.x == 0 && tid < SP) A.sys[tid] = st[tid];
    // the last block to leave sets the counters back for the next launch
    if (tid == 0 && count_arrival(tickets + kExitSlot) == (unsigned)B - 1) {
        tickets[kBarSlot] = 0u;
        tickets[kExitSlot] = 0u;
    }
}

}  // namespace sv
}  // namespace mtgpu
