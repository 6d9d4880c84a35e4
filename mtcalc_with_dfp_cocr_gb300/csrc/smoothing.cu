// Receiver output by subdomain L2-projection smoothing: the reference's
// default E/H output path (Code/OutputNu: Give_out_vec_mt::Give_out_on_hex
// with OutputResultant3d, give_out_vec_mt.cpp:200-237, OutputResultant3d.cpp:
// 76-199, 293-450; Subdomain::Init / AsmGlobalMatrix / AsmGlobalVector,
// Subdomain.cpp:132-661).  Per receiver output type:
//
//   * the receivers are located in the first brick (index order) whose box
//     grown by 1e-6 holds them; for A the air (material 0) is skipped;
//   * curl A is smoothed over one subdomain of all materials, A over one
//     subdomain per material holding a receiver; a subdomain is its
//     receivers' bricks grown `levels` times by every brick of its material
//     sharing a node with it;
//   * in each subdomain the brick-centre values (A or curl A of the edge
//     solution) are projected onto the nodal trilinear functions:
//     M u = f with M the nodal mass matrix and f_i = sum over the bricks at
//     node i of (the brick matrix's row sum) x (the centre value);
//   * the receiver value is the trilinear interpolant of u in its brick.
//
// The reference factorises M with PARDISO and solves one value type at a
// time.  Here every (subdomain, value type, system) is one column, solved by
// iterative refinement: FP64 right-hand sides, solutions and residuals f - M u,
// corrections by Jacobi-preconditioned conjugate gradients in FP32 (the
// diagonally scaled trilinear mass matrix has a condition number below ~30,
// so about 20 iterations gain five digits), until the FP64 residual is below
// 1e-14 of the right-hand side: three to four rounds.  One block holds one
// subdomain and two or four columns from the right-hand side to the solution:
// no launches between iterations, and the matrix, read from L2, serves all of
// its columns; where few columns leave SMs idle, a cluster of up to eight
// blocks shares the subdomain's nodes.  (CG in FP64, four launches an
// iteration, took 5.9 ms for 96 columns of 6,600 nodes; GB300 runs FP64 at 1/64
// of FP32, and 27 multiply-adds a node, column and iteration are 27 us of its
// FP64 pipes.)
// The subdomains, the mass matrix and the interpolation weights are built
// once per receiver set on the host; the per-call work (centre values,
// right-hand sides, projection, interpolation) runs on the device.
//
// Vector layout: [column][padded node], column = value * S + system with
// values (x re, x im, y re, y im, z re, z im); FP32 vectors [group
// of columns][padded node][column].  Conforming (tensor) meshes only: no
// terminal nodes.
#include "rcv_eval.cuh"
#include "receivers.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>

namespace mtgpu {
namespace {

constexpr int kPad = 32;             // padding unit of a subdomain's nodes
constexpr int kSolve = 512;          // threads of a solving block
constexpr double kTol2 = 1e-28;      // (relative residual 1e-14)^2
// A residual that has stopped falling is at FP64's own accuracy; accepted
// below this square
constexpr double kFloor2 = 1e-24;
constexpr int kMaxOuter = 60;        // guards; four rounds of ~20 are needed
constexpr int kMaxInner = 60;
constexpr float kInner2 = 1e-10f;    // (a round's FP32 residual reduction)^2

// brick-centre values: one thread per (brick of a subdomain, system)
__global__ void k_sm_centre(int ncell, int S, const int *__restrict__ cell,
                            const int *__restrict__ cell_sub, const int *__restrict__ nver,
                            int nver_stride, const int *__restrict__ ed, int ed_stride,
                            const double *__restrict__ xyz, long long x_stride,
                            const double2 *__restrict__ x, double *val)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (i >= ncell || k >= S) return;
    const long long g = cell[i];
    const int v0 = nver[g * nver_stride], v7 = nver[g * nver_stride + 7];
    const double hx = xyz[3 * v7] - xyz[3 * v0], hy = xyz[3 * v7 + 1] - xyz[3 * v0 + 1],
                 hz = xyz[3 * v7 + 2] - xyz[3 * v0 + 2];
    const double2 *xs = x + (long long)k * x_stride;
    double2 v[12];
#pragma unroll
    for (int j = 0; j < 12; j++) v[j] = xs[ed[g * ed_stride + j]];
    double2 A[3], C[3];
    rcv::brick_eval(v, 0.0, 0.0, 0.0, hx, hy, hz, A, C);
    const double2 *f = cell_sub[i] == 0 ? C : A;
    for (int d = 0; d < 3; d++) {
        val[((long long)(2 * d) * S + k) * ncell + i] = f[d].x;
        val[((long long)(2 * d + 1) * S + k) * ncell + i] = f[d].y;
    }
}

constexpr int kSlots = 27;           // matrix entries per node, padded

// C FP32 values, one per column of the block
template <int C>
struct alignas(4 * C) vec {
    float a[C];
};
template <int C>
__device__ __forceinline__ vec<C> splat(float s)
{
    vec<C> v;
#pragma unroll
    for (int c = 0; c < C; c++) v.a[c] = s;
    return v;
}
template <int C>
__device__ __forceinline__ vec<C> operator*(vec<C> x, vec<C> y)
{
#pragma unroll
    for (int c = 0; c < C; c++) x.a[c] *= y.a[c];
    return x;
}
template <int C>
__device__ __forceinline__ vec<C> fma_(vec<C> x, vec<C> y, vec<C> z)
{
#pragma unroll
    for (int c = 0; c < C; c++) z.a[c] = fmaf(x.a[c], y.a[c], z.a[c]);
    return z;
}
// x / y where y > 0, else 0
template <int C>
__device__ __forceinline__ vec<C> quot(vec<C> x, vec<C> y)
{
#pragma unroll
    for (int c = 0; c < C; c++) x.a[c] = y.a[c] > 0.f ? x.a[c] / y.a[c] : 0.f;
    return x;
}

// Q blocks that share a subdomain are a cluster (CL): barriers of all its
// threads, after which each sees what the others stored before theirs, and
// stores into the other blocks' shared memory.
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_addr(const void *own, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(own)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_store(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_store(unsigned a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
constexpr int kMaxCluster = 8;

// Sums of C values per thread over the block, in a fixed order, to all
// threads; buf: [warps] slots, alternated by the caller between calls.  Of a
// cluster, block `rank` of Q then gives its sums to all blocks (all: [block]
// slots, alternated likewise), and every thread adds them in block order.
template <int C, bool CL, class T>
__device__ __forceinline__ void block_sum(T (&v)[C], T (*buf)[C], T (*all)[C], int Q, int rank)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // halve the values a lane holds while lane bits are left to pick them,
    // then add the lanes of each value
    int o = 16, first = 0;
#pragma unroll
    for (int h = C / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
        first += up ? h : 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const T mine = up ? v[i + h] : v[i], give = up ? v[i] : v[i + h];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    const int rest = o;
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    if ((lane & (2 * rest - 1)) == 0) buf[w][first] = v[0];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < C; c++) {
        T s = buf[0][c];
#pragma unroll
        for (int q = 1; q < kSolve / 32; q++) s += buf[q][c];
        v[c] = s;
    }
    if (CL) {
        if (threadIdx.x < Q) {
            const unsigned a = cluster_addr(all[rank], threadIdx.x);
#pragma unroll
            for (int c = 0; c < C; c++) cluster_store(a + c * (unsigned)sizeof(T), v[c]);
        }
        cluster_barrier();
#pragma unroll
        for (int c = 0; c < C; c++) {
            v[c] = 0;
            for (int q = 0; q < Q; q++) v[c] += all[q][c];
        }
    }
}

struct SolveArgs {
    int npad, ncol, ncell;
    const int *off, *nn;                     // per subdomain: first padded node, nodes
    const int *nc_ptr, *nc;                  // node -> bricks
    const double *cell_g, *val;
    // the mass matrix, kSlots entries a node (padded with zeros), slot by slot
    // for every 32 nodes so that a warp reads whole lines: column within the
    // subdomain and FP32 value, FP64 value
    const int2 *m32;
    const double *m64;
    const float *dinv;                       // 1 / diagonal
    double *x, *f, *r;                       // [column][padded node]
    float *w;                                // FP32 vectors, 4 x [group][padded node][C]
    int pcap;                                // bytes of shared memory for p
    int q;                                   // blocks a subdomain (a cluster)
    int *out;                                // columns that did not converge; largest iteration count
};

// the projection of C columns of one subdomain (blockIdx.y); CL: by a cluster of
// A.q blocks, each a range of the nodes, with p in global memory
template <int C, bool CL>
__global__ void __launch_bounds__(kSolve, 1)
k_sm_solve(SolveArgs A)
{
    using V = vec<C>;
    extern __shared__ __align__(16) unsigned char psh[];
    __shared__ double dbuf[2][kSolve / 32][C];
    __shared__ float fbuf[2][kSolve / 32][C];
    __shared__ double dall[2][CL ? kMaxCluster : 1][C];
    __shared__ float fall[2][CL ? kMaxCluster : 1][C];
    const int Q = CL ? A.q : 1, rank = CL ? blockIdx.x % Q : 0, group = CL ? blockIdx.x / Q : blockIdx.x;
    const int sub = blockIdx.y, n0 = A.off[sub], nn = A.nn[sub];
    // this block's nodes
    const int share = CL ? (nn + 32 * Q - 1) / (32 * Q) * 32 : nn;
    const int first = share * rank + threadIdx.x, end = min(nn, share * (rank + 1));
    const int c0 = C * group, nc = min(C, A.ncol - c0);
    const long long nw = (long long)(gridDim.x / Q) * A.npad;
    V *const w = reinterpret_cast<V *>(A.w) + (long long)group * A.npad + n0;
    V *const p = !CL && nn * (int)sizeof(V) <= A.pcap ? reinterpret_cast<V *>(psh) : w;
    V *const r32 = w + nw, *const d32 = w + 2 * nw, *const q32 = w + 3 * nw;
    const float *const dinv = A.dinv + n0;
    const int2 *const m32 = A.m32 + (long long)n0 * kSlots;
    const double *const m64 = A.m64 + (long long)n0 * kSlots;
    auto slots = [](int n) { return (n >> 5) * (32 * kSlots) + (n & 31); };
    double *x[C], *f[C], *r[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
        const long long o = (long long)(c0 + min(c, nc - 1)) * A.npad + n0;
        x[c] = A.x + o;
        f[c] = A.f + o;
        r[c] = A.r + o;
    }
    int flip = 0, total = 0;
    auto everyone = [&] {
        if (CL) cluster_barrier();
        else __syncthreads();
    };
    auto sum = [&](V v) {
        block_sum<C, CL>(v.a, fbuf[flip], fall[flip], Q, rank);
        flip ^= 1;
        return v;
    };
    if (CL) cluster_barrier();               // the other blocks have started
    // f = sum over the node's bricks of g_c val_c; x = 0, so r = f
    double ff[C] = {}, rr[C], last[C] = {};
    for (int n = first; n < end; n += kSolve)
        for (int c = 0; c < nc; c++) {
            double s = 0.0;
            for (int j = A.nc_ptr[n0 + n]; j < A.nc_ptr[n0 + n + 1]; j++) {
                const int e = A.nc[j];
                s += A.cell_g[e] * A.val[(long long)(c0 + c) * A.ncell + e];
            }
            f[c][n] = s;
            r[c][n] = s;
            x[c][n] = 0.0;
#pragma unroll
            for (int q = 0; q < C; q++)
                if (q == c) ff[q] += s * s;
        }
    block_sum<C, CL>(ff, dbuf[flip], dall[flip], Q, rank);
    flip ^= 1;
#pragma unroll
    for (int c = 0; c < C; c++) {
        rr[c] = ff[c];
        // no projection of an infinity or a NaN (or of squares beyond FP64): the
        // column is done at once, and not with x = 0
        if (c < nc && !(ff[c] <= DBL_MAX))
            for (int n = first; n < end; n += kSolve) x[c][n] = nan("");
    }
    bool done[C];
    int open = 0;
    for (int round = 0; round < kMaxOuter; round++) {
        open = 0;
#pragma unroll
        for (int c = 0; c < C; c++) {
            // (an infinity or a NaN ends its column, as does a zero right-hand side)
            done[c] = c >= nc || !(rr[c] > kTol2 * ff[c]) ||
                      (round > 0 && rr[c] > 0.25 * last[c] && rr[c] <= kFloor2 * ff[c]);
            open += !done[c];
            last[c] = rr[c];
        }
        if (open == 0) break;
        // FP32 correction M d = r / |r| of the open columns
        double norm[C], scale[C];
#pragma unroll
        for (int c = 0; c < C; c++) {
            norm[c] = done[c] ? 0.0 : sqrt(rr[c]);
            scale[c] = norm[c] > 0.0 ? 1.0 / norm[c] : 0.0;
        }
        V rz = splat<C>(0.f);
        for (int n = first; n < end; n += kSolve) {
            V v;
#pragma unroll
            for (int c = 0; c < C; c++) v.a[c] = done[c] ? 0.f : (float)(r[c][n] * scale[c]);
            const V z = v * splat<C>(dinv[n]);
            r32[n] = v;
            d32[n] = splat<C>(0.f);
            p[n] = z;
            rz = fma_(v, z, rz);
        }
        rz = sum(rz);
        for (int it = 0; it < kMaxInner; it++) {
            V pq = splat<C>(0.f);
            for (int n = first; n < end; n += kSolve) {
                V s = splat<C>(0.f);
                const int2 *m = m32 + slots(n);
#pragma unroll 9
                for (int j = 0; j < kSlots; j++) {
                    const int2 e = __ldg(m + 32 * j);
                    s = fma_(splat<C>(__int_as_float(e.y)), p[e.x], s);
                }
                q32[n] = s;
                pq = fma_(p[n], s, pq);
            }
            pq = sum(pq);
            total++;
            const V al = quot(rz, pq), nal = al * splat<C>(-1.f);
            V rz2 = splat<C>(0.f), r2 = rz2;
            for (int n = first; n < end; n += kSolve) {
                d32[n] = fma_(al, p[n], d32[n]);
                const V v = fma_(nal, q32[n], r32[n]);
                r32[n] = v;
                r2 = fma_(v, v, r2);
                rz2 = fma_(v, v * splat<C>(dinv[n]), rz2);
            }
            r2 = sum(r2);
            bool more = false;
#pragma unroll
            for (int c = 0; c < C; c++) more |= r2.a[c] > kInner2;
            if (!more) break;
            rz2 = sum(rz2);
            const V be = quot(rz2, rz);
            rz = rz2;
            for (int n = first; n < end; n += kSolve) p[n] = fma_(be, p[n], r32[n] * splat<C>(dinv[n]));
            everyone();
        }
        // x += |r| d, r = f - M x in FP64
        for (int n = first; n < end; n += kSolve) {
            const V d = d32[n];
#pragma unroll
            for (int c = 0; c < C; c++)
                if (!done[c]) x[c][n] += norm[c] * (double)d.a[c];
        }
        everyone();
        double s2[C] = {};
        for (int n = first; n < end; n += kSolve) {
            double s[C];
#pragma unroll
            for (int c = 0; c < C; c++) s[c] = done[c] ? 0.0 : f[c][n];
            const int at = slots(n);
#pragma unroll 3
            for (int j = 0; j < kSlots; j++) {
                const double m = m64[at + 32 * j];
                const int col = m32[at + 32 * j].x;
#pragma unroll
                for (int c = 0; c < C; c++)
                    if (!done[c]) s[c] -= m * x[c][col];
            }
#pragma unroll
            for (int c = 0; c < C; c++)
                if (!done[c]) {
                    r[c][n] = s[c];
                    s2[c] += s[c] * s[c];
                }
        }
        block_sum<C, CL>(s2, dbuf[flip], dall[flip], Q, rank);
        flip ^= 1;
#pragma unroll
        for (int c = 0; c < C; c++)
            if (!done[c]) rr[c] = s2[c];
    }
    if (rank == 0 && threadIdx.x == 0) {
        if (open > 0) atomicAdd(A.out, open);
        atomicMax(A.out + 1, total);
    }
}

// receiver values (trilinear interpolation of the nodal solutions) and the
// total fields: one thread per (receiver, system)
__global__ void k_sm_receivers(int nrec, int S, int npad, const int *__restrict__ rn,
                               const double *__restrict__ rw, const double *__restrict__ u,
                               const double *__restrict__ omega, const int *__restrict__ alfa,
                               int n1d, const double *__restrict__ z1d,
                               const double *__restrict__ usin, const double *__restrict__ ucos,
                               const double4 *__restrict__ loc, double2 *e_out, double2 *h_out,
                               double2 *scal)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;
    if (r >= nrec || k >= S) return;
    double2 F[2][3] = {};   // curl A, A
    for (int t = 0; t < 2; t++) {
        const int *nn = rn + (r * 2 + t) * 8;
        const double *ww = rw + (r * 2 + t) * 8;
        if (nn[0] < 0) continue;
        for (int v = 0; v < 6; v++) {
            const double *uc = u + ((long long)v * S + k) * npad;
            double s = 0.0;
            for (int l = 0; l < 8; l++) s += ww[l] * uc[nn[l]];
            if (v & 1)
                F[t][v >> 1].y = s;
            else
                F[t][v >> 1].x = s;
        }
    }
    const long long o = (long long)k * nrec + r;
    rcv::total_fields(F[1], F[0], omega[k], alfa[k], loc[r].w, n1d, z1d,
                      usin + (long long)k * n1d, ucos + (long long)k * n1d, e_out + 3 * o,
                      h_out + 3 * o, scal + o);
}

// ------------------------------------------------------------- host set-up
// Blocks a subdomain: where the groups of columns leave SMs without a block, 2, 4
// or 8 (a portable cluster), as many as run side by side (76 clusters of 2, 36 of
// 4, 15 of 8 here) and with at least this many nodes each.  The GPU's time at
// 1, 2, 4, 8 blocks: 59,904 nodes, one system 26.4 / 12.3 / 6.6 / 3.7 ms, eight 31.3 / 14.7
// (and 8.4 in two waves of 4); 8,112 nodes, one 3.0 / 2.0 / 1.3 / 0.94, with four
// systems 3.0 / 2.0 / 1.3 and 1.6 beyond what fits; 3,072 nodes 1.23 / 1.11 / 0.84 / 0.69; 343
// nodes 0.39 / 0.61 / 0.62 / 0.63.  (Conjugate gradients in FP64 over the whole grid: 7.8 ms for one
// system on 59,904 nodes, 13.4 for two, 47.7 for eight.)
constexpr int kClusterNodes = 1024;

// launch of the projection by clusters of q blocks
cudaLaunchConfig_t cluster_config(cudaLaunchAttribute *at, int q, int groups, int nsub)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups * q, nsub);
    cfg.blockDim = kSolve;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = q;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

struct SubBuild {
    std::vector<int> cells, nodes;   // ascending global indices
};

// Subdomain.cpp:132-246: seed bricks, then `levels` rounds of every allowed
// brick sharing a node with the current node set
SubBuild grow_subdomain(const ::mtgpu_assembly_s &a, const std::vector<int> &seed, int material,
                        int levels)
{
    const int kpar = a.P.kpar, kuz = a.P.kuzlov, ns = a.nver_stride;
    std::vector<unsigned char> in_cell(kpar, 0), in_node(kuz, 0);
    auto allowed = [&](int c) { return material < 0 || a.nvkat[c] == material; };
    for (int c : seed) {
        if (c < 0 || !allowed(c) || in_cell[c]) continue;
        in_cell[c] = 1;
        for (int j = 0; j < 8; j++) in_node[a.nver[(size_t)c * ns + j]] = 1;
    }
    std::vector<int> fresh;
    for (int lv = 0; lv < levels; lv++) {
        fresh.clear();
        for (int c = 0; c < kpar; c++) {
            if (in_cell[c] || !allowed(c)) continue;
            for (int j = 0; j < 8; j++)
                if (in_node[a.nver[(size_t)c * ns + j]]) {
                    fresh.push_back(c);
                    break;
                }
        }
        for (int c : fresh) {
            in_cell[c] = 1;
            for (int j = 0; j < 8; j++) in_node[a.nver[(size_t)c * ns + j]] = 1;
        }
    }
    SubBuild s;
    for (int c = 0; c < kpar; c++)
        if (in_cell[c]) s.cells.push_back(c);
    for (int n = 0; n < kuz; n++)
        if (in_node[n]) s.nodes.push_back(n);
    return s;
}

// T_Brick::Phi_node at a point of a brick (T_Brick.cpp:866-887, 2010-2023)
void trilinear_weights(const double *lo, const double *hi, const double *p, double *w)
{
    double l0[3], l1[3];
    for (int d = 0; d < 3; d++) {
        const double t = (2.0 * p[d] - lo[d] - hi[d]) / (hi[d] - lo[d]);
        l0[d] = 0.5 * (1.0 - t);
        l1[d] = 0.5 * (1.0 + t);
    }
    for (int j = 0; j < 8; j++)
        w[j] = ((j & 1) ? l1[0] : l0[0]) * ((j & 2) ? l1[1] : l0[1]) * ((j & 4) ? l1[2] : l0[2]);
}

}  // namespace

void Smoothing::release()
{
    dev_free(d_cell);
    dev_free(d_cell_sub);
    dev_free(d_cell_g);
    dev_free(d_nc_ptr);
    dev_free(d_nc);
    dev_free(d_m64);
    dev_free(d_off);
    dev_free(d_nn);
    dev_free(d_m32);
    dev_free(d_dinv);
    dev_free(d_rn);
    dev_free(d_rw);
    dev_free(d_val);
    dev_free(d_x);
    dev_free(d_r);
    dev_free(d_f);
    dev_free(d_w);
    dev_free(d_out);
    S_cap = 0;
}

template <class T>
static int upload(T **d, const std::vector<T> &h, cudaStream_t st)
{
    int rc = dev_alloc(d, h.size());
    if (rc) return rc;
    if (!h.empty())
        MTGPU_TRY(cudaMemcpyAsync(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, st));
    return MTGPU_OK;
}

int smoothing_build(Smoothing &sm, const ::mtgpu_assembly_s &a, int nrec, const double *xyz_rec,
                    cudaStream_t st)
{
    const ParamMatrix &P = a.P;
    const int ns = a.nver_stride;
    // receiver bricks: curl A (all materials) and A (air skipped), boxes + 1e-6
    std::vector<int> eb(nrec), ea(nrec);
    {
        int *d_e = nullptr;
        double *d_rec = nullptr;
        int rc;
        if ((rc = dev_alloc(&d_e, (size_t)2 * nrec)) || (rc = dev_alloc(&d_rec, (size_t)3 * nrec))) {
            dev_free(d_e);
            return rc;
        }
        cudaError_t e = cudaMemcpyAsync(d_rec, xyz_rec, sizeof(double) * 3 * nrec,
                                        cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            rc = locate_receivers(P, nrec, d_rec, 1e-6, false, d_e, st);
            if (!rc) rc = locate_receivers(P, nrec, d_rec, 1e-6, true, d_e + nrec, st);
            if (!rc) {
                e = cudaMemcpyAsync(eb.data(), d_e, sizeof(int) * nrec, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(ea.data(), d_e + nrec, sizeof(int) * nrec,
                                        cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            }
        }
        dev_free(d_e);
        dev_free(d_rec);
        if (rc) return rc;
        if (e != cudaSuccess) {
            set_last_error(e, "smoothing receiver location", __FILE__, __LINE__);
            return MTGPU_ERR_CUDA;
        }
        for (int r = 0; r < nrec; r++) {
            if (eb[r] == INT_MAX) eb[r] = -1;
            if (ea[r] == INT_MAX) ea[r] = -1;
        }
    }
    // subdomains: curl A over all materials, A per material with a receiver
    std::vector<int> mats;
    for (int r = 0; r < nrec; r++)
        if (ea[r] >= 0) mats.push_back(a.nvkat[ea[r]]);
    std::sort(mats.begin(), mats.end());
    mats.erase(std::unique(mats.begin(), mats.end()), mats.end());
    std::vector<SubBuild> subs;
    std::vector<int> sub_mat;
    subs.push_back(grow_subdomain(a, eb, -1, sm.levels));
    sub_mat.push_back(-1);
    for (int m : mats) {
        subs.push_back(grow_subdomain(a, ea, m, sm.levels));
        sub_mat.push_back(m);
    }
    sm.nsub = (int)subs.size();
    sm.sub_cells.clear();
    sm.sub_nodes.clear();
    sm.sub_material = sub_mat;
    // padded node numbering, bricks, mass matrix, node -> bricks
    std::vector<int> node_off(sm.nsub + 1, 0), cell_off(sm.nsub + 1, 0);
    for (int s = 0; s < sm.nsub; s++) {
        const int nn = (int)subs[s].nodes.size();
        node_off[s + 1] = node_off[s] + (nn + kPad - 1) / kPad * kPad;
        cell_off[s + 1] = cell_off[s] + (int)subs[s].cells.size();
        sm.sub_cells.push_back((int)subs[s].cells.size());
        sm.sub_nodes.push_back(nn);
    }
    sm.npad = node_off[sm.nsub];
    sm.ncell = cell_off[sm.nsub];
    std::vector<int> cell(sm.ncell), cell_sub(sm.ncell);
    std::vector<double> cell_g(sm.ncell);
    std::vector<float> dinv(sm.npad, 1.f);
    std::vector<int2> m32((size_t)sm.npad * kSlots, make_int2(0, 0));
    std::vector<double> m64((size_t)sm.npad * kSlots, 0.0);
    std::vector<int> nc_ptr(sm.npad + 1, 0), nc;
    std::vector<int> loc(P.kuzlov, -1);
    for (int s = 0; s < sm.nsub; s++) {
        const SubBuild &B = subs[s];
        const int n0 = node_off[s], nn = (int)B.nodes.size();
        for (int i = 0; i < nn; i++) loc[B.nodes[i]] = i;
        // rows of up to 27 (column, value) slots
        std::vector<int> rc(27 * (size_t)nn, -1), cnt(nn, 0);
        std::vector<double> rv(27 * (size_t)nn, 0.0);
        std::vector<std::vector<int>> adj(nn);
        for (size_t ci = 0; ci < B.cells.size(); ci++) {
            const int c = B.cells[ci], gi = cell_off[s] + (int)ci;
            cell[gi] = c;
            cell_sub[gi] = s;
            const int *nv = &a.nver[(size_t)c * ns];
            const double *x0 = &a.xyz[3 * (size_t)nv[0]], *x7 = &a.xyz[3 * (size_t)nv[7]];
            // Hex_Local_Matrix.cpp:120-198
            const double t2 = (x7[0] - x0[0]) * (x7[1] - x0[1]) * (x7[2] - x0[2]);
            const double t[4] = {t2 / 27.0, t2 / 54.0, t2 / 108.0, t2 / 216.0};
            double g = 0.0;   // row sum (Subdomain.cpp:504-505), corner 0
            for (int k = 0; k < 8; k++) g += t[__builtin_popcount(k)];
            cell_g[gi] = g;
            int li[8];
            for (int j = 0; j < 8; j++) li[j] = loc[nv[j]];
            for (int j = 0; j < 8; j++) {
                adj[li[j]].push_back(gi);
                for (int k = 0; k < 8; k++) {
                    const double bv = t[__builtin_popcount(j ^ k)];
                    const size_t base = 27 * (size_t)li[j];
                    int q = 0;
                    while (q < cnt[li[j]] && rc[base + q] != li[k]) q++;
                    if (q == cnt[li[j]]) {
                        if (q == 27) {
                            set_last_message("smoothing: a node with more than 27 neighbours "
                                             "(the mesh is not a conforming hexahedral mesh)");
                            return MTGPU_ERR_ARG;
                        }
                        rc[base + q] = li[k];
                        rv[base + q] = 0.0;
                        cnt[li[j]]++;
                    }
                    rv[base + q] += bv;
                }
            }
        }
        for (int i = 0; i < nn; i++) {
            const size_t base = 27 * (size_t)i;
            std::vector<std::pair<int, double>> row(cnt[i]);
            for (int q = 0; q < cnt[i]; q++) row[q] = {rc[base + q], rv[base + q]};
            std::sort(row.begin(), row.end());
            const size_t at = (size_t)n0 * kSlots + (size_t)(i >> 5) * (32 * kSlots) + (i & 31);
            for (int q = 0; q < cnt[i]; q++) {
                const float v32 = (float)row[q].second;
                m32[at + 32 * q].x = row[q].first;
                memcpy(&m32[at + 32 * q].y, &v32, sizeof(float));
                m64[at + 32 * q] = row[q].second;
                if (row[q].first == i) dinv[n0 + i] = (float)(1.0 / row[q].second);
            }
            for (int c : adj[i]) nc.push_back(c);
            nc_ptr[n0 + i + 1] = (int)nc.size();
        }
        for (int i = nn; i < node_off[s + 1] - n0; i++) nc_ptr[n0 + i + 1] = (int)nc.size();   // padding rows
        for (int i = 0; i < nn; i++) loc[B.nodes[i]] = -1;
    }
    // receivers: padded nodes and trilinear weights of their brick, per type
    std::vector<int> rn((size_t)nrec * 16, -1);
    std::vector<double> rw((size_t)nrec * 16, 0.0);
    for (int r = 0; r < nrec; r++) {
        for (int t = 0; t < 2; t++) {
            const int c = t == 0 ? eb[r] : ea[r];
            if (c < 0) continue;
            int s = 0;
            if (t == 1) s = 1 + (int)(std::lower_bound(mats.begin(), mats.end(), a.nvkat[c]) -
                                      mats.begin());
            const SubBuild &B = subs[s];
            const int *nv = &a.nver[(size_t)c * ns];
            for (int j = 0; j < 8; j++) {
                auto it = std::lower_bound(B.nodes.begin(), B.nodes.end(), nv[j]);
                rn[(size_t)(r * 2 + t) * 8 + j] = node_off[s] + (int)(it - B.nodes.begin());
            }
            trilinear_weights(&a.xyz[3 * (size_t)nv[0]], &a.xyz[3 * (size_t)nv[7]],
                              xyz_rec + 3 * (size_t)r, &rw[(size_t)(r * 2 + t) * 8]);
        }
    }
    int rc;
    if ((rc = upload(&sm.d_cell, cell, st)) || (rc = upload(&sm.d_cell_sub, cell_sub, st)) ||
        (rc = upload(&sm.d_cell_g, cell_g, st)) || (rc = upload(&sm.d_nc_ptr, nc_ptr, st)) ||
        (rc = upload(&sm.d_nc, nc, st)) || (rc = upload(&sm.d_m64, m64, st)) ||
        (rc = upload(&sm.d_m32, m32, st)) || (rc = upload(&sm.d_dinv, dinv, st)) ||
        (rc = upload(&sm.d_off, node_off, st)) || (rc = upload(&sm.d_nn, sm.sub_nodes, st)) ||
        (rc = upload(&sm.d_rn, rn, st)) || (rc = upload(&sm.d_rw, rw, st)) ||
        (rc = dev_alloc(&sm.d_out, 2)))
        return rc;
    MTGPU_TRY(cudaStreamSynchronize(st));   // the host vectors go out of scope
    // clusters of q blocks that run side by side
    for (int q = 2; q <= kMaxCluster; q *= 2) {
        cudaLaunchAttribute at[1];
        cudaLaunchConfig_t cfg = cluster_config(at, q, 1, 1);
        sm.clusters[q] = 0;
        if (cudaOccupancyMaxActiveClusters(&sm.clusters[q], k_sm_solve<2, true>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            sm.clusters[q] = 0;
        }
    }
    return MTGPU_OK;
}

int smoothing_fields(Smoothing &sm, const ParamMatrix &P, int nrec, int S, long long x_stride,
                     const double2 *d_x, const double *d_omega, const int *d_alfa, int n1d,
                     const double *d_z1d, const double *d_us, const double *d_uc,
                     const double4 *d_loc, double2 *d_e, double2 *d_h, double2 *d_scal,
                     cudaStream_t st)
{
    // grow-only work arrays
    const int ncol = 6 * S;
    if (S > sm.S_cap) {
        for (double **p : {&sm.d_val, &sm.d_x, &sm.d_r, &sm.d_f}) dev_free(*p);
        dev_free(sm.d_w);
        sm.S_cap = 0;
        const size_t nv = (size_t)ncol * sm.npad;
        int rc;
        if ((rc = dev_alloc(&sm.d_val, (size_t)ncol * std::max(sm.ncell, 1))) ||
            (rc = dev_alloc(&sm.d_x, nv)) || (rc = dev_alloc(&sm.d_r, nv)) ||
            (rc = dev_alloc(&sm.d_f, nv)) || (rc = dev_alloc(&sm.d_w, (size_t)4 * (ncol + 3) * sm.npad)))
            return rc;
        sm.S_cap = S;
    }
    unsigned long long launches = 0;
    sm.iterations = 0;
    if (sm.npad > 0) {
        k_sm_centre<<<dim3(ceil_div(sm.ncell, kThreads), S), kThreads, 0, st>>>(
            sm.ncell, S, sm.d_cell, sm.d_cell_sub, P.d_nver, P.nver_stride, P.d_ed, P.ed_stride,
            P.d_xyz, x_stride, d_x, sm.d_val);
        // four columns a block share the matrix's reads; two where four would
        // leave more than a third of the SMs without a block
        int dev = 0, nsm = 1;
        MTGPU_TRY(cudaGetDevice(&dev));
        MTGPU_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        const int C = 3LL * ceil_div(ncol, 4) * sm.nsub >= 2LL * nsm ? 4 : 2, groups = ceil_div(ncol, C);
        // p of a subdomain in shared memory where it fits (12,800 nodes at
        // four columns), else in L2
        constexpr int kSmem = 200 * 1024;
        int widest = 0;
        for (int n : sm.sub_nodes) widest = std::max(widest, n);
        int q = 1;
        if (C == 2)
            while (q < kMaxCluster && widest >= kClusterNodes * 2 * q && groups * sm.nsub <= sm.clusters[2 * q]) q *= 2;
        const int smem = q > 1 ? 0 : (int)std::min<long long>(kSmem, (long long)widest * 4 * C);
        const SolveArgs A{sm.npad, ncol, sm.ncell, sm.d_off, sm.d_nn, sm.d_nc_ptr, sm.d_nc, sm.d_cell_g,
                          sm.d_val, sm.d_m32, sm.d_m64, sm.d_dinv, sm.d_x, sm.d_f, sm.d_r, sm.d_w, smem,
                          q, sm.d_out};
        MTGPU_TRY(cudaMemsetAsync(sm.d_out, 0, 2 * sizeof(int), st));
        if (q > 1) {
            cudaLaunchAttribute at[1];
            cudaLaunchConfig_t cfg = cluster_config(at, q, groups, sm.nsub);
            cfg.stream = st;
            MTGPU_TRY(cudaLaunchKernelEx(&cfg, k_sm_solve<2, true>, A));
        } else {
            const void *solve = C == 4 ? (const void *)k_sm_solve<4, false> : (const void *)k_sm_solve<2, false>;
            MTGPU_TRY(cudaFuncSetAttribute(solve, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
            if (C == 4) k_sm_solve<4, false><<<dim3(groups, sm.nsub), kSolve, smem, st>>>(A);
            else k_sm_solve<2, false><<<dim3(groups, sm.nsub), kSolve, smem, st>>>(A);
        }
        launches += 2;
        MTGPU_TRY(cudaGetLastError());
        int out[2] = {0, 0};
        MTGPU_TRY(cudaMemcpyAsync(out, sm.d_out, sizeof(out), cudaMemcpyDeviceToHost, st));
        MTGPU_TRY(cudaStreamSynchronize(st));
        sm.iterations = out[1];
        if (out[0] > 0) {
            set_last_message("receiver smoothing: the projection solve did not converge");
            note_launches(launches);
            return MTGPU_MAXITER;
        }
    }
    k_sm_receivers<<<dim3(ceil_div(nrec, 128), S), 128, 0, st>>>(
        nrec, S, sm.npad, sm.d_rn, sm.d_rw, sm.d_x, d_omega, d_alfa, n1d, d_z1d, d_us, d_uc,
        d_loc, d_e, d_h, d_scal);
    note_launches(launches + 1);
    MTGPU_TRY(cudaGetLastError());
    return MTGPU_OK;
}

}  // namespace mtgpu
