// Batched double-float COCR survey solver.
//
// All systems of a survey (frequencies x polarisations) share the mesh, hence
// the sparsity pattern and the frequency-independent matrices of
// A_k = K + i omega_k M.  One launch works on every system: a thread owns one
// (row, system) pair, the SP systems of a row sit in adjacent lanes, so K, M
// and the column indices are read once per row for all systems and every
// gather of a vector row is one contiguous SP-wide segment.
//
// Arithmetic.  GB300 issues FP32 at 64x its FP64 rate.  Plain FP32 Krylov
// iterations do not converge on these systems: the air (sigma = 1e-8 S/m)
// leaves the gradient null space of the curl-curl operator regularised only
// at ~1e-12 of its scale, below FP32 resolution.  So every quantity here is a
// double-float (dfloat.cuh: hi + lo FP32 pair, 48-bit significand) computed
// on the FP32 pipes; the iteration then follows the FP64 reference, iteration
// for iteration.
//
// Algorithm.  The reference's preconditioned COCR
// (Code/COCR_FP/pcocr_rci.cpp:52-181) with the folded preconditioner
// (FoldedPreconditioner.cpp:578-630) and the MRS-smoothed stop test
// (MRS.cpp:85-153, rci.cpp:66-75), per system; when a system stops, its true
// residual ||b - A x|| / ||b|| is computed in FP64 and, if `verify` is set and
// it is not below eps, the system keeps iterating or restarts on its FP64
// residual (iterative refinement, FP64 solution).  One iteration is the node
// gather, the edge gather + (a, w), the updates + the MRS smoothing, and the
// SpMV + (z, s) (one kernel for a stored matrix, two for the matrix-free
// forms), captured in a CUDA graph several iterations at a time, with p and x
// brought up to date once per group of iterations; all per-system decisions are
// taken on the device by the block of each kernel that finishes last.  Small
// problems run a group's iterations in one cooperative kernel (survey_small.cuh).
#include "survey_impl.cuh"

#include <algorithm>
#include <chrono>
#include <climits>
#include <cstdlib>
#include <cstring>

namespace mtgpu {

using namespace dfl;
using namespace sv;

void Survey::release()
{
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
    dev_free(kc); dev_free(mc); dev_free(kr);
    dev_free(gv32); dev_free(tv32);
    dev_free(da); dev_free(ds);
    dev_free(omega); dev_free(omega64); dev_free(gkg); dev_free(gmg);
    dev_free(sys);
    dev_free(r); dev_free(s); dev_free(hist); dev_free(p); dev_free(a);
    dev_free(z); dev_free(w); dev_free(sm); dev_free(h); dev_free(a2);
    prec_tile = false;
    dev_free(b64); dev_free(xacc);
    dev_free(uoff); dev_free(ucol); dev_free(lc); dev_free(lr);
    ntiles = 0;
    tiles_built = false;
    dev_free(partials);
    if (hsys) cudaFreeHost(hsys);
    hsys = nullptr;
    G.release();
    mf.release();
}

void MatFree::release()
{
    dev_free(pos);
    dev_free(w);
    dev_free(f);
    dev_free(g);
    dev_free(dir);
    ndir = 0;
    on = false;
    lattice = false;
    tiled = false;
    tile_checked = false;
    gface = false;
}

namespace {

// counts the G rows that differ from k_node_lat's lattice form
__global__ void k_g_lattice_check(MF M, int m, const int *__restrict__ gp, const int *__restrict__ gj,
                                  const float *__restrict__ gv, int *bad)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m) return;
    const int ix = M.nx - 2, iy = M.ny - 2;
    const int i = v % ix + 1, t = v / ix, j = t % iy + 1, kk = t / iy + 1;
    const int e0 = mf_edge_in(M, 0, i, j, kk);
    const int es[6] = {e0 + 2 - M.plane, e0 + 1 - M.l3, e0 - 3, e0, e0 + 1, e0 + 2};
    int nbad = gp[v + 1] - gp[v] != 6;
    if (!nbad)
        for (int q = 0; q < 6; q++)
            if (gj[gp[v] + q] != es[q] || gv[gp[v] + q] != (q < 3 ? 0.5f : -0.5f)) nbad = 1;
    if (nbad) atomicAdd(bad, 1);
}

// Two row-major vectors of double-float values, the lanes of the batch's S
// systems: out[0], out[1] the largest |a - b| and |b| (bits of a double),
// out[2] whether any value differs, out[3] whether any is a NaN.
// The magnitudes are FP32 (FP64 values and an atomic per thread took 590 us
// for 19.5M complex values): |a - b| to 2^-47 |b| and 2^-23 of itself, for
// the tolerances; equality is out[2]'s, word by word.
__global__ void k_maxdiff(long long n, int S, int SP, const float4 *__restrict__ a,
                          const float4 *__restrict__ b, unsigned long long *out)
{
    float dm = 0.f, bm = 0.f;
    bool differs = false, nan = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        if ((int)(i & (SP - 1)) >= S) continue;       // lanes that nothing writes
        const float4 u = a[i], v = b[i];
        differs |= !(u.x == v.x && u.y == v.y && u.z == v.z && u.w == v.w);
        const float re = (u.x - v.x) + (u.z - v.z), im = (u.y - v.y) + (u.w - v.w);
        nan |= re != re || im != im;
        dm = fmaxf(dm, fmaxf(fabsf(re), fabsf(im)));
        bm = fmaxf(bm, fmaxf(fabsf(v.x + v.z), fabsf(v.y + v.w)));
    }
    __shared__ unsigned int mx[4];
    if (threadIdx.x < 4) mx[threadIdx.x] = 0u;
    __syncthreads();
    // the order of non-negative floats is that of their bits
    atomicMax(&mx[0], __float_as_uint(dm));
    atomicMax(&mx[1], __float_as_uint(bm));
    if (differs) mx[2] = 1u;
    if (nan) mx[3] = 1u;
    __syncthreads();
    if (threadIdx.x < 2)
        atomicMax(out + threadIdx.x,
                  (unsigned long long)__double_as_longlong((double)__uint_as_float(mx[threadIdx.x])));
    else if (threadIdx.x < 4 && mx[threadIdx.x])
        atomicMax(out + threadIdx.x, 1ull);
}
struct MaxDiff {
    unsigned long long w[4] = {0, 0, 1, 1};
    bool equal() const { return w[2] == 0; }
    // |a - b| / |b| by the largest of each; 1 where there is nothing to compare or a NaN
    double relative() const
    {
        double d, m;
        memcpy(&d, &w[0], sizeof(double));
        memcpy(&m, &w[1], sizeof(double));
        return m > 0.0 && w[3] == 0 ? d / m : 1.0;
    }
};

// a fixed pseudo-random test vector (double-float values in [-1, 1))
__global__ void k_pattern(long long n, float4 *v)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        unsigned h = (unsigned)i * 2654435761u + 12345u;
        float q[4];
        for (int t = 0; t < 4; t++) {
            h ^= h >> 15;
            h *= 2246822519u;
            h ^= h >> 13;
            q[t] = (float)(h & 0xffffffu) / 8388608.0f - 1.0f;
        }
        v[i] = make_float4(q[0], q[2] * (1.f + 0.25f * q[1] * q[3]), 0.f, 0.f);
    }
}

// pass 0 (write == 0): count[t] = distinct columns of tile t; pass 1: the
// distinct columns to ucol[uoff[t]..] and every slot's local index.  A tile
// with more than kTileMaxKeys slots sets *overflow.
__global__ void __launch_bounds__(kTileThreads)
k_tile_cols(int nslices, int T, const long long *pc, const long long *pr, const int *col_c,
            const int *col_r, const int *uoff, int *count, int *ucol, unsigned short *lc,
            unsigned short *lr, int *overflow, int write)
{
    extern __shared__ int keys[];              // [kTileMaxKeys], then unique [kTileMaxKeys]
    int *uniq = keys + kTileMaxKeys;
    __shared__ int part[kTileThreads];
    const int t = blockIdx.x;
    const int s0 = t * T, s1 = min(s0 + T, nslices);
    const long long c0 = pc[s0], nc = pc[s1] - c0, q0 = pr[s0], nr = pr[s1] - q0;
    const long long n = nc + nr;
    if (n > kTileMaxKeys) {
        if (threadIdx.x == 0) atomicExch(overflow, 1);
        return;
    }
    int np2 = 1;
    while (np2 < n) np2 <<= 1;
    for (int i = threadIdx.x; i < np2; i += blockDim.x)
        keys[i] = i < nc ? col_c[c0 + i] : (i < n ? col_r[q0 + i - nc] : INT_MAX);
    __syncthreads();
    // bitonic sort
    for (int size = 2; size <= np2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < np2; i += blockDim.x) {
                const int j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0;
                    const int a = keys[i], b = keys[j];
                    if ((a > b) == up) {
                        keys[i] = b;
                        keys[j] = a;
                    }
                }
            }
            __syncthreads();
        }
    // distinct values: a contiguous chunk per thread, then a scan of the chunk counts
    const int chunk = (int)((n + blockDim.x - 1) / blockDim.x);
    const int a0 = threadIdx.x * chunk, a1 = min((long long)a0 + chunk, n);
    int cnt = 0;
    for (int i = a0; i < a1; i++) cnt += (i == 0 || keys[i] != keys[i - 1]);
    part[threadIdx.x] = cnt;
    __syncthreads();
    for (int off = 1; off < (int)blockDim.x; off <<= 1) {
        const int v = threadIdx.x >= off ? part[threadIdx.x - off] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    const int total = part[blockDim.x - 1];
    if (!write) {
        if (threadIdx.x == 0) count[t] = total;
        return;
    }
    int pos = part[threadIdx.x] - cnt;
    for (int i = a0; i < a1; i++)
        if (i == 0 || keys[i] != keys[i - 1]) uniq[pos++] = keys[i];
    __syncthreads();
    for (int i = threadIdx.x; i < total; i += blockDim.x) ucol[uoff[t] + i] = uniq[i];
    // local index of every slot: binary search in uniq
    for (long long i = threadIdx.x; i < n; i += blockDim.x) {
        const int c = i < nc ? col_c[c0 + i] : col_r[q0 + i - nc];
        int lo = 0, hi = total - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (uniq[mid] < c) lo = mid + 1; else hi = mid;
        }
        if (i < nc) lc[c0 + i] = (unsigned short)lo;
        else lr[q0 + i - nc] = (unsigned short)lo;
    }
}

// System-major [S][nb] FP64 <-> row-major [nb][SP], FP64 or double-float.
// With more than kFewLanes lanes a block moves 32 rows of all systems through
// shared memory, so that both sides are read and written in whole lines:
// element by element in the row-major order, a warp of 32 systems touched 32
// lines of the system-major side for 16 bytes of each (32 systems x 610k rows:
// 283 -> 150 us in, 345 -> 150 us out).  With few lanes a warp's elements are whole
// lines on both sides as they are, and a block of 32 rows leaves most of its
// threads idle: a product with both transposes on 1.8M rows took 190 us that way
// against 129 at 1 lane, 247 against 204 at 2, 390 against 374 at 4; 704 both at 8.
constexpr int kTRows = 32;
__device__ __forceinline__ void row_store(double2 *p, double2 v) { *p = v; }
__device__ __forceinline__ void row_store(float4 *p, double2 v) { *p = to4(from_d2(v)); }
__device__ __forceinline__ double2 row_load(const double2 *p) { return *p; }
__device__ __forceinline__ double2 row_load(const float4 *p) { return to_d2(*p); }

template <class T>
__global__ void __launch_bounds__(kB)
k_to_rows(int nb, int S, int SP, const double2 *__restrict__ src, T *__restrict__ dst)
{
    __shared__ double2 t[32][kTRows + 1];
    const int r0 = blockIdx.x * kTRows, l = threadIdx.x % kTRows;
    if (r0 + l < nb)
        for (int k = threadIdx.x / kTRows; k < S; k += kB / kTRows) t[k][l] = src[(long long)k * nb + r0 + l];
    __syncthreads();
    for (int i = threadIdx.x; i < kTRows * SP; i += kB) {
        const int k = i % SP, r = i / SP;
        if (r0 + r < nb) row_store(dst + (long long)r0 * SP + i, k < S ? t[k][r] : make_double2(0.0, 0.0));
    }
}

template <class T>
__global__ void __launch_bounds__(kB)
k_from_rows(int nb, int S, int SP, const T *__restrict__ src, double2 *__restrict__ dst)
{
    __shared__ double2 t[32][kTRows + 1];
    const int r0 = blockIdx.x * kTRows, l = threadIdx.x % kTRows;
    for (int i = threadIdx.x; i < kTRows * SP; i += kB) {
        const int k = i % SP, r = i / SP;
        if (r0 + r < nb && k < S) t[k][r] = row_load(src + (long long)r0 * SP + i);
    }
    __syncthreads();
    if (r0 + l < nb)
        for (int k = threadIdx.x / kTRows; k < S; k += kB / kTRows) dst[(long long)k * nb + r0 + l] = t[k][l];
}

// element by element in the row-major order; SP = 1 << lg
template <class T>
__global__ void __launch_bounds__(kB)
k_to_rows_few(int nb, int S, int lg, const double2 *__restrict__ src, T *__restrict__ dst)
{
    const long long i = (long long)blockIdx.x * kB + threadIdx.x, row = i >> lg;
    const int k = (int)i & ((1 << lg) - 1);
    if (row < nb) row_store(dst + i, k < S ? src[(long long)k * nb + row] : make_double2(0.0, 0.0));
}

template <class T>
__global__ void __launch_bounds__(kB)
k_from_rows_few(int nb, int S, int lg, const T *__restrict__ src, double2 *__restrict__ dst)
{
    const long long i = (long long)blockIdx.x * kB + threadIdx.x, row = i >> lg;
    const int k = (int)i & ((1 << lg) - 1);
    if (row < nb && k < S) dst[(long long)k * nb + row] = row_load(src + i);
}

constexpr int kFewLanes = 4;
template <class T>
void to_rows(const Survey &V, const double2 *src, T *dst)
{
    const int lg = __builtin_ctz(V.SP);
    if (V.SP <= kFewLanes)
        k_to_rows_few<<<(unsigned)((((long long)V.nb << lg) + kB - 1) / kB), kB, 0, V.st>>>(V.nb, V.S, lg, src, dst);
    else
        k_to_rows<<<(unsigned)ceil_div(V.nb, kTRows), kB, 0, V.st>>>(V.nb, V.S, V.SP, src, dst);
    note_launches(1);
}
template <class T>
void from_rows(const Survey &V, const T *src, double2 *dst)
{
    const int lg = __builtin_ctz(V.SP);
    if (V.SP <= kFewLanes)
        k_from_rows_few<<<(unsigned)((((long long)V.nb << lg) + kB - 1) / kB), kB, 0, V.st>>>(V.nb, V.S, lg, src, dst);
    else
        k_from_rows<<<(unsigned)ceil_div(V.nb, kTRows), kB, 0, V.st>>>(V.nb, V.S, V.SP, src, dst);
    note_launches(1);
}

// ------------------------------------------------------- conversions
__global__ void k_to_df(long long n, const double *src, float2 *dst)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const df v = from_double(src[i]);
        dst[i] = make_float2(v.h, v.l);
    }
}

// D_A[row][k] = 1 / (K_ii + i omega_k M_ii), computed in FP64
__global__ void k_diag_a(int nb, int SP, const int *nc, const long long *pc, const int *col_c,
                         const double *kcd, const double *mcd, const double *omega64, float4 *da)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nb * SP) return;
    const int k = (int)(i % SP);
    const int row = (int)(i / SP);
    double kk = 0.0, mm = 0.0;
    for (int q = 0; q < nc[row]; q++) {
        const long long t = slot(pc, row, q);
        if (col_c[t] == row) {
            kk = kcd[t];
            mm = mcd[t];
        }
    }
    const double2 inv = cdiv(make_double2(1.0, 0.0), make_double2(kk, omega64[k] * mm));
    da[i] = to4(from_d2(inv));
}

// D_S[v][k] = 1 / (diag(G K G^T) + i omega_k diag(G M G^T)), in FP64
__global__ void k_diag_s(int m, int SP, const double *gkg, const double *gmg,
                         const double *omega64, float4 *ds)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)m * SP) return;
    const int k = (int)(i % SP);
    const int v = (int)(i / SP);
    const double2 inv = cdiv(make_double2(1.0, 0.0), make_double2(gkg[v], omega64[k] * gmg[v]));
    ds[i] = to4(from_d2(inv));
}

// diag(G K G^T) and diag(G M G^T), FP64, in the reference's summation order
// (row k of A by increasing column, unfused multiply-add; see folded.cu),
// in two passes: one thread per G entry j = (v, k) forms t_j = sum over row
// k of A of A[k][c] G[v][c]; then one thread per node v adds t_j G[v][k]
// over its entries in G's order — the sums and their order of the single
// pass, without its per-node serial chain
__global__ void k_gdiag_entry(int m, const int *__restrict__ gp, const int *__restrict__ gj,
                              const double *__restrict__ gv, const int *__restrict__ rowof,
                              const int *__restrict__ nc_row, const int *__restrict__ nr_row,
                              const long long *__restrict__ pc, const long long *__restrict__ pr,
                              const int *__restrict__ col_c, const double *__restrict__ kc,
                              const double *__restrict__ mc, const int *__restrict__ col_r,
                              const double *__restrict__ kr, double *tkv, double *tmv)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= gp[m]) return;
    const int v = rowof[j];
    const int b0 = gp[v], e0 = gp[v + 1];
    const int k = gj[j];
    const int nc = nc_row[k], nr = nr_row[k];
    double tk = 0.0, tm = 0.0;
    int qc = 0, qr = 0;
    while (qc < nc || qr < nr) {
        const int cc = qc < nc ? col_c[slot(pc, k, qc)] : 0x7fffffff;
        const int cr = qr < nr ? col_r[slot(pr, k, qr)] : 0x7fffffff;
        double kv, mv;
        int c;
        if (cc < cr) {
            const long long t = slot(pc, k, qc++);
            kv = kc[t];
            mv = mc[t];
            c = cc;
        } else {
            kv = kr[slot(pr, k, qr++)];
            mv = 0.0;
            c = cr;
        }
        for (int u = b0; u < e0; u++)
            if (gj[u] == c) {
                tk = __dadd_rn(tk, __dmul_rn(kv, gv[u]));
                tm = __dadd_rn(tm, __dmul_rn(mv, gv[u]));
            }
    }
    tkv[j] = tk;
    tmv[j] = tm;
}

// The first pass on meshes with the compact G^T, one thread per edge k: row
// k of A is read slot by slot (a warp's 32 rows side by side in the slice),
// and both of column k's G entries (v_a, k) and (v_b, k) are formed, v_a and
// v_b the G rows of k's first and second node.  G[v][c] is -1/2 where v is
// the row of c's first node and +1/2 where it is its second's, so every
// term and its place in the sum are those of k_gdiag_entry.  t[k] holds
// (t of v_a, t of v_b).
__global__ void k_gdiag_edge(int nb, const int2 *__restrict__ tn, const int *__restrict__ nc_row,
                             const int *__restrict__ nr_row, const long long *__restrict__ pc,
                             const long long *__restrict__ pr, const int *__restrict__ col_c,
                             const double *__restrict__ kc, const double *__restrict__ mc,
                             const int *__restrict__ col_r, const double *__restrict__ kr,
                             double2 *tk, double2 *tm)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nb) return;
    const int2 me = tn[k];
    if (me.x < 0 && me.y < 0) return;
    const int nc = nc_row[k], nr = nr_row[k];
    double ak = 0.0, am = 0.0, bk = 0.0, bm = 0.0;
    int qc = 0, qr = 0;
    int cc = nc > 0 ? col_c[slot(pc, k, 0)] : 0x7fffffff;
    int cr = nr > 0 ? col_r[slot(pr, k, 0)] : 0x7fffffff;
    while (qc < nc || qr < nr) {
        double kv, mv;
        int c;
        if (cc < cr) {
            const long long t = slot(pc, k, qc++);
            kv = kc[t];
            mv = mc[t];
            c = cc;
            cc = qc < nc ? col_c[slot(pc, k, qc)] : 0x7fffffff;
        } else {
            kv = kr[slot(pr, k, qr++)];
            mv = 0.0;
            c = cr;
            cr = qr < nr ? col_r[slot(pr, k, qr)] : 0x7fffffff;
        }
        const int2 o = __ldg(tn + c);
        const double ga = me.x < 0 ? 0.0 : (o.x == me.x ? -0.5 : (o.y == me.x ? 0.5 : 0.0));
        const double gb = me.y < 0 ? 0.0 : (o.x == me.y ? -0.5 : (o.y == me.y ? 0.5 : 0.0));
        if (ga != 0.0) {
            ak = __dadd_rn(ak, __dmul_rn(kv, ga));
            am = __dadd_rn(am, __dmul_rn(mv, ga));
        }
        if (gb != 0.0) {
            bk = __dadd_rn(bk, __dmul_rn(kv, gb));
            bm = __dadd_rn(bm, __dmul_rn(mv, gb));
        }
    }
    tk[k] = make_double2(ak, bk);
    tm[k] = make_double2(am, bm);
}

// the second pass over k_gdiag_edge's per-edge values: node v's entries in
// G's order, each t taken from the side of its edge that v is
__global__ void k_gdiag_nodes(int m, const int *__restrict__ gp, const int *__restrict__ gj,
                              const double *__restrict__ gv, const int2 *__restrict__ tn,
                              const double2 *__restrict__ tk, const double2 *__restrict__ tm,
                              double *gkg, double *gmg)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m) return;
    double sk = 0.0, sm = 0.0;
    for (int j = gp[v]; j < gp[v + 1]; j++) {
        const int e = gj[j];
        const bool first = tn[e].x == v;
        const double2 a = tk[e], b = tm[e];
        sk = __dadd_rn(sk, __dmul_rn(first ? a.x : a.y, gv[j]));
        sm = __dadd_rn(sm, __dmul_rn(first ? b.x : b.y, gv[j]));
    }
    gkg[v] = sk;
    gmg[v] = sm;
}

__global__ void k_gdiag_rows(int m, const int *__restrict__ gp, int *rowof)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m) return;
    for (int j = gp[v]; j < gp[v + 1]; j++) rowof[j] = v;
}

__global__ void k_gdiag(int m, const int *__restrict__ gp, const double *__restrict__ gv,
                        const double *__restrict__ tkv, const double *__restrict__ tmv,
                        double *gkg, double *gmg)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= m) return;
    double sk = 0.0, sm = 0.0;
    for (int j = gp[v]; j < gp[v + 1]; j++) {
        sk = __dadd_rn(sk, __dmul_rn(tkv[j], gv[j]));
        sm = __dadd_rn(sm, __dmul_rn(tmv[j], gv[j]));
    }
    gkg[v] = sk;
    gmg[v] = sm;
}

__global__ void k_f64_to_f32(long long n, const double *src, float *dst)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = (float)src[i];
}

const Ops &ops_of(int sp)
{
    switch (sp) {
    case 1: return ops1();
    case 2: return ops2();
    case 4: return ops4();
    case 8: return ops8();
    case 16: return ops16();
    default: return ops32();
    }
}
#define MTGPU_SP_DISPATCH(SPV, CALL) ops_of(SPV).CALL

int sync_sys(Survey &V)
{
    MTGPU_TRY(cudaMemcpyAsync(V.hsys, V.sys, sizeof(SysState) * kSysSlots, cudaMemcpyDeviceToHost, V.st));
    MTGPU_TRY(cudaStreamSynchronize(V.st));
    return MTGPU_OK;
}

}  // namespace

namespace {

// Tiles of the x-staged SpMV: TileCfg<SP>::T slices per tile, covered by
// a block of TileCfg<SP>::NT threads in whole passes.  Leaves
// V.ntiles = 0 (variant unavailable) when a tile does not fit the set-up
// sort or the shared memory of a block.
int build_tiles(Survey &V, int nsm)
{
    const ParamMatrix &P = *V.P;
    MTGPU_SP_DISPATCH(V.SP, tile_slices_of(&V.tile_T));
    const int nt = ceil_div(P.nslices, V.tile_T);
    int *d_count = nullptr, *d_over = nullptr;
    int rc;
    if ((rc = dev_alloc(&d_count, nt)) || (rc = dev_alloc(&d_over, 1)) ||
        (rc = dev_alloc(&V.uoff, nt + 1)) || (rc = dev_alloc(&V.lc, P.len_c)) ||
        (rc = dev_alloc(&V.lr, P.len_r))) {
        dev_free(d_count);
        dev_free(d_over);
        return rc;
    }
    auto done = [&](int code) {
        dev_free(d_count);
        dev_free(d_over);
        return code;
    };
    const int sort_smem = 2 * kTileMaxKeys * (int)sizeof(int);
    MTGPU_TRY(cudaFuncSetAttribute((const void *)k_tile_cols,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, sort_smem));
    MTGPU_TRY(cudaMemsetAsync(d_over, 0, sizeof(int), V.st));
    k_tile_cols<<<nt, kTileThreads, sort_smem, V.st>>>(P.nslices, V.tile_T, P.d_pc, P.d_pr,
                                                      P.d_col_c, P.d_col_r, V.uoff, d_count,
                                                      nullptr, V.lc, V.lr, d_over, 0);
    note_launches(1);
    MTGPU_TRY(cudaGetLastError());
    std::vector<int> count(nt), off(nt + 1, 0);
    std::vector<long long> pc(P.nslices + 1), pr(P.nslices + 1);
    int over = 0;
    MTGPU_TRY(cudaMemcpyAsync(&over, d_over, sizeof(int), cudaMemcpyDeviceToHost, V.st));
    MTGPU_TRY(cudaMemcpyAsync(count.data(), d_count, sizeof(int) * nt, cudaMemcpyDeviceToHost, V.st));
    MTGPU_TRY(cudaMemcpyAsync(pc.data(), P.d_pc, sizeof(long long) * pc.size(), cudaMemcpyDeviceToHost, V.st));
    MTGPU_TRY(cudaMemcpyAsync(pr.data(), P.d_pr, sizeof(long long) * pr.size(), cudaMemcpyDeviceToHost, V.st));
    MTGPU_TRY(cudaStreamSynchronize(V.st));
    if (over) return done(MTGPU_OK);
    long long smem = 0, smem_x = 0;
    for (int t = 0; t < nt; t++) {
        off[t + 1] = off[t] + count[t];
        const int s0 = t * V.tile_T, s1 = std::min(s0 + V.tile_T, P.nslices);
        smem = std::max(smem, tile_bytes(count[t], V.SP, pc[s1] - pc[s0], pr[s1] - pr[s0]));
        smem_x = std::max(smem_x, tile_bytes(count[t], V.SP, 0, 0));
    }
    int max_smem = 0;
    int dev = 0;
    MTGPU_TRY(cudaGetDevice(&dev));
    MTGPU_TRY(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (smem > max_smem - 26 * 1024) return done(MTGPU_OK);   // too large (with the static reduction buffers): variant off
    if ((rc = dev_alloc(&V.ucol, std::max(off[nt], 1)))) return done(rc);
    MTGPU_TRY(cudaMemcpyAsync(V.uoff, off.data(), sizeof(int) * (nt + 1), cudaMemcpyHostToDevice, V.st));
    k_tile_cols<<<nt, kTileThreads, sort_smem, V.st>>>(P.nslices, V.tile_T, P.d_pc, P.d_pr,
                                                      P.d_col_c, P.d_col_r, V.uoff, d_count,
                                                      V.ucol, V.lc, V.lr, d_over, 1);
    note_launches(1);
    MTGPU_TRY(cudaGetLastError());
    MTGPU_TRY(cudaStreamSynchronize(V.st));
    V.tile_smem = (int)smem;
    V.tile_smem_x = (int)smem_x;
    cudaError_t e = cudaSuccess;
    MTGPU_SP_DISPATCH(V.SP, tile_attr(V, &e));
    if (e != cudaSuccess) {
        cudaGetLastError();   // clear it: the variant is just unavailable
        return done(MTGPU_OK);
    }
    V.ntiles = nt;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    return done(MTGPU_OK);
}

}  // namespace

namespace {

// Set-up of the matrix-free tables on the device.  k_mfb_nodes checks
// every node against the lattice (coordinates on the node lines, surface
// nodes Dirichlet) and every edge against RegularMeshBuilder's numbering
// (the +d edge of node (i, j, k) at its closed-form number joins n and its
// +d neighbour) and writes the edge's row position; k_mfb_cells checks the
// cells' nodes and materials and writes the weights.  bad[0] counts
// mismatches of the structure, bad[1] edges whose Dirichlet flag (both
// nodes Dirichlet) differs from the lattice rule.
struct MfbLines {
    const double *x, *y, *z;   // node lines
    const double *mu, *sigma;  // per material
    int nmat;
};

__global__ void k_mfb_nodes(MF M, MfbLines L, int nb, const double *__restrict__ xyz,
                            const unsigned char *__restrict__ bnode, const int *__restrict__ edges,
                            unsigned *pos, int *bad)
{
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = M.nx, ny = M.ny, nz = M.nz;
    if (n >= (long long)nx * ny * nz) return;
    const int i = (int)(n % nx), j = (int)((n / nx) % ny), k = (int)(n / ((long long)nx * ny));
    int nbad = 0, nlat = 0;
    if (xyz[3 * n] != L.x[i] || xyz[3 * n + 1] != L.y[j] || xyz[3 * n + 2] != L.z[k]) nbad++;
    const bool bi = i == 0 || i == nx - 1, bj = j == 0 || j == ny - 1, bk = k == 0 || k == nz - 1;
    if ((bi || bj || bk) && !bnode[n]) nbad++;
    const int step[3] = {1, nx, nx * ny};
    const bool has[3] = {i < nx - 1, j < ny - 1, k < nz - 1};
    const bool want[3] = {bj || bk, bi || bk, bi || bj};
    for (int d = 0; d < 3; d++) {
        if (!has[d]) continue;
        const int e = mf_edge(M, d, i, j, k);
        if (e < 0 || e >= nb) {
            nbad++;
            continue;
        }
        const int n2 = (int)n + step[d];
        if (edges[2 * e] != (int)n || edges[2 * e + 1] != n2) nbad++;
        const bool be = bnode[n] && bnode[n2];
        if (be != want[d]) nlat++;
        // rows plane by plane, in a plane its x-, y-, then z-edges (i
        // fastest): a warp's rows share their direction except at the two
        // boundaries of a plane, and the three edges of a node, adjacent in
        // the vectors, are read within one plane's sweep
        const long long xr = (long long)(nx - 1) * ny, yr = (long long)nx * (ny - 1);
        long long row = (long long)k * (xr + yr + (long long)nx * ny);
        if (d == 0) row += (long long)j * (nx - 1) + i;
        else if (d == 1) row += xr + (long long)j * nx + i;
        else row += xr + yr + (long long)j * nx + i;
        pos[row] = (unsigned)i | ((unsigned)j << 10) | ((unsigned)k << 20) | ((unsigned)d << 30);
    }
    if (nbad) atomicAdd(&bad[0], nbad);
    if (nlat) atomicAdd(&bad[1], nlat);
}

// weights of cell c: wF / 3 = 2 h_d / (h_t1 h_t2) / mu / 3 and
// wM / 9 = sigma h_t1 h_t2 / h_d / 9 (times omega of a host SLAE), the
// expressions and their order as FP64 on the host
__global__ void k_mfb_cells(MF M, MfbLines L, const int *__restrict__ nver, int stride,
                            const int *__restrict__ nvkat, double om, int scale, float2 *w, int *bad)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nx = M.nx, ny = M.ny, nxy = nx * ny;
    const int cx = nx - 1, cy = ny - 1;
    if (c >= M.ncell) return;
    const int i = (int)(c % cx), j = (int)((c / cx) % cy), k = (int)(c / ((long long)cx * cy));
    int nbad = 0;
    const int n0 = (k * ny + j) * nx + i;
    const int want[8] = {n0, n0 + 1, n0 + nx, n0 + nx + 1,
                         n0 + nxy, n0 + nxy + 1, n0 + nxy + nx, n0 + nxy + nx + 1};
    for (int t = 0; t < 8; t++)
        if (nver[(size_t)c * stride + t] != want[t]) nbad++;
    const int mat = nvkat[c];
    if (mat < 0 || mat >= L.nmat || !(L.mu[mat] > 0.0)) {
        atomicAdd(&bad[0], nbad + 1);
        return;
    }
    if (nbad) atomicAdd(&bad[0], nbad);
    const double h[3] = {L.x[i + 1] - L.x[i], L.y[j + 1] - L.y[j], L.z[k + 1] - L.z[k]};
    for (int d = 0; d < 3; d++) {
        const int t1 = (d + 1) % 3, t2 = (d + 2) % 3;
        const double wf = 2.0 * h[d] / (h[t1] * h[t2]) / L.mu[mat] / 3.0;
        double wm = L.sigma[mat] * h[t1] * h[t2] / h[d] / 9.0;
        if (scale) wm *= om;
        const df f = from_double(wf), m = from_double(wm);
        w[(size_t)d * M.ncell + c] = make_float2(f.h, f.l);
        w[(size_t)(3 + d) * M.ncell + c] = make_float2(m.h, m.l);
    }
}

// The matrix-free variant's tables, when the assembly's mesh is a tensor
// mesh numbered as RegularMeshBuilder numbers it (nodes x fastest, cells
// likewise, edges per node +x, +y, +z, every node of the outer surface a
// Dirichlet node); anything else leaves the variant off.  The node lines
// come from the host coordinates, every table check and every table from
// the device mesh tables.  A set-up check compares one matrix-free product
// with the stored-matrix product and leaves the variant off unless they
// agree to 1e-9.
int matfree_build(Survey &V, const MatFreeMesh &a, const DevMesh &dm, int kuz, int kpar, int nsm)
{
    MatFree &F = V.mf;
    F.release();
    const ParamMatrix &P = *V.P;
    const double *xyz = a.xyz;
    if (!xyz || !dm.xyz || !dm.nver || !dm.nvkat || !dm.edges || !dm.bnode || kuz < 27 ||
        a.nver_stride < 8 || dm.nn != kuz)
        return MTGPU_OK;
    int nx = 1;
    while (nx < kuz && xyz[3 * nx + 1] == xyz[1] && xyz[3 * nx + 2] == xyz[2]) nx++;
    int nxy = nx;
    while (nxy < kuz && xyz[3 * nxy + 2] == xyz[2]) nxy++;
    if (nxy % nx || kuz % nxy) return MTGPU_OK;
    const int ny = nxy / nx, nz = kuz / nxy;
    if (nx < 3 || ny < 3 || nz < 3 || nx > 1024 || ny > 1024 || nz > 1024) return MTGPU_OK;
    std::vector<double> lines((size_t)nx + ny + nz);
    double *X = lines.data(), *Y = X + nx, *Z = Y + ny;
    for (int i = 0; i < nx; i++) X[i] = xyz[3 * i];
    for (int j = 0; j < ny; j++) Y[j] = xyz[3 * (j * nx) + 1];
    for (int k = 0; k < nz; k++) Z[k] = xyz[3 * (k * nxy) + 2];
    for (int i = 1; i < nx; i++) if (!(X[i] > X[i - 1])) return MTGPU_OK;
    for (int j = 1; j < ny; j++) if (!(Y[j] > Y[j - 1])) return MTGPU_OK;
    for (int k = 1; k < nz; k++) if (!(Z[k] > Z[k - 1])) return MTGPU_OK;
    const long long ncell = (long long)(nx - 1) * (ny - 1) * (nz - 1);
    if (ncell != kpar) return MTGPU_OK;
    const long long nex = (long long)(nx - 1) * ny * nz, ney = (long long)nx * (ny - 1) * nz,
                    nez = (long long)nx * ny * (nz - 1);
    if (nex + ney + nez != P.nb) return MTGPU_OK;
    // 32-bit indexing in the kernels: edges, faces and weights times systems
    const long long nfaces = (long long)nx * (ny - 1) * (nz - 1) +
                             (long long)(nx - 1) * ny * (nz - 1) +
                             (long long)(nx - 1) * (ny - 1) * nz;
    if ((long long)P.nb * V.SP >= (1LL << 31) || 6 * ncell >= (1LL << 31) ||
        nfaces * V.SP >= (1LL << 31))
        return MTGPU_OK;
    const int nmat = (int)std::min(a.mu.size(), a.sigma.size());
    if (nmat < 1) return MTGPU_OK;
    // a host SLAE's M carries omega_true: the ratio of its diagonal to the
    // mass coefficient of the edge itself (4 times the 4 cells' wM) on an
    // interior x-edge; the set-up check below confirms it on every row
    double om = 1.0;
    const int scale = a.idi && a.di;
    if (scale) {
        const int i = (nx - 1) / 2, j = ny / 2, k = nz / 2;
        const long long e = (long long)k * ((ny - 1) * (3LL * nx - 1) + (2LL * nx - 1)) +
                            (long long)j * (3LL * nx - 1) + 3LL * i;   // +x edge of an interior node
        double wsum = 0.0;
        for (int b1 = -1; b1 <= 0; b1++)
            for (int b2 = -1; b2 <= 0; b2++) {
                const size_t c = ((size_t)(k + b2) * (ny - 1) + (j + b1)) * (nx - 1) + i;
                const int mat = a.nvkat[c];
                if (mat < 0 || mat >= nmat) return MTGPU_OK;
                const double h[3] = {X[i + 1] - X[i], Y[j + b1 + 1] - Y[j + b1], Z[k + b2 + 1] - Z[k + b2]};
                wsum += a.sigma[mat] * h[1] * h[2] / h[0] / 9.0;
            }
        if (a.idi[e + 1] - a.idi[e] != 2 || !(wsum > 0.0)) return MTGPU_OK;
        om = a.di[a.idi[e] + 1] / (4.0 * wsum);
        if (!(om > 0.0)) return MTGPU_OK;
    }
    F.nx = nx;
    F.ny = ny;
    F.nz = nz;
    F.nfx = (long long)nx * (ny - 1) * (nz - 1);
    F.nfy = (long long)(nx - 1) * ny * (nz - 1);
    F.nfz = (long long)(nx - 1) * (ny - 1) * nz;
    // the edges on the outer surface: both transverse coordinates' lines of a
    // direction that touch it, numbered as mf_edge does
    std::vector<int> surface;
    for (int k = 0; k < nz; k++)
        for (int j = 0; j < ny; j++) {
            const bool sk = k == 0 || k == nz - 1, sj = j == 0 || j == ny - 1;
            const int ey = j < ny - 1, ez = k < nz - 1;
            const int line = k * ((ny - 1) * (3 * nx - 1) + 2 * nx - 1) + j * (ez ? 3 * nx - 1 : 2 * nx - 1);
            for (int i = 0; i < nx; i++) {
                const bool si = i == 0 || i == nx - 1;
                if (!si && !sj && !sk) {          // no surface edge along the rest of the line
                    i = nx - 2;
                    continue;
                }
                const int ex = i < nx - 1, e = line + i * (1 + ey + ez);
                if (ex && (sj || sk)) surface.push_back(e);
                if (ey && (si || sk)) surface.push_back(e + ex);
                if (ez && (si || sj)) surface.push_back(e + ex + ey);
            }
        }
    F.ndir = (int)surface.size();
    double *d_lines = nullptr;
    int *d_bad = nullptr;
    int rc;
    if ((rc = dev_alloc(&F.pos, (size_t)P.nb)) || (rc = dev_alloc(&F.dir, surface.size())) ||
        (rc = dev_alloc(&F.w, (size_t)6 * ncell)) ||
        (rc = dev_alloc(&F.f, (size_t)(F.nfx + F.nfy + F.nfz) * V.SP)) ||
        (rc = dev_alloc(&F.g, (size_t)(F.nfx + F.nfy + F.nfz) * V.SP)) ||
        (rc = dev_alloc(&d_lines, lines.size() + 2 * (size_t)nmat)) || (rc = dev_alloc(&d_bad, 2))) {
        dev_free(d_lines);
        F.release();
        return rc;
    }
    cudaError_t err = cudaMemcpyAsync(d_lines, lines.data(), sizeof(double) * lines.size(),
                                      cudaMemcpyHostToDevice, V.st);
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(F.dir, surface.data(), sizeof(int) * surface.size(), cudaMemcpyHostToDevice, V.st);
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(d_lines + lines.size(), a.mu.data(), sizeof(double) * nmat,
                              cudaMemcpyHostToDevice, V.st);
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(d_lines + lines.size() + nmat, a.sigma.data(), sizeof(double) * nmat,
                              cudaMemcpyHostToDevice, V.st);
    if (err == cudaSuccess) err = cudaMemsetAsync(d_bad, 0, sizeof(int) * 2, V.st);
    int bad[2] = {0, 0};
    if (err == cudaSuccess) {
        MF M{};
        M.nx = nx;
        M.ny = ny;
        M.nz = nz;
        M.ncell = ncell;
        M.nfx = F.nfx;
        M.nfy = F.nfy;
        M.nfz = F.nfz;
        mf_strides(M);
        const MfbLines L{d_lines, d_lines + nx, d_lines + nx + ny, d_lines + lines.size(),
                         d_lines + lines.size() + nmat, nmat};
        k_mfb_nodes<<<ceil_div(kuz, kB), kB, 0, V.st>>>(M, L, P.nb, dm.xyz, dm.bnode, dm.edges,
                                                       F.pos, d_bad);
        k_mfb_cells<<<ceil_div(ncell, kB), kB, 0, V.st>>>(M, L, dm.nver, dm.nver_stride, dm.nvkat, om,
                                                         scale, F.w, d_bad);
        note_launches(2);
        err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaMemcpyAsync(bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost, V.st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(V.st);
    dev_free(d_lines);
    dev_free(d_bad);
    if (err != cudaSuccess) {
        F.release();
        set_last_error(err, "matrix-free tables", __FILE__, __LINE__);
        return MTGPU_ERR_CUDA;
    }
    if (bad[0] != 0 || bad[1] != 0) {
        // not a tensor mesh in the builder's numbering, or Dirichlet edges
        // other than the lattice's: variant off
        F.release();
        return MTGPU_OK;
    }
    // the kernels derive the Dirichlet edges from the lattice: an edge is
    // Dirichlet iff one of its two transverse node lines is on the surface
    F.lattice = true;
    F.on = true;
    // set-up check against the stored-matrix SpMV on a test vector
    const int ch = V.ch;
    std::vector<SysState> init(32);
    for (int k = 0; k < 32; k++) {
        SysState q{};
        q.status = k < V.S ? kRun : MTGPU_OK;
        q.maxiter = 1;
        host_scalars(q);
        init[k] = q;
    }
    const long long n = (long long)V.nb * V.SP;
    unsigned long long *d_mx = nullptr;
    if ((rc = dev_alloc(&d_mx, 4))) return rc;
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    k_pattern<<<4 * nsm, kB, 0, V.st>>>(n, V.s);
    V.ch = 4;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
    MTGPU_TRY(cudaMemcpyAsync(V.w, V.z, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    V.ch = kMatFree;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
    MTGPU_TRY(cudaMemsetAsync(d_mx, 0, sizeof(MaxDiff), V.st));
    k_maxdiff<<<4 * nsm, kB, 0, V.st>>>(n, V.S, V.SP, V.z, V.w, d_mx);
    note_launches(5);
    MaxDiff mx;
    err = cudaGetLastError();
    if (err == cudaSuccess)
        err = cudaMemcpyAsync(mx.w, d_mx, sizeof(mx), cudaMemcpyDeviceToHost, V.st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(V.st);
    dev_free(d_mx);
    V.ch = ch;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    if (err != cudaSuccess) {
        set_last_error(err, "matrix-free SpMV set-up check", __FILE__, __LINE__);
        return MTGPU_ERR_CUDA;
    }
    const double check = mx.relative();
    if (!(check < 1e-9)) {
        F.release();   // not this matrix's operator: variant off, memory back
        F.check = check;
        return MTGPU_OK;
    }
    F.check = check;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    {
        // the D^T (F f) form rounds differently from variant 32 (products of
        // the face values summed per face first): it must agree to 1e-12
        F.gface = true;
        k_pattern<<<4 * nsm, kB, 0, V.st>>>(n, V.s);
        MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
        V.ch = kMatFree;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
        MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
        MTGPU_TRY(cudaMemcpyAsync(V.w, V.z, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
        MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
        V.ch = kMatFree + 3;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
        MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
        V.ch = ch;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
        if ((rc = dev_alloc(&d_mx, 4))) return rc;
        MTGPU_TRY(cudaMemsetAsync(d_mx, 0, sizeof(MaxDiff), V.st));
        k_maxdiff<<<4 * nsm, kB, 0, V.st>>>(n, V.S, V.SP, V.z, V.w, d_mx);
        note_launches(4 + spmv_extra_launches(kMatFree) + spmv_extra_launches(kMatFree + 3));
        err = cudaGetLastError();
        if (err == cudaSuccess)
            err = cudaMemcpyAsync(mx.w, d_mx, sizeof(mx), cudaMemcpyDeviceToHost, V.st);
        if (err == cudaSuccess) err = cudaStreamSynchronize(V.st);
        dev_free(d_mx);
        if (err != cudaSuccess) {
            set_last_error(err, "face-mass matrix-free SpMV set-up check", __FILE__, __LINE__);
            return MTGPU_ERR_CUDA;
        }
        F.gface = mx.relative() < 1e-12;
    }
    return MTGPU_OK;
}

// Variant 34 sums in the same order as variant 32: it is enabled only if
// its product on a pseudo-random vector equals variant 32's bit for bit.
// Run on the first request of the variant.
int matfree_tile_check(Survey &V, int nsm)
{
    MatFree &F = V.mf;
    F.tile_checked = true;
    F.tiled = F.on && F.lattice && V.g_mft > 0 && V.g_mft <= V.pblocks;
    if (!F.tiled) return MTGPU_OK;
    std::vector<SysState> init(32);
    for (int k = 0; k < 32; k++) {
        SysState q{};
        q.status = k < V.S ? kRun : MTGPU_OK;
        q.maxiter = 1;
        host_scalars(q);
        init[k] = q;
    }
    const int ch = V.ch;
    const long long n = (long long)V.nb * V.SP;
    k_pattern<<<4 * nsm, kB, 0, V.st>>>(n, V.s);
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    V.ch = kMatFree;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
    MTGPU_TRY(cudaMemcpyAsync(V.w, V.z, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    V.ch = kMatFree + 2;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
    V.ch = ch;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    unsigned long long *d_mx = nullptr;
    int rc = dev_alloc(&d_mx, 4);
    if (rc) return rc;
    MTGPU_TRY(cudaMemsetAsync(d_mx, 0, sizeof(MaxDiff), V.st));
    k_maxdiff<<<4 * nsm, kB, 0, V.st>>>(n, V.S, V.SP, V.z, V.w, d_mx);
    note_launches(4 + spmv_extra_launches(kMatFree));
    MaxDiff mx;
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaMemcpyAsync(mx.w, d_mx, sizeof(mx), cudaMemcpyDeviceToHost, V.st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(V.st);
    dev_free(d_mx);
    if (err != cudaSuccess) {
        F.tiled = false;
        set_last_error(err, "tiled matrix-free SpMV set-up check", __FILE__, __LINE__);
        return MTGPU_ERR_CUDA;
    }
    F.tiled = mx.equal();
    return MTGPU_OK;
}

}  // namespace

// What variant v needs beyond the set-up, built on its first request: the
// stored matrix's tiles (variants 0, 1), the tiled variant's check (34)
int survey_prepare_variant(Survey &V, int v)
{
    int dev = 0, nsm = 0;
    MTGPU_TRY(cudaGetDevice(&dev));
    MTGPU_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    int rc;
    if ((v == 0 || v == 1) && !V.tiles_built) {
        V.tiles_built = true;
        if ((rc = build_tiles(V, nsm))) return rc;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    }
    if (v == kMatFree + 2 && !V.mf.tile_checked && (rc = matfree_tile_check(V, nsm))) return rc;
    return MTGPU_OK;
}

namespace {

// The fused preconditioner (prec_tile.cuh), on request (MTGPU_PREC_TILE=1
// in the environment: on GB300 it measured slower than the node and edge
// kernels on every benchmark workload, 0.72 against 0.59 ms per iteration
// on c2 at 2 systems, 3.8 against 2.1 ms on c3 at 32) and where the mesh
// allows it: a tensor mesh with the lattice's Dirichlet edges, every
// interior node a row of G in node order, the compact G^T.  A set-up check
// runs one step of both forms on the same pseudo-random vectors and keeps
// the fused one only if a and w agree bit for bit.
int prec_tile_setup(Survey &V, int nsm)
{
    V.prec_tile = false;
    const char *force = getenv("MTGPU_PREC_TILE");
    if (!force || *force != '1') return MTGPU_OK;
    if (!V.mf.on || !V.mf.lattice || !V.G.d_tn) return MTGPU_OK;
    const long long mi = (long long)(V.mf.nx - 2) * (V.mf.ny - 2) * (V.mf.nz - 2);
    if (V.G.m != mi) return MTGPU_OK;
    MTGPU_SP_DISPATCH(V.SP, prec_grid(V, nsm));
    if (V.g_pt < 1 || V.g_pt > V.pblocks) return MTGPU_OK;
    const long long n = (long long)V.nb * V.SP;
    int rc;
    if (!V.a2 && (rc = dev_alloc(&V.a2, (size_t)n))) return rc;
    std::vector<SysState> init(32);
    for (int k = 0; k < 32; k++) {
        SysState q{};
        q.status = k < V.S ? kRun : MTGPU_OK;
        q.maxiter = INT_MAX;
        q.zs = make_double2(1.0, 0.0);
        q.beta = make_double2(0.375, -0.25);
        host_scalars(q);
        init[k] = q;
    }
    float4 *ref = nullptr;
    unsigned long long *d_mx = nullptr;
    if ((rc = dev_alloc(&ref, (size_t)2 * n)) || (rc = dev_alloc(&d_mx, 4))) {
        dev_free(ref);
        return rc;
    }
    // the same z and a for both, from the pattern
    for (float4 *v : {V.z, V.a}) k_pattern<<<4 * nsm, kB, 0, V.st>>>(n, v);
    note_launches(2);
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    // unfused: k_edge updates a in place; its input is kept for the fused form
    MTGPU_TRY(cudaMemcpyAsync(V.p, V.a, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
    MTGPU_SP_DISPATCH(V.SP, precond_step(V, false, V.a, V.a));
    MTGPU_TRY(cudaMemcpyAsync(ref, V.w, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
    MTGPU_TRY(cudaMemcpyAsync(ref + n, V.a, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
    // lanes beyond the batch's systems are written by neither
    MTGPU_TRY(cudaMemcpyAsync(V.a2, V.a, sizeof(float4) * n, cudaMemcpyDeviceToDevice, V.st));
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    MTGPU_SP_DISPATCH(V.SP, precond_step(V, true, V.p, V.a2));
    MTGPU_TRY(cudaMemsetAsync(d_mx, 0, sizeof(MaxDiff), V.st));
    k_maxdiff<<<4 * nsm, kB, 0, V.st>>>(n, V.S, V.SP, V.w, ref, d_mx);
    k_maxdiff<<<4 * nsm, kB, 0, V.st>>>(n, V.S, V.SP, V.a2, ref + n, d_mx);
    note_launches(5);
    MaxDiff mx;
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaMemcpyAsync(mx.w, d_mx, sizeof(mx), cudaMemcpyDeviceToHost, V.st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(V.st);
    dev_free(ref);
    dev_free(d_mx);
    if (err != cudaSuccess) {
        set_last_error(err, "fused preconditioner set-up check", __FILE__, __LINE__);
        return MTGPU_ERR_CUDA;
    }
    if (!mx.equal()) {   // not bit-equal: keep the two-kernel form
        dev_free(V.a2);
        return MTGPU_OK;
    }
    // both forms' whole iterations timed, for the record
    float t_un = 0.f, t_fu = 0.f;
    V.prec_tile = false;
    if ((rc = survey_iter_timed(V, 2, &t_un)) || (rc = survey_iter_timed(V, 4, &t_un))) return rc;
    V.prec_tile = true;
    if ((rc = survey_iter_timed(V, 2, &t_fu)) || (rc = survey_iter_timed(V, 4, &t_fu))) return rc;
    V.prec_ms[0] = t_un / 4.f;
    V.prec_ms[1] = t_fu / 4.f;
    return MTGPU_OK;
}

}  // namespace

namespace {
// iterations per group: 16, fewer where their s vectors would take more than
// a quarter of the free memory (1: no more memory than without groups)
int group_length(const Survey &V, int *group)
{
    size_t mem_free = 0, mem_total = 0;
    MTGPU_TRY(cudaMemGetInfo(&mem_free, &mem_total));
    const size_t vec = sizeof(float4) * (size_t)V.nb * V.SP;
    int g = kGroupIters;
    while (g > 1 && (size_t)(g + 1) * vec > mem_free / 4) g /= 2;
    *group = g;
    return MTGPU_OK;
}
}  // namespace

int survey_lengthen_group(Survey &V)
{
    int g = 1, rc;
    if ((rc = group_length(V, &g)) || g <= V.group) return rc;
    float4 *s = nullptr;
    if (dev_alloc(&s, (size_t)(g + 1) * V.nb * V.SP)) {
        cudaGetLastError();       // (other users of the GPU: the short group stays)
        return MTGPU_OK;
    }
    dev_free(V.s);
    V.s = s;
    V.group = g;
    return MTGPU_OK;
}

int survey_setup(const ParamMatrix &P, const mtgpu_mesh_desc &mesh, int S, const double *omega,
                 Survey &V, cudaStream_t st, const mtgpu_assembly_s *a, const MatFreeMesh *mfm,
                 int pin_variant)
{
    PhaseTrace trace(st, "survey set-up");
    V.release();
    V.autotuned = false;
    MTGPU_CHECK_ARG(S >= 1 && S <= 32, "a survey batch holds 1 to 32 systems");
    V.P = &P;
    V.st = st;
    V.nb = P.nb;
    V.S = S;
    V.SP = 1;
    while (V.SP < S) V.SP <<= 1;
    int dev = 0, nsm = 0;
    MTGPU_TRY(cudaGetDevice(&dev));
    MTGPU_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int rpb = kB / V.SP;
    V.grid_rows = std::max(1, ceil_div(V.nb, rpb));
    int rc;
    // the mesh tables on the device: the assembly's own, or uploads of a
    // host SLAE's mesh
    DevMeshUpload dmu;
    if (a && P.d_nver && P.d_nvkat && P.d_edges && P.d_bnode && P.d_xyz)
        rc = dmu.over_device(P.kpar, P.nb, P.kuzlov, P.nver_stride, P.d_xyz, P.d_nver, P.d_nvkat,
                             P.d_edges, P.d_bnode, a->sigflag.data(), (int)a->sigflag.size(), st);
    else
        rc = dmu.upload(mesh, mfm ? mfm->xyz : nullptr, st);
    if (rc) return rc;
    trace.mark("mesh tables");
    bool conforming = false;
    if ((rc = folded_build_g_device(dmu.view, V.G, st, &conforming))) return rc;
    if (!conforming && (rc = folded_build_g(mesh, V.G, st))) return rc;
    trace.mark("preconditioner G");
    const int m = V.G.m, mm = std::max(m, 1);
    V.grid_nodes = std::max(1, ceil_div(mm, rpb));
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    const int gmax = std::max({V.g_init, V.g_node, V.g_edge, V.g_update, V.g_true, V.g_spmv});
    const size_t nv = (size_t)V.nb * V.SP;
    if ((rc = dev_alloc(&V.kc, P.len_c)) || (rc = dev_alloc(&V.mc, P.len_c)) ||
        (rc = dev_alloc(&V.kr, P.len_r)) || (rc = dev_alloc(&V.da, nv)) ||
        (rc = dev_alloc(&V.ds, (size_t)mm * V.SP)) || (rc = dev_alloc(&V.gkg, mm)) ||
        (rc = dev_alloc(&V.gmg, mm)) || (rc = dev_alloc(&V.omega, 32)) ||
        (rc = dev_alloc(&V.omega64, 32)) || (rc = dev_alloc(&V.sys, kSysSlots)) ||
        (rc = dev_alloc(&V.r, nv)) || (rc = dev_alloc(&V.p, nv)) || (rc = dev_alloc(&V.a, nv)) ||
        (rc = dev_alloc(&V.z, nv)) || (rc = dev_alloc(&V.w, nv)) || (rc = dev_alloc(&V.sm, nv)) ||
        (rc = dev_alloc(&V.h, (size_t)mm * V.SP)) || (rc = dev_alloc(&V.b64, nv)) ||
        (rc = dev_alloc(&V.xacc, nv)) || (rc = dev_alloc(&V.hist, 2 * 32 * kGroupIters)) ||
        (rc = dev_alloc(&V.partials, partial_slots(std::max(gmax, nsm * 32), V.SP))))
        return rc;
    V.pblocks = std::max(gmax, nsm * 32);
    MTGPU_CHECK_ARG(ceil_div(V.pblocks, kGroupBlocks) <= kMaxGroups, "more blocks than the grid sums have tickets");
    // the s vectors of a group of iterations.  Of a survey of several batches,
    // 1 for now: the batches set up after this one need their memory first
    // (survey_lengthen_group)
    V.group = 1;
    if (V.alone && (rc = group_length(V, &V.group))) return rc;
    if ((rc = dev_alloc(&V.s, (size_t)(V.group + 1) * nv))) return rc;
    MTGPU_TRY(cudaMemsetAsync(V.partials, 0, sizeof(float4) * kTicketSlots, st));
    MTGPU_TRY(cudaMemsetAsync(V.sys, 0, sizeof(SysState) * kSysSlots, st));
    MTGPU_TRY(cudaMallocHost((void **)&V.hsys, sizeof(SysState) * kSysSlots));
    trace.mark("allocations");
    std::vector<float2> omdf(32, make_float2(0.f, 0.f));
    std::vector<double> om64(32, 0.0);
    for (int k = 0; k < S; k++) {
        const dfl::df v = dfl::from_double(omega[k]);
        omdf[k] = make_float2(v.h, v.l);
        om64[k] = omega[k];
    }
    MTGPU_TRY(cudaMemcpyAsync(V.omega, omdf.data(), sizeof(float2) * 32, cudaMemcpyHostToDevice, st));
    MTGPU_TRY(cudaMemcpyAsync(V.omega64, om64.data(), sizeof(double) * 32, cudaMemcpyHostToDevice, st));
    k_to_df<<<(unsigned)((P.len_c + kB - 1) / kB), kB, 0, st>>>(P.len_c, P.d_kc, V.kc);
    k_to_df<<<(unsigned)((P.len_c + kB - 1) / kB), kB, 0, st>>>(P.len_c, P.d_mc, V.mc);
    k_to_df<<<(unsigned)((P.len_r + kB - 1) / kB), kB, 0, st>>>(P.len_r, P.d_kr, V.kr);
    k_diag_a<<<(unsigned)((nv + kB - 1) / kB), kB, 0, st>>>(V.nb, V.SP, P.d_nc, P.d_pc, P.d_col_c,
                                                          P.d_kc, P.d_mc, V.omega64, V.da);
    trace.mark("double-float K, M, D_A");
    {
        int nnz = 0;
        MTGPU_TRY(cudaMemcpyAsync(&nnz, V.G.d_gp + m, sizeof(int), cudaMemcpyDeviceToHost, st));
        MTGPU_TRY(cudaStreamSynchronize(st));
        if ((rc = dev_alloc(&V.gv32, std::max(nnz, 1))) || (rc = dev_alloc(&V.tv32, std::max(nnz, 1))))
            return rc;
        if (nnz > 0) {
            k_f64_to_f32<<<(nnz + kB - 1) / kB, kB, 0, st>>>(nnz, V.G.d_gv, V.gv32);
            k_f64_to_f32<<<(nnz + kB - 1) / kB, kB, 0, st>>>(nnz, V.G.d_tv, V.tv32);
        }
    }
    // MTGPU_GDIAG_ENTRIES=1 (environment): the per-entry passes on every mesh
    const char *ge = getenv("MTGPU_GDIAG_ENTRIES");
    const bool per_edge = V.G.d_tn && !(ge && *ge == '1');
    if (m > 0 && per_edge) {
        double2 *tk = nullptr, *tm = nullptr;
        if ((rc = dev_alloc(&tk, V.nb)) || (rc = dev_alloc(&tm, V.nb))) {
            dev_free(tk);
            return rc;
        }
        k_gdiag_edge<<<ceil_div(V.nb, kB), kB, 0, st>>>(V.nb, V.G.d_tn, P.d_nc, P.d_nr, P.d_pc,
                                                        P.d_pr, P.d_col_c, P.d_kc, P.d_mc,
                                                        P.d_col_r, P.d_kr, tk, tm);
        k_gdiag_nodes<<<ceil_div(m, kB), kB, 0, st>>>(m, V.G.d_gp, V.G.d_gj, V.G.d_gv, V.G.d_tn,
                                                      tk, tm, V.gkg, V.gmg);
        note_launches(2);
        cudaStreamSynchronize(st);
        dev_free(tk);
        dev_free(tm);
        const size_t nm = (size_t)m * V.SP;
        k_diag_s<<<(unsigned)((nm + kB - 1) / kB), kB, 0, st>>>(m, V.SP, V.gkg, V.gmg, V.omega64, V.ds);
    } else if (m > 0) {
        int nnz = 0;
        MTGPU_TRY(cudaMemcpyAsync(&nnz, V.G.d_gp + m, sizeof(int), cudaMemcpyDeviceToHost, st));
        MTGPU_TRY(cudaStreamSynchronize(st));
        double *tkv = nullptr, *tmv = nullptr;
        int *rowof = nullptr;
        if ((rc = dev_alloc(&tkv, std::max(nnz, 1))) || (rc = dev_alloc(&tmv, std::max(nnz, 1))) ||
            (rc = dev_alloc(&rowof, std::max(nnz, 1)))) {
            dev_free(tkv);
            dev_free(tmv);
            return rc;
        }
        k_gdiag_rows<<<ceil_div(m, kB), kB, 0, st>>>(m, V.G.d_gp, rowof);
        if (nnz > 0)
            k_gdiag_entry<<<ceil_div(nnz, 128), 128, 0, st>>>(m, V.G.d_gp, V.G.d_gj, V.G.d_gv, rowof,
                                                              P.d_nc, P.d_nr, P.d_pc, P.d_pr,
                                                              P.d_col_c, P.d_kc, P.d_mc, P.d_col_r,
                                                              P.d_kr, tkv, tmv);
        k_gdiag<<<ceil_div(m, kB), kB, 0, st>>>(m, V.G.d_gp, V.G.d_gv, tkv, tmv, V.gkg, V.gmg);
        note_launches(2);
        cudaStreamSynchronize(st);
        dev_free(tkv);
        dev_free(tmv);
        dev_free(rowof);
        const size_t nm = (size_t)m * V.SP;
        k_diag_s<<<(unsigned)((nm + kB - 1) / kB), kB, 0, st>>>(m, V.SP, V.gkg, V.gmg, V.omega64, V.ds);
    }
    MTGPU_TRY(cudaGetLastError());
    MTGPU_TRY(cudaStreamSynchronize(st));
    note_launches(8);
    trace.mark("vectors, diagonals");
    if (a) {
        MatFreeMesh mm;
        mm.xyz = a->xyz.data();
        mm.nver_stride = a->nver_stride;
        mm.nvkat = a->nvkat.data();
        mm.mu.resize(P.n_materials);
        mm.sigma.resize(P.n_materials);
        MTGPU_TRY(cudaMemcpyAsync(mm.mu.data(), P.d_mu, sizeof(double) * P.n_materials,
                                  cudaMemcpyDeviceToHost, st));
        MTGPU_TRY(cudaMemcpyAsync(mm.sigma.data(), P.d_sig, sizeof(double) * P.n_materials,
                                  cudaMemcpyDeviceToHost, st));
        MTGPU_TRY(cudaStreamSynchronize(st));
        if ((long long)a->xyz.size() == 3LL * P.kuzlov &&
            (rc = matfree_build(V, mm, dmu.view, P.kuzlov, P.kpar, nsm)))
            return rc;
    } else if (mfm && (rc = matfree_build(V, *mfm, dmu.view, mesh.n_nodes_c, mesh.kpar, nsm))) {
        return rc;
    }
    // G in the lattice form (k_node_lat): every interior node a row, in
    // node order, its six edges in order
    V.g_lat = false;
    if (V.mf.on && V.G.m > 0 &&
        (long long)V.G.m == (long long)(V.mf.nx - 2) * (V.mf.ny - 2) * (V.mf.nz - 2)) {
        int *d_bad = nullptr, bad = 1;
        if ((rc = dev_alloc(&d_bad, 1))) return rc;
        cudaError_t e = cudaMemsetAsync(d_bad, 0, sizeof(int), st);
        if (e == cudaSuccess) {
            MF M{};
            MTGPU_SP_DISPATCH(V.SP, mfd_into(V, M));
            k_g_lattice_check<<<ceil_div(V.G.m, kB), kB, 0, st>>>(M, V.G.m, V.G.d_gp, V.G.d_gj,
                                                                 V.gv32, d_bad);
            note_launches(1);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        dev_free(d_bad);
        if (e != cudaSuccess) {
            set_last_error(e, "lattice G check", __FILE__, __LINE__);
            return MTGPU_ERR_CUDA;
        }
        V.g_lat = bad == 0;
    }
    if (V.g_lat) {
        // both node kernels on the same pseudo-random z, a and beta: the
        // lattice form is kept only if its h equals the CSR form's
        std::vector<SysState> init(32);
        for (int k = 0; k < 32; k++) {
            SysState q{};
            q.status = k < V.S ? kRun : MTGPU_OK;
            q.beta = make_double2(0.375, -0.25);
            host_scalars(q);
        init[k] = q;
        }
        const long long n = (long long)V.nb * V.SP, nh = (long long)V.G.m * V.SP;
        unsigned long long *d_mx = nullptr;
        if ((rc = dev_alloc(&d_mx, 4))) return rc;
        k_pattern<<<4 * nsm, kB, 0, st>>>(n, V.z);
        k_pattern<<<4 * nsm, kB, 0, st>>>(n, V.p);
        cudaError_t e = cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            MTGPU_SP_DISPATCH(V.SP, node(V, V.z, V.p, 1));   // lattice form -> h
            e = cudaMemcpyAsync(V.w, V.h, sizeof(float4) * nh, cudaMemcpyDeviceToDevice, st);
        }
        if (e == cudaSuccess) {
            V.g_lat = false;
            MTGPU_SP_DISPATCH(V.SP, node(V, V.z, V.p, 1));   // CSR form -> h
            e = cudaMemsetAsync(d_mx, 0, sizeof(MaxDiff), st);
        }
        if (e == cudaSuccess) {
            k_maxdiff<<<4 * nsm, kB, 0, st>>>(nh, V.S, V.SP, V.h, V.w, d_mx);
            note_launches(5);
            e = cudaGetLastError();
        }
        MaxDiff mx;
        if (e == cudaSuccess) e = cudaMemcpyAsync(mx.w, d_mx, sizeof(mx), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        dev_free(d_mx);
        if (e != cudaSuccess) {
            set_last_error(e, "lattice G check", __FILE__, __LINE__);
            return MTGPU_ERR_CUDA;
        }
        V.g_lat = mx.equal();
    }
    trace.mark(!V.mf.on ? "no matrix-free tables" : (V.g_lat ? "matrix-free, lattice G" : "matrix-free tables"));
    // the stored matrix's tiles (variants 0, 1) where there is no
    // matrix-free operator; with one they are built only on request
    if (!V.mf.on && (rc = survey_prepare_variant(V, 0))) return rc;
    trace.mark("SpMV tiles");
    // the SpMV variant: by rule (below), a kept timing, or timing each candidate.
    // MTGPU_SPMV_VARIANT (environment) pins an available variant instead:
    // runs under a profiler, which serialises and cold-starts every launch,
    // would otherwise tune to other variants than plain runs do
    const char *pin = getenv("MTGPU_SPMV_VARIANT");
    const int pin_env = pin && *pin ? atoi(pin) : -1;
    if (pin_env >= 0 && (rc = survey_prepare_variant(V, pin_env))) return rc;
    if (pin_variant >= 0 && (rc = survey_prepare_variant(V, pin_variant))) return rc;
    // Variant 35 without timing for two systems and more, and for one where its
    // iterations run in one kernel.  Whole iterations, 32 / 33 / 35: 229,000 edges
    // x systems at 2 lanes 43.2 / 42.5 / 43.2 us, 296,000 46.9 / 48.0 / 45.2, 1.6M
    // 150 / 148 / 131; at 4 lanes 283,000 46.9 / 47.9 / 44.9, at 8 360,000 55.1 / 56.1 /
    // 50.3, at 16 423,000 57.8 / 57.5 / 53.7, at 32 847,000 92.6 / 93.7 / 80.3, and
    // further apart beyond.  For one system the sides change (346,000 edges 49.6
    // / 52.1, 811,000 85.8 / 82.8): timed.  The timing took 1.6 of a forward
    // model's 63 ms (126,000 edges x 8).
    auto g_form = [&]() {
        if (!V.mf.on || !V.mf.gface) return false;
        V.ch = kMatFree + 3;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
        return V.SP >= 2 || V.g_small > 0;
    };
    if (pin_env >= 0 && spmv_variant_available(V, pin_env)) {
        V.ch = pin_env;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    } else if (g_form()) {
        // (its grids are set)
    } else if (pin_variant >= 0 && spmv_variant_available(V, pin_variant)) {
        V.ch = pin_variant;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    } else {
        // with the matrix-free operator the stored-matrix variants and the
        // tiled matrix-free one measured slower on every tensor mesh (whole
        // iterations on c2 at 2 systems: 0.67 ms and more against 0.57-0.60),
        // so only the matrix-free forms are timed
        const int cand[kSpmvVariants] = {0, 1, 2, 4, 8, kRowVariant + 2, kRowVariant + 4, kMatFree,
                                         kMatFree + 1, kMatFree + 2, kMatFree + 3};
        auto tried = [&](int v) {
            if (!V.mf.on) return true;
            return v == kMatFree || v == kMatFree + 1 || v == kMatFree + 3;
        };
        float best = 1e30f;
        int best_ch = 4;
        for (int c = 0; c < kSpmvVariants; c++) {
            if (!tried(cand[c]) || !spmv_variant_available(V, cand[c])) continue;
            V.ch = cand[c];
            MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
            float ms = 0.f;
            if ((rc = survey_iter_timed(V, 1, &ms))) return rc;   // warm-up
            if ((rc = survey_iter_timed(V, 3, &ms))) return rc;
            V.tune_ms[c] = ms / 3.f;
            if (ms < best) {
                best = ms;
                best_ch = cand[c];
            }
        }
        V.ch = best_ch;
        V.autotuned = true;
        MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    }
    trace.mark("SpMV autotuning");
    rc = prec_tile_setup(V, nsm);
    trace.mark("fused preconditioner");
    return rc;
}

int survey_set_variant(Survey &V, int variant)
{
    int dev = 0, nsm = 0;
    MTGPU_TRY(cudaGetDevice(&dev));
    MTGPU_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    V.ch = variant;
    MTGPU_SP_DISPATCH(V.SP, grids(V, nsm));
    if (V.graph) cudaGraphExecDestroy(V.graph);   // captured with the old variant
    V.graph = nullptr;
    V.graph_iters = 0;
    return MTGPU_OK;
}

// Times the SpMV as the iteration launches it: mode 1 (z = A s, (z, s), the
// stop test and beta), every system running.  The state set here (no stop
// threshold, no iteration limit) keeps all systems running across the
// launches; a solve re-initialises the state and the vectors it touches.
int survey_spmv_timed(Survey &V, int reps, float *ms)
{
    std::vector<SysState> init(32);
    for (int k = 0; k < 32; k++) {
        SysState s{};
        s.status = k < V.S ? kRun : MTGPU_OK;
        s.maxiter = INT_MAX;
        s.eps_k = -1.0;
        s.r_old = 1.0;
        s.mrs_mode = 2;
        s.mrs_w = 0.5;
        host_scalars(s);
        init[k] = s;
    }
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    const size_t nv = sizeof(float4) * (size_t)V.nb * V.SP;
    MTGPU_TRY(cudaMemsetAsync(V.s, 0, nv, V.st));
    cudaEvent_t e0, e1;
    MTGPU_TRY(cudaEventCreate(&e0));
    MTGPU_TRY(cudaEventCreate(&e1));
    MTGPU_TRY(cudaEventRecord(e0, V.st));
    for (int q = 0; q < reps; q++) MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 1));
    note_launches((unsigned long long)reps);
    MTGPU_TRY(cudaEventRecord(e1, V.st));
    MTGPU_TRY(cudaEventSynchronize(e1));
    MTGPU_TRY(cudaEventElapsedTime(ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    MTGPU_TRY(cudaGetLastError());
    return MTGPU_OK;
}

// Times `reps` whole iterations (node, edge and update kernels, SpMV) on
// pattern-filled vectors with every system running: the autotuning ranks
// the SpMV variants by these, since the kernels before the SpMV leave the
// cache as it finds it inside a solve.  The values go to NaN within a few
// iterations, which changes neither the work nor its speed; no state
// reaches a stop (no threshold, no iteration limit, and the breakdown test
// of (a, w) does not fire on NaN).  A solve re-initialises everything.
int survey_iter_timed(Survey &V, int reps, float *ms)
{
    std::vector<SysState> init(32);
    for (int k = 0; k < 32; k++) {
        SysState s{};
        s.status = k < V.S ? kRun : MTGPU_OK;
        s.maxiter = INT_MAX;
        s.eps_k = -1.0;
        s.r_old = 1.0;
        s.mrs_mode = 2;
        s.mrs_w = 0.5;
        s.zs = make_double2(1.0, 0.0);
        s.alpha = make_double2(1e-3, 0.0);
        s.beta = make_double2(0.5, 0.0);
        host_scalars(s);
        init[k] = s;
    }
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    const long long nv = (long long)V.nb * V.SP;
    for (float4 *v : {V.r, V.s, V.p, V.a, V.z, V.w, V.sm})
        k_pattern<<<1024, kB, 0, V.st>>>(nv, v);
    if (V.G.m > 0) k_pattern<<<1024, kB, 0, V.st>>>((long long)V.G.m * V.SP, V.h);
    note_launches(V.G.m > 0 ? 8 : 7);
    cudaEvent_t e0, e1;
    MTGPU_TRY(cudaEventCreate(&e0));
    MTGPU_TRY(cudaEventCreate(&e1));
    MTGPU_TRY(cudaEventRecord(e0, V.st));
    for (int q = 0; q < reps; q++) MTGPU_SP_DISPATCH(V.SP, iteration(V, q, small_used(V) ? reps : INT_MAX));
    note_launches((unsigned long long)reps * iteration_launches(V) + (small_used(V) ? 2u * ceil_div(reps, V.group) : 0u));
    MTGPU_TRY(cudaEventRecord(e1, V.st));
    MTGPU_TRY(cudaEventSynchronize(e1));
    MTGPU_TRY(cudaEventElapsedTime(ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    MTGPU_TRY(cudaGetLastError());
    return MTGPU_OK;
}

// y_k = A_k x_k for every system with the current SpMV variant: FP64
// system-major x, y [S][nb] complex in and out, through the double-float
// vectors of the iteration.  It overwrites the survey's work vectors; a
// solve re-initialises them.
int survey_spmv(Survey &V, const double2 *x_sys_major, double2 *y_sys_major)
{
    std::vector<SysState> init(32);
    for (int k = 0; k < 32; k++) {
        SysState s{};
        s.status = k < V.S ? kRun : MTGPU_OK;
        s.maxiter = 1;
        host_scalars(s);
        init[k] = s;
    }
    MTGPU_TRY(cudaMemcpyAsync(V.sys, init.data(), sizeof(SysState) * 32, cudaMemcpyHostToDevice, V.st));
    to_rows(V, x_sys_major, V.s);
    MTGPU_SP_DISPATCH(V.SP, spmv_only(V, 0));
    from_rows(V, V.z, y_sys_major);
    MTGPU_TRY(cudaGetLastError());
    MTGPU_TRY(cudaStreamSynchronize(V.st));
    return MTGPU_OK;
}

namespace {

int upload_sys(Survey &V)
{
    MTGPU_TRY(cudaMemcpyAsync(V.sys, V.hsys, sizeof(SysState) * kSysSlots, cudaMemcpyHostToDevice, V.st));
    return sync_sys(V);
}

int upload_flags(int *d, const std::vector<int> &h, cudaStream_t st)
{
    MTGPU_TRY(cudaMemcpyAsync(d, h.data(), sizeof(int) * 32, cudaMemcpyHostToDevice, st));
    return MTGPU_OK;
}

}  // namespace

// The solution is accumulated in FP64: a group of iterations adds its
// double-float increment at its end (k_group), so the rounding of the x
// updates is relative to the increment, not to x: that keeps the true
// residual at the FP64 solver's level down to 1e-3 Hz.  The iteration solves
// A d = b - A x0 with the reference's stop rule relative to ||b||.  When the
// systems have stopped, their true residuals are evaluated in FP64 from the
// FP64 matrix; with verify, a system above eps keeps iterating with a tighter
// stop threshold while that still lowers its true residual.  A system whose
// smoothed residual stops decreasing (the double-float operator's own
// accuracy: very low frequencies on fine meshes, where omega sigma_air is
// ~1e-13 of the curl-curl scale) or that does not reach eps ends with
// MTGPU_MAXITER; the caller re-solves those in FP64.
//
// A solve is a sequence of steps so that several batches (groups of up to 32
// systems, or the systems of different meshes) can run interleaved on their
// own streams: survey_begin (initial residual, start, graph), then
// survey_launch (one graph launch if a system is running, asynchronous) and
// survey_collect (wait, then the host's decisions) until done, then
// survey_finish.
namespace {
constexpr int kMaxContinue = 4;      // continuations after the first stop
// stalled: the smoothed residual has not halved for max(kStallWindow,
// iterations before its last halving) iterations (COCR plateaus that end
// are shorter than the way down to them)
constexpr int kStallWindow = 1000;
}  // namespace

void SurveyRun::release()
{
    dev_free(d_flag);
}

int survey_begin(Survey &V, const double2 *b_sys_major, double2 *x_sys_major, double eps,
                 int maxiter, int verify, int iters_per_launch, SurveyRun &R)
{
    R = SurveyRun{};
    R.x_out = x_sys_major;
    R.eps = eps;
    R.maxiter = maxiter;
    R.verify = verify;
    V.eps = eps;
    if (iters_per_launch <= 0) iters_per_launch = 16;
    R.ipl = iters_per_launch + (iters_per_launch & 1);
    for (int k = 0; k < 32; k++) {
        SysState s{};
        s.status = k < V.S ? kRun : MTGPU_OK;
        s.maxiter = maxiter;
        s.residual_rel = 1.0;
        s.true_rel = -1.0;
        s.eps_k = eps;
        V.hsys[k] = s;
    }
    V.hsys[kBarState] = SysState{};
    int rc;
    // (the ticket slots: a launch that gave up leaves its counters behind)
    MTGPU_TRY(cudaMemsetAsync(V.partials, 0, sizeof(float4) * kTicketSlots, V.st));
    if (barrier_polls() != kBarPolls)
        MTGPU_TRY(cudaMemsetAsync((unsigned int *)V.partials + kBarSlot, 0xff, sizeof(unsigned int), V.st));
    if ((rc = upload_sys(V))) return rc;
    to_rows(V, b_sys_major, V.b64);
    to_rows(V, x_sys_major, V.xacc);
    if ((rc = dev_alloc(&R.d_flag, 32))) return rc;
    // inner right-hand side r0 = b - A x0 (FP64), threshold relative to ||b||
    for (int k = 0; k < 32; k++) R.flag[k] = k < V.S;
    if ((rc = upload_flags(R.d_flag, R.flag, V.st))) return rc;
    MTGPU_SP_DISPATCH(V.SP, res64(V, R.d_flag, 1));
    if ((rc = sync_sys(V))) return rc;
    for (int k = 0; k < V.S; k++) {
        SysState &q = V.hsys[k];
        q.checks = 0;
        q.true_rel = -1.0;
        q.eps_k = (q.rnorm > 0.0 && q.bnorm > 0.0) ? eps * q.bnorm / q.rnorm : eps;
    }
    if ((rc = upload_sys(V))) return rc;
    MTGPU_SP_DISPATCH(V.SP, start(V));
    MTGPU_TRY(cudaGetLastError());
    if ((rc = sync_sys(V))) return rc;
    if (!V.graph || V.graph_iters != R.ipl) {
        if (V.graph) cudaGraphExecDestroy(V.graph);
        V.graph = nullptr;
        cudaGraph_t g;
        MTGPU_TRY(cudaStreamBeginCapture(V.st, cudaStreamCaptureModeThreadLocal));
        // an even count: the fused preconditioner's a is back in V.a after the graph
        for (int k = 0; k < R.ipl; k++) MTGPU_SP_DISPATCH(V.SP, iteration(V, k, R.ipl));
        MTGPU_TRY(cudaStreamEndCapture(V.st, &g));
        cudaError_t e = cudaGraphInstantiate(&V.graph, g, 0);
        cudaGraphDestroy(g);
        MTGPU_TRY(e);
        V.graph_iters = R.ipl;
    }
    R.guard_max = (long long)maxiter + (long long)(kMaxContinue + 1) * 4 * R.ipl + 64;
    // MTGPU_SURVEY_GUARD_ITERS (environment) lowers the guard: the device
    // stops every system at maxiter, so only this makes the guard's error
    // path run in a test
    if (const char *g = getenv("MTGPU_SURVEY_GUARD_ITERS"))
        if (atoll(g) > 0) R.guard_max = std::min(R.guard_max, atoll(g));
    return MTGPU_OK;
}

// one graph launch (asynchronous) if a system is running
int survey_launch(Survey &V, SurveyRun &R)
{
    R.launched = false;
    if (R.done) return MTGPU_OK;
    bool running = false;
    for (int k = 0; k < V.S; k++) running |= V.hsys[k].status == kRun;
    if (!running) return MTGPU_OK;
    cudaError_t e = cudaGraphLaunch(V.graph, V.st);
    if (e != cudaSuccess) {
        set_last_error(e, "cudaGraphLaunch", __FILE__, __LINE__);
        return MTGPU_ERR_CUDA;
    }
    const unsigned long long kpi = iteration_launches(V);
    note_launches(kpi * (unsigned long long)R.ipl + (small_used(V) ? 2u : 1u) * ceil_div(R.ipl, V.group));
    R.guard += R.ipl;
    // the state arrives with the launch's end (read in survey_collect)
    MTGPU_TRY(cudaMemcpyAsync(V.hsys, V.sys, sizeof(SysState) * kSysSlots, cudaMemcpyDeviceToHost, V.st));
    R.launched = true;
    return MTGPU_OK;
}

// the host's decisions after a launch, or, once every system has stopped,
// the FP64 true residuals and the continuation decisions
int survey_collect(Survey &V, SurveyRun &R)
{
    if (R.done) return MTGPU_OK;
    int rc;
    if (R.launched) {
        MTGPU_TRY(cudaStreamSynchronize(V.st));
        if (R.guard > R.guard_max) {
            set_last_message("survey solve did not finish within its iteration guard");
            return MTGPU_ERR_TIMEOUT;
        }
        if (V.hsys[kBarState].status != 0) {
            set_last_message("survey solve: a grid barrier did not complete");
            return MTGPU_ERR_TIMEOUT;
        }
        bool changed = false;
        for (int k = 0; k < V.S; k++) {
            SysState &q = V.hsys[k];
            if (q.status != kRun) continue;
            if (q.residual_rel < 0.5 * R.best[k]) {
                R.best[k] = q.residual_rel;
                R.best_it[k] = q.iter;
            } else if (q.iter - R.best_it[k] > std::max(kStallWindow, R.best_it[k])) {
                q.status = MTGPU_MAXITER;   // stalled
                R.stalled[k] = 1;
                changed = true;
            }
        }
        if (changed && (rc = upload_sys(V))) return rc;
        return MTGPU_OK;
    }
    // every system has stopped: FP64 true residual of those that stopped
    // on their threshold (first time, or again after further iterations)
    bool any = false;
    for (int k = 0; k < 32; k++) {
        R.flag[k] = k < V.S && !R.final_[k] && V.hsys[k].status == MTGPU_OK;
        any |= R.flag[k] != 0;
    }
    if (!any) {
        R.done = true;
        return MTGPU_OK;
    }
    if ((rc = upload_flags(R.d_flag, R.flag, V.st))) return rc;
    MTGPU_SP_DISPATCH(V.SP, res64(V, R.d_flag, 0));
    if ((rc = sync_sys(V))) return rc;
    bool resume = false;
    for (int k = 0; k < V.S; k++) {
        if (!R.flag[k]) continue;
        SysState &q = V.hsys[k];
        if (!R.verify || q.true_rel < R.eps) {
            R.final_[k] = 1;
        } else if (q.iter < q.maxiter && R.cont[k] < kMaxContinue &&
                   q.true_rel < 0.9 * R.last_true[k]) {
            // the Krylov iteration still lowers the true residual: go on,
            // asking the recurrence for the missing factor (and a margin)
            R.cont[k]++;
            q.eps_k *= fmin(0.9, fmax(0.05, 0.8 * R.eps / q.true_rel));
            q.status = kRun;
            q.iter += 1;
            resume = true;
        } else {
            q.status = MTGPU_MAXITER;   // not converged: left to the caller
            R.final_[k] = 1;
        }
        R.last_true[k] = q.true_rel;
    }
    if (!resume) {
        R.done = true;
        return MTGPU_OK;
    }
    return upload_sys(V);
}

int survey_finish(Survey &V, SurveyRun &R, mtgpu_survey_stats *stats, int stat_offset)
{
    int rc;
    // true residual of the systems that ended without a check
    bool any = false;
    for (int k = 0; k < 32; k++) {
        R.flag[k] = k < V.S && V.hsys[k].checks == 0 && V.hsys[k].status != MTGPU_X0_NULL;
        any |= R.flag[k] != 0;
    }
    if (any) {
        if ((rc = upload_flags(R.d_flag, R.flag, V.st))) return rc;
        MTGPU_SP_DISPATCH(V.SP, res64(V, R.d_flag, 0));
        if ((rc = sync_sys(V))) return rc;
    }
    from_rows(V, V.xacc, R.x_out);
    MTGPU_TRY(cudaGetLastError());
    MTGPU_TRY(cudaStreamSynchronize(V.st));
    int worst = MTGPU_OK;
    for (int k = 0; k < V.S; k++) {
        const SysState &q = V.hsys[k];
        if (stats) {
            const int o = stat_offset + k;
            stats->status[o] = q.status;
            stats->iterations[o] = q.iter;
            stats->verifications[o] = q.checks;
            stats->fp64_iterations[o] = 0;
            stats->true_residual_rel[o] = q.true_rel;
            stats->residual_rel[o] = q.residual_rel;
        }
        if (q.status != MTGPU_OK && worst == MTGPU_OK) worst = q.status;
    }
    return worst;
}

int survey_solve(Survey &V, const double2 *b_sys_major, double2 *x_sys_major, double eps,
                 int maxiter, int verify, int iters_per_launch, mtgpu_survey_stats *stats)
{
    SurveyRun R;
    int rc = survey_begin(V, b_sys_major, x_sys_major, eps, maxiter, verify, iters_per_launch, R);
    while (!rc && !R.done) {
        if (!(rc = survey_launch(V, R))) rc = survey_collect(V, R);
    }
    if (!rc) rc = survey_finish(V, R, stats, 0);
    R.release();
    return rc;
}

}  // namespace mtgpu
