// Element-level formulas shared by the assembly and the adjoint kernels:
// local edge geometry of a brick, its curl-curl and mass entries, and the
// 1-D table interpolation of the normal field.
#pragma once
#include "mtgpu_internal.cuh"

namespace mtgpu {

// local edge -> direction (0 x, 1 y, 2 z), the grouping of T_Portrait.h:37-51
__device__ __forceinline__ int ldir(int l) { return l >> 2; }

// side (0/1) of local edge l along axis a (a != its direction), from the
// edge midpoints of T_Brick.h:201-214
__device__ __forceinline__ int lpos(int l, int a)
{
    // bit 0 / bit 1 of the position inside the direction group:
    // x-edges (y, z) = (l&1, l>>1 &1); y-edges (x, z) = (l>>1 &1, l&1);
    // z-edges (x, y) = (l&1, l>>1 &1)
    const int d = l >> 2, k = l & 3;
    if (d == 0) return a == 1 ? (k & 1) : ((k >> 1) & 1);
    if (d == 1) return a == 0 ? ((k >> 1) & 1) : (k & 1);
    return a == 0 ? (k & 1) : ((k >> 1) & 1);
}

// entries (i, j) of the local curl-curl b and mass c matrices of a brick
// (closed forms of T_Brick.cpp:123-455 in tensor-product form; see
// oracle/mtcalc_oracle.c orc_brick_bc for the derivation)
__device__ __forceinline__ void brick_entry(int i, int j, const double h[3], double &b, double &c)
{
    const int da = ldir(i), db = ldir(j);
    if (da == db) {
        const int t1 = (da + 1) % 3, t2 = (da + 2) % 3;
        const bool s1 = lpos(i, t1) == lpos(j, t1);
        const bool s2 = lpos(i, t2) == lpos(j, t2);
        const double M1 = s1 ? 2.0 / 3.0 : 1.0 / 3.0, M2 = s2 ? 2.0 / 3.0 : 1.0 / 3.0;
        const double K1 = s1 ? 1.0 : -1.0, K2 = s2 ? 1.0 : -1.0;
        const double m1 = 2.0 * h[t1] / (h[da] * h[t2]);
        const double m2 = 2.0 * h[t2] / (h[da] * h[t1]);
        b = m1 * K2 * M1 + m2 * K1 * M2;
        c = (h[t1] * h[t2] / h[da]) * M1 * M2;
    } else {
        const int q = 3 - da - db;
        const double sa = lpos(i, db) ? 1.0 : -1.0;
        const double sb = lpos(j, da) ? 1.0 : -1.0;
        const double Mq = lpos(i, q) == lpos(j, q) ? 2.0 / 3.0 : 1.0 / 3.0;
        b = -(2.0 * h[q] / (h[da] * h[db])) * sa * sb * Mq;
        c = 0.0;
    }
}

// The entries of one row i of a brick's matrices: brick_entry's values (the
// same operations), with what does not depend on the column formed once, and
// b / mu once per distinct |b|: 13 FP64 divides a row and cell instead of ~45
struct BrickRow {
    int d, i;
    double bs[4], cs[4];      // same direction, by [on the same side along t1] + 2 [t2]: b / mu, c
    double bo[3][2];          // direction db: |b| / mu by [same side along the third axis]
    __device__ __forceinline__ void init(int row, const double h[3], double mu)
    {
        i = row;
        d = ldir(row);
        const int t1 = (d + 1) % 3, t2 = (d + 2) % 3;
        const double m1 = 2.0 * h[t1] / (h[d] * h[t2]);
        const double m2 = 2.0 * h[t2] / (h[d] * h[t1]);
        const double cc = h[t1] * h[t2] / h[d];
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const double M1 = s & 1 ? 2.0 / 3.0 : 1.0 / 3.0, M2 = s & 2 ? 2.0 / 3.0 : 1.0 / 3.0;
            const double K1 = s & 1 ? 1.0 : -1.0, K2 = s & 2 ? 1.0 : -1.0;
            bs[s] = __ddiv_rn(m1 * K2 * M1 + m2 * K1 * M2, mu);
            cs[s] = cc * M1 * M2;
        }
#pragma unroll
        for (int db = 0; db < 3; db++) {
            if (db == d) continue;
            const int q = 3 - d - db;
            const double f = 2.0 * h[q] / (h[d] * h[db]);
            bo[db][0] = __ddiv_rn(f * (1.0 / 3.0), mu);
            bo[db][1] = __ddiv_rn(f * (2.0 / 3.0), mu);
        }
    }
    // b / mu and c of column j
    __device__ __forceinline__ void entry(int j, double &b, double &c) const
    {
        const int db = ldir(j);
        if (db == d) {
            const int t1 = (d + 1) % 3, t2 = (d + 2) % 3;
            const int s = (lpos(i, t1) == lpos(j, t1)) + 2 * (lpos(i, t2) == lpos(j, t2));
            b = s == 0 ? bs[0] : (s == 1 ? bs[1] : (s == 2 ? bs[2] : bs[3]));
            c = s == 0 ? cs[0] : (s == 1 ? cs[1] : (s == 2 ? cs[2] : cs[3]));
        } else {
            const int q = 3 - d - db;
            const bool same = lpos(i, q) == lpos(j, q);
            double v = 0.0;
#pragma unroll
            for (int t = 0; t < 3; t++)
                if (t == db) v = same ? bo[t][1] : bo[t][0];
            // the sign -sa sb of brick_entry
            b = lpos(i, db) == lpos(j, d) ? -v : v;
            c = 0.0;
        }
    }
};

__device__ __forceinline__ void cell_h(const double *xyz, const int *nver, int stride, int cell,
                                       double h[3])
{
    const int n0 = nver[(long long)cell * stride], n7 = nver[(long long)cell * stride + 7];
    h[0] = xyz[3 * n7 + 0] - xyz[3 * n0 + 0];
    h[1] = xyz[3 * n7 + 1] - xyz[3 * n0 + 1];
    h[2] = xyz[3 * n7 + 2] - xyz[3 * n0 + 2];
}

// interval lo and position xi in it of x in the ascending table z[n]
// (For_Solvers.cpp:236-270), found by bisection; outside the table the first
// or last value (xi = 0 or 1)
__device__ __forceinline__ void table_interval(double x, int n, const double *z, int &at, double &xi)
{
    int lo = 0, hi = n - 2;
    if (x < z[0]) {
        at = 0;
        xi = 0.0;
        return;
    }
    if (x > z[n - 1]) {
        at = n - 2;
        xi = 1.0;
        return;
    }
    while (lo < hi) {   // smallest t with x <= z[t+1]
        const int mid = (lo + hi) >> 1;
        if (x <= z[mid + 1]) hi = mid; else lo = mid + 1;
    }
    at = lo;
    xi = (x - z[lo]) / (z[lo + 1] - z[lo]);
}

// linear interpolation of a 1-D table
__device__ __forceinline__ double spline(double x, int n, const double *z, const double *v)
{
    if (x < z[0]) return v[0];
    if (x > z[n - 1]) return v[n - 1];
    int lo;
    double xi;
    table_interval(x, n, z, lo, xi);
    return (1.0 - xi) * v[lo] + xi * v[lo + 1];
}

}  // namespace mtgpu
