// Assembly of a whole sweep from frequency-independent moments.
//
// The distance of a point pair of the RWG pair (m, n) differs from the
// distance R0 = |C_m - C_n| of the two basis functions' centres by at most
// delta, twice the reach of a basis function (plus the softening length), so
//     e^{-jkR} = e^{-jkR0} e^{-jx t},   t = (R - R0) / delta in [-1, 1],
//     x = k delta,   e^{-jx t} ~ sum_{n < N} a_n(x) t^n,
// with the a_n of the Chebyshev expansion J_0(x) + 2 sum (-j)^n J_n(x) T_n(t)
// (Abramowitz & Stegun 9.1.44/45), whose remainder is about 2 |x/2|^N / N!.
// Every entry of every frequency then follows from 2 N real numbers,
//     A_n = sum W (f_m . f_n) t^n / (4 pi R),   S_n = sum W div_m div_n t^n / (4 pi R)
// (sums over the point pairs of the entry's four triangle pairs; f = c (rho - d),
// div = 2 c):
//     Z(m, n; k) = e^{-jkR0} sum_n a_n(k delta) (alpha A_n + beta S_n).
// N is the smallest compiled count whose remainder is below 4e-17 for the
// sweep's largest |k|: the series then replaces e^{-jkR} to less than its
// FP64 rounding.  The sums are FP64 throughout and in a fixed order.
//
// Three kernels once per sweep -- the special (near, self, adjacent) triangle
// pairs' moments, the regular pairs of every entry, the special pairs' share
// of the entries -- and one per batch of frequencies, which reads an entry's
// moments once and writes every frequency's entry: an entry and frequency
// cost about 2 N + 30 FP64 instructions and its 16 bytes of Z instead of nine
// point pairs' phases, a pair value written to memory and four read back.
// Measured (one B200, 3-point rule, Ne 6968, N = 12): 4.7 ms per sweep and
// 0.18 ms per frequency, against 1.22 ms per frequency with the pair values;
// 6-point rule with 9216-point-pair near pairs, Ne 1074, 21 frequencies:
// 2.6 ms against 54.
#include <algorithm>
#include <cmath>
#include <complex>
#include <type_traits>
#include <vector>

#include "efie_internal.h"
#include "quad.cuh"
#include "warp.cuh"

namespace {

constexpr int TE = 32;   // entries per tile side

// tile t of the upper triangle of TE x TE tiles, bm <= bn
__device__ __forceinline__ void tri_tile(int t, int &bm, int &bn) {
    int j = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((j + 1) * (j + 2) / 2 <= t) j++;
    while (j * (j + 1) / 2 > t) j--;
    bn = j;
    bm = t - j * (j + 1) / 2;
}

struct SeriesGeom {
    int Ne, Nt;
    const int *etri;        // triangle per RWG side, [2][Ne], -1 = none
    const double4 *ecd;     // free vertex - origin, c, [2][Ne]
    const double4 *origin;  // [Nt]
    const double4 *ctr;     // RWG centres [Ne]
    const uint8_t *mask;    // 1 = special pair, [Nt][Nt]
};

// ---------------------------------------------------------------------------
// Centres (mean of the centroids of an RWG's triangles) and reach: the largest
// distance of a quadrature point -- with `vtx`, also of a vertex -- of its
// triangles from the centre, and the largest softening length; reach[0..1] as
// the bit patterns of non-negative doubles (their order is the integers').
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_series_reach(int Ne, const int *__restrict__ etri,
                                                      const double4 *__restrict__ origin, int nr,
                                                      const double4 *__restrict__ reg, int nn,
                                                      const double4 *__restrict__ near, int ns,
                                                      const double4 *__restrict__ self,
                                                      const double4 *__restrict__ vtx, int NsS,
                                                      const double *__restrict__ self_a,
                                                      const double *__restrict__ aeq, double near_alpha,
                                                      double4 *__restrict__ ctr, unsigned long long *__restrict__ reach) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= Ne) return;
    int t[2] = {etri[e], etri[Ne + e]};
    if (t[0] < 0) t[0] = t[1];
    if (t[1] < 0) t[1] = t[0];
    if (t[0] < 0) {   // no triangle: the row of Z is zero
        ctr[e] = make_double4(0, 0, 0, 0);
        return;
    }
    const double4 o0 = origin[t[0]], o1 = origin[t[1]];
    const double4 c = make_double4(0.5 * (o0.x + o1.x), 0.5 * (o0.y + o1.y), 0.5 * (o0.z + o1.z), 0.0);
    ctr[e] = c;
    double r2 = 0.0, a = 0.0;
    for (int s = 0; s < 2; s++) {
        const double4 o = s ? o1 : o0;
        const double dx = o.x - c.x, dy = o.y - c.y, dz = o.z - c.z;
        auto far = [&](const double4 *p, int n) {
            for (int i = 0; i < n; i++) {
                const double4 q = p[(size_t)t[s] * n + i];
                const double x = q.x + dx, y = q.y + dy, z = q.z + dz;
                r2 = fmax(r2, x * x + y * y + z * z);
            }
        };
        far(reg, nr);
        if (near) far(near, nn);
        if (self) far(self, ns);
        if (vtx) far(vtx, 3);
        if (self_a)
            for (int i = 0; i < NsS; i++) a = fmax(a, fabs(self_a[(size_t)t[s] * NsS + i]));
        if (aeq) a = fmax(a, fabs(near_alpha * aeq[t[s]]));
    }
    atomicMax(reach, (unsigned long long)__double_as_longlong(sqrt(r2)));
    atomicMax(reach + 1, (unsigned long long)__double_as_longlong(a));
}

// ---------------------------------------------------------------------------
// Moments of the special triangle pairs about their own base distance Rb
// (the centroids' distance of a near pair, else 0):
// sp[(n * 8 + comp) * nsp + pair], comp = S0, S1xyz (rho, first triangle),
// S2xyz (rho'), S3 of W t^n / (4 pi R), t = (R - Rb) / delta.  One warp per
// pair.
// ---------------------------------------------------------------------------
enum { SP_NEAR = 0, SP_SELF = 1 };

struct SpecialArgs {
    int n_pairs, first;          // pairs of this kind, index of the first in the store
    const int2 *list;            // (t1, t2), t1 <= t2 (near, adjacent); self: t = pair index
    int P, per_sub;              // points per triangle, points per sub-triangle (self)
    int parts;                   // parts of the inner points' loop (near, self)
    const double4 *origin, *pts, *vtx;
    const double *aeq, *self_a;  // softening
    double near_alpha;
    int NsS;
};

// Near and self pairs, NT powers from NT * blockIdx.y on.  A lane keeps one
// outer point p (and one of `parts` equal parts of the inner points) at a
// time: its 4 NT sums of t^n {1, rho'} take five instructions per power and
// point pair, and the factors 1 and rho_p come in once per outer point, where
// the eight components are summed over the warp.  Bound by the FP64 pipe:
// 25 + 5 NT instructions per point pair (eight accumulators per power: 25 + 10
// per power in chunks of eight, 4.8 ms for 21783 pairs of 96 x 96 points and
// 14 powers; this form 1.8).
template <int KIND, int NT>
__global__ void __launch_bounds__(64) k_series_pairs(const SpecialArgs q, double inv_delta, int N, size_t nsp,
                                                     double *__restrict__ sp) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= q.n_pairs) return;
    const int n0 = NT * blockIdx.y, P = q.P, items = P * q.parts, len = P / q.parts;
    int2 pr = make_int2(w, w);
    if (KIND == SP_NEAR) pr = q.list[w];
    const int t1 = pr.x, t2 = pr.y;
    double dox = 0.0, doy = 0.0, doz = 0.0, a2 = 0.0, Rb = 0.0;
    if (KIND == SP_NEAR) {
        const double4 o1 = q.origin[t1], o2 = q.origin[t2];
        dox = o1.x - o2.x;
        doy = o1.y - o2.y;
        doz = o1.z - o2.z;
        const double a = q.near_alpha * fmin(q.aeq[t1], q.aeq[t2]);
        a2 = a * a;
        Rb = sqrt(dox * dox + doy * doy + doz * doz);
    }
    constexpr int NG = (NT + 3) / 4;   // groups of four powers: 32 sums, one per lane
    double sum[NG];
#pragma unroll
    for (int g = 0; g < NG; g++) sum[g] = 0.0;
    const double4 *in = q.pts + (size_t)t2 * P;
#pragma unroll 1
    for (int it = lane; it - lane < items; it += 32) {
        double T[NT], X[NT], Y[NT], Z[NT];
#pragma unroll
        for (int n = 0; n < NT; n++) T[n] = X[n] = Y[n] = Z[n] = 0.0;
        double4 pp = make_double4(0, 0, 0, 0);
        if (it < items) {
            const int p = it % P, r0 = (it / P) * len;
            pp = q.pts[(size_t)t1 * P + p];
            const double px = dox + pp.x, py = doy + pp.y, pz = doz + pp.z, wp = pp.w * (1.0 / (4.0 * kPi));
            double b2 = 0.0;
            int s0 = P, s1 = P;   // the inner points of the same sub-triangle
            if (KIND == SP_SELF) {
                const int sa = p / q.per_sub;
                const double aS = q.self_a[(size_t)t1 * q.NsS + sa];
                b2 = aS * aS;
                s0 = sa * q.per_sub;
                s1 = s0 + q.per_sub;
            }
#pragma unroll 1
            for (int r = r0; r < r0 + len; r++) {
                const double4 pq = in[r];
                const double dx = px - pq.x, dy = py - pq.y, dz = pz - pq.z;
                double R2 = dx * dx + dy * dy + dz * dz + (KIND == SP_NEAR ? a2 : 0.0);
                if (KIND == SP_SELF && r >= s0 && r < s1) R2 += b2;
                R2 = fmax(R2, 1e-30);
                const double rs = rsqrt(R2);
                const double t = (R2 * rs - Rb) * inv_delta;
                double u = wp * pq.w * rs;
                for (int i = 0; i < n0; i++) u *= t;
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    T[n] += u;
                    X[n] = fma(u, pq.x, X[n]);
                    Y[n] = fma(u, pq.y, Y[n]);
                    Z[n] = fma(u, pq.z, Z[n]);
                    u *= t;
                }
            }
        }
#pragma unroll
        for (int g = 0; g < NG; g++) {
            constexpr int last = NT % 4;
            double d[32];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                if (4 * g + m >= NT) break;
                const int n = 4 * g + m;
                d[8 * m] = T[n];
                d[8 * m + 1] = T[n] * pp.x;
                d[8 * m + 2] = T[n] * pp.y;
                d[8 * m + 3] = T[n] * pp.z;
                d[8 * m + 4] = X[n];
                d[8 * m + 5] = Y[n];
                d[8 * m + 6] = Z[n];
                d[8 * m + 7] = pp.x * X[n] + pp.y * Y[n] + pp.z * Z[n];
            }
            if (last && g == NG - 1) {
                double h[16];
#pragma unroll
                for (int i = 0; i < 16; i++) h[i] = d[i];
                sum[g] += warp_sums<16>(h, lane);
            } else {
                sum[g] += warp_sums<32>(d, lane);
            }
        }
    }
#pragma unroll
    for (int g = 0; g < NG; g++) {   // the lane is left with power 4 g + lane / 8, component lane mod 8
        const int l = 4 * g + (lane >> 3), n = n0 + l;
        if (l < NT && n < N) sp[((size_t)n * 8 + (lane & 7)) * nsp + q.first + w] = sum[g];
    }
}

// Adjacent pairs of the extraction scheme, eight powers per blockIdx.y: the
// static part (n = 0) is analytic over the inner triangle, the powers from
// n = 1 on take the rule's point pairs, so few that the lanes share them.
__global__ void __launch_bounds__(64) k_series_adjacent(const SpecialArgs q, double inv_delta, int N, size_t nsp,
                                                        double *__restrict__ sp) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= q.n_pairs) return;
    const int n0 = 8 * blockIdx.y, P = q.P;
    const int2 pr = q.list[w];
    const int t1 = pr.x, t2 = pr.y;
    const double4 o1 = q.origin[t1], o2 = q.origin[t2];
    const double dox = o1.x - o2.x, doy = o1.y - o2.y, doz = o1.z - o2.z;
    double v[2][32];   // powers n0 .. n0 + 3, n0 + 4 .. n0 + 7
#pragma unroll
    for (int i = 0; i < 32; i++) v[0][i] = v[1][i] = 0.0;
    constexpr double k4pi = 1.0 / (4.0 * kPi);
    for (int e = lane; e < P * P; e += 32) {
        const int p = e / P, r = e - p * P;
        const double4 pp = q.pts[(size_t)t1 * P + p], pq = q.pts[(size_t)t2 * P + r];
        const double dx = dox + pp.x - pq.x, dy = doy + pp.y - pq.y, dz = doz + pp.z - pq.z;
        const double t = sqrt(dx * dx + dy * dy + dz * dz) * inv_delta;
        double u = pp.w * pq.w * k4pi * inv_delta;   // W t^n / (4 pi R) = W t^(n - 1) / (4 pi delta)
        for (int i = 1; i < n0; i++) u *= t;
        const double dd = pp.x * pq.x + pp.y * pq.y + pp.z * pq.z;
#pragma unroll
        for (int n = 0; n < 8; n++) {
            if (n == 0 && n0 == 0) continue;
            double *a = &v[n >> 2][8 * (n & 3)];
            a[0] += u;
            a[1] += u * pp.x;
            a[2] += u * pp.y;
            a[3] += u * pp.z;
            a[4] += u * pq.x;
            a[5] += u * pq.y;
            a[6] += u * pq.z;
            a[7] += u * dd;
            u *= t;
        }
    }
    if (n0 == 0 && lane < P) {
        // static part: outer point on t1, 1/R integrated analytically over t2
        const double4 pp = q.pts[(size_t)t1 * P + lane];
        const double3 r = make_double3(pp.x + dox, pp.y + doy, pp.z + doz);
        const double4 v0 = q.vtx[3 * (size_t)t2], v1 = q.vtx[3 * (size_t)t2 + 1], v2 = q.vtx[3 * (size_t)t2 + 2];
        double I0;
        double3 J;
        potential_integrals(make_double3(v0.x, v0.y, v0.z), make_double3(v1.x, v1.y, v1.z),
                            make_double3(v2.x, v2.y, v2.z), r, I0, J);
        const double sx = J.x + r.x * I0, sy = J.y + r.y * I0, sz = J.z + r.z * I0;
        const double wt = pp.w * k4pi;
        v[0][0] += wt * I0;
        v[0][1] += wt * I0 * pp.x;
        v[0][2] += wt * I0 * pp.y;
        v[0][3] += wt * I0 * pp.z;
        v[0][4] += wt * sx;
        v[0][5] += wt * sy;
        v[0][6] += wt * sz;
        v[0][7] += wt * (pp.x * sx + pp.y * sy + pp.z * sz);
    }
    __syncwarp();
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const double s = warp_sums<32>(v[g], lane);
        const int n = n0 + 4 * g + (lane >> 3);
        if (n < N) sp[((size_t)n * 8 + (lane & 7)) * nsp + q.first + w] = s;
    }
}

// ---------------------------------------------------------------------------
// Regular pairs of every entry of a tile: lane = row m, a warp's turn = column
// n, so the column's points are broadcast reads and the row's are
// conflict-free ([component][row] in shared memory).  A thread holds the 2 N
// sums in registers over the entry's up to four triangle pairs; the powers of
// t run in two chains (even and odd) to halve the dependent multiplications.
// Bound by the FP64 pipe: about 24 + 3 N instructions per point pair, at N = 12
// 83 operations by the counters and 18.2 TFLOP/s (Ne 4110: 1.42 ms), half of
// what cuBLAS DGEMM reaches with nothing but fused multiply-adds.
// mom[((tile - tile0) * 2 N + comp) * 1024 + column * 32 + row], comp = A_0.., S_0...
// ---------------------------------------------------------------------------
template <int NQ>
struct EntrySmem {
    double d[2][2 * NQ * 7][TE];   // rho xyz, f xyz (c w (rho - d)), 2 c w per side and point
    double o[2][6][TE];            // triangle origins per side
    double c[2][3][TE];            // RWG centres
    int t[2][2][TE];
};

template <int NQ, int N>
__global__ void __launch_bounds__(128, (N <= 14 ? 4 : 3)) k_series_entries(const SeriesGeom G, int tile0,
                                                                          const double4 *__restrict__ pts,
                                                                          double inv_delta,
                                                                          double *__restrict__ mom,
                                                                          int *__restrict__ special) {
    extern __shared__ __align__(16) unsigned char raw[];
    EntrySmem<NQ> &S = *reinterpret_cast<EntrySmem<NQ> *>(raw);
    int bm, bn;
    tri_tile(tile0 + blockIdx.x, bm, bn);
    const int tid = threadIdx.x;
    for (int i = tid; i < 2 * 2 * TE; i += 128) {
        const int r = i & 31, s = (i >> 5) & 1, w = i >> 6;
        const int e = (w ? bn : bm) * TE + r;
        int t = -1;
        double4 cd = make_double4(0, 0, 0, 0), o = cd, c = cd;
        if (e < G.Ne) {
            t = G.etri[(size_t)s * G.Ne + e];
            cd = G.ecd[(size_t)s * G.Ne + e];
            c = G.ctr[e];
            if (t >= 0) o = G.origin[t];
        }
        S.t[w][s][r] = t;
        S.o[w][3 * s][r] = o.x;
        S.o[w][3 * s + 1][r] = o.y;
        S.o[w][3 * s + 2][r] = o.z;
        if (s == 0) S.c[w][0][r] = c.x, S.c[w][1][r] = c.y, S.c[w][2][r] = c.z;
        // 1 / (4 pi) goes with the rows
        const double cc = w ? cd.w : cd.w * (1.0 / (4.0 * kPi));
        for (int p = 0; p < NQ; p++) {
            const double4 q = t >= 0 ? pts[(size_t)t * NQ + p] : make_double4(0, 0, 0, 0);
            double(*D)[TE] = &S.d[w][(s * NQ + p) * 7];
            const double cw = cc * q.w;
            D[0][r] = q.x;
            D[1][r] = q.y;
            D[2][r] = q.z;
            D[3][r] = cw * (q.x - cd.x);
            D[4][r] = cw * (q.y - cd.y);
            D[5][r] = cw * (q.z - cd.z);
            D[6][r] = 2.0 * cw;
        }
    }
    __syncthreads();
    const int tx = tid & 31, cols = TE / gridDim.y;   // this CTA's columns of the tile
    const int m = bm * TE + tx;
    double *out = mom + (size_t)blockIdx.x * 2 * N * TE * TE + tx;
    bool any = false;   // a special pair among this CTA's entries
#pragma unroll 1
    for (int j = blockIdx.y * cols + (tid >> 5); j < (blockIdx.y + 1) * cols; j += 4) {
        const int n = bn * TE + j;
        const bool on = m < G.Ne && n < G.Ne && !(bm == bn && tx > j);
        double A[N], C[N];
#pragma unroll
        for (int i = 0; i < N; i++) A[i] = 0.0, C[i] = 0.0;
        const double cx = S.c[0][0][tx] - S.c[1][0][j], cy = S.c[0][1][tx] - S.c[1][1][j],
                     cz = S.c[0][2][tx] - S.c[1][2][j];
        const double t0 = -sqrt(cx * cx + cy * cy + cz * cz) * inv_delta;
#pragma unroll 1
        for (int ab = 0; ab < 4; ab++) {
            const int a = ab >> 1, b = ab & 1;
            const int t1 = S.t[0][a][tx], t2 = S.t[1][b][j];
            if (t2 < 0) continue;
            if (!on || t1 < 0) continue;
            if (G.mask[(size_t)t1 + (size_t)G.Nt * t2]) {
                any = true;
                continue;
            }
            const double ox = S.o[0][3 * a][tx] - S.o[1][3 * b][j], oy = S.o[0][3 * a + 1][tx] - S.o[1][3 * b + 1][j],
                         oz = S.o[0][3 * a + 2][tx] - S.o[1][3 * b + 2][j];
#pragma unroll 1
            for (int p = 0; p < NQ; p++) {
                const double(*M)[TE] = &S.d[0][(a * NQ + p) * 7];
                const double px = ox + M[0][tx], py = oy + M[1][tx], pz = oz + M[2][tx];
                const double fx = M[3][tx], fy = M[4][tx], fz = M[5][tx], sw = M[6][tx];
#pragma unroll 1
                for (int q = 0; q < NQ; q++) {
                    const double(*Q)[TE] = &S.d[1][(b * NQ + q) * 7];
                    const double dx = px - Q[0][j], dy = py - Q[1][j], dz = pz - Q[2][j];
                    const double R2 = fmax(dx * dx + dy * dy + dz * dz, 1e-30);
                    const double rs = rsqrt(R2);
                    const double t = fma(R2 * rs, inv_delta, t0), tt = t * t;
                    const double ua = rs * (fx * Q[3][j] + fy * Q[4][j] + fz * Q[5][j]);
                    const double us = rs * (sw * Q[6][j]);
                    double pe = 1.0, po = t;
#pragma unroll
                    for (int i = 0; i < N; i += 2) {
                        A[i] = fma(ua, pe, A[i]);
                        C[i] = fma(us, pe, C[i]);
                        A[i + 1] = fma(ua, po, A[i + 1]);
                        C[i + 1] = fma(us, po, C[i + 1]);
                        if (i + 2 < N) {
                            pe *= tt;
                            po *= tt;
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            out[(size_t)i * TE * TE + j * TE] = A[i];
            out[(size_t)(N + i) * TE * TE + j * TE] = C[i];
        }
    }
    any = __syncthreads_or(any);
    if (tid == 0) special[blockIdx.x * gridDim.y + blockIdx.y] = any;
}

// ---------------------------------------------------------------------------
// The special pairs' share of the entries: the pair's moments combined for the
// two basis functions, moved from its base distance to the entry's R0 --
// int (t + s)^n from int t^n, s = (Rb - R0) / delta, in N - 1 passes
// M_n += s M_{n-1} -- and added to the entry's sums.  Four CTAs per tile: the
// tiles along the diagonal hold most of the special pairs, so their columns
// are spread (127 us with one CTA per tile at Ne 1074).
// ---------------------------------------------------------------------------
struct SpecialIndex {
    const int2 *list;   // near or adjacent pairs, ordered by (t2, t1)
    int n_list;
    bool adj;           // adjacent pairs (self pairs among them, all bases 0); else near pairs, then self
};

template <int N>
__global__ void __launch_bounds__(256) k_series_add(const SeriesGeom G, int tile0, const SpecialIndex X, size_t nsp,
                                                    const double *__restrict__ sp, double inv_delta,
                                                    double *__restrict__ mom, const int *__restrict__ special,
                                                    int split) {
    // most tiles hold no special pair: k_series_entries has seen every one
    bool any = false;
    for (int i = 0; i < split; i++) any |= special[blockIdx.x * split + i] != 0;
    if (!any) return;
    int bm, bn;
    tri_tile(tile0 + blockIdx.x, bm, bn);
    const int tx = threadIdx.x & 31;
    const int m = bm * TE + tx;
    if (m >= G.Ne) return;
    const int cols = TE / gridDim.y;
#pragma unroll 1
    for (int j = blockIdx.y * cols + (threadIdx.x >> 5); j < (blockIdx.y + 1) * cols; j += 8) {
        const int n = bn * TE + j;
        if (n >= G.Ne || (bm == bn && tx > j)) continue;
#pragma unroll 1
        for (int ab = 0; ab < 4; ab++) {
            const int a = ab >> 1, b = ab & 1;
            const int t1 = G.etri[(size_t)a * G.Ne + m], t2 = G.etri[(size_t)b * G.Ne + n];
            if (t1 < 0 || t2 < 0 || !G.mask[(size_t)t1 + (size_t)G.Nt * t2]) continue;
            const int lo = min(t1, t2), hi = max(t1, t2);
            size_t idx;
            double Rb = 0.0;
            if (!X.adj && lo == hi) {
                idx = (size_t)X.n_list + lo;
            } else {
                int l = 0, r = X.n_list;   // first pair not before (lo, hi)
                while (l < r) {
                    const int c = (l + r) >> 1;
                    const int2 p = X.list[c];
                    if (p.y < hi || (p.y == hi && p.x < lo)) l = c + 1;
                    else r = c;
                }
                if (l >= X.n_list) continue;
                idx = l;
                if (!X.adj) {
                    const double4 o1 = G.origin[lo], o2 = G.origin[hi];
                    const double x = o1.x - o2.x, y = o1.y - o2.y, z = o1.z - o2.z;
                    Rb = sqrt(x * x + y * y + z * z);
                }
            }
            const double4 dm = G.ecd[(size_t)a * G.Ne + m], dn = G.ecd[(size_t)b * G.Ne + n];
            const double cc = dm.w * dn.w, dd = dm.x * dn.x + dm.y * dn.y + dm.z * dn.z;
            const bool sw = t1 > t2, mean = X.adj && lo == hi;
            double A[N], C[N];
#pragma unroll
            for (int i = 0; i < N; i++) {
                double s[8];
#pragma unroll
                for (int k = 0; k < 8; k++) s[k] = sp[((size_t)i * 8 + k) * nsp + idx];
                if (mean) {   // self pair of the extraction scheme: the mean of both outer/inner orders
#pragma unroll
                    for (int k = 1; k < 4; k++) s[k] = s[k + 3] = 0.5 * (s[k] + s[k + 3]);
                } else if (sw) {   // stored for (t2, t1)
#pragma unroll
                    for (int k = 1; k < 4; k++) {
                        const double x = s[k];
                        s[k] = s[k + 3];
                        s[k + 3] = x;
                    }
                }
                A[i] = cc * (s[7] - (dn.x * s[1] + dn.y * s[2] + dn.z * s[3]) -
                             (dm.x * s[4] + dm.y * s[5] + dm.z * s[6]) + dd * s[0]);
                C[i] = 4.0 * cc * s[0];
            }
            const double4 c1 = G.ctr[m], c2 = G.ctr[n];
            const double x = c1.x - c2.x, y = c1.y - c2.y, z = c1.z - c2.z;
            const double s = (Rb - sqrt(x * x + y * y + z * z)) * inv_delta;
#pragma unroll
            for (int k = 1; k < N; k++)
#pragma unroll
                for (int i = N - 1; i >= k; i--) {
                    A[i] = fma(s, A[i - 1], A[i]);
                    C[i] = fma(s, C[i - 1], C[i]);
                }
            double *out = mom + (size_t)blockIdx.x * 2 * N * TE * TE + j * TE + tx;
#pragma unroll
            for (int i = 0; i < N; i++) {
                out[(size_t)i * TE * TE] += A[i];
                out[(size_t)(N + i) * TE * TE] += C[i];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Every frequency's entries of a tile from its moments: the 2 N sums are read
// once into registers, then each frequency costs two polynomials, the phase
// (a sincos of k R0, or, in an equally spaced run, one multiplication by the
// step's phase, restarted every fourth frequency) and the stores: Z's upper
// triangle, its 128 x 128 diagonal blocks in full (what the symmetric GMRES
// product reads) and, with `planes`, the complex64 planes' lower triangle.
// Bound by HBM: 16 bytes written per entry and frequency (24 with the planes)
// and 16 N read per entry.
// coef[f]: kr, ki, alr, ali, ber, bei, 0, 0, then N complex coefficients a_n.
// ---------------------------------------------------------------------------
constexpr int CF = 8;

template <int N, bool LOSSY>
__global__ void __launch_bounds__(256) k_series_eval(int Ne, int tile0, const double *__restrict__ mom,
                                                     const double4 *__restrict__ ctr, int nf,
                                                     const double *__restrict__ coef, int even,
                                                     double2 *__restrict__ Zb, size_t zstride,
                                                     float *__restrict__ planes, size_t pstride, int ld) {
    extern __shared__ double cs[];
    constexpr int CS = CF + 2 * N;
    for (int i = threadIdx.x; i < nf * CS; i += 256) cs[i] = coef[i];
    __syncthreads();
    int bm, bn;
    tri_tile(tile0 + blockIdx.x, bm, bn);
    const int tx = threadIdx.x & 31;
    const int m = bm * TE + tx;
    const bool mirror = bm != bn && bm / 4 == bn / 4;
    const double *in = mom + (size_t)blockIdx.x * 2 * N * TE * TE;
    const int cols = TE / gridDim.y;
#pragma unroll 1
    for (int j = blockIdx.y * cols + (threadIdx.x >> 5); j < (blockIdx.y + 1) * cols; j += 8) {
        const int n = bn * TE + j;
        if (m >= Ne || n >= Ne) continue;
        // below the diagonal of a diagonal tile: the transposed entry
        const int at = (bm == bn && tx > j) ? tx * TE + j : j * TE + tx;
        double A[N], C[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            A[i] = __ldcs(in + (size_t)i * TE * TE + at);
            C[i] = __ldcs(in + (size_t)(N + i) * TE * TE + at);
        }
        const double4 c1 = ctr[min(m, n)], c2 = ctr[max(m, n)];
        const double x = c1.x - c2.x, y = c1.y - c2.y, z = c1.z - c2.z;
        const double R0 = sqrt(x * x + y * y + z * z);
        double str = 1.0, sti = 0.0, er = 1.0, ei = 0.0;
        if (even) {
            double sn, cn;
            sincos((cs[CS] - cs[0]) * R0, &sn, &cn);
            str = cn;
            sti = -sn;
            if (LOSSY) {
                const double d = exp((cs[CS + 1] - cs[1]) * R0);
                str *= d;
                sti *= d;
            }
        }
#pragma unroll 1
        for (int f = 0; f < nf; f++) {
            const double *c = cs + f * CS;
            if (!even || (f & 3) == 0) {
                double sn, cn;
                sincos(c[0] * R0, &sn, &cn);
                er = cn;
                ei = -sn;
                if (LOSSY) {
                    const double d = exp(c[1] * R0);
                    er *= d;
                    ei *= d;
                }
            } else {
                const double r = er * str - ei * sti;
                ei = er * sti + ei * str;
                er = r;
            }
            double ar = 0.0, ai = 0.0, sr = 0.0, si = 0.0;
#pragma unroll
            for (int i = 0; i < N; i++) {
                const double gr = c[CF + 2 * i], gi = c[CF + 2 * i + 1];
                if (LOSSY || (i & 1) == 0) {   // real k: even coefficients are real, odd ones imaginary
                    ar = fma(gr, A[i], ar);
                    sr = fma(gr, C[i], sr);
                }
                if (LOSSY || (i & 1) == 1) {
                    ai = fma(gi, A[i], ai);
                    si = fma(gi, C[i], si);
                }
            }
            const double vr = (c[2] * ar - c[3] * ai) + (c[4] * sr - c[5] * si);
            const double vi = (c[2] * ai + c[3] * ar) + (c[4] * si + c[5] * sr);
            const double zr = er * vr - ei * vi, zi = er * vi + ei * vr;
            double2 *Z = Zb + zstride * f;
            Z[(size_t)m + (size_t)Ne * n] = make_double2(zr, zi);
            if (mirror) Z[(size_t)n + (size_t)Ne * m] = make_double2(zr, zi);
            if (planes) {   // row n, column m of the lower triangle
                float *pr = planes + pstride * f + (size_t)n * ld + m;
                pr[0] = (float)zr;
                pr[(size_t)ld * Ne] = (float)zi;
            }
        }
    }
}

// N terms compiled, smallest first
constexpr int kTerms[] = {8, 10, 12, 14, 16, 20, 24};

// the largest |a_n| remainder of N terms at |x|: 2 sum_{n >= N} |J_n(x)|, with
// |J_n(x)| <= |x/2|^n e^{|Im x|} / n! (A&S 9.1.62)
double remainder(int N, double ax, double im) {
    double u = 2.0 * std::exp(im);
    for (int n = 1; n <= N; n++) u *= 0.5 * ax / n;
    return u / (1.0 - 0.5 * ax / (N + 1));
}

// a_n (n < N) of e^{-jxt} in powers of t
void coefficients(int N, std::complex<double> x, double *out) {
    typedef std::complex<long double> cl;
    const cl h = cl(x.real(), x.imag()) * (long double)0.5;
    std::vector<cl> a(N, cl(0)), J(N);
    cl lead = 1;
    for (int n = 0; n < N; n++) {
        if (n) lead *= h / (long double)n;
        cl term = lead, s = lead;   // J_n = sum_m (-1)^m (x/2)^{2m+n} / (m! (m+n)!)
        for (int i = 1; i < 40; i++) {
            term *= -h * h / ((long double)i * (long double)(i + n));
            s += term;
        }
        J[n] = s;
    }
    // T_n in powers of t
    std::vector<long double> t0(N + 1, 0), t1(N + 1, 0), t2(N + 1, 0);
    t0[0] = 1;
    t1[1] = 1;
    cl mj(0, -1), pj = 1;
    for (int n = 0; n < N; n++) {
        const std::vector<long double> &T = n == 0 ? t0 : t1;
        const cl w = (n ? (long double)2 : (long double)1) * pj * J[n];
        for (int i = 0; i <= n; i++) a[i] += w * T[i];
        pj *= mj;
        if (n >= 1) {
            for (int i = 0; i <= N; i++) t2[i] = (i ? 2 * t1[i - 1] : 0) - t0[i];
            t0 = t1;
            t1 = t2;
        }
    }
    for (int n = 0; n < N; n++) {
        out[2 * n] = (double)a[n].real();
        out[2 * n + 1] = (double)a[n].imag();
    }
}

SeriesGeom series_geom(const GeomDev &g) {
    return SeriesGeom{g.Ne, g.Nt, g.edge_tri.as<int>(), g.edge_cd.as<double4>(), g.origin.as<double4>(),
                      g.ser_ctr.as<double4>(), g.near_mask.as<uint8_t>()};
}

size_t special_pairs(const GeomDev &g) {
    return g.scheme == EFIE_SCHEME_EXTRACT ? (size_t)g.n_adj : (size_t)g.n_near + g.Nt;
}

// CTAs per tile (at most `most`): enough for four per SM where the tiles of a
// small problem are few
unsigned tile_split(int tiles, int most) {
    unsigned y = 1;
    while ((int)y < most && tiles * (int)y < 600) y *= 2;
    return y;
}

template <int NQ, int N>
efie_status launch_entries(const GeomDev &g, cudaStream_t s, int tile0, int nt, double inv_delta, double *mom,
                           int *special) {
    constexpr size_t bytes = sizeof(EntrySmem<NQ>);
    if (bytes > 48 * 1024)
        EFIE_CUDA(cudaFuncSetAttribute(k_series_entries<NQ, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    k_series_entries<NQ, N><<<dim3(nt, tile_split(nt, 8)), 128, bytes, s>>>(series_geom(g), tile0, g.reg_pts.as<double4>(), inv_delta, mom,
                                                                                      special);
    return efie_cuda_check(cudaGetLastError(), "series entries");
}

// Parts of the inner points' loop: the fewest that keep the lanes busiest
int pair_parts(int P) {
    int best = 1;
    double eff = 0.0;
    for (int parts : {1, 2, 4, 8}) {
        if (P % parts) continue;
        const int items = P * parts;
        const double e = items / (32.0 * ((items + 31) / 32));
        if (e > eff + 1e-9) eff = e, best = parts;
    }
    return best;
}

template <int KIND>
efie_status launch_pairs(SpecialArgs q, double inv_delta, int N, size_t nsp, double *sp, cudaStream_t s) {
    q.parts = pair_parts(q.P);
    const unsigned nx = (q.n_pairs + 1) / 2;
    // all powers in one pass up to 16 (4 sums each in registers), else in two
    switch (N) {
    case 8: k_series_pairs<KIND, 8><<<nx, 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    case 10: k_series_pairs<KIND, 10><<<nx, 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    case 12: k_series_pairs<KIND, 12><<<nx, 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    case 14: k_series_pairs<KIND, 14><<<nx, 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    case 16: k_series_pairs<KIND, 16><<<nx, 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    case 20: k_series_pairs<KIND, 10><<<dim3(nx, 2), 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    case 24: k_series_pairs<KIND, 12><<<dim3(nx, 2), 64, 0, s>>>(q, inv_delta, N, nsp, sp); break;
    default: return efie_fail(EFIE_ERR_ARGS, "series: unknown term count");
    }
    return efie_cuda_check(cudaGetLastError(), "series pairs");
}

template <int N>
efie_status launch_tiles(efie_ctx *ctx, const GeomDev &g, int tile0, int nt, double *mom) {
    cudaStream_t s = ctx->stream;
    const double inv = 1.0 / g.ser_delta;
    int *flags = g.ser_flag.as<int>();
    size_t tok = ctx->log.begin(s);
    switch (g.Nq) {
    case 1: EFIE_TRY((launch_entries<1, N>(g, s, tile0, nt, inv, mom, flags))); break;
    case 3: EFIE_TRY((launch_entries<3, N>(g, s, tile0, nt, inv, mom, flags))); break;
    case 6: EFIE_TRY((launch_entries<6, N>(g, s, tile0, nt, inv, mom, flags))); break;
    case 7: EFIE_TRY((launch_entries<7, N>(g, s, tile0, nt, inv, mom, flags))); break;
    default: return efie_fail(EFIE_ERR_ARGS, "series: unsupported rule");
    }
    const bool adj = g.scheme == EFIE_SCHEME_EXTRACT;
    const SpecialIndex X{adj ? g.adj_list.as<int2>() : g.near_list.as<int2>(), adj ? g.n_adj : g.n_near, adj};
    k_series_add<N><<<dim3(nt, 4), 256, 0, s>>>(series_geom(g), tile0, X, special_pairs(g), g.ser_sp.as<double>(), inv, mom,
                                              flags, (int)tile_split(nt, 8));
    EFIE_CUDA(cudaGetLastError());
    // point pairs: four triangle pairs per entry
    ctx->log.end(EFIE_K_QUAD, s, tok, 4.0 * (double)g.Nq * g.Nq * (double)nt * TE * TE, 2);
    return EFIE_OK;
}

template <int N>
efie_status launch_eval(efie_ctx *ctx, const GeomDev &g, int tile0, int nt, const double *mom, int nf, bool lossy,
                        bool even, void *Z, size_t zstride, const PlanesOut *po) {
    cudaStream_t s = ctx->stream;
    const size_t sm = sizeof(double) * nf * (CF + 2 * N);
    double2 *Zd = static_cast<double2 *>(Z);
    float *pl = po ? po->p : nullptr;
    const size_t ps = po ? po->pstride : 0;
    const int ld = po ? po->ld : 0;
    const dim3 grid(nt, tile_split(nt, 4));
    size_t tok = ctx->log.begin(s);
    if (lossy)
        k_series_eval<N, true><<<grid, 256, sm, s>>>(g.Ne, tile0, mom, g.ser_ctr.as<double4>(), nf,
                                                   g.ser_coef.as<double>(), even, Zd, zstride, pl, ps, ld);
    else
        k_series_eval<N, false><<<grid, 256, sm, s>>>(g.Ne, tile0, mom, g.ser_ctr.as<double4>(), nf,
                                                    g.ser_coef.as<double>(), even, Zd, zstride, pl, ps, ld);
    EFIE_CUDA(cudaGetLastError());
    // algorithmic bytes: the moments once, Z (and the planes) of every frequency
    ctx->log.end(EFIE_K_GATHER, s, tok, (double)nt * TE * TE * (16.0 * N + (po ? 24.0 : 16.0) * nf));
    return EFIE_OK;
}

// fn(integral_constant<int, N>) for the compiled term count N
template <class Fn>
efie_status with_terms(int N, Fn fn) {
    switch (N) {
    case 8: return fn(std::integral_constant<int, 8>());
    case 10: return fn(std::integral_constant<int, 10>());
    case 12: return fn(std::integral_constant<int, 12>());
    case 14: return fn(std::integral_constant<int, 14>());
    case 16: return fn(std::integral_constant<int, 16>());
    case 20: return fn(std::integral_constant<int, 20>());
    case 24: return fn(std::integral_constant<int, 24>());
    }
    return efie_fail(EFIE_ERR_ARGS, "series: unknown term count");
}

}  // namespace

efie_status efie_series_begin(efie_ctx *ctx, GeomDev &g, double kabs, double kimag, bool *use) {
    *use = false;
    g.ser_n = 0;
    if (!g.symmetric || g.Ne < 1 || (g.Nq != 1 && g.Nq != 3 && g.Nq != 6 && g.Nq != 7)) return EFIE_OK;
    cudaStream_t s = ctx->stream;
    const bool ref = g.scheme == EFIE_SCHEME_REF;
    if (!(g.ser_delta > 0)) {
        EFIE_TRY(g.ser_ctr.reserve(sizeof(double4) * g.Ne));
        EFIE_TRY(g.ser_coef.reserve(sizeof(double) * 2));
        EFIE_CUDA(cudaMemsetAsync(g.ser_coef.p, 0, sizeof(double) * 2, s));
        k_series_reach<<<(g.Ne + 127) / 128, 128, 0, s>>>(
            g.Ne, g.edge_tri.as<int>(), g.origin.as<double4>(), g.Nq, g.reg_pts.as<double4>(), g.NsN * g.Nq2,
            ref ? g.near_pts.as<double4>() : nullptr, g.NsS * g.Nq2, ref ? g.self_pts.as<double4>() : nullptr,
            ref ? nullptr : g.tri_vtx.as<double4>(), g.NsS, ref ? g.self_a.as<double>() : nullptr,
            ref ? g.aeq.as<double>() : nullptr, g.near_alpha, g.ser_ctr.as<double4>(),
            g.ser_coef.as<unsigned long long>());
        EFIE_CUDA(cudaGetLastError());
        double r[2] = {0, 0};
        EFIE_CUDA(cudaMemcpyAsync(r, g.ser_coef.p, sizeof(r), cudaMemcpyDeviceToHost, s));
        EFIE_CUDA(cudaStreamSynchronize(s));
        g.ser_delta = (2.0 * r[0] + r[1]) * (1.0 + 1e-9);
    }
    if (!(g.ser_delta > 0) || !std::isfinite(g.ser_delta)) return EFIE_OK;
    const double ax = kabs * g.ser_delta, im = std::abs(kimag) * g.ser_delta;
    if (!(ax <= 3.0)) return EFIE_OK;   // past it the terms grow and the shifts of the special pairs lose digits
    int N = 0;
    for (int c : kTerms)
        if (remainder(c, ax, im) < 4e-17) {
            N = c;
            break;
        }
    if (!N) return EFIE_OK;
    // the moments share the buffer of the pair values, within a third of free
    // memory; what does not fit is made a part at a time, for every batch
    const size_t nb = (g.Ne + TE - 1) / TE, tiles = nb * (nb + 1) / 2;
    const size_t per = sizeof(double) * 2 * N * TE * TE, old = g.moments.bytes;
    if (tiles > (size_t)1 << 30) return EFIE_OK;
    if (old < tiles * per) {
        size_t freeb = 0, total = 0;
        if (cudaMemGetInfo(&freeb, &total) != cudaSuccess) return EFIE_OK;
        const size_t most = (freeb + efie_pool_cached(ctx->device) + old) / 3 / per;
        const size_t want = std::min(tiles, most) * per;
        if (want > old) {
            EFIE_CUDA(cudaStreamSynchronize(s));   // an earlier assembly may still read it
            g.moments.release();
            g.mf = 0;
            // no room after all: the sweep takes the pair values, which reserve what they need
            if (g.moments.reserve(want) != EFIE_OK) return EFIE_OK;
        }
    }
    const size_t cap = g.moments.bytes / per;
    if (cap < 1) return EFIE_OK;
    const size_t nsp = special_pairs(g);   // the special pairs' moments
    if (g.ser_sp.reserve(sizeof(double) * 8 * N * std::max<size_t>(nsp, 1)) != EFIE_OK ||
        g.ser_flag.reserve(sizeof(int) * 8 * std::min(cap, tiles)) != EFIE_OK)
        return EFIE_OK;
    g.ser_n = N;
    g.ser_cap = std::min(cap, tiles);
    g.ser_tiles = tiles;
    g.ser_done = false;
    SpecialArgs q{};
    q.origin = g.origin.as<double4>();
    const double inv = 1.0 / g.ser_delta;
    size_t tok = ctx->log.begin(s);
    int nl = 0;
    double qpe = 0;
    if (ref) {
        q.n_pairs = g.n_near;
        q.first = 0;
        q.list = g.near_list.as<int2>();
        q.P = g.NsN * g.Nq2;
        q.pts = g.near_pts.as<double4>();
        q.aeq = g.aeq.as<double>();
        q.near_alpha = g.near_alpha;
        if (g.n_near > 0) {
            EFIE_TRY(launch_pairs<SP_NEAR>(q, inv, N, nsp, g.ser_sp.as<double>(), s));
            nl++;
            qpe += (double)q.n_pairs * q.P * q.P;
        }
        q.n_pairs = g.Nt;
        q.first = g.n_near;
        q.P = g.NsS * g.Nq2;
        q.per_sub = g.Nq2;
        q.pts = g.self_pts.as<double4>();
        q.self_a = g.self_a.as<double>();
        q.NsS = g.NsS;
        EFIE_TRY(launch_pairs<SP_SELF>(q, inv, N, nsp, g.ser_sp.as<double>(), s));
        nl++;
        qpe += (double)q.n_pairs * q.P * q.P;
    } else if (g.n_adj > 0) {
        q.n_pairs = g.n_adj;
        q.list = g.adj_list.as<int2>();
        q.P = g.Nq;
        q.pts = g.reg_pts.as<double4>();
        q.vtx = g.tri_vtx.as<double4>();
        k_series_adjacent<<<dim3((g.n_adj + 1) / 2, (N + 7) / 8), 64, 0, s>>>(q, inv, N, nsp, g.ser_sp.as<double>());
        nl++;
        qpe += (double)q.n_pairs * q.P * (q.P + 1);
    }
    EFIE_CUDA(cudaGetLastError());
    ctx->log.end(EFIE_K_NEARSELF, s, tok, qpe, nl);
    *use = true;
    return EFIE_OK;
}

efie_status efie_series_assemble(efie_ctx *ctx, GeomDev &g, const Physics *ph, int nf, void *Z, size_t zstride,
                                 const PlanesOut *po) {
    const int N = g.ser_n;
    const int cs = CF + 2 * N;
    std::vector<double> c((size_t)nf * cs, 0.0);
    bool lossy = false, even = nf > 2;
    for (int f = 0; f < nf; f++) {
        double *r = c.data() + (size_t)f * cs;
        r[0] = ph[f].kr; r[1] = ph[f].ki;
        r[2] = ph[f].alr; r[3] = ph[f].ali; r[4] = ph[f].ber; r[5] = ph[f].bei;
        coefficients(N, std::complex<double>(ph[f].kr, ph[f].ki) * g.ser_delta, r + CF);
        lossy = lossy || ph[f].ki != 0.0;
    }
    // k_f = k_{f-1} + dk to rounding, so that the step's phase carries over
    for (int f = 1; f < nf && even; f++) {
        const double er = ph[f].kr - ph[f - 1].kr - (ph[1].kr - ph[0].kr);
        const double ei = ph[f].ki - ph[f - 1].ki - (ph[1].ki - ph[0].ki);
        if (std::hypot(er, ei) > 1e-15 * std::hypot(ph[f].kr, ph[f].ki)) even = false;
    }
    EFIE_TRY(g.ser_coef.reserve(sizeof(double) * c.size()));
    EFIE_CUDA(cudaMemcpyAsync(g.ser_coef.p, c.data(), sizeof(double) * c.size(), cudaMemcpyHostToDevice, ctx->stream));
    double *mom = g.moments.as<double>();
    for (size_t t0 = 0; t0 < g.ser_tiles; t0 += g.ser_cap) {
        const int nt = (int)std::min(g.ser_cap, g.ser_tiles - t0);
        EFIE_TRY(with_terms(N, [&](auto n) -> efie_status {
            constexpr int M = decltype(n)::value;
            if (!g.ser_done) EFIE_TRY(launch_tiles<M>(ctx, g, (int)t0, nt, mom));
            return launch_eval<M>(ctx, g, (int)t0, nt, mom, nf, lossy, even, Z, zstride, po);
        }));
    }
    if (g.ser_cap >= g.ser_tiles) g.ser_done = true;   // every later batch reads the stored moments
    return EFIE_OK;
}
