// Initial guesses of a batch from the solutions of the sweep's solved
// frequencies (snapshots).
//
// The currents of a sweep move in a space of few dimensions, so the combination
// of the nearest snapshots x_j that minimises || b - Z(f) sum c_j x_j || starts
// the refinement of frequency f far below any fixed interpolation weights:
// measured (Ne 1074, 2-3 GHz, snapshots 60 MHz apart solved to 1e-10), four
// snapshots leave 3e-5 of ||b||, eight 4e-10 and twelve 1e-11, where the
// quadratic through three leaves 5e-3.  From twelve on most frequencies meet
// the residual target before their first GMRES step.
//
//   W = Z(f) [x_1 .. x_k]   one product kernel for all vectors (k_symv_multi)
//   [W b] = Q R             tall-skinny Householder QR, two launches
//   c = R^-1 Q^H b          (nearly dependent columns get c = 0), x0 = sum c_j x_j
// The Householder form keeps the digits that the snapshots' near dependence
// would cost the normal equations; the refinement then starts from the true
// residual of x0, so the guess never decides what counts as solved.
#include <algorithm>
#include <vector>

#include "efie_internal.h"
#include "solve.h"
#include "tma.h"
#include "warp.cuh"

namespace {

using namespace efie_tma;

constexpr int KMAX = EFIE_SNAP_MAX;   // snapshots per frequency
// columns of [W b] in the QR: 16 (up to 15 snapshots) or 24
static_assert(KMAX == 23, "the wider QR holds 24 columns");

// ---------------------------------------------------------------------------
// W_f = Z_f X_f for up to 8 NG vectors, Z symmetric (upper triangle and full
// 128 x 128 diagonal blocks stored).  An item is a block of 128 rows I of one
// frequency: its y_I stays in registers over all blocks J, from tile (I, J)
// as stored for J >= I and from the stored tile (J, I) transposed below, so
// there are no partial vectors and no sums across tiles; Z is read twice
// (once from L2 where the two readers meet), which the FP64 pipe hides: a
// 64 KB chunk of 16 vectors costs 2048 multiply-adds per lane of the SM's 128.
// Chunks are 32 of the contraction's entries, through a ring of three stages:
// boxes of 8 rows (128 bytes) in the 128-byte swizzle.
// The products are FP64 matrix instructions (16 x 8 x 8): warp w forms rows
// 16 (w & 7) .. + 15 of eight vectors, four products per step (re re, re im,
// -im im, im re) from six shared-memory reads, where a lane that forms its
// own row reads every vector's entry for four multiply-adds.  Row r of an
// eight-row box is held by lane group 2 (r & 3) + (r >> 2), so that the eight
// lanes of a shared-memory phase (two groups x four contraction entries) meet
// eight different 16-byte banks of the swizzle, as stored and transposed;
// the vectors' slices are 64 bytes apart modulo 128 for the same reason.
// One more warp issues the copies.  Bound by the FP64 pipe: Ne 6968, 22
// frequencies, 15 vectors: 5.05 ms, 76 % of it (nine rounds of items over the
// SMs where 8.2 would do); one row per lane of sixteen warps with plain
// multiply-adds took 7.3 ms.
// ---------------------------------------------------------------------------
constexpr int MB = 128;                             // rows per item
constexpr int MC = 32;                              // contraction entries per chunk
constexpr int MR = 3;                               // stages
constexpr uint32_t MZ = MB * MC * sizeof(double2);  // 64 KB of Z per chunk
constexpr uint32_t MX = MC * sizeof(double2) + 64;  // one vector's slice

template <int NG>   // the swizzle follows address bits: stages start on 1024 bytes
constexpr uint32_t multi_stage = (MZ + 8 * NG * MX + 1023u) & ~1023u;
template <int NG>
constexpr size_t multi_smem = MR * (size_t)multi_stage<NG> + 1024 + 64;

// d += a b on 16 x 8 x 8: a row major, b column major
__device__ __forceinline__ void dmma(double (&d)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

struct SnapIdx {
    const int *k;     // [nf] snapshots of each frequency
    const int *pos;   // [nf][KMAX] their rows of xall, nearest first
};   // a launch takes vectors v0 .. v0 + 8 NG - 1 into those columns of W [nf][ldw][N]

template <int NG>
__global__ void __launch_bounds__(256 * NG + 32, 1) k_symv_multi(const __grid_constant__ CUtensorMap dmap,
                                                       const __grid_constant__ CUtensorMap tmap, int N, int nb, int nf,
                                                       const double2 *__restrict__ xall, const SnapIdx S,
                                                       double2 *__restrict__ W, int v0, int ldw, char *ctl) {
    extern __shared__ unsigned char dsm[];
    __shared__ int fail;
    constexpr int K = 8 * NG, MT = 256 * NG + 32;
    constexpr uint32_t STAGE = multi_stage<NG>;
    unsigned char *ring = dsm + (((smem_u32(dsm) + 1023u) & ~1023u) - smem_u32(dsm));
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + MR * STAGE);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool feeder = warp == 8 * NG;   // the last warp issues the copies
    const int G = gridDim.x, items = nb * nf;
    // slices past row N are not copied: what a stage holds there must be finite
    constexpr int NX = K * (int)(MX / sizeof(double2));
    for (int i = tid; i < MR * NX; i += MT)
        reinterpret_cast<double2 *>(ring + (i / NX) * STAGE + MZ)[i % NX] = make_double2(0.0, 0.0);
    int p_it = blockIdx.x, p_q = 0, issued = 0;   // producer (feeder's lane 0): chunk p_q of item p_it is next
    auto produce = [&]() {
        if (p_it >= items) return;
        const int f = p_it / nb, I = p_it - f * nb, J = p_q >> 2, n0 = J * MB + (p_q & 3) * MC;
        unsigned char *st = ring + (issued % MR) * STAGE;
        uint64_t *bar = full + issued % MR;
        const int kf = min(K, max(0, S.k[f] - v0)), cnt = max(0, min(MC, N - n0));
        mbar_expect_tx(bar, MZ + (uint32_t)(kf * cnt) * sizeof(double2));
        if (J >= I)
            for (int b = 0; b < MB / 8; b++) tma_load_3d(&dmap, st + b * 4096, 2 * (I * MB + 8 * b), n0, f, bar);
        else
            for (int b = 0; b < MC / 8; b++) tma_load_3d(&tmap, st + b * 16384, 2 * (n0 + 8 * b), I * MB, f, bar);
        if (cnt > 0)
            for (int v = 0; v < kf; v++)
                bulk_g2s(st + MZ + v * MX, xall + (size_t)N * S.pos[f * KMAX + v0 + v] + n0,
                         (uint32_t)cnt * sizeof(double2), bar);
        issued++;
        if (++p_q == 4 * nb) p_q = 0, p_it += G;
    };
    if (tid == 0) {
        for (int s = 0; s < MR; s++) mbar_init(full + s, 1);
        mbar_init_fence();
        fail = 0;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the zeros before the copies
    __syncthreads();
    if (feeder && lane == 0)
        for (int s = 0; s < MR; s++) produce();
    const int g = lane >> 2, t = lane & 3, row = (g & 1) * 4 + (g >> 1), w8 = warp & 7, v8 = 8 * (warp >> 3);
    int cc = 0;
    for (int it = blockIdx.x; it < items; it += G) {
        const int f = it / nb, I = it - f * nb;
        double yr[4] = {0.0, 0.0, 0.0, 0.0}, yi[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
        for (int q = 0; q < 4 * nb; q++) {
            if (!feeder && !mbar_wait_bounded(full + cc % MR, (uint32_t)(cc / MR) & 1u)) fail = 1;
            const unsigned char *st = ring + (cc % MR) * STAGE;
            if (!feeder && __all_sync(0xffffffffu, !fail)) {   // matrix instructions want whole warps
                const unsigned char *X = st + MZ + (v8 + g) * MX + t * sizeof(double2);
                // rows r and r + 8 of the warp, contraction entries c = 8 k + t and + 4: box,
                // row and 16-byte chunk of the swizzle as stored, or transposed (block-uniform)
                const bool direct = (q >> 2) >= I;
                const unsigned char *zb = direct ? st + w8 * 8192 + t * 128 : st + (16 * w8 + row) * 128;
                const int r8 = direct ? 4096 : 1024, c4 = direct ? 512 : 0, c8 = direct ? 1024 : 16384;
                const int x0 = (row ^ t) << 4, x4 = x0 ^ 64;
#pragma unroll
                for (int k = 0; k < MC / 8; k++) {
                    const unsigned char *p = zb + k * c8;
                    const double2 a0 = *reinterpret_cast<const double2 *>(p + x0);
                    const double2 a1 = *reinterpret_cast<const double2 *>(p + r8 + x0);
                    const double2 a2 = *reinterpret_cast<const double2 *>(p + c4 + x4);
                    const double2 a3 = *reinterpret_cast<const double2 *>(p + r8 + c4 + x4);
                    const double2 b0 = *reinterpret_cast<const double2 *>(X + k * 128);
                    const double2 b1 = *reinterpret_cast<const double2 *>(X + k * 128 + 64);
                    const double zr[4] = {a0.x, a1.x, a2.x, a3.x}, zi[4] = {a0.y, a1.y, a2.y, a3.y};
                    const double xr[2] = {b0.x, b1.x}, xi[2] = {b0.y, b1.y}, xn[2] = {-b0.y, -b1.y};
                    dmma(yr, zr, xr);
                    dmma(yi, zr, xi);
                    dmma(yr, zi, xn);
                    dmma(yi, zi, xr);
                }
            }
            __syncthreads();   // every warp is done with the stage
            if (fail) {
                // a chunk never arrived: every frequency of the launch falls back
                if (tid < nf) atomicExch(reinterpret_cast<int *>(ctl + 64 * tid + 36), 3);
                if (feeder && lane == 0)
                    for (int k = cc + 1; k < issued; k++)
                        if (!mbar_wait_bounded(full + k % MR, (uint32_t)(k / MR) & 1u)) break;
                return;
            }
            if (feeder && lane == 0) produce();
            cc++;
        }
        if (feeder) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int m = I * MB + 16 * w8 + 8 * (i >> 1) + row, v = v0 + v8 + 2 * t + (i & 1);
            if (m < N && v < ldw) W[((size_t)f * ldw + v) * N + m] = make_double2(yr[i], yi[i]);
        }
    }
}

// ---------------------------------------------------------------------------
// Householder reduction of a block of 256 rows x QC complex columns, one row
// per thread in registers: afterwards threads 0..QC-1 hold the rows of R.  Per
// column one reduction gives x^H a_c of every column; with v = x - alpha e_j
// (alpha opposite to the pivot), v^H a_c = x^H a_c - conj(alpha) a_jc.
// ---------------------------------------------------------------------------
template <int QC>
struct QrSmem {
    double part[8][2 * QC];
    double sum[2 * QC];
    double2 piv[QC];
};

// x^H a_c over the warp for the n / 2 columns from c0 on
template <int n, int QC>
__device__ __forceinline__ double column_dots(const double2 (&a)[QC], double2 x, int c0, bool on, int lane) {
    double d[n];
#pragma unroll
    for (int c = 0; c < n / 2; c++) {
        const double2 y = a[c0 + c];
        d[2 * c] = on ? x.x * y.x + x.y * y.y : 0.0;
        d[2 * c + 1] = on ? x.x * y.y - x.y * y.x : 0.0;
    }
    return warp_sums<n>(d, lane);
}

template <int QC>
__device__ __forceinline__ void householder(double2 (&a)[QC], QrSmem<QC> &S) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int j = 0; j < QC - 1; j++) {
        const bool on = tid >= j;
        // columns before j are finished; their sums are not used
        S.part[warp][lane] = column_dots<32>(a, a[j], 0, on, lane);
        if (QC == 24) {
            const double d = column_dots<16>(a, a[j], QC - 8, on, lane);
            if (lane < 16) S.part[warp][2 * QC - 16 + lane] = d;
        }
        if (tid == j)
#pragma unroll
            for (int c = 0; c < QC; c++) S.piv[c] = a[c];
        __syncthreads();
        if (tid < 2 * QC) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < 8; w++) s += S.part[w][tid];
            S.sum[tid] = s;
        }
        __syncthreads();
        const double n2 = S.sum[2 * j];
        if (n2 > 0.0) {   // uniform
            const double nrm = sqrt(n2), ap = hypot(S.piv[j].x, S.piv[j].y);
            const double2 u = ap > 0.0 ? make_double2(S.piv[j].x / ap, S.piv[j].y / ap) : make_double2(1.0, 0.0);
            const double2 alpha = make_double2(-u.x * nrm, -u.y * nrm);
            const double tau = 1.0 / (nrm * (nrm + ap));
            const double2 v = tid == j ? make_double2(a[j].x - alpha.x, a[j].y - alpha.y) : a[j];
            if (on) {
#pragma unroll
                for (int c = j + 1; c < QC; c++) {
                    const double2 p = S.piv[c];
                    const double wr = tau * (S.sum[2 * c] - (alpha.x * p.x + alpha.y * p.y));
                    const double wi = tau * (S.sum[2 * c + 1] - (alpha.x * p.y - alpha.y * p.x));
                    a[c].x -= v.x * wr - v.y * wi;
                    a[c].y -= v.x * wi + v.y * wr;
                }
                a[j] = tid == j ? alpha : make_double2(0.0, 0.0);
            }
        }
        __syncthreads();   // sum, piv and part are free for the next column
    }
}

// R of each block of 256 rows of [W b]: R[f][block][QC][QC]
template <int QC>
__global__ void __launch_bounds__(256) k_tsqr_local(int N, int ldw, const int *__restrict__ kf,
                                                    const double2 *__restrict__ W, const double2 *__restrict__ b,
                                                    double2 *__restrict__ R) {
    __shared__ QrSmem<QC> S;
    const int f = blockIdx.y, n = blockIdx.x * 256 + threadIdx.x, k = kf[f];
    double2 a[QC];
#pragma unroll
    for (int c = 0; c < QC - 1; c++)
        a[c] = n < N && c < k ? W[((size_t)f * ldw + c) * N + n] : make_double2(0.0, 0.0);
    a[QC - 1] = n < N ? b[n] : make_double2(0.0, 0.0);
    householder<QC>(a, S);
    if (threadIdx.x < QC) {
        double2 *out = R + (((size_t)f * gridDim.x + blockIdx.x) * QC + threadIdx.x) * QC;
#pragma unroll
        for (int c = 0; c < QC; c++) out[c] = a[c];
    }
}

// The blocks' R stacked below the result so far and reduced, as many as 256
// rows hold at a time, then the coefficients coef[f][KMAX] by back
// substitution; a column that depends on the ones before it to 1e-13 of its
// norm gets none.
template <int QC>
__global__ void __launch_bounds__(256) k_tsqr_combine(int nblk, const int *__restrict__ kf,
                                                      const double2 *__restrict__ R, double2 *__restrict__ coef) {
    __shared__ QrSmem<QC> S;
    __shared__ double2 T[QC][QC];
    const int f = blockIdx.x, tid = threadIdx.x;
    constexpr int PASS = 256 / QC - 1;
    double2 a[QC];
#pragma unroll
    for (int c = 0; c < QC; c++) a[c] = make_double2(0.0, 0.0);
    for (int b0 = 0; b0 < nblk; b0 += PASS) {
        const int p = tid / QC - 1, blk = b0 + p, row = tid % QC;
        if (tid >= QC) {
            const bool in_range = p < PASS && blk < nblk;
            const double2 *in = R + (((size_t)f * nblk + (in_range ? blk : 0)) * QC + row) * QC;
#pragma unroll
            for (int c = 0; c < QC; c++) a[c] = in_range ? in[c] : make_double2(0.0, 0.0);
        }
        householder<QC>(a, S);
    }
    if (tid < QC)
#pragma unroll
        for (int c = 0; c < QC; c++) T[tid][c] = a[c];
    __syncthreads();
    if (tid == 0) {
        double2 x[QC - 1];
        const int k = kf[f];
        for (int j = QC - 2; j >= 0; j--) {
            double2 s = T[j][QC - 1];
            double col = 0.0;
            for (int i = 0; i <= j; i++) col += T[i][j].x * T[i][j].x + T[i][j].y * T[i][j].y;
            for (int i = j + 1; i < k; i++) {
                s.x -= T[j][i].x * x[i].x - T[j][i].y * x[i].y;
                s.y -= T[j][i].x * x[i].y + T[j][i].y * x[i].x;
            }
            const double2 d = T[j][j];
            const double dn = d.x * d.x + d.y * d.y;
            x[j] = j < k && dn > 1e-26 * col
                       ? make_double2((s.x * d.x + s.y * d.y) / dn, (s.y * d.x - s.x * d.y) / dn)
                       : make_double2(0.0, 0.0);
            if (j < k) coef[f * KMAX + j] = x[j];
        }
    }
}

// x_f = sum_j c_j x_j
__global__ void __launch_bounds__(256) k_snap_x(int N, const double2 *__restrict__ xall, const SnapIdx S,
                                                const double2 *__restrict__ coef, double2 *__restrict__ x) {
    const int f = blockIdx.y, n = blockIdx.x * 256 + threadIdx.x;
    if (n >= N) return;
    double2 s = make_double2(0.0, 0.0);
    const int k = S.k[f];
    for (int j = 0; j < k; j++) {
        const double2 c = coef[f * KMAX + j], v = xall[(size_t)N * S.pos[f * KMAX + j] + n];
        s.x += c.x * v.x - c.y * v.y;
        s.y += c.x * v.y + c.y * v.x;
    }
    x[(size_t)N * f + n] = s;
}

// The two maps of Z (all slots) as doubles [B][N][2N]: boxes of 8 rows x 32
// columns (tiles as stored) and 8 rows x 128 columns (tiles read transposed)
efie_status multi_maps(int N, int B, const void *Z, size_t zstride, CUtensorMap *d, CUtensorMap *t) {
    const cuuint64_t dims[3] = {2 * (cuuint64_t)N, (cuuint64_t)N, (cuuint64_t)B};
    const cuuint64_t strides[2] = {sizeof(double2) * (cuuint64_t)N, sizeof(double2) * (cuuint64_t)zstride};
    const cuuint32_t bd[3] = {16, MC, 1}, bt[3] = {16, MB, 1};
    EFIE_TRY(efie_encode_tiled(d, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void *>(Z), dims, strides, bd,
                               CU_TENSOR_MAP_SWIZZLE_128B));
    return efie_encode_tiled(t, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void *>(Z), dims, strides, bt,
                             CU_TENSOR_MAP_SWIZZLE_128B);
}

template <int NG>
efie_status launch_multi(efie_ctx *ctx, const CUtensorMap &d, const CUtensorMap &t, int N, int nf,
                         const double2 *xall, const SnapIdx &S, double2 *W, int v0, int ldw, char *ctl) {
    const int nb = (N + MB - 1) / MB;
    EFIE_CUDA(cudaFuncSetAttribute(k_symv_multi<NG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)multi_smem<NG>));
    k_symv_multi<NG><<<std::min(ctx->num_sms, nb * nf), 256 * NG + 32, multi_smem<NG>, ctx->stream>>>(d, t, N, nb, nf, xall, S, W,
                                                                                           v0, ldw, ctl);
    return efie_cuda_check(cudaGetLastError(), "snapshot products");
}

}  // namespace

efie_status efie_snapshot_guess(efie_ctx *ctx, SolveWork &w, const void *Z, size_t zstride, const void *xall,
                                const void *b, int nf, const SnapSpec &spec, void *x) {
    cudaStream_t s = ctx->stream;
    const int N = w.N, nblk = (N + 255) / 256;
    int kmax = 0;
    for (int f = 0; f < nf; f++) kmax = std::max(kmax, spec.k[f]);
    if (nf < 1 || kmax < 1 || kmax > KMAX) return efie_fail(EFIE_ERR_ARGS, "snapshot guess: bad snapshot count");
    // up to eight or sixteen vectors per product launch
    const int ldw = kmax <= 8 ? 8 : kmax <= 15 ? 15 : 23;
    const int QC = ldw <= 15 ? 16 : 24;
    // W [nf][ldw][N], R [nf][nblk][QC][QC], coefficients [nf][KMAX], spec
    const size_t nW = (size_t)nf * ldw * N, nR = (size_t)nf * nblk * QC * QC, nC = (size_t)nf * KMAX;
    EFIE_TRY(w.snap.reserve(sizeof(double2) * (nW + nR + nC) + sizeof(SnapSpec)));
    double2 *W = w.snap.as<double2>(), *R = W + nW, *coef = R + nR, *xd = static_cast<double2 *>(x);
    int *dspec = reinterpret_cast<int *>(coef + nC);
    EFIE_CUDA(cudaMemcpyAsync(dspec, &spec, sizeof(SnapSpec), cudaMemcpyHostToDevice, s));
    const SnapIdx S{dspec, dspec + EFIE_MAX_BATCH};
    const double2 *xa = static_cast<const double2 *>(xall), *bd = static_cast<const double2 *>(b);
    CUtensorMap d, t;
    EFIE_TRY(multi_maps(N, w.B, Z, zstride, &d, &t));
    size_t tok = ctx->log.begin(s);
    char *ctl = w.ctl.as<char>();
    if (ldw > 8)
        EFIE_TRY(launch_multi<2>(ctx, d, t, N, nf, xa, S, W, 0, ldw, ctl));
    if (ldw != 15)
        EFIE_TRY(launch_multi<1>(ctx, d, t, N, nf, xa, S, W, ldw > 8 ? 16 : 0, ldw, ctl));
    const int nprod = ldw > 15 ? 2 : 1;
    ctx->log.end(EFIE_K_RESIDUAL, s, tok, nprod * 8.0 * (double)N * N * nf, nprod);
    tok = ctx->log.begin(s);
    const dim3 rows(nblk, nf);
    if (QC == 16) {
        k_tsqr_local<16><<<rows, 256, 0, s>>>(N, ldw, S.k, W, bd, R);
        k_tsqr_combine<16><<<nf, 256, 0, s>>>(nblk, S.k, R, coef);
    } else {
        k_tsqr_local<24><<<rows, 256, 0, s>>>(N, ldw, S.k, W, bd, R);
        k_tsqr_combine<24><<<nf, 256, 0, s>>>(nblk, S.k, R, coef);
    }
    k_snap_x<<<rows, 256, 0, s>>>(N, xa, S, coef, xd);
    EFIE_CUDA(cudaGetLastError());
    ctx->log.end(EFIE_K_OTHER, s, tok, 0.0, 3);
    return EFIE_OK;
}

// Test entries: guesses from host arrays (Z column-major N x N, xs [nx][N]).
extern "C" efie_status efie_debug_snapshot_guesses(efie_ctx *ctx, int32_t N, int32_t nf, int32_t nx, const int32_t *k,
                                                   const int32_t *pos, const efie_c128 *Z, const efie_c128 *xs,
                                                   const efie_c128 *b, efie_c128 *x) {
    if (!ctx || N < 1 || nf < 1 || nf > EFIE_MAX_BATCH || nx < 1 || !k || !pos || !Z || !xs || !b || !x)
        return efie_fail(EFIE_ERR_ARGS, "efie_debug_snapshot_guesses: bad arguments");
    SnapSpec sp{};
    for (int f = 0; f < nf; f++) {
        sp.k[f] = k[f];
        bool ok = k[f] >= 1 && k[f] <= KMAX;
        for (int j = 0; ok && j < k[f]; j++) {
            sp.pos[f][j] = pos[f * KMAX + j];
            ok = sp.pos[f][j] >= 0 && sp.pos[f][j] < nx;
        }
        if (!ok) return efie_fail(EFIE_ERR_ARGS, "efie_debug_snapshot_guesses: bad snapshot list");
    }
    DeviceGuard dg(ctx->device);
    ctx->log.reset(false);
    cudaStream_t s = ctx->stream;
    SolveWork w;
    w.N = N;
    w.B = nf;
    EFIE_TRY(w.ctl.reserve(64 * (size_t)nf));
    EFIE_CUDA(cudaMemsetAsync(w.ctl.p, 0, 64 * (size_t)nf, s));
    DevBuf dZ, dx, db, dg0;
    const size_t v = sizeof(efie_c128) * (size_t)N;
    EFIE_TRY(dZ.reserve(v * N * nf));
    EFIE_TRY(dx.reserve(v * nx));
    EFIE_TRY(db.reserve(v));
    EFIE_TRY(dg0.reserve(v * nf));
    EFIE_CUDA(cudaMemcpyAsync(dZ.p, Z, v * N * nf, cudaMemcpyHostToDevice, s));
    EFIE_CUDA(cudaMemcpyAsync(dx.p, xs, v * nx, cudaMemcpyHostToDevice, s));
    EFIE_CUDA(cudaMemcpyAsync(db.p, b, v, cudaMemcpyHostToDevice, s));
    EFIE_TRY(efie_snapshot_guess(ctx, w, dZ.p, (size_t)N * N, dx.p, db.p, nf, sp, dg0.p));
    std::vector<char> ctl(64 * (size_t)nf);
    EFIE_CUDA(cudaMemcpyAsync(ctl.data(), w.ctl.p, ctl.size(), cudaMemcpyDeviceToHost, s));
    EFIE_CUDA(cudaMemcpyAsync(x, dg0.p, v * nf, cudaMemcpyDeviceToHost, s));
    EFIE_CUDA(cudaStreamSynchronize(s));
    for (int f = 0; f < nf; f++)
        if (*reinterpret_cast<const int *>(ctl.data() + 64 * f + 36))
            return efie_fail(EFIE_ERR_TIMEOUT, "efie_debug_snapshot_guesses: device error flag");
    return EFIE_OK;
}

extern "C" efie_status efie_debug_snapshot_guess(efie_ctx *ctx, int32_t N, int32_t k, const efie_c128 *Z,
                                                 const efie_c128 *xs, const efie_c128 *b, efie_c128 *x) {
    int32_t pos[KMAX];
    for (int j = 0; j < KMAX; j++) pos[j] = j;
    return efie_debug_snapshot_guesses(ctx, N, 1, k, &k, pos, Z, xs, b, x);
}
