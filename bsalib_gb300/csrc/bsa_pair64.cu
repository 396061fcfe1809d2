// bsa_pair64.cu -- the Classic FP64 analysis over distinct frequency pairs.
//
// Every nodal quantity of the path depends on |f| (the spectra and c^|f|), so on the grid
// f_i = i df, i = -N .. N, A(f_i) = A(f_-i): N + 1 distinct rows.  With
// E(x, y)[(a, b), j] = sum_k Q[k][a] A(x)[k][b] A(y)[k][j], the three terms of the BFM at a grid
// point (functionsImpl.F90:1494-1538) are elements of E at two of |f1|, |f2|, |f1 + f2|
//   T1(f1, f2)[m, n, o] = E(f1, f2)[(m, n), o]
//   T2(f1, f2)[m, n, o] = E(f1 + f2, f2)[(n, m), o]
//   T3(f1, f2)[m, n, o] = E(f1, f1 + f2)[(o, n), m]
// and E(x, y)[(a, b), j] = E(y, x)[(a, j), b].  The whole grid therefore needs E(x, y) for
// 0 <= x <= y only: (N + 1)(N + 2) / 2 products of 2 K NM^3 flop instead of (2 N + 1)^2 points of
// 4 K NM^3 (one sixteenth of the flop; GB300 issues two FP64 FMAs an SM and clock, so the flop
// count is the time).  The analytic S(f1 + f2) (classic_trunc off) adds the rows N + 1 .. 2 N and
// the pairs (x, y) with y > N, y - x <= N.
//
// The products go to HBM in chunks of first rows x (k_pair_gemm), then k_pair_moments adds each
// element into the third moments with the FRF products and weights of every grid point that reads
// it.  B(-f1, -f2) = B(f1, f2) on the grid, so half of the points stand for both (weight 2).
// With Hx = H(x), Hy = H(y), P = H(x + y), D = H(y - x) and, per row (a, b) and column j,
//   alpha = Re[Hx_a Hy_b conj P_j],  beta = Re[Hx_a conj Hy_b D_j],
//   gamma = Re[Hy_a conj P_b Hx_j],  delta = Re[Hy_a conj D_b conj Hx_j]
// the twelve contributions of an element are
//   T1 at (x, +-y):      (m, n, o) = (a, b, j)   w1 (alpha + beta)
//   T1 at (y, +-x):                  (a, j, b)   w1 (gamma + delta)
//   T2 at (x -+ y, +-y):             (b, a, j)   w2m gamma + w2p delta
//   T3 at (y, +-x - y):              (b, j, a)   w2m alpha + w2p beta
//   T3 at (x, +-y - x):              (j, b, a)   w3m gamma + w3p delta
//   T2 at (y -+ x, +-x):             (j, a, b)   w3m alpha + w3p beta
// with w1 the weight of the grid points (x, +-y), w2p / w2m of (x - y, y) / (x + y, -y) and
// w3p / w3m of (x, y - x) / (x, -x - y), zero beyond the grid (two contributions share a weight
// because the weights are symmetric under f1 <-> f2 and under the central symmetry).  A product
// with x = y feeds all at half weight (its transpose is in the same product), x = 0 has no minus
// partners.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/bsa_gpu.h"
#include "bsa_engine.cuh"
#include "bsa_kernels.cuh"
#include "bsa_pair64.cuh"

namespace bsa {
namespace p64 {

constexpr int kKT = 16;
constexpr int kKinds = 9;           // K1 .. K6 (the order above: abj, ajb, baj, jba, jab, bja), M1, M2, M3
constexpr int kBatch = 8;           // pairs a thread takes between two barriers
constexpr int kRow = 10;            // doubles of a row's factors

// E of one product tile, or of a quarter of its rows: 256 threads, ROWS / 32 x 4 elements each, K staged
// 16 at a time; the row operand Q[k][a] A(x)[k][b] is formed while staging.  FP64-pipe bound (one
// product in 32 for the staging); a problem of few tiles spreads over more SMs by quarters (the
// 30-node tower's 45 tiles: 40 -> 20 us).
template <int ROWS>
__global__ __launch_bounds__(256) void k_pair_gemm(Chunk c, const double *__restrict__ A, const double *__restrict__ Q) {
    after_previous();
    constexpr int RPT = ROWS / 32, KS = 256 / ROWS;
    __shared__ double As[kKT][ROWS], Bs[kKT][kTN];
    const int t = threadIdx.x, qn = c.qn, an = c.an, rx = c.rx(), K = c.K;
    const long long item = blockIdx.x;
    const int lo = tile_row(c, item);
    const RowTile rt = c.rt[lo];
    const int ct = rt.ct0 + (int)(item - rt.item0);
    const int rt0 = blockIdx.y * ROWS, r0 = lo * kTM + rt0, rows = (c.x1 - c.x0) * rx;
    // this thread's staging row and column
    const int sr = t % ROWS, kr = t / ROWS;              // As: KS k rows of ROWS rows at a time
    const bool rv = r0 + sr < rows;
    const int rr = rv ? r0 + sr : 0, x = c.x0 + rr / rx, ab = rr % rx, a = ab / an, b = ab % an;
    const double *Qa = Q + a, *Ab = A + (size_t)x * K * an + b;
    const int sc = t & (kTN - 1), kc = t >> 5;           // Bs: 8 k rows of 32 columns at a time
    const int col = ct * kTN + sc, y = col / an, j = col - y * an;
    const bool cv = y <= c.hi;
    const double *Aj = A + (size_t)(cv ? y : 0) * K * an + j;
    const int tr = (t >> 3) * RPT, tc = (t & 7) * 4;
    double acc[RPT][4];
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = 0.0;
    for (int k0 = 0; k0 < K; k0 += kKT) {
        const int kn = min(kKT, K - k0);
#pragma unroll
        for (int u = 0; u < kKT / KS; ++u) {
            const int k = kr + KS * u;
            As[k][sr] = (rv && k < kn) ? Qa[(size_t)(k0 + k) * qn] * Ab[(size_t)(k0 + k) * an] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kKT / 8; ++u) {
            const int k = kc + 8 * u;
            Bs[k][sc] = (cv && k < kn) ? Aj[(size_t)(k0 + k) * an] : 0.0;
        }
        __syncthreads();
        for (int k = 0; k < kn; ++k) {
            double ar[RPT], br[4];
#pragma unroll
            for (int i = 0; i < RPT; ++i) ar[i] = As[k][tr + i];
#pragma unroll
            for (int q = 0; q < 4; ++q) br[q] = Bs[k][tc + q];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[i][q] = fma(ar[i], br[q], acc[i][q]);
        }
        __syncthreads();
    }
    const size_t ld = (size_t)rt.nct * kTN;
    double *out = c.E + rt.base + (size_t)(ct - rt.ct0) * kTN + tc;
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) out[(size_t)(rt0 + tr + i) * ld + q] = acc[i][q];
}

// H of the kept modes at i df, i = 0 .. 2 N.
__global__ void k_frf_rows(int n, int nm, double df, FrfPar frf, double2 *__restrict__ H) {
    after_previous();
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n * nm) return;
    const int m = u % nm;
    double hr, hi;
    frf_eval(frf.M[m], frf.K[m], frf.C[m], (double)(u / nm) * df * kPi2, hr, hi);
    H[u] = make_double2(hr, hi);
}

struct MomPar {
    int N, vect;            // vect: edge weights of intgSpectraVect_, else uniform
    long long npairs;       // pairs (x, y) of the chunk
    const long long *pre;   // pairs before first row x0 + i, and the total
    const double2 *H;       // [2 N + 1][nm]
    double *part;           // [groups][kKinds][nm^2][nm]
    int first;              // first chunk: the partials are written, not added to
    int RT, PL, PB;         // rows (a, b) of a block, pair lanes, pairs of a batch (at most kBatch PL)
};

// Relative weight of grid point (i1, i2) (BsaClassicImpl.F90:596-632, vertex -1/2), 0 beyond it.
template <typename T>
__device__ __forceinline__ T wrel(int i1, int i2, int N, int vect) {
    const int u = abs(i1), v = abs(i2);
    if (u > N || v > N) return T(0);
    if (!vect) return T(1);
    return u == N ? (v == N ? T(-0.5) : T(0.5)) : (v == N ? T(0.5) : T(1));
}

// T: double, or float where the weights (multiples of 1/8, exact in either) are formed per element
template <typename T>
struct PairWeights {
    int x, y, region;        // 0: every weight 1; 1: w1 = w2p = w3p = 1, w2m = w3m = 0; 2: general
    T w1, w2p, w2m, w3p, w3m, wm1, wm2, wm3;
};

using PairInfo = PairWeights<double>;

template <typename T>
__device__ __forceinline__ PairWeights<T> pair_info(int x, int y, int N, int vect) {
    PairWeights<T> f;
    f.x = x;
    f.y = y;
    const T s = (x == y ? T(0.5) : T(1)) * (x == 0 && y == 0 ? T(0.5) : T(1)), sm = x == 0 ? T(0) : s;
    // plus partners (x, y), (x - y, y), (x, y - x); minus partners (x, -y), (x + y, -y), (x, -x - y)
    const T a1 = wrel<T>(x, y, N, vect);
    f.w1 = s * a1;
    f.w2p = s * wrel<T>(x - y, y, N, vect);
    f.w3p = s * wrel<T>(x, y - x, N, vect);
    f.w2m = sm * wrel<T>(x + y, y, N, vect);
    f.w3m = sm * wrel<T>(x, x + y, N, vect);
    f.wm1 = f.w1 + sm * a1;
    f.wm2 = f.w2p + f.w2m;
    f.wm3 = f.w3p + f.w3m;
    f.region = 2;
    if (x > 0 && x < y && f.w1 == T(1) && f.w2p == T(1) && f.w3p == T(1)) {
        if (f.w2m == T(1) && f.w3m == T(1)) f.region = 0;
        else if (f.w2m == T(0) && f.w3m == T(0)) f.region = 1;
    }
    return f;
}

// One block per (tile of RT rows (a, b), group of pairs); a thread holds one element (a, b, j) and
// takes the pairs of its lane.  Per batch of PB pairs: the pairs and weights, then the
// products of the row factors (10 doubles a row) and the columns' FRF values in shared memory, then
// 9 (all weights one), 13 (no sums on the grid) or 27 FP64 operations an element and pair.  Bound by
// the FP64 pipe (84 % busy): 2145 pairs of 24 modes 0.88 ms, the sums of row factors formed
// once a row.
__global__ __launch_bounds__(256) void k_pair_moments(Chunk c, MomPar P) {
    after_previous();
    extern __shared__ double sm[];
    const int t = threadIdx.x, nm = c.an, nm2 = nm * nm;
    const int PB = P.PB, RT = P.RT, EL = RT * nm;
    double *rowf = sm;                                 // [PB][RT][kRow]
    double2 *colf = (double2 *)(rowf + (size_t)PB * RT * kRow);  // [PB][nm][3]: Hx, P, D
    PairInfo *info = (PairInfo *)(colf + (size_t)PB * nm * 3);
    const int pl = t / EL, el = t - pl * EL;
    const int rl = el / nm, j = el - rl * nm, ab = blockIdx.x * RT + rl;
    const bool live = pl < P.PL && ab < nm2;
    const int G = gridDim.y;
    double K1 = 0, K2 = 0, K3 = 0, K4 = 0, K5 = 0, K6 = 0, M1 = 0, M2 = 0, M3 = 0;
    double Kc = 0, Kd = 0, Mc = 0, K56 = 0, K34 = 0, M23 = 0;
    for (long long p0 = (long long)blockIdx.y * PB; p0 < P.npairs; p0 += (long long)G * PB) {
        const int np = (int)min((long long)PB, P.npairs - p0);
        __syncthreads();
        if (t < np) {
            const long long p = p0 + t;
            int lo = 0, up = c.x1 - c.x0 - 1;
            while (lo < up) {
                const int mid = (lo + up + 1) >> 1;
                if (P.pre[mid] <= p) lo = mid; else up = mid - 1;
            }
            const int x = c.x0 + lo;
            PairInfo f = pair_info<double>(x, x + (int)(p - P.pre[lo]), P.N, P.vect);
            info[t] = f;
        }
        __syncthreads();
        double e[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int s = u * P.PL + pl;
            e[u] = 0.0;
            if (live && s < np) {
                const int r = (info[s].x - c.x0) * nm2 + ab, mt = r / kTM;
                const RowTile rt = c.rt[mt];
                e[u] = c.E[rt.base + (size_t)(r - mt * kTM) * rt.nct * kTN + (info[s].y * nm + j - rt.ct0 * kTN)];
            }
        }
        for (int q = t; q < np * nm * 3; q += 256) {
            const int s = q / (nm * 3), z = q - s * nm * 3, w = z / nm, m = z - w * nm;
            const int x = info[s].x, y = info[s].y;
            const int i = w == 0 ? x : w == 1 ? x + y : y - x;
            // x + y <= 2 N wherever its value is used (a pair with y > N has w1 = 0, w2m = w3m = 0 beyond)
            colf[((size_t)s * nm + m) * 3 + w] = P.H[(size_t)min(i, 2 * P.N) * nm + m];
        }
        for (int q = t; q < np * RT; q += 256) {
            const int s = q / RT, rr = blockIdx.x * RT + (q - s * RT);
            if (rr >= nm2) continue;
            const int a = rr / nm, b = rr - a * nm, x = info[s].x, y = info[s].y;
            const double2 xa = P.H[(size_t)x * nm + a], ya = P.H[(size_t)y * nm + a], yb = P.H[(size_t)y * nm + b];
            const double2 pb = P.H[(size_t)min(x + y, 2 * P.N) * nm + b], db = P.H[(size_t)(y - x) * nm + b];
            double *o = rowf + (size_t)q * kRow;
            o[0] = xa.x * yb.x - xa.y * yb.y;  // q1 = Hx_a Hy_b
            o[1] = xa.x * yb.y + xa.y * yb.x;
            o[2] = xa.x * yb.x + xa.y * yb.y;  // q2 = Hx_a conj Hy_b
            o[3] = xa.y * yb.x - xa.x * yb.y;
            o[4] = ya.x * pb.x + ya.y * pb.y;  // c = Hy_a conj P_b
            o[5] = ya.y * pb.x - ya.x * pb.y;
            o[6] = ya.x * db.x + ya.y * db.y;  // d = Hy_a conj D_b
            o[7] = ya.y * db.x - ya.x * db.y;
            o[8] = o[4] + o[6];
            o[9] = o[7] - o[5];
        }
        __syncthreads();
        if (live) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int s = u * P.PL + pl;
                if (s >= np) continue;
                const PairInfo &f = info[s];
                const double *o = rowf + ((size_t)s * RT + rl) * kRow;
                const double2 *h = colf + ((size_t)s * nm + j) * 3;
                const double2 hx = h[0], hp = h[1], hd = h[2];
                const double v = e[u];
                const double beta = fma(o[2], hd.x, -(o[3] * hd.y));
                if (f.region == 0) {
                    const double ab_ = fma(o[0], hp.x, fma(o[1], hp.y, beta));
                    // gamma + delta
                    const double gd = fma(o[8], hx.x, o[9] * hx.y);
                    Kc = fma(v, ab_, Kc);
                    Kd = fma(v, gd, Kd);
                    Mc += v;
                } else if (f.region == 1) {
                    const double ab_ = fma(o[0], hp.x, fma(o[1], hp.y, beta));
                    const double dl = fma(o[6], hx.x, o[7] * hx.y);
                    const double gd = fma(o[4], hx.x, fma(-o[5], hx.y, dl));
                    K1 = fma(v, ab_, K1);
                    K56 = fma(v, beta, K56);
                    K2 = fma(v, gd, K2);
                    K34 = fma(v, dl, K34);
                    M23 += v;
                } else {
                    const double al = fma(o[0], hp.x, o[1] * hp.y);
                    const double dl = fma(o[6], hx.x, o[7] * hx.y);
                    const double ga = fma(o[4], hx.x, -(o[5] * hx.y));
                    const double w1m = f.wm1 - f.w1;
                    const double va = v * al, vb = v * beta, vg = v * ga, vd = v * dl;
                    K1 = fma(f.w1, va, fma(w1m, vb, K1));
                    K2 = fma(f.w1, vg, fma(w1m, vd, K2));
                    K3 = fma(f.w2p, vd, fma(f.w2m, vg, K3));
                    K6 = fma(f.w2p, vb, fma(f.w2m, va, K6));
                    K4 = fma(f.w3p, vd, fma(f.w3m, vg, K4));
                    K5 = fma(f.w3p, vb, fma(f.w3m, va, K5));
                    M1 = fma(f.wm1, v, M1);
                    M2 = fma(f.wm2, v, M2);
                    M3 = fma(f.wm3, v, M3);
                }
            }
        }
    }
    double k[kKinds] = {K1 + Kc,         K2 + Kd,         K3 + Kd + K34,       K4 + Kd + K34,      K5 + Kc + K56,
                        K6 + Kc + K56,   M1 + 2.0 * (Mc + M23), M2 + 2.0 * Mc + M23, M3 + 2.0 * Mc + M23};
    // lanes of one element, then the block's partial
    double *red = sm;
#pragma unroll
    for (int q = 0; q < kKinds; ++q) {
        double s = k[q];
        if (P.PL > 1) {
            __syncthreads();
            if (pl < P.PL) red[t] = s;
            __syncthreads();
            if (pl == 0)
                for (int z = 1; z < P.PL; ++z) s += red[z * EL + el];
        }
        if (pl == 0 && ab < nm2) {
            double *o = P.part + (((size_t)blockIdx.y * kKinds + q) * nm2 + ab) * nm + j;
            *o = P.first ? s : *o + s;
        }
    }
}

// m3[m + nm n + nm^2 o] from the groups' partials [group][kKinds][(a, b)][j], lanes over the groups;
// w4 = 2 (the BFM's factor) x 2 (a point and its mirror) x d^2.
__global__ void k_pair_finish(int nm, int G, double w4, const double *__restrict__ S, double *__restrict__ m3mf,
                              double *__restrict__ m3mr, EndFlags fl) {
    after_previous();
    end_flags(fl);
    const int x = blockIdx.x * 32 + threadIdx.x, nm2 = nm * nm, nm3 = nm2 * nm, xe = x < nm3 ? x : 0;
    const int m = xe % nm, n = (xe / nm) % nm, o = xe / nm2;
    double mr = 0.0, mf = 0.0;
    for (int g = threadIdx.y; g < G; g += kRedLanes) {
        const double *s = S + (size_t)g * kKinds * nm3;
        auto at = [&](int kind, int a, int b, int j) { return s[((size_t)kind * nm2 + a * nm + b) * nm + j]; };
        mr += ((at(0, m, n, o) + at(1, m, o, n)) + (at(2, n, m, o) + at(3, o, n, m))) + (at(4, n, o, m) + at(5, o, m, n));
        mf += ((at(6, m, n, o) + at(6, m, o, n)) + (at(7, n, m, o) + at(7, o, m, n))) + (at(8, o, n, m) + at(8, n, o, m));
    }
    red_lanes(mr, mf);
    if (threadIdx.y == 0 && x < nm3) {
        m3mr[x] = w4 * mr;
        m3mf[x] = w4 * mf;
    }
}

// E(x, y)[(a, b), j] of a chunk that holds every product.
__device__ __forceinline__ double pair_at(const Chunk &c, int x, int y, int a, int b, int j) {
    if (x > y) {
        const int t = x;
        x = y;
        y = t;
        const int u = b;
        b = j;
        j = u;
    }
    const int r = x * c.rx() + a * c.an + b, mt = r / kTM;
    const RowTile rt = c.rt[mt];
    return c.E[rt.base + (size_t)(r - mt * kTM) * rt.nct * kTN + (y * c.an + j - rt.ct0 * kTN)];
}

// Force and response bispectra of every grid point from the products: one block per point (i1, i2) =
// (p % nf - N, p / nf - N), the layout and FRF product of k_bfm_fp64.  65 x 65 points of 60 nodes, 6
// modes: 0.55 ms by three contractions a point, 0.02 ms with the products.
__global__ __launch_bounds__(256) void k_pair_points(Chunk c, int N, const double2 *__restrict__ H, double *__restrict__ bf,
                                                     double *__restrict__ br) {
    after_previous();
    __shared__ double2 h[3][64];
    const int nm = c.an, nm2 = nm * nm, nm3 = nm2 * nm, nf = 2 * N + 1, p = blockIdx.x;
    const int i1 = p % nf - N, i2 = p / nf - N, i3 = i1 + i2, x = abs(i1), y = abs(i2), z = abs(i3);
    for (int q = threadIdx.x; q < 3 * nm; q += blockDim.x) {
        const int w = q / nm, i = w == 0 ? i1 : w == 1 ? i2 : i3;
        double2 v = H[(size_t)abs(i) * nm + (q - w * nm)];
        if (i < 0) v.y = -v.y;
        h[w][q - w * nm] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nm3; e += blockDim.x) {
        const int m = e % nm, n = (e / nm) % nm, o = e / nm2;
        double v = pair_at(c, x, y, m, n, o);                                                  // T1
        if (z <= c.hi) v += pair_at(c, z, y, n, m, o) + pair_at(c, x, z, o, n, m);             // T2 + T3
        const double2 h1 = h[0][m], h2 = h[1][n], h3 = h[2][o];
        const double cr = h2.x * h3.x + h2.y * h3.y, ci = h2.y * h3.x - h2.x * h3.y;
        const double F = h1.x * cr - h1.y * ci, b = 2.0 * v;
        if (bf) bf[(size_t)p * nm3 + e] = b;
        if (br) br[(size_t)p * nm3 + e] = b * F;
    }
}

// Diagonal-only spectra: the products are P_m(x, y) = sum_k Q_km L_km^2 S_k(x) S_k(y), rows (x, m),
// columns y, and with a = b = j = m the twelve contributions collapse to
// 2 (w1 + w2m + w3m) alpha + 2 (w1- + w2p + w3p) beta.  One block per (mode, group of x), a warp per
// x with its lanes over y; part[group][0: force, 1: response][m].  Bound by the FP64 pipe (20
// instructions an element): 513 x 513 points of 24 modes 60 us with the weights formed in FP64, 44 in FP32.
__global__ __launch_bounds__(256) void k_pair_moments_diag(Chunk c, int N, int analytic, int vect, double w4,
                                                           const double2 *__restrict__ H, double *__restrict__ part) {
    after_previous();
    __shared__ double red[2][8];
    const int m = blockIdx.x, nm = c.qn, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double sf = 0.0, sr = 0.0;
    for (int x = c.x0 + blockIdx.y * 8 + warp; x < c.x1; x += 8 * gridDim.y) {
        const int r = (x - c.x0) * nm + m, mt = r / kTM, y1 = analytic ? min(c.hi, x + N) : N;
        const RowTile rt = c.rt[mt];
        const double *e = c.E + rt.base + (size_t)(r - mt * kTM) * rt.nct * kTN - rt.ct0 * kTN;
        const double2 hx = H[(size_t)x * nm + m];
        for (int y = x + lane; y <= y1; y += 32) {
            const PairWeights<float> f = pair_info<float>(x, y, N, vect);
            const double2 hy = H[(size_t)y * nm + m], p = H[(size_t)min(x + y, 2 * N) * nm + m], d = H[(size_t)(y - x) * nm + m];
            const double qr = hx.x * hy.x, qi = hx.y * hy.y, ur = hx.x * hy.y, ui = hx.y * hy.x;
            const double al = (qr - qi) * p.x + (ur + ui) * p.y, be = (qr + qi) * d.x - (ui - ur) * d.y;
            const double g = (double)(f.w1 + f.w2m + f.w3m) * al + (double)(f.wm1 - f.w1 + f.w2p + f.w3p) * be;
            const double v = 2.0 * e[y];
            sr = fma(v, g, sr);
            sf = fma(v, (double)(f.wm1 + f.wm2 + f.wm3), sf);
        }
    }
    for (int h = 16; h > 0; h >>= 1) {
        sf += __shfl_down_sync(0xffffffffu, sf, h);
        sr += __shfl_down_sync(0xffffffffu, sr, h);
    }
    if (lane == 0) {
        red[0][warp] = sf;
        red[1][warp] = sr;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += red[threadIdx.x][w];
        part[((size_t)blockIdx.y * 2 + threadIdx.x) * nm + m] = w4 * s;
    }
}

}  // namespace p64

// Third moments of the whole Classic grid (circular-frequency convention, every row) in FP64 from
// the products of distinct frequency pairs; dA (dS for the diagonal-only spectra) holds the rows of
// i df, i = 0 .. N (truncated S(f1 + f2)) or 0 .. 2 N (analytic).
// With bf_host / br_host the bispectra of every grid point instead (every product in one chunk:
// pair64_points).
int Engine::contract_pair64(int N, double df, bool analytic, bool vect, double wval, double *m3mf, double *m3mr,
                            double *bf_host, double *br_host) {
    using namespace p64;
    const bool diag = set.onlyd != 0;
    const int nm = nme, an = diag ? 1 : nm, rx = nm * an, hi = analytic ? 2 * N : N;
    const long long nb = dim_bisp();  // outputs: nm^3, or nm
    const double *A = diag ? dS.as<double>() : dA.as<double>(), *Q = diag ? dWd3.as<double>() : dQ.as<double>();
    cudaError_t e;
    auto ylast = [&](int x) { return analytic ? std::min(hi, x + N) : N; };  // last partner of first row x
    const long long pairs_all = (long long)(N + 1) * (N + 2) / 2 + (analytic ? (long long)N * (N + 1) / 2 : 0);
    // moment kernel: rows of a block, pair lanes, pairs of a batch (fewer for small grids, so that the
    // groups still fill the chip) and groups: one wave of resident blocks (a third wave of a few blocks
    // cost 0.3 of 1.1 ms)
    const int RT = std::max(1, std::min(rx, 256 / nm)), PL = std::max(1, std::min(8, 256 / (RT * nm)));
    const int tiles = (rx + RT - 1) / RT;
    auto smem_of = [&](int PB) {
        return std::max((size_t)256 * sizeof(double), sizeof(double) * (size_t)PB * RT * kRow +
                        sizeof(double2) * (size_t)PB * nm * 3 + sizeof(PairInfo) * (size_t)PB);
    };
    int dev = 0, nsm = 0, occ = 1;
    if ((e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) ||
        (e = cudaFuncSetAttribute(k_pair_moments, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_of(kBatch * PL))) ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_pair_moments, 256, smem_of(kBatch * PL))))
        return cuda_fail(e, "pair moments kernel");
    const long long want = std::max(1, std::max(1, occ) * nsm / tiles);
    const int PB = PL * (int)std::max(1LL, std::min<long long>(kBatch, pairs_all / (want * PL)));
    const int G = diag ? std::min(64, (N + 8) / 8) : (int)std::max(1LL, std::min(want, (pairs_all + PB - 1) / PB));
    const size_t smem = smem_of(PB);
    // Products on the tensor cores (bsa_pair64_tc.cu) where they outweigh the digits' preparation.
    // Measured contraction in ms, FP64 pipe / tensor cores: 4.1e6 FMAs, K = 30: 0.069 / 0.080; 1.1e7, K = 24:
    // 0.096 / 0.103; 1.6e7, K = 30: 0.115 / 0.102; from K = 40 on 7.3e6, K = 60: 0.082 / 0.080; 1.2e7, K = 40:
    // 0.090 / 0.089; 1.4e7, K = 400: 0.168 / 0.091.  (K is padded to 16 and the moments do not get faster.)
    const bool tensor = K >= 24 && pairs_all * nb * K >= (K < 40 ? 15000000LL : 7000000LL);
    // chunks of first rows: at most 4 GB of products and of row digits each
    const long long cap = 1LL << 29;
    const int Kd = (K + 63) / 64 * 64 * 2;  // digits of a row in doubles
    struct Plan { int x0, x1, ntiles; long long items, elems, npairs; size_t rt0, pre0; };
    std::vector<Plan> plans;
    std::vector<RowTile> rts;
    std::vector<long long> pre;
    long long emax = 0, rmax = 0, imax = 0;
    const bool pts = bf_host || br_host;
    for (int x0 = 0; x0 <= N;) {
        Plan p{x0, x0, 0, 0, 0, 0, rts.size(), pre.size()};
        long long el = 0;
        while (p.x1 <= N) {
            const long long add = (long long)rx * std::max((ylast(p.x1) - p.x1 + 1) * (long long)an + 2 * kTN, (long long)Kd);
            if (!pts && p.x1 > x0 && el + add > cap) break;
            el += add;
            pre.push_back(p.npairs);
            p.npairs += ylast(p.x1) - p.x1 + 1;
            ++p.x1;
        }
        const long long rows = (long long)(p.x1 - x0) * rx;
        for (long long r = 0; r < rows; r += kTM) {
            const int xa = x0 + (int)(r / rx), xb = x0 + (int)((std::min(rows, r + kTM) - 1) / rx);
            RowTile t;
            t.ct0 = xa * an / kTN;
            t.nct = (int)(((long long)(ylast(xb) + 1) * an + kTN - 1) / kTN) - t.ct0;
            t.base = p.elems;
            t.item0 = p.items;
            p.items += t.nct;
            p.elems += (long long)t.nct * kTN * kTM;
            rts.push_back(t);
        }
        p.ntiles = (int)(rts.size() - p.rt0);
        emax = std::max(emax, p.elems);
        rmax = std::max(rmax, rows);
        imax = std::max(imax, p.items);
        plans.push_back(p);
        x0 = p.x1;
    }
    const size_t rtb = sizeof(RowTile) * rts.size(), preb = sizeof(long long) * pre.size();
    const size_t hb = sizeof(double2) * (size_t)(2 * N + 1) * nm, nparts = diag ? G * plans.size() : G;
    const long long plen = diag ? 2 * nb : kKinds * nb;
    const size_t ptb = sizeof(double) * (size_t)(2 * N + 1) * (2 * N + 1) * nb;
    const bool two = !diag && G > 64;
    auto room = [&](DevBuf &b, size_t bytes) { return !e && (e = b.reserve(bytes)) == cudaErrorMemoryAllocation; };
    e = cudaSuccess;
    if (room(dMixA, sizeof(double) * (size_t)emax) || (tensor && room(dMixB, tc_col_bytes(hi + 1, an, K))) ||
        (tensor && room(dMshT, tc_row_bytes(rmax, K, imax))) || room(dMixH, hb) || room(dMshIdx, rtb + preb) ||
        room(dPartF, sizeof(double) * nparts * plen) || (two && room(dPartR, sizeof(double) * (size_t)plen)) ||
        room(dOut, sizeof(double) * out_doubles()) || (tensor && room(dFlag, 256)) ||
        (bf_host && room(dBF, ptb)) || (br_host && room(dBR, ptb)))
        return kNoRoom;
    if (e) return cuda_fail(e, "allocating pair products");
    double *o = dOut.as<double>() + 3 * (size_t)dim_psd();
    char *idx = (char *)dMshIdx.p;
    std::vector<char> lists(rtb + preb);
    std::memcpy(lists.data(), rts.data(), rtb);
    std::memcpy(lists.data() + rtb, pre.data(), preb);
    if ((e = cudaMemcpyAsync(idx, lists.data(), lists.size(), cudaMemcpyHostToDevice, stream))) return cuda_fail(e, "pair lists");
    h2d += (double)(rtb + preb);
    if ((e = cudaEventRecord(ev2, stream)) || (e = cudaEventRecord(evg0, stream))) return cuda_fail(e, "event");
    const int nh = (2 * N + 1) * nm;
    launch_next(k_frf_rows, (nh + 127) / 128, 128, 0, stream, 2 * N + 1, nm, df, frf(), dMixH.as<double2>());
    if (tensor && ((e = cudaMemsetAsync(dFlag.as<int>() + 1, 0, sizeof(int), stream)) ||
                   (e = tc_prep_cols(stream, hi + 1, an, K, A, dMixB.p))))
        return cuda_fail(e, "pair product operands");
    if (tensor) kernels += 2;
    for (size_t q = 0; q < plans.size(); ++q) {
        const Plan &p = plans[q];
        Chunk c{p.x0, p.x1, nm, an, K, hi, p.ntiles, p.items, (const RowTile *)idx + p.rt0, dMixA.as<double>(), rx, nullptr, wait_test_pair1};
        wait_test_pair1 = 0;  // one launch only
        if (tensor) {
            if ((e = tc_products(stream, c, hi + 1, A, Q, dMixB.p, dMshT.p, dFlag.as<int>() + 1)))
                return cuda_fail(e, "pair product kernel");
            kernels += 3;
        } else {
            if (p.items < 304) launch_next(k_pair_gemm<32>, dim3((unsigned)p.items, kTM / 32), 256, 0, stream, c, A, Q);
            else launch_next(k_pair_gemm<kTM>, dim3((unsigned)p.items, 1), 256, 0, stream, c, A, Q);
        }
        if (pts) {
            launch_next(k_pair_points, (2 * N + 1) * (2 * N + 1), 256, 0, stream, c, N, dMixH.as<double2>(), bf_host ? dBF.as<double>() : nullptr,
                                                                         br_host ? dBR.as<double>() : nullptr);
        } else if (diag) {
            launch_next(k_pair_moments_diag, dim3(nm, G), 256, 0, stream, c, N, analytic ? 1 : 0, vect ? 1 : 0, 4.0 * wval,
                                                                  dMixH.as<double2>(), dPartF.as<double>() + q * G * plen);
        } else {
            MomPar mp{N, vect ? 1 : 0, p.npairs, (const long long *)(idx + rtb) + p.pre0, dMixH.as<double2>(),
                      dPartF.as<double>(), q == 0 ? 1 : 0, RT, PL, PB};
            launch_next(k_pair_moments, dim3((unsigned)tiles, (unsigned)G), 256, smem, stream, c, mp);
        }
        kernels += 2;
    }
    if ((e = cudaGetLastError())) return cuda_fail(e, "pair contraction kernels");
    if ((e = cudaEventRecord(evg1, stream))) return cuda_fail(e, "event");
    if (pts) {
        const size_t bytes = ptb;
        int flags[2] = {0, 0};
        const bool pend = atable_pending;
        if (((tensor || pend) && (e = cudaMemcpyAsync(flags, dFlag.p, sizeof flags, cudaMemcpyDeviceToHost, stream))) ||
            (bf_host && (e = fetch(stream, bf_host, dBF.p, bytes))) || (br_host && (e = fetch(stream, br_host, dBR.p, bytes))) ||
            (e = cudaEventRecord(ev1, stream)) || (e = cudaStreamSynchronize(stream)))
            return cuda_fail(e, "bispectrum copy");
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ev2, ev1);
        last_ms_contraction = ms;
        cudaEventElapsedTime(&ms, evg0, evg1);
        last_ms_gemm = ms;
        d2h += (double)bytes * ((bf_host ? 1 : 0) + (br_host ? 1 : 0));
        return pipeline_flags(flags, pend, tensor);
    }
    const bool pend = atable_pending;
    const EndFlags fl{pend ? dFlag.as<int>() : nullptr, tensor ? dFlag.as<int>() + 1 : nullptr, out_flags()};
    if (diag) {
        if ((e = launch_reduce_groups(stream, (int)nparts, plen, dPartF.as<double>(), o, nullptr, nullptr, fl)))
            return cuda_fail(e, "reduction kernel");
    } else {
        // many groups (few outputs) are summed kind by kind first: 304 groups of 4 modes 9 + 4 us, by
        // k_pair_finish alone 39; from 64 groups down it is the other way
        if (two && (e = launch_reduce_groups(stream, G, plen, dPartF.as<double>(), dPartR.as<double>(), nullptr, nullptr)))
            return cuda_fail(e, "reduction kernel");
        launch_next(k_pair_finish, (unsigned)((nb + 31) / 32), dim3(32, kRedLanes), 0, stream,
            nm, two ? 1 : G, 4.0 * wval, two ? dPartR.as<double>() : dPartF.as<double>(), o, o + nb, fl);
    }
    if ((e = cudaGetLastError())) return cuda_fail(e, "reduction kernel");
    kernels += two ? 3 : 2;
    float ms = 0.f, ms_gemm = 0.f;
    if ((e = results(&ms, &ms_gemm))) return cuda_fail(e, "moment copy");
    int rc;
    if ((rc = pipeline_flags((const int *)(hRes.data() + out_doubles() - 1), pend, tensor))) return rc;
    last_ms_contraction = ms;
    last_ms_gemm = ms_gemm;
    d2h += 2.0 * sizeof(double) * (double)nb;
    const double *h = hRes.data() + 3 * (size_t)dim_psd();
    if (m3mf) std::memcpy(m3mf, h, sizeof(double) * nb);
    if (m3mr) std::memcpy(m3mr, h + nb, sizeof(double) * nb);
    return BSA_OK;
}

}  // namespace bsa
