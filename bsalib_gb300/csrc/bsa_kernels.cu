// bsa_kernels.cu -- FP64 kernels of the BFM hot path (nodal spectra, per-frequency
// factor A(f), force PSD / second-order moments, and the plain FP64 contraction with the
// FRF product and the weighted moment reduction fused into its epilogue).
#include "bsa_kernels.cuh"

#include <algorithm>

namespace bsa {

// ------------------------------------------------------------------------------------
// Stage (a): nodal turbulence PSD.  One thread per (f, itc, node), node fastest so the
// stores are coalesced.  Model formulas: vonKarmanPSD_ (WindPSDImpl.F90:149-226, u form
// for tc == 1, v/w form otherwise), kaimalPSD_ (:231-243, identically zero),
// davenportPSD_Greisch_ (:249-277), davenportPSD_Uliege_ (:283-316); divided by 4 pi
// under the circular-frequency convention (:142-143).  R = double for the FP64 paths; the
// split-precision paths, whose A(f) tables take sqrt(S) in FP32, evaluate the same formulas
// in FP32 (R = float: relative error ~1e-7, where FP64's pow costs ~100 FP64 instructions).
// ------------------------------------------------------------------------------------
// y^(5/6) and y^(4/3): in FP64 from the square and cube roots (45 and 25 FP64 instructions, the general
// power about 100; 205 600 spectra of Davenport's form 62 us by pow, 29 so), within its 2 ulp.
template <typename R>
__device__ __forceinline__ R pow56(R y) {
    if constexpr (sizeof(R) == 8) return sqrt(y) * cbrt(y);
    else return pow(y, R(5.0 / 6.0));
}
template <typename R>
__device__ __forceinline__ R pow43(R y) {
    if constexpr (sizeof(R) == 8) return y * cbrt(y);
    else return pow(y, R(4.0 / 3.0));
}

template <typename R>
__global__ void k_nodal_psd(int nf, const double *__restrict__ f, int ntc, int4 tcs, int nnl,
                            const PsdNode *__restrict__ par, int psd_type, int scaling, double *__restrict__ S,
                            double *__restrict__ expt) {
    after_previous();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long tot = (long long)nf * ntc * nnl;
    // expt (FP64 only): sqrt(S) instead of S, and the A kernel's exponential table
    if (sizeof(R) == 8 && expt && blockIdx.x == 0) expt[threadIdx.x] = exp2((double)threadIdx.x / kExpTab);
    if (t >= tot) return;
    const int i = (int)(t % nnl);
    const long long r = t / nnl;
    const int itc = (int)(r % ntc);
    const int fi = (int)(r / ntc);
    const int tc = itc == 0 ? tcs.x : (itc == 1 ? tcs.y : tcs.z);
    const PsdNode p = par[itc * nnl + i];
    const R fr = (R)f[fi], Ls = (R)p.Ls, U = (R)p.U, Uref = (R)p.Uref, sg = (R)p.sigma;
    const R sig2 = sg * sg;
    // FP64: the scaling goes into each form's denominator, a division less
    const R sc = sizeof(R) == 8 && scaling == 1 ? R(kPi4) : R(1);
    R v = 0;
    switch (psd_type) {
    case 1:
        if (tc == 1) {
            const R rt = Ls / U;
            R x = fabs(fr) * rt;
            x = x * x;
            x = pow56(R(1) + R(70.7) * x);
            v = R(4) * (rt * sig2) / (x * sc);
        } else {
            R d = R(2) * (fr * (Ls / U));
            d = d * d;
            const R y = R(1) + R(70.7) * d;
            const R r2 = (sizeof(R) == 8 ? y * pow56(y) : pow(y, R(11.0 / 6.0))) * U * sc;
            const R r3 = Ls * (R(1) + R(188.4) * d) / r2 * sig2;
            const R a = r3 + r3;
            v = a + a;
        }
        break;
    case 2:
        v = 0;
        break;
    case 3: {
        const R cst1 = R(0.65 * 1200.0);
        const R x = cst1 * fr / Uref;
        v = cst1 * sig2 / Uref / (pow56(R(1) + x * x) * sc);
    } break;
    case 5: {
        const R clu = Ls / U;
        const R cf = fabs(fr) * clu;
        v = ((R(2.0 / 3.0)) * cf * clu * sig2) / (pow43(R(1) + cf * cf) * sc);
    } break;
    default:
        v = 0;
    }
    if (sizeof(R) == 4 && scaling == 1) v = v / R(kPi4);
    S[t] = (sizeof(R) == 8 && expt) ? sqrt((double)v) : (double)v;
}

cudaError_t launch_nodal_psd(cudaStream_t st, int nf, const double *f, int ntc, const int *tcs_host,
                             int nnl, const PsdNode *par, int psd_type, int scaling, double *S, bool fp32, double *expt) {
    const long long tot = (long long)nf * ntc * nnl;
    if (tot == 0) return cudaSuccess;
    int4 tcs = make_int4(tcs_host[0], ntc > 1 ? tcs_host[1] : 0, ntc > 2 ? tcs_host[2] : 0, 0);
    const int blk = kExpTab;
    const unsigned grid = (unsigned)((tot + blk - 1) / blk);
    if (fp32)
        launch_next(k_nodal_psd<float>, grid, blk, 0, st, nf, f, ntc, tcs, nnl, par, psd_type, scaling, S, expt);
    else
        launch_next(k_nodal_psd<double>, grid, blk, 0, st, nf, f, ntc, tcs, nnl, par, psd_type, scaling, S, expt);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Stage (a)+(b) factor: A(f)[(itc,i)][m] = sqrt(S_i) sum_j c_ij^|f| sqrt(S_j) L[(itc,j)][m].
// The coherent cross-PSD c_ij^|f| sqrt(S_i S_j) (functionsImpl.F90:1450-1477,
// getFullNodalPSD WindPSDImpl.F90:76-108) is generated on the fly from log c_ij and never
// stored as an NNL^2 x NF tensor.  c^0 = 1 for every c (Fortran 0**0 = 1).
//
// Bound by the FP64 pipe (two FMAs an SM and clock): per (i, j) one exponential and nm FMAs.  Block:
// 64 rows i x all modes, j streamed in tiles of 32; a thread holds one row and every fourth mode,
// MPT of them, so nm is padded to a multiple of 4 only (8 threads a row and 8 slots each, tested
// one by one, cost 12 modes a third of the pipe).  The exponential is expc, 10 FP64 instructions
// where exp() spends about 25, and sqrt(S) comes from k_nodal_psd.  150 nodes, 12 modes, 3333
// frequencies: 13.1 -> 3.9 ms.
// ------------------------------------------------------------------------------------
template <int MPT>
__global__ __launch_bounds__(256) void k_atable(int nf, const double *__restrict__ f, int ntc, int nnl,
                                                int nm, const double *__restrict__ logc,
                                                const double *__restrict__ expt,
                                                const double *__restrict__ rootS,
                                                const double *__restrict__ L, double *__restrict__ A,
                                                const int *__restrict__ only) {
    after_previous();
    if (only && !*only) return;
    constexpr int RI = 64, JT = 32, NML = 4 * MPT;
    const int fi = blockIdx.x / ntc, itc = blockIdx.x % ntc;
    const int i0 = blockIdx.y * RI;
    __shared__ double T[kExpTab];
    __shared__ double Gs[JT][RI + 1];
    __shared__ double Ls[JT][NML];
    const double af = fabs(f[fi]);
    const double *Sf = rootS + ((size_t)fi * ntc + itc) * nnl;
    const double *lc = logc + (size_t)itc * nnl * nnl;
    const double *Lt = L + (size_t)itc * nnl * nm;
    const int t = threadIdx.x, il = t >> 2, mg = t & 3;
    T[t] = expt[t];
    double acc[MPT];
#pragma unroll
    for (int u = 0; u < MPT; ++u) acc[u] = 0.0;
    __syncthreads();
    for (int j0 = 0; j0 < nnl; j0 += JT) {
#pragma unroll
        for (int u = 0; u < RI * JT / 256; ++u) {
            const int e = t + 256 * u, ii = e >> 5, jj = e & 31, gi = i0 + ii, gj = j0 + jj;
            double g = 0.0;
            if (gi < nnl && gj < nnl) g = (af == 0.0) ? 1.0 : expc(af * lc[(size_t)gi * nnl + gj], T);
            Gs[jj][ii] = g;
        }
        for (int e = t; e < JT * NML; e += 256) {
            const int jj = e / NML, m = e % NML, gj = j0 + jj;
            Ls[jj][m] = (gj < nnl && m < nm) ? Sf[gj] * Lt[(size_t)gj * nm + m] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int jj = 0; jj < JT; ++jj) {
            const double g = Gs[jj][il];
#pragma unroll
            for (int u = 0; u < MPT; ++u) acc[u] = fma(g, Ls[jj][mg + 4 * u], acc[u]);
        }
        __syncthreads();
    }
    const int gi = i0 + il;
    if (gi < nnl) {
        const double si = Sf[gi];
        double *out = A + (((size_t)fi * ntc + itc) * nnl + gi) * nm;
#pragma unroll
        for (int u = 0; u < MPT; ++u) {
            const int m = mg + 4 * u;
            if (m < nm) out[m] = si * acc[u];
        }
    }
}

// log c_ij of every loaded node pair from the packed upper triangle (util_getCorrVectIndex,
// src/utils/utility.F90:60-71), in FP64 and FP32; the host side of this expansion and its copy were
// 0.6 ms of a 400-node, two-component analysis.
__global__ void k_log_coh(int ntc, int nnl, int nn, long long ncorr, const int *__restrict__ nodes,
                          const double *__restrict__ corr, double *__restrict__ lc, float *__restrict__ lc32,
                          int *__restrict__ bad) {
    after_previous();
    const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= (long long)ntc * nnl * nnl) return;
    const int j = (int)(x % nnl), i = (int)(x / nnl % nnl), c = (int)(x / nnl / nnl);
    const long long a = min(nodes[i], nodes[j]), b = max(nodes[i], nodes[j]);
    const double w = corr[c * ncorr + (a - 1) * nn + b - (a * a - a) / 2 - 1];
    if (!(w >= 0.0 && w <= 1.0) || (i == j && w != 1.0)) *bad = 1;
    const double v = log(w);
    lc[x] = v;
    lc32[x] = (float)v;
}

int *log_coh_bad(const double *lc, size_t n) { return (int *)(lc + n + kExpTab); }

cudaError_t launch_log_coh(cudaStream_t st, int ntc, int nnl, int nn, long long ncorr, const int *nodes, const double *corr,
                           double *lc, float *lc32) {
    const long long n = (long long)ntc * nnl * nnl;
    if (n == 0) return cudaSuccess;
    int *bad = log_coh_bad(lc, (size_t)n);
    cudaError_t e = cudaMemsetAsync(bad, 0, sizeof(int), st);
    if (e != cudaSuccess) return e;
    launch_next(k_log_coh, (unsigned)((n + 255) / 256), 256, 0, st, ntc, nnl, nn, ncorr, nodes, corr, lc, lc32, bad);
    return cudaGetLastError();
}

// Projection of the wind coefficients onto the kept modes and the tables made of it, a thread per (k, m).
// Launch-bound; on the host, with five tables to copy in the place of their inputs, it was the longest
// part of a small analysis (400 nodes, two components, 24 modes: 0.2 of 0.72 ms, now 0.03).
__global__ void k_project(int K, int nm, int nl, int nnl, const double *__restrict__ wfc, const double *__restrict__ phi,
                          double *__restrict__ L, double *__restrict__ Q, double *__restrict__ W3, double *__restrict__ W2,
                          float *__restrict__ L32) {
    after_previous();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= K * nm) return;
    const int k = x / nm, m = x - k * nm;
    double l = 0.0, q = 0.0;
    if (nl == 0) {
        l = wfc[x];
        q = wfc[(size_t)K * nm + x];
    } else {
        const double *p = phi + ((size_t)m * nnl + k % nnl) * nl, *wl = wfc + (size_t)k * nl, *wq = wl + (size_t)K * nl;
        for (int z = 0; z < nl; ++z) {
            l = fma(wl[z], p[z], l);
            q = fma(wq[z], p[z], q);
        }
    }
    L[x] = l;
    Q[x] = q;
    W3[x] = q * l * l;
    W2[x] = l * l;
    L32[x] = (float)l;
}

cudaError_t launch_project(cudaStream_t st, int K, int nm, int nl, const double *wfc, const double *phi, int nnl, double *L,
                           double *Q, double *W3, double *W2, float *L32) {
    launch_next(k_project, (K * nm + 127) / 128, 128, 0, st, K, nm, nl, nnl, wfc, phi, L, Q, W3, W2, L32);
    return cudaGetLastError();
}

size_t log_coh_bytes(size_t n) { return sizeof(double) * (n + kExpTab + 1); }

cudaError_t launch_atable(cudaStream_t st, int nf, const double *f, int ntc, int nnl, int nm,
                          const double *logc, const double *rootS, const double *L, double *A, const int *only) {
    if (nf == 0) return cudaSuccess;
    if (nm > 64) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)nf * ntc, (unsigned)((nnl + 63) / 64));
    const double *expt = logc + (size_t)ntc * nnl * nnl;
#define BSA_AT_CASE(V)                                                                          \
    if (nm <= 4 * V) {                                                                          \
        launch_next(k_atable<V>, grid, 256, 0, st, nf, f, ntc, nnl, nm, logc, expt, rootS, L, A, only);  \
        return cudaGetLastError();                                                              \
    }
    BSA_AT_CASE(1)
    BSA_AT_CASE(2)
    BSA_AT_CASE(3)
    BSA_AT_CASE(4)
    BSA_AT_CASE(5)
    BSA_AT_CASE(6)
    BSA_AT_CASE(8)
    BSA_AT_CASE(10)
    BSA_AT_CASE(12)
    BSA_AT_CASE(14)
    BSA_AT_CASE(16)
#undef BSA_AT_CASE
    return cudaErrorInvalidValue;
}

// ------------------------------------------------------------------------------------
// Second-order path: force PSD and m2 moments (functionsImpl.F90:1548-1560, 1653-1676;
// BsaClassicImpl.F90:149-154, 197-210).
// ------------------------------------------------------------------------------------
// psd[f][n + nm o] = sum_k L[k][o] A[f][k][n]: 32 pairs (n, o) by 8 lanes over k per block (16 where the
// blocks are few: 291 blocks of 173 k 11 -> 8 us, 650 of 800 43 -> 50), the lanes' sums added in shared
// memory in a fixed order.  One thread a pair walking all k, in one block a frequency, was bound by load
// latency: 65 rows of the 400-node, 24-mode building 0.56 -> 0.06 ms.  L^T S(f) L is symmetric, so the
// pairs n <= o stand for both: 59 -> 43 us there.
template <int LANES>
__global__ __launch_bounds__(32 * LANES) void k_force_psd(int ntc, int nnl, int nm, const double *__restrict__ L,
                                                   const double *__restrict__ A, double *__restrict__ psd) {
    after_previous();
    __shared__ double red[LANES][32];
    const int fi = blockIdx.x, nm2 = nm * nm, K = ntc * nnl;
    const int pr = blockIdx.y * 32 + (threadIdx.x & 31), lane = threadIdx.x >> 5, np = nm * (nm + 1) / 2;
    // pr = o (o + 1) / 2 + n, at most 2080 pairs: the root is right to less than one
    int o = (int)((sqrtf(8.f * (float)pr + 1.f) - 1.f) * 0.5f);
    if (o * (o + 1) / 2 > pr) --o;
    if ((o + 1) * (o + 2) / 2 <= pr) ++o;
    const int n = pr - o * (o + 1) / 2;
    const double *Af = A + (size_t)fi * K * nm + n, *Lo = L + o;
    double s = 0.0;
    if (pr < np)
#pragma unroll 4
        for (int k = lane; k < K; k += LANES) s = fma(Lo[(size_t)k * nm], Af[(size_t)k * nm], s);
    red[lane][threadIdx.x & 31] = s;
    __syncthreads();
    if (lane == 0 && pr < np) {
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < LANES; ++q) v += red[q][threadIdx.x];
        psd[(size_t)fi * nm2 + n + nm * o] = v;
        psd[(size_t)fi * nm2 + o + nm * n] = v;
    }
}

cudaError_t launch_force_psd(cudaStream_t st, int nf, int ntc, int nnl, int nm, const double *L,
                             const double *A, double *psd) {
    if (nf == 0) return cudaSuccess;
    const dim3 grid(nf, (nm * (nm + 1) / 2 + 31) / 32);
    if ((long long)grid.x * grid.y <= 304) launch_next(k_force_psd<16>, grid, 512, 0, st, ntc, nnl, nm, L, A, psd);
    else launch_next(k_force_psd<8>, grid, 256, 0, st, ntc, nnl, nm, L, A, psd);
    return cudaGetLastError();
}

// The same from the FP32 tables of the split path: FP32 products summed in FP32 over runs of
// 32 k and the runs in FP64 (GB300's FP64 rate makes the all-FP64 form the slow one; the
// operands are FP32-rounded anyway, and the runs keep the sum to ~1e-7).  A lane takes every eighth
// run: 1025 rows of 800 k, 24 modes 0.46 -> 0.21 ms.
__global__ __launch_bounds__(256) void k_force_psd32(int ntc, int nnl, int nm, const float *__restrict__ L,
                                                     const float *__restrict__ A, double *__restrict__ psd) {
    after_previous();
    __shared__ double red[8][32];
    const int fi = blockIdx.x, nm2 = nm * nm, K = ntc * nnl;
    const int pr = blockIdx.y * 32 + (threadIdx.x & 31), lane = threadIdx.x >> 5;
    const int n = pr % nm, o = pr / nm;
    const float *Af = A + (size_t)fi * K * nm + n, *Lo = L + o;
    double s = 0.0;
    if (pr < nm2)
        for (int k0 = lane * 32; k0 < K; k0 += 256) {
            const int k1 = min(K, k0 + 32);
            float r = 0.f;
#pragma unroll 8
            for (int k = k0; k < k1; ++k) r = fmaf(Lo[(size_t)k * nm], Af[(size_t)k * nm], r);
            s += (double)r;
        }
    red[lane][threadIdx.x & 31] = s;
    __syncthreads();
    if (lane == 0 && pr < nm2) {
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) v += red[q][threadIdx.x];
        psd[(size_t)fi * nm2 + pr] = v;
    }
}

cudaError_t launch_force_psd32(cudaStream_t st, int nf, int ntc, int nnl, int nm, const float *L,
                               const float *A, double *psd) {
    if (nf == 0) return cudaSuccess;
    launch_next(k_force_psd32, dim3(nf, (nm * nm + 31) / 32), 256, 0, st, ntc, nnl, nm, L, A, psd);
    return cudaGetLastError();
}

// One block per (n, o) pair; threads stride over frequencies, fixed-order tree reduction.
// diag != 0: psd[f][m] holds the same-mode spectra (length nm), pair (n, o) = (m, m).
__global__ void k_m2(int k0, int k1, int nm, int diag, const double *__restrict__ f, const double *__restrict__ wf,
                     const double *__restrict__ psd, FrfPar frf, double *m2mf, double *m2mr,
                     double *m2o2mr) {
    after_previous();
    const int nm2 = diag ? nm : nm * nm;
    const int pr = blockIdx.x;
    const int n = diag ? pr : pr % nm, o = diag ? pr : pr / nm;
    double sf = 0.0, sr = 0.0, so = 0.0;
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const double w = f[k] * kPi2;
        double hnr, hni, hor, hoi;
        frf_eval(frf.M[n], frf.K[n], frf.C[n], w, hnr, hni);
        frf_eval(frf.M[o], frf.K[o], frf.C[o], w, hor, hoi);
        const double p = psd[(size_t)k * nm2 + pr];
        const double pr_ = p * (hor * hnr + hoi * hni);
        sf += wf[k] * p;
        sr += wf[k] * pr_;
        so += wf[k] * (pr_ * w * w);
    }
    __shared__ double red[3][256];
    red[0][threadIdx.x] = sf;
    red[1][threadIdx.x] = sr;
    red[2][threadIdx.x] = so;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h)
            for (int q = 0; q < 3; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (m2mf) m2mf[pr] = red[0][0];
        if (m2mr) m2mr[pr] = red[1][0];
        if (m2o2mr) m2o2mr[pr] = red[2][0];
    }
}

cudaError_t launch_m2(cudaStream_t st, int k0, int k1, int nm, int diag, const double *f, const double *wf,
                      const double *psd, FrfPar frf, double *m2mf, double *m2mr, double *m2o2mr) {
    launch_next(k_m2, diag ? nm : nm * nm, 256, 0, st, k0, k1, nm, diag, f, wf, psd, frf, m2mf, m2mr, m2o2mr);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Stages (b)+(c) in FP64, one block per (point group, tile of NOT (n,o) pairs).
// ------------------------------------------------------------------------------------
constexpr int KC = 32;

// PAIR: the three terms of a point are read from products E(x, y) of its frequency pairs
// (bsa_list64.cu) instead of formed from the A rows.
template <int NOT, int MT, bool PAIR>
__global__ __launch_bounds__(256) void k_bfm_fp64(const double *__restrict__ A,
                                                  const double *__restrict__ Q, int K, int nm,
                                                  PointSrc ps, long long npts, FrfPar frf, PairPts pp,
                                                  double *__restrict__ part_mf,
                                                  double *__restrict__ part_mr,
                                                  double *__restrict__ bf_out,
                                                  double *__restrict__ br_out) {
    after_previous();
    constexpr int MG = 256 / NOT;  // m-groups; thread owns m = mg + MG * u, u < MT
    const int tile = blockIdx.x, pg = blockIdx.y, G = gridDim.y;
    const int t = threadIdx.x, nol = t % NOT, mg = t / NOT;
    const int nm2 = nm * nm;
    const long long nm3 = (long long)nm2 * nm;
    const int no = tile * NOT + nol;
    const bool ok = no < nm2;
    const int n = ok ? no % nm : 0, o = ok ? no / nm : 0;
    extern __shared__ double sm[];
    double *Qs = sm;
    double *Zs = Qs + KC * nm;
    double *Ps = Zs + KC * nm;
    double *Rs = Ps + KC * NOT;
    double *Hs = PAIR ? sm : Rs + KC * NOT;  // [3][nm][2]
    double smf[MT], smr[MT];
#pragma unroll
    for (int u = 0; u < MT; ++u) smf[u] = smr[u] = 0.0;
    const size_t tab = (size_t)K * nm;
    for (long long p = pg; p < npts; p += G) {
        int ix, iy, iz;
        double w, f1, f2;
        get_point(ps, p, ix, iy, iz, w, f1, f2);
        const double *X = A + (size_t)ix * tab;
        const double *Y = A + (size_t)iy * tab;
        const double *Z = iz >= 0 ? A + (size_t)iz * tab : nullptr;
        double acc[MT];
#pragma unroll
        for (int u = 0; u < MT; ++u) acc[u] = 0.0;
        if constexpr (PAIR) {
            // T1 = E(x, y)[(m, n), o], T2 = E(z, y)[(n, m), o], T3 = E(x, z)[(o, n), m]; a product kept
            // as E(y, x) is read with its last two indices exchanged
            const int *e3 = pp.pe + 3 * p;
            auto src = [&](int w) { return e3[w] >= 0 ? pp.E + (size_t)(e3[w] >> 1) * nm3 : nullptr; };
            const double *E1 = src(0), *E2 = src(1), *E3 = src(2);
            const int t1 = e3[0] & 1, t2 = e3[1] & 1, t3 = e3[2] & 1;
            const int i1 = t1 ? o * nm + n : n * nm + o;           // + m nm^2
            const int s2 = t2 ? 1 : nm, i2 = n * nm2 + (t2 ? o * nm : o);   // + m s2
            const int s3 = t3 ? nm : 1, i3 = o * nm2 + (t3 ? n : n * nm);   // + m s3
#pragma unroll
            for (int u = 0; u < MT; ++u) {
                const int m = mg + MG * u;
                if (ok && m < nm) {
                    double v = E1 ? E1[(size_t)m * nm2 + i1] : 0.0;
                    if (E2) v += E2[i2 + m * s2];
                    if (E3) v += E3[i3 + m * s3];
                    acc[u] = v;
                }
            }
        }
        for (int k0 = 0; !PAIR && k0 < K; k0 += KC) {
            const int kc = min(KC, K - k0);
            for (int e = t; e < kc * nm; e += 256) {
                Qs[e] = Q[(size_t)k0 * nm + e];
                Zs[e] = Z ? Z[(size_t)k0 * nm + e] : 0.0;
            }
            for (int e = t; e < kc * NOT; e += 256) {
                const int kk = e / NOT, jl = e % NOT, pr = tile * NOT + jl;
                double pv = 0.0, rv = 0.0;
                if (pr < nm2) {
                    const int nn = pr % nm, oo = pr / nm;
                    const size_t r = (size_t)(k0 + kk) * nm;
                    const double x = X[r + nn], y = Y[r + oo], qn = Q[r + nn], qo = Q[r + oo];
                    pv = x * y;
                    rv = fma(qn, y, x * qo);
                }
                Ps[e] = pv;
                Rs[e] = rv;
            }
            __syncthreads();
            if (ok) {
                for (int kk = 0; kk < kc; ++kk) {
                    const double pv = Ps[kk * NOT + nol], rv = Rs[kk * NOT + nol];
                    const double *qr = Qs + kk * nm, *zr = Zs + kk * nm;
#pragma unroll
                    for (int u = 0; u < MT; ++u) {
                        const int m = mg + MG * u;
                        if (m < nm) acc[u] = fma(qr[m], pv, fma(zr[m], rv, acc[u]));
                    }
                }
            }
            __syncthreads();
        }
        if (ps.cptr) {
            // listed BRM points (triangular zones): G = sum_e c_e Re[H_m(w1_e) H_n(w2_e) conj H_o(w1_e + w2_e)]
            double g[MT];
#pragma unroll
            for (int u = 0; u < MT; ++u) g[u] = 0.0;
            const long long e1 = ps.cptr[p + 1];
            for (long long e = ps.cptr[p]; e < e1; ++e) {
                const double v1 = ps.cq[3 * e] * kPi2, v2 = ps.cq[3 * e + 1] * kPi2, ce = ps.cq[3 * e + 2];
                if (t < nm) {
                    frf_eval(frf.M[t], frf.K[t], frf.C[t], v1, Hs[2 * t], Hs[2 * t + 1]);
                    frf_eval(frf.M[t], frf.K[t], frf.C[t], v2, Hs[2 * nm + 2 * t], Hs[2 * nm + 2 * t + 1]);
                    frf_eval(frf.M[t], frf.K[t], frf.C[t], v1 + v2, Hs[4 * nm + 2 * t], Hs[4 * nm + 2 * t + 1]);
                }
                __syncthreads();
                if (ok) {
                    const double h2r = Hs[2 * nm + 2 * n], h2i = Hs[2 * nm + 2 * n + 1];
                    const double h3r = Hs[4 * nm + 2 * o], h3i = Hs[4 * nm + 2 * o + 1];
                    const double cr = h2r * h3r + h2i * h3i, ci = h2i * h3r - h2r * h3i;
#pragma unroll
                    for (int u = 0; u < MT; ++u) {
                        const int m = mg + MG * u;
                        if (m < nm) g[u] = fma(ce, Hs[2 * m] * cr - Hs[2 * m + 1] * ci, g[u]);
                    }
                }
                __syncthreads();
            }
            if (ok) {
#pragma unroll
                for (int u = 0; u < MT; ++u) {
                    const int m = mg + MG * u;
                    if (m < nm) {
                        const double bfv = 2.0 * acc[u];
                        smf[u] = fma(w, bfv, smf[u]);
                        smr[u] = fma(g[u], bfv, smr[u]);
                    }
                }
            }
            continue;
        }
        if (ps.zones) {
            // Mesher zone point: the force bispectrum of this BFM lattice point enters every
            // BRM lattice point of its bilinear support with weight lambda; accumulate
            // G = sum_q lambda_q w_q Re[H_m(w1_q) H_n(w2_q) conj H_o(w1_q + w2_q)].
            const ZoneDev z = ps.zones[ps.zid[p]];
            const long long off = ps.zoff ? ps.zoff[ps.zid[p]] : -1;
            if (off >= 0) {
                // lattice along the axes: f1 changes along one lattice direction (a) only and f2 along the
                // other (b), so G = Re sum_a H_m(a) S_no(a), S_no(a) = sum_b w_ab H_n(b) conj H_o(a, b):
                // the inner sum once per (n, o), one a per m group at a time, the FRF values from the
                // zone's table.  Evaluated per point and block by one warp and summed per (m, n, o), the FRF
                // part took 3.0 ms of the 200-node, 16-mode building's 128 zones (1523 points); now 0.4.
                const bool ax = z.dIj == 0.0 && z.dJi == 0.0;  // f1 along the I direction
                const int la = ax ? ps.zi[p] : ps.zj[p], lb = ax ? ps.zj[p] : ps.zi[p];
                const int Fa = ax ? z.Fi : z.Fj, Fb = ax ? z.Fj : z.Fi;
                const int Na = ((ax ? z.ni : z.nj) - 1) * Fa, Nb = ((ax ? z.nj : z.ni) - 1) * Fb;
                const int a0 = max(0, la * Fa + 1 - Fa), a1 = min(Na, la * Fa + Fa - 1);
                const int b0 = max(0, lb * Fb + 1 - Fb), b1 = min(Nb, lb * Fb + Fb - 1);
                const double2 *H1 = ps.zH + off, *H2 = H1 + (size_t)(Na + 1) * nm, *H3 = H2 + (size_t)(Nb + 1) * nm;
                const double wz = z.sym * (z.wI / z.Fi) * (z.wJ / z.Fj), ra = 1.0 / Fa, rb = 1.0 / Fb;
                double2 *Ss = (double2 *)Hs;  // [MG][NOT]
                double g[MT];
#pragma unroll
                for (int u = 0; u < MT; ++u) g[u] = 0.0;
                for (int ac = a0; ac <= a1; ac += MG) {
                    const int qa = ac + mg;
                    double sr = 0.0, si = 0.0;
                    if (ok && qa <= a1) {
                        for (int qb = b0; qb <= b1; ++qb) {
                            const double wb = (1.0 - abs(qb - lb * Fb) * rb) * ((qb == 0 || qb == Nb) ? 0.5 : 1.0);
                            const double2 h2 = H2[(size_t)qb * nm + n], h3 = H3[((size_t)qa * (Nb + 1) + qb) * nm + o];
                            const double xr = wb * h2.x, xi = wb * h2.y;
                            sr = fma(xr, h3.x, fma(xi, h3.y, sr));
                            si = fma(xi, h3.x, fma(-xr, h3.y, si));
                        }
                        const double wa = wz * (1.0 - abs(qa - la * Fa) * ra) * ((qa == 0 || qa == Na) ? 0.5 : 1.0);
                        sr *= wa;
                        si *= wa;
                    }
                    __syncthreads();
                    Ss[mg * NOT + nol] = make_double2(sr, si);
                    __syncthreads();
                    if (ok) {
                        const int na = min(MG, a1 - ac + 1);
                        for (int q = 0; q < na; ++q) {
                            const double2 s2 = Ss[q * NOT + nol];
#pragma unroll
                            for (int u = 0; u < MT; ++u) {
                                const int m = mg + MG * u;
                                if (m < nm) {
                                    const double2 h1 = H1[(size_t)(ac + q) * nm + m];
                                    g[u] = fma(h1.x, s2.x, fma(-h1.y, s2.y, g[u]));
                                }
                            }
                        }
                    }
                }
                if (ok) {
#pragma unroll
                    for (int u = 0; u < MT; ++u) {
                        const int m = mg + MG * u;
                        if (m < nm) {
                            const double bfv = 2.0 * acc[u];
                            smf[u] = fma(w, bfv, smf[u]);
                            smr[u] = fma(g[u], bfv, smr[u]);
                        }
                    }
                }
                __syncthreads();
                continue;
            }
            const int li = ps.zi[p], lj = ps.zj[p];
            const int NI = (z.ni - 1) * z.Fi, NJ = (z.nj - 1) * z.Fj;  // last BRM index
            double g[MT];
#pragma unroll
            for (int u = 0; u < MT; ++u) g[u] = 0.0;
            for (int di = 1 - z.Fi; di < z.Fi; ++di) {
                const int qi = li * z.Fi + di;
                if (qi < 0 || qi > NI) continue;
                for (int dj = 1 - z.Fj; dj < z.Fj; ++dj) {
                    const int qj = lj * z.Fj + dj;
                    if (qj < 0 || qj > NJ) continue;
                    const double lam = (1.0 - (double)abs(di) / z.Fi) * (1.0 - (double)abs(dj) / z.Fj);
                    const double ti = (qi == 0 || qi == NI) ? 0.5 : 1.0, tj = (qj == 0 || qj == NJ) ? 0.5 : 1.0;
                    const double wq = z.sym * (z.wI / z.Fi) * (z.wJ / z.Fj) * ti * tj * lam;
                    const double a = (double)qi / z.Fi, bq = (double)qj / z.Fj;
                    const double q1 = z.fi0 + a * z.dIi + bq * z.dJi, q2 = z.fj0 + a * z.dIj + bq * z.dJj;
                    const double v1 = q1 * kPi2, v2 = q2 * kPi2;
                    if (t < nm) {
                        frf_eval(frf.M[t], frf.K[t], frf.C[t], v1, Hs[2 * t], Hs[2 * t + 1]);
                        frf_eval(frf.M[t], frf.K[t], frf.C[t], v2, Hs[2 * nm + 2 * t], Hs[2 * nm + 2 * t + 1]);
                        frf_eval(frf.M[t], frf.K[t], frf.C[t], v1 + v2, Hs[4 * nm + 2 * t], Hs[4 * nm + 2 * t + 1]);
                    }
                    __syncthreads();
                    if (ok) {
                        const double h2r = Hs[2 * nm + 2 * n], h2i = Hs[2 * nm + 2 * n + 1];
                        const double h3r = Hs[4 * nm + 2 * o], h3i = Hs[4 * nm + 2 * o + 1];
                        const double cr = h2r * h3r + h2i * h3i, ci = h2i * h3r - h2r * h3i;
#pragma unroll
                        for (int u = 0; u < MT; ++u) {
                            const int m = mg + MG * u;
                            if (m < nm) g[u] = fma(wq, Hs[2 * m] * cr - Hs[2 * m + 1] * ci, g[u]);
                        }
                    }
                    __syncthreads();
                }
            }
            if (ok) {
#pragma unroll
                for (int u = 0; u < MT; ++u) {
                    const int m = mg + MG * u;
                    if (m < nm) {
                        const double bfv = 2.0 * acc[u];
                        smf[u] = fma(w, bfv, smf[u]);
                        smr[u] = fma(g[u], bfv, smr[u]);
                    }
                }
            }
            continue;
        }
        const double w1 = f1 * kPi2, w2 = f2 * kPi2;
        if (t < nm) {
            frf_eval(frf.M[t], frf.K[t], frf.C[t], w1, Hs[2 * t], Hs[2 * t + 1]);
            frf_eval(frf.M[t], frf.K[t], frf.C[t], w2, Hs[2 * nm + 2 * t], Hs[2 * nm + 2 * t + 1]);
            frf_eval(frf.M[t], frf.K[t], frf.C[t], w1 + w2, Hs[4 * nm + 2 * t], Hs[4 * nm + 2 * t + 1]);
        }
        __syncthreads();
        if (ok) {
            const double h2r = Hs[2 * nm + 2 * n], h2i = Hs[2 * nm + 2 * n + 1];
            const double h3r = Hs[4 * nm + 2 * o], h3i = Hs[4 * nm + 2 * o + 1];
            // H_n(w2) conj(H_o(w1+w2))
            const double cr = h2r * h3r + h2i * h3i, ci = h2i * h3r - h2r * h3i;
#pragma unroll
            for (int u = 0; u < MT; ++u) {
                const int m = mg + MG * u;
                if (m < nm) {
                    const double F = Hs[2 * m] * cr - Hs[2 * m + 1] * ci;
                    const double bfv = 2.0 * acc[u];
                    const double brv = bfv * F;
                    smf[u] = fma(w, bfv, smf[u]);
                    smr[u] = fma(w, brv, smr[u]);
                    const size_t idx = (size_t)p * nm3 + m + (size_t)nm * no;
                    if (bf_out) bf_out[idx] = bfv;
                    if (br_out) br_out[idx] = brv;
                }
            }
        }
        __syncthreads();
    }
    if (ok) {
#pragma unroll
        for (int u = 0; u < MT; ++u) {
            const int m = mg + MG * u;
            if (m < nm) {
                const size_t idx = (size_t)pg * nm3 + m + (size_t)nm * no;
                part_mf[idx] = !pp.first ? part_mf[idx] + smf[u] : smf[u];
                part_mr[idx] = !pp.first ? part_mr[idx] + smr[u] : smr[u];
            }
        }
    }
}

static int not_for(int nm) {
    const int nm2 = nm * nm;
    return nm2 >= 64 ? 64 : (nm2 > 16 ? 32 : 16);
}

int bfm_fp64_groups(long long npts, int nm) {
    const int NOT = not_for(nm);
    const int tiles = (nm * nm + NOT - 1) / NOT;
    long long g = (1216 + tiles - 1) / tiles;  // about 8 blocks per SM on 152 SMs
    g = std::min<long long>(g, npts);
    g = std::min<long long>(g, 65535);
    return (int)std::max<long long>(g, 1);
}

template <int NOT, int MT>
static cudaError_t launch_bfm_t(cudaStream_t st, const double *A, const double *Q, int K, int nm,
                                const PointSrc &ps, long long npts, FrfPar frf, const PairPts &pp, int n_groups,
                                double *part_mf, double *part_mr, double *bf_out, double *br_out) {
    const size_t smem = sizeof(double) * ((pp.E ? 0 : 2 * KC * nm + 2 * KC * NOT) + std::max(6 * nm, ps.zoff ? 2 * 256 : 0));
    const auto kern = pp.E ? k_bfm_fp64<NOT, MT, true> : k_bfm_fp64<NOT, MT, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((nm * nm + NOT - 1) / NOT), (unsigned)n_groups);
    launch_next(kern, grid, 256, smem, st, A, Q, K, nm, ps, npts, frf, pp, part_mf, part_mr, bf_out, br_out);
    return cudaGetLastError();
}

// MT = smallest supported count >= ceil(nm / MG), so no thread carries idle mode slots.
template <int NOT>
static cudaError_t launch_bfm_n(cudaStream_t st, const double *A, const double *Q, int K, int nm,
                                const PointSrc &ps, long long npts, FrfPar frf, const PairPts &pp, int n_groups,
                                double *part_mf, double *part_mr, double *bf_out, double *br_out) {
    constexpr int MG = 256 / NOT;
    const int need = (nm + MG - 1) / MG;
#define BSA_MT_CASE(V)                                                                                       \
    if (need <= V)                                                                                           \
        return launch_bfm_t<NOT, V>(st, A, Q, K, nm, ps, npts, frf, pp, n_groups, part_mf, part_mr, bf_out, br_out);
    BSA_MT_CASE(1)
    BSA_MT_CASE(2)
    BSA_MT_CASE(4)
    BSA_MT_CASE(6)
    BSA_MT_CASE(8)
    BSA_MT_CASE(12)
    BSA_MT_CASE(16)
#undef BSA_MT_CASE
    return cudaErrorInvalidValue;
}

// The zones' FRF tables (PointSrc::zH): a thread per value.
__global__ void k_zone_frf(int nz, int nm, const ZoneDev *__restrict__ zones, const long long *__restrict__ zoff,
                           long long total, FrfPar frf, double2 *__restrict__ H) {
    after_previous();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    int lo = 0, up = nz - 1;  // last zone that has a table starting at or before t (zoff[nz + k]: running starts)
    while (lo < up) {
        const int mid = (lo + up + 1) >> 1;
        if (zoff[nz + mid] <= t) lo = mid; else up = mid - 1;
    }
    const ZoneDev z = zones[lo];
    const bool ax = z.dIj == 0.0 && z.dJi == 0.0;
    const int Fa = ax ? z.Fi : z.Fj, Fb = ax ? z.Fj : z.Fi;
    const int Na = ((ax ? z.ni : z.nj) - 1) * Fa + 1, Nb = ((ax ? z.nj : z.ni) - 1) * Fb + 1;
    const long long r = (t - zoff[nz + lo]) / nm;
    const int m = (int)((t - zoff[nz + lo]) - r * nm);
    auto f1 = [&](int a) { return (z.fi0 + (double)a / Fa * (ax ? z.dIi : z.dJi)) * kPi2; };
    auto f2 = [&](int b) { return (z.fj0 + (double)b / Fb * (ax ? z.dJj : z.dIj)) * kPi2; };
    double w;
    if (r < Na) w = f1((int)r);
    else if (r < Na + Nb) w = f2((int)(r - Na));
    else {
        const long long q = r - Na - Nb;
        w = f1((int)(q / Nb)) + f2((int)(q % Nb));
    }
    double hr, hi;
    frf_eval(frf.M[m], frf.K[m], frf.C[m], w, hr, hi);
    H[t] = make_double2(hr, hi);
}

cudaError_t launch_zone_frf(cudaStream_t st, int nz, int nm, const ZoneDev *zones, const long long *zoff, long long total,
                            FrfPar frf, double2 *H) {
    if (total == 0) return cudaSuccess;
    launch_next(k_zone_frf, (unsigned)((total + 255) / 256), 256, 0, st, nz, nm, zones, zoff, total, frf, H);
    return cudaGetLastError();
}

cudaError_t launch_bfm_fp64(cudaStream_t st, const double *A, const double *Q, int K, int nm,
                            const PointSrc &ps, long long npts, FrfPar frf, int n_groups,
                            double *part_mf, double *part_mr, double *bf_out, double *br_out, const PairPts &pp) {
    if (nm > 64 || nm < 1) return cudaErrorInvalidValue;
    if (npts == 0) return cudaSuccess;
    switch (not_for(nm)) {
    case 64:
        return launch_bfm_n<64>(st, A, Q, K, nm, ps, npts, frf, pp, n_groups, part_mf, part_mr, bf_out, br_out);
    case 32:
        return launch_bfm_n<32>(st, A, Q, K, nm, ps, npts, frf, pp, n_groups, part_mf, part_mr, bf_out, br_out);
    default:
        return launch_bfm_n<16>(st, A, Q, K, nm, ps, npts, frf, pp, n_groups, part_mf, part_mr, bf_out, br_out);
    }
}

// Sum over the groups of part[g][x], fixed order: 32 x per block (coalesced), blockDim.y lanes over
// the groups and a shared-memory tree.  One thread per x walking every group was bound by load
// latency: the 30-node tower's 1216 groups of 64 elements took 0.50 ms.
__global__ void k_reduce_groups(int n_groups, long long len, const double *__restrict__ part,
                                double *__restrict__ out, const double *__restrict__ part2,
                                double *__restrict__ out2, EndFlags fl) {
    after_previous();
    end_flags(fl);
    __shared__ double red[2][32][33];
    const long long x = (long long)blockIdx.x * 32 + threadIdx.x;
    const int ty = threadIdx.y;
    double s = 0.0, s2 = 0.0;
    if (x < len)
        for (int g = ty; g < n_groups; g += blockDim.y) {
            s += part[(size_t)g * len + x];
            if (part2) s2 += part2[(size_t)g * len + x];
        }
    red[0][ty][threadIdx.x] = s;
    red[1][ty][threadIdx.x] = s2;
    for (int h = blockDim.y >> 1; h > 0; h >>= 1) {
        __syncthreads();
        if (ty < h) {
            red[0][ty][threadIdx.x] += red[0][ty + h][threadIdx.x];
            red[1][ty][threadIdx.x] += red[1][ty + h][threadIdx.x];
        }
    }
    if (ty == 0 && x < len) {
        out[x] = red[0][0][threadIdx.x];
        if (out2) out2[x] = red[1][0][threadIdx.x];
    }
}

cudaError_t launch_reduce_groups(cudaStream_t st, int n_groups, long long len, const double *part,
                                 double *out, const double *part2, double *out2, EndFlags fl) {
    if (len == 0) return cudaSuccess;
    // a lane sums at most four groups where the block allows it
    int ny = 1;
    while (ny < 32 && 4 * ny < n_groups) ny *= 2;
    launch_next(k_reduce_groups, (unsigned)((len + 31) / 32), dim3(32, ny), 0, st, n_groups, len, part, out, part2, out2, fl);
    return cudaGetLastError();
}

}  // namespace bsa
