// bsa_kernels.cuh -- launchers of the FP64 kernels (internal C++ interface of libbsagpu).
#pragma once
#include "bsa_common.cuh"

namespace bsa {

// Nodal PSD S[f][itc][i] for nf frequencies (evalPSD_ and the model functions,
// src/wind/WindPSDImpl.F90:123-316).  tcs: turbulent component ids (1..3) per itc.  expt
// (FP64): sqrt(S) instead, and the A kernel's exponential table into expt.
cudaError_t launch_nodal_psd(cudaStream_t st, int nf, const double *f, int ntc, const int *tcs_host,
                             int nnl, const PsdNode *par, int psd_type, int scaling, double *S, bool fp32 = false,
                             double *expt = nullptr);

// log c_ij [itc][i][j] of the loaded nodes (1-based ids) from the packed coherences corr[itc][ncorr] of
// nn nodes, in FP64 and FP32.  lc has room for the A kernel's exponential table behind it
// and a flag (log_coh_bad) that says whether a coherence lies outside [0, 1] or a node's own is not 1
// (log_coh_bytes(n) in all, n = ntc nnl^2).
size_t log_coh_bytes(size_t n);
int *log_coh_bad(const double *lc, size_t n);
cudaError_t launch_log_coh(cudaStream_t st, int ntc, int nnl, int nn, long long ncorr, const int *nodes, const double *corr,
                           double *lc, float *lc32);

// A[f][k][m] = sqrt(S_i(f)) sum_j c_ij^|f| sqrt(S_j(f)) L[(itc,j)][m]  (FP64); rootS = sqrt(S), logc
// followed by the exponential's table (launch_nodal_psd's expt).  only: form nothing where *only is 0.
cudaError_t launch_atable(cudaStream_t st, int nf, const double *f, int ntc, int nnl, int nm,
                          const double *logc, const double *rootS, const double *L, double *A, const int *only = nullptr);

// The same on the tensor cores (bsa_atable64_tc.cu); leaves A alone where *bad is set (then launch_atable
// with only = bad forms it).  scratch: atable64_tc_scratch(nf, ntc, nnl, nm) bytes; err receives a
// nonzero code if a pipeline wait ran out of its budget.  test_skip1: pass + 1 whose ready signal block 0 omits.
size_t atable64_tc_scratch(int nf, int ntc, int nnl, int nm);
cudaError_t launch_atable64_tc(cudaStream_t st, int nf, const double *f, int ntc, int nnl, int nm, const double *logc,
                               const double *rootS, const double *L, const int *bad, double *A, void *scratch, int *err,
                               int test_skip1 = 0);


// The FP32 table on the tensor cores (bsa_atable_tc.cu): tf32 hi/lo split, FP32 accumulation;
// err receives a nonzero code if a pipeline wait ran out of its budget.  nm <= 64.
// scratch: atable_tc_scratch(ntc, nnl, nm) bytes (the split B tables).
size_t atable_tc_scratch(int ntc, int nnl, int nm);
cudaError_t launch_atable_tc(cudaStream_t st, int nf, const double *f, int ntc, int nnl, int nm,
                             const float *logc, const double *S, const float *L, float *A, void *scratch, int *err);

// Force PSD on the grid psd[f][n + nm*o] = sum_k L[k][o] A[f][k][n]
// (functionsImpl.F90:1548-1560), then the second-order moments
// m2mf, m2mr (x Re[H_o conj H_n]), m2o2mr (x w^2) with per-frequency weights wf.
cudaError_t launch_force_psd(cudaStream_t st, int nf, int ntc, int nnl, int nm, const double *L,
                             const double *A, double *psd);
cudaError_t launch_force_psd32(cudaStream_t st, int nf, int ntc, int nnl, int nm, const float *L,
                               const float *A, double *psd);
// Second-order moments over the grid frequencies k in [k0, k1); diag != 0 for the
// same-mode spectra psd[f][m].
cudaError_t launch_m2(cudaStream_t st, int k0, int k1, int nm, int diag, const double *f, const double *wf,
                      const double *psd, FrfPar frf, double *m2mf, double *m2mr, double *m2o2mr);

// Projected wind coefficients (bsa_kernels.cu): L, Q, Q L^2, L^2 [k][m] and L in FP32; nl = 0: wfc holds the
// projections.
cudaError_t launch_project(cudaStream_t st, int K, int nm, int nl, const double *wfc, const double *phi, int nnl, double *L,
                           double *Q, double *W3, double *W2, float *L32);

// Diagonal-only force PSD psd[f][m] = sum_k W2[k][m] S[f][k], W2 = L^2 (functionsImpl.F90:1924-1947).
cudaError_t launch_force_psd_diag(cudaStream_t st, int nf, int K, int nm, const double *S, const double *W2,
                                  double *psd);

// FP64 BFM contraction + FRF + weighted reduction over a point set.
//   B_F[m,n,o](p) = 2 sum_k ( Q_km X_kn Y_ko + Z_km (Q_kn Y_ko + X_kn Q_ko) ),
//   X = A(f1), Y = A(f2), Z = A(f1+f2)   (the exact factorisation of the nodal triple sum
//   of functionsImpl.F90:1494-1538), B_R = B_F * Re[H_m(w1) H_n(w2) conj H_o(w1+w2)].
// part_mf / part_mr receive one nm^3 partial per point group (n_groups of them);
// bf_out / br_out (optional) receive B_F / B_R per point, (nm^3, npts).
// pp.E set: the points' terms from pair products E[pair][a nm + b][j] instead of A and Q; point p reads
// pairs pp.pe[3 p + 0 .. 2] (f1 f2, f1+f2 f2, f1 f1+f2) = 2 pair + (product kept with its two
// frequencies exchanged), or -1 for a zero term; !pp.first: the partials are added to.
struct PairPts {
    const double *E = nullptr;
    const int *pe = nullptr;
    int first = 1;
};
cudaError_t launch_bfm_fp64(cudaStream_t st, const double *A, const double *Q, int K, int nm,
                            const PointSrc &ps, long long npts, FrfPar frf, int n_groups,
                            double *part_mf, double *part_mr, double *bf_out, double *br_out, const PairPts &pp = PairPts());
int bfm_fp64_groups(long long npts, int nm);

// The FRF tables of PointSrc::zH (total values): zoff holds nz offsets (< 0: zone without a table), then
// the nz running starts.
cudaError_t launch_zone_frf(cudaStream_t st, int nz, int nm, const ZoneDev *zones, const long long *zoff, long long total,
                            FrfPar frf, double2 *H);

// out[x] = sum_g part[g * len + x] (fixed order); optional second array.
cudaError_t launch_reduce_groups(cudaStream_t st, int n_groups, long long len, const double *part,
                                 double *out, const double *part2, double *out2, EndFlags fl = EndFlags());

}  // namespace bsa
