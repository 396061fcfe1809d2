// bsa_pair64_tc.cu -- FP64 products on the tensor cores, by error-free splitting (K. Ozaki,
// T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59, 2012; on half-precision tensor cores:
// D. Mukunoki, K. Ozaki, T. Ogita, T. Imamura, ISC 2020).
//
// Each operand row (fixed x, a, b or y, j; contiguous k) is scaled by a power of two above its
// largest magnitude, rounded to a 62-bit integer and cut into eight balanced base-256 digits
// |d| <= 128, stored as bf16 (exact).  The digit products s + t = l < 8 are summed in FP32 in TMEM:
// at most 8 x 128 products of at most 2^14, so every partial sum is an integer within 2^24 and
// exact; longer K is cut into passes of 128 whose sums meet in 64-bit integers.  The eight level
// sums combine exactly in integers and round once to FP64, with no FP64 instruction (the pipe is
// two lanes an SM and clock).
//
// Error: rounding the rows at 2^-63 of their scale and leaving out the levels s + t >= 8 is an absolute
// error of at most K 2^-59 of the row's scale times the column's.  Against the FP64 FMAs' bound K 2^-53
// sum |a_k b_k| that is no more wherever the sum is at least 2^-6 of the scales; an element whose terms are
// all smaller (two modes that move different nodes) is found and computed again on the FP64 pipe
// (k_pair_mend), so every element keeps FP64's own precision.  With seven digits the bound was met only from
// four times the scales up: elements between two groups of nodes 50 m apart were off by 2e-11 of themselves.
//
// Cost: 36 digit products of bf16 against the DFMA kernel's one FP64 FMA: 36 / 4096 clocks of an SM
// against 1 / 2.  Tile: 128 rows by 32 columns; the B digits of the tile are stacked along N (256
// rows), so A digit s meets B digits 0 .. 7 - s in one MMA of N = (8 - s) 32 whose columns land on
// levels s .. 7: 8 MMAs a K step instead of 36, and 512 TMEM columns hold two tiles.  Bound by shared
// memory at long K (operand reads and TMA writes exceed the MMA clocks), by the drain of the
// level sums at short K: 16 warps share it.  400 nodes x 2 components, 24 modes, 65 rows: FP64 pipe
// 40.5 ms; 1.32 ms here (8.5e11 digit FMAs), row digits 0.10 ms, the search for small elements 0.09 ms; 173
// nodes, 11 modes, 97 rows 86 us, 13 and 28.  Seven digits: 1.19 ms and 79 us.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "bsa_digits.cuh"
#include "bsa_pair64.cuh"

namespace bsa {
namespace p64 {

using namespace tc;

constexpr int kPassK = kPassMax / kBK;   // K blocks of one exact pass
constexpr int kRingA = kDig;             // A digit tiles in flight (16 KB each): digit s in slot s
constexpr int kRingB = 2;                // B tiles in flight (32 KB each)
constexpr int kTileA = kTM * 128, kTileB = kDig * kTN * 128;
constexpr int kEpiW = 16;                // epilogue warps: four a TMEM lane quarter, a quarter of the columns each
constexpr int kTcThreads = 64 + 32 * kEpiW, kEpiC = kTN * 4 / kEpiW;
constexpr float kSmall = 1.f / 64;       // k_pair_mend
constexpr long long kSmallHi = 1LL << 30;
constexpr size_t kTcSmem = 1024 + (size_t)kRingA * kTileA + (size_t)kRingB * kTileB + 512;

// Column operand: exponent e[c] with |A[y][k][j]| < 2^e[c], c = y an + j.
__global__ __launch_bounds__(256) void k_col_exp(int an, int K, const double *__restrict__ A, int *__restrict__ ec) {
    after_previous();
    __shared__ int mx[64];
    const int y = blockIdx.x;
    if (threadIdx.x < 64) mx[threadIdx.x] = 0;
    __syncthreads();
    const double *a = A + (size_t)y * K * an;
    // a thread keeps one column: 256 / an lanes over k
    const int lanes = 256 / an, j = threadIdx.x % an, lane = threadIdx.x / an;
    int m = 0;
    if (lane < lanes)
        for (int k = lane; k < K; k += lanes) m = max(m, expo(a[(size_t)k * an + j]));
    atomicMax(&mx[j], m);
    __syncthreads();
    if ((int)threadIdx.x < an) {
        const int e = mx[threadIdx.x];
        ec[y * an + threadIdx.x] = e == 2047 ? kBad : e == 0 ? kNone : expo_row(e - 1022);
    }
}

// Row operand: |Q[k][a] A(x)[k][b]| < 2^e[r] from the factors' exponents (at most a bit above).
// 32 rows by 16 or 8 lanes over k per block: where the blocks fit the chip at once a lane's chain of loads
// is the time and 16 lanes halve it (K = 800, 24 rows of 257 frequencies: 26 -> 17 us), where they do not the
// lanes' join counts (K = 150, 144 rows of 2222: 67 us by 8, 81 by 16; these by the high words alone, which do
// not tell the smallest denormals from zero: 73 us by 8 with both words, 43 instead of 36 for 576 rows of 65).
// Zeros, fields and infinities are kept apart until the end: with expo_pair for every k 86 and 55 us.
template <int LANES>
__global__ __launch_bounds__(32 * LANES) void k_row_exp(Chunk c, const double *__restrict__ A, const double *__restrict__ Q,
                                                 int *__restrict__ er) {
    after_previous();
    __shared__ int mx[LANES][32];
    const int qn = c.qn, an = c.an, rx = c.rx(), ab = blockIdx.y * 32 + (threadIdx.x & 31), lane = threadIdx.x >> 5;
    const int x = c.xmap ? c.xmap[blockIdx.x] : c.x0 + blockIdx.x, a = ab / an, b = ab - a * an;
    const double *q = Q + a, *p = A + (size_t)x * c.K * an + b;
    int m = -1, top = 0;  // largest sum of two fields, none yet; largest high word
    if (ab < rx)
#pragma unroll 8
        for (int k = lane; k < c.K; k += LANES) {
            const double u = q[(size_t)k * qn], v = p[(size_t)k * an];
            const int hu = __double2hiint(u) & 0x7fffffff, hv = __double2hiint(v) & 0x7fffffff;
            const unsigned nz = min((unsigned)(hu | __double2loint(u)), (unsigned)(hv | __double2loint(v)));
            m = max(m, nz ? (hu >> 20) + (hv >> 20) : -1);
            top = max(top, max(hu, hv));
        }
    if (top >= 0x7ff00000) m = kBad;
    mx[lane][threadIdx.x & 31] = m;
    __syncthreads();
    if (lane == 0 && ab < rx) {
#pragma unroll
        for (int z = 1; z < LANES; ++z) m = max(m, mx[z][threadIdx.x]);
        er[(size_t)blockIdx.x * c.rpad + ab] = m == kBad ? kBad : m < 0 ? kNone : expo_row(m - 2044);
    }
}

// Column digits [ct][digit][32 columns][Kp]; block: one column tile, 128 k.
__global__ __launch_bounds__(256) void k_col_digits(int nr, int an, int K, int Kp, const double *__restrict__ A,
                                                    const int *__restrict__ ec, __nv_bfloat16 *__restrict__ D) {
    after_previous();
    const int ct = blockIdx.x, col = threadIdx.x & 31, k0 = blockIdx.y * 128 + (threadIdx.x >> 5) * 16;
    if (k0 >= Kp) return;
    const int c = ct * kTN + col, y = c / an, j = c - y * an;
    const bool ok = y < nr;
    const int e = ok ? ec[c] : kNone;
    const bool some = e != kNone && e != kBad;
    double v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = (some && k0 + i < K) ? A[((size_t)y * K + k0 + i) * an + j] : 0.0;
    put_digits<16>(v, some ? e : 0, D + ((size_t)ct * kDig * kTN + col) * Kp + k0, (size_t)kTN * Kp);
}

// Column digits of a pair list [block][digit][bw columns][Kp]; exponents [block][32].
__global__ __launch_bounds__(256) void k_block_digits(int nm, int np, int bw, int K, int Kp, const double *__restrict__ A,
                                                      const int *__restrict__ ec, int *__restrict__ eb,
                                                      __nv_bfloat16 *__restrict__ D) {
    after_previous();
    const int blk = blockIdx.x, col = threadIdx.x & 31, k0 = blockIdx.y * 128 + (threadIdx.x >> 5) * 16;
    const int y = blk / np, j = (blk - y * np) * bw + col;
    const bool ok = col < bw && j < nm;
    const int e = ok ? ec[y * nm + j] : kNone;
    if (blockIdx.y == 0 && threadIdx.x < 32) eb[blk * 32 + col] = e;
    if (k0 >= Kp || col >= bw) return;
    const bool some = e != kNone && e != kBad;
    double v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = (some && k0 + i < K) ? A[((size_t)y * K + k0 + i) * nm + j] : 0.0;
    put_digits<16>(v, some ? e : 0, D + ((size_t)blk * kDig * bw + col) * Kp + k0, (size_t)bw * Kp);
}

// Row digits [mt][digit][128 rows][Kp]; block: one x, 64 k, every (a, b).  Eight lanes cover a row's 64 k,
// so that a warp's store of a digit is four whole 128-byte rows (16 bytes a row at a time, 32 rows a
// store, ran at 1.3 TB/s: 0.36 ms for 65 x 576 rows of 800 k, now 0.11 ms).
__global__ __launch_bounds__(256) void k_row_digits(Chunk c, int Kp, const double *__restrict__ A,
                                                    const double *__restrict__ Q, const int *__restrict__ er,
                                                    __nv_bfloat16 *__restrict__ D) {
    after_previous();
    constexpr int LD = 66;  // [mode][64 k] with 16-byte aligned, staggered rows
    extern __shared__ __align__(16) double sm[];
    const int qn = c.qn, an = c.an, rx = c.rx(), K = c.K, xl = blockIdx.x, kb = blockIdx.y * 64;
    double *As = sm, *Qs = sm + LD * an;
    const int n = max(0, min(64, K - kb));
    const double *a = A + ((size_t)(c.xmap ? c.xmap[xl] : c.x0 + xl) * K + kb) * an, *q = Q + (size_t)kb * qn;
    for (int i = threadIdx.x; i < 64 * an; i += 256) As[i % an * LD + i / an] = i < n * an ? a[i] : 0.0;
    for (int i = threadIdx.x; i < 64 * qn; i += 256) Qs[i % qn * LD + i / qn] = i < n * qn ? q[i] : 0.0;
    __syncthreads();
    const int kq = (threadIdx.x & 7) * 8;
    for (int ab = threadIdx.x >> 3; ab < rx; ab += 32) {
        const int ia = ab / an, ib = ab - ia * an;
        const long long r = (long long)xl * c.rpad + ab;
        const int e = er[r];
        const bool some = e != kNone && e != kBad;
        const double2 *pa = reinterpret_cast<const double2 *>(As + ib * LD + kq), *pq = reinterpret_cast<const double2 *>(Qs + ia * LD + kq);
        double v[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double2 u = pa[i], w = pq[i];
            v[2 * i] = some ? w.x * u.x : 0.0;
            v[2 * i + 1] = some ? w.y * u.y : 0.0;
        }
        put_digits<8>(v, some ? e : 0, D + ((r / kTM) * kDig * kTM + r % kTM) * (size_t)Kp + kb + kq, (size_t)kTM * Kp);
    }
}

// LIST: the items and column blocks of a pair list instead of the chunk's tile rows.
template <bool LIST>
__global__ void __launch_bounds__(kTcThreads, 1)
    k_pair_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, Chunk c, PairList pl,
              int nk, int ks_last, const int *__restrict__ er, const int *__restrict__ ec, uint8_t *__restrict__ small, int *err) {
    after_previous();
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sa = smem, *sb = smem + (size_t)kRingA * kTileA;
    uint64_t *bars = (uint64_t *)(sb + (size_t)kRingB * kTileB);
    uint64_t *fa = bars, *ea = fa + kRingA, *fb = ea + kRingA, *eb = fb + kRingB, *tfull = eb + kRingB, *tempty = tfull + 2,
             *done = tempty + 2;
    uint32_t *tmem_slot = (uint32_t *)(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRingA; ++s) {
            mbar_init(&fa[s], 1);
            mbar_init(&ea[s], 1);
        }
        for (int s = 0; s < kRingB; ++s) {
            mbar_init(&fb[s], 1);
            mbar_init(&eb[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 32 * kEpiW);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(su32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            uint32_t ia = 0, ib = 0;
            bool ok = true;
            for (long long item = blockIdx.x; item < c.items && ok; item += gridDim.x) {
                int mt, ct = 0;
                int4 it = make_int4(0, 0, 0, 0);
                if (LIST) {
                    it = pl.items[item];
                    mt = it.x;
                } else {
                    mt = tile_row(c, item);
                    ct = c.rt[mt].ct0 + (int)(item - c.rt[mt].item0);
                }
                for (int kb = 0; kb < nk && ok; ++kb, ++ib) {
                    const int sB = ib % kRingB;
                    if (!mbar_wait(&eb[sB], ((ib / kRingB) & 1u) ^ 1u, err, 1)) { ok = false; break; }
                    if (LIST) {
                        // blocks side by side within each digit's 32 rows; columns past them hold what was there
                        mbar_expect_tx(&fb[sB], (uint32_t)(it.z * kDig * pl.bw * 128));
                        for (int q = 0; q < it.z; ++q) {
                            const int y = pl.blk[it.y + q] * kDig * pl.bw;
                            for (int t = 0; t < kDig; ++t)
                                tma_2d(sb + sB * kTileB + (t * kTN + q * pl.bw) * 128, &tmB, &fb[sB], kb * kBK, y + t * pl.bw);
                        }
                    } else {
                        mbar_expect_tx(&fb[sB], kTileB);
                        tma_2d(sb + sB * kTileB, &tmB, &fb[sB], kb * kBK, ct * kDig * kTN);
                    }
                    for (int s = 0; s < kDig; ++s, ++ia) {
                        if (!mbar_wait(&ea[s], (ib & 1u) ^ 1u, err, 1)) { ok = false; break; }
                        mbar_expect_tx(&fa[s], kTileA);
                        tma_2d(sa + s * kTileA, &tmA, &fa[s], kb * kBK, (mt * kDig + s) * kTM);
                    }
                }
            }
            // copies in flight land before the block leaves
            for (uint32_t q = (ia > (uint32_t)kRingA ? ia - kRingA : 0); q < ia; ++q) {
                const uint64_t t0 = gtime();
                while (!mbar_try(&fa[q % kRingA], (q / kRingA) & 1u) && gtime() - t0 < kWaitNs) {
                }
            }
            for (uint32_t q = (ib > (uint32_t)kRingB ? ib - kRingB : 0); q < ib; ++q) {
                const uint64_t t0 = gtime();
                while (!mbar_try(&fb[q % kRingB], (q / kRingB) & 1u) && gtime() - t0 < kWaitNs) {
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            uint32_t ib = 0, tile = 0;
            bool ok = true;
            for (long long item = blockIdx.x; item < c.items && ok; item += gridDim.x) {
                for (int k0 = 0; k0 < nk && ok; k0 += kPassK, ++tile) {
                    const int buf = tile & 1;
                    if (!mbar_wait(&tempty[buf], ((tile >> 1) & 1u) ^ 1u, err, 2)) { ok = false; break; }
                    fence_after();
                    const uint32_t d = tmem + buf * 256;
                    const int k1 = min(nk, k0 + kPassK);
                    for (int kb = k0; kb < k1 && ok; ++kb, ++ib) {
                        const int sB = ib % kRingB;
                        if (!mbar_wait(&fb[sB], (ib / kRingB) & 1u, err, 3)) { ok = false; break; }
                        const uint32_t bb = su32(sb + sB * kTileB);
                        const int nks = kb == nk - 1 ? ks_last : kBK / 16;
                        // unrolled: with the loops kept, issuing took longer than the MMAs (a product
                        // of 400 nodes x 2 components, 24 modes, 65 rows 1.80 ms, unrolled 1.33 ms)
#pragma unroll
                        for (int s = 0; s < kDig; ++s) {
                            if (!mbar_wait(&fa[s], ib & 1u, err, 3)) { ok = false; break; }
                            fence_after();
                            const uint32_t ab = su32(sa + s * kTileA);
                            // N = (8 - s) 32 columns from level s on
                            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                                   ((uint32_t)((kDig - s) * kTN >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);
#pragma unroll
                            for (int ks = 0; ks < kBK / 16; ++ks)
                                if (ks < nks)
                                    mma_n(d + s * kTN, sdesc(ab + ks * 32), sdesc(bb + ks * 32), idesc,
                                          (kb > k0 || ks > 0 || s > 0) ? 1u : 0u);
                            mma_commit(&ea[s]);
                        }
                        if (ok) mma_commit(&eb[sB]);
                    }
                    if (ok && !(c.test_skip1 == (int)tile + 1 && blockIdx.x == 0)) mma_commit(&tfull[buf]);
                }
            }
            mma_commit(done);
            const uint64_t t0 = gtime();
            while (!mbar_try(done, 0) && gtime() - t0 < kWaitNs) {
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: 128 rows, kEpiC columns of one a thread ----------------
        const int quarter = warp & 3, row = quarter * 32 + lane, c0 = ((warp - 2) >> 2) * kEpiC;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16) + c0;
        const int nrows = (c.x1 - c.x0) * c.rx(), ncols = (c.hi + 1) * c.an;
        uint32_t tile = 0;
        bool ok = true;
        for (long long item = blockIdx.x; item < c.items && ok; item += gridDim.x) {
            int mt, ct = 0;
            RowTile rt{};
            int4 it = make_int4(0, 0, 0, 0);
            if (LIST) {
                it = pl.items[item];
                mt = it.x;
            } else {
                mt = tile_row(c, item);
                rt = c.rt[mt];
                ct = rt.ct0 + (int)(item - rt.item0);
            }
            long long hi[kEpiC], lo[kEpiC];
#pragma unroll
            for (int q = 0; q < kEpiC; ++q) hi[q] = lo[q] = 0;
            for (int k0 = 0; k0 < nk && ok; k0 += kPassK, ++tile) {
                const int buf = tile & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(&tfull[buf], (tile >> 1) & 1u, err, 4));
                if (!ok) break;
                fence_after();
#pragma unroll
                for (int cg = 0; cg < kEpiC / 8; ++cg) {
#pragma unroll
                    for (int z = 0; z < 2; ++z) {  // levels 0 .. 3, then 4 .. 7
                        uint32_t v[4][8];
#pragma unroll
                        for (int l = 0; l < 4; ++l) tmem_ld8(lane_base + buf * 256 + (4 * z + l) * kTN + cg * 8, v[l]);
                        tmem_wait_ld();
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            int D[4];
#pragma unroll
                            for (int l = 0; l < 4; ++l) D[l] = __float2int_rn(__uint_as_float(v[l][q]));
                            (z ? lo : hi)[cg * 8 + q] += join_levels(D);
                        }
                    }
                }
                fence_before();
                mbar_arrive(&tempty[buf]);
            }
            // value = 2^(er + ec - 68) (hi 2^32 + lo); bit q of the mask: |value| < kSmall 2^(er + ec) or fp64_only, k_pair_mend looks
            uint32_t mask = 0;
            auto value = [&](int q, int eu, int ev) {
                if (fp64_only(eu, ev)) {
                    mask |= 1u << q;
                    return 0.0;
                }
                if (eu == kNone || ev == kNone) return 0.0;
                const long long h = hi[q] + (lo[q] >> 32);
                if (h < kSmallHi && h >= -kSmallHi) mask |= 1u << q;
                return combine(hi[q], lo[q], eu + ev - 68);
            };
            if (LIST) {
                const int nm = c.an, r = (mt % pl.tiles_x) * kTM + row;
                if (ok && r < c.rx()) {
                    const int eu = er[mt * kTM + row];
#pragma unroll
                    for (int q = 0; q < kEpiC; ++q) {
                        const int cc = c0 + q, s = (cc >= pl.bw) + (cc >= 2 * pl.bw) + (cc >= 3 * pl.bw);
                        if (s >= it.z) continue;
                        const int blk = pl.blk[it.y + s], cq = cc - s * pl.bw, j = (blk % pl.np) * pl.bw + cq;
                        if (j < nm)
                            c.E[((size_t)pl.pair[it.y + s] * c.rx() + r) * nm + j] = value(q, eu, ec[blk * 32 + cq]);
                    }
                }
            } else {
                const int r = mt * kTM + row;
                if (ok && r < nrows) {
                    const int eu = er[r];
                    double *o = c.E + rt.base + (size_t)row * rt.nct * kTN + (size_t)(ct - rt.ct0) * kTN + c0;
#pragma unroll
                    for (int q = 0; q < kEpiC; q += 2) {
                        const int col = ct * kTN + c0 + q;
                        *reinterpret_cast<double2 *>(o + q) = make_double2(value(q, eu, col < ncols ? ec[col] : kNone),
                                                                           value(q + 1, eu, col + 1 < ncols ? ec[col + 1] : kNone));
                    }
                }
            }
            if (ok) small[((size_t)item * kTM + row) * (kTN / kEpiC) + (c0 / kEpiC)] = (uint8_t)mask;
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Products whose terms are all small against the scales: k_pair_tc's error is absolute, at most
// K 2^-59 2^(er + ec) (a term's two roundings at 2^-63 and the seven products of level 8), where K FP64
// FMAs are within K 2^-53 sum |a_k b_k|.  So an element keeps its digits only where sum |a_k b_k| >=
// 2^-6 2^(er + ec) = kSmall 2^(er + ec): there the bound is the FMAs' own.  |E| is a lower bound of that
// sum; for the elements below it (mask) the sum itself is formed in FP32, over 16 k spread along K at a time until it
// suffices, and what stays below is computed again as k_pair_gemm does it.  Measured error relative to
// the sum at the threshold, digits / FMAs: K = 24 6e-17 / 1.4e-16, 173 1.0e-16 / 3.6e-16, 800 2.0e-16 /
// 7.9e-16; at 2^-10 of the scales the digits are 4 times the FMAs' error, at 2^-20 4000 times.
// Elements whose row or column exponent is kBad go there at once (fp64_only).
// One block per product tile, most of which end at the first test.
template <bool LIST>
__global__ __launch_bounds__(256) void k_pair_mend(Chunk c, PairList pl, const double *__restrict__ A, const double *__restrict__ Q,
                                                   const int *__restrict__ er, const int *__restrict__ ec,
                                                   const uint32_t *__restrict__ small) {
    after_previous();
    constexpr int KT = 16;
    __shared__ __align__(16) double As[KT][kTM], Bs[KT][kTN];
    const int t = threadIdx.x, tr = (t >> 3) * 4, tc = (t & 7) * 4, qn = c.qn, an = c.an, rx = c.rx(), K = c.K;
    const long long item = blockIdx.x;
    uint32_t bits = 0;  // element (i, q) of this thread: bit 4 i + q
#pragma unroll
    for (int i = 0; i < 4; ++i) bits |= ((small[item * kTM + tr + i] >> tc) & 15u) << (4 * i);
    if (!__syncthreads_or(bits != 0)) return;
    int4 it = make_int4(0, 0, 0, 0);
    RowTile rt{};
    int mt, ct = 0;
    if (LIST) {
        it = pl.items[item];
        mt = it.x;
    } else {
        mt = tile_row(c, item);
        rt = c.rt[mt];
        ct = rt.ct0 + (int)(item - rt.item0);
    }
    // row of the tile: its A row and its place among the rows (a, b) of that; column: A row and mode
    auto row_of = [&](int row, int &x, int &ab) {
        if (LIST) {
            x = c.xmap[mt / pl.tiles_x];
            ab = (mt % pl.tiles_x) * kTM + row;
            return ab < rx;
        }
        const int r = mt * kTM + row;
        x = c.x0 + r / rx;
        ab = r % rx;
        return x < c.x1;
    };
    auto col_of = [&](int cc, int &y, int &j, int &e) {
        if (LIST) {
            const int s = cc / pl.bw;
            if (s >= it.z) return false;
            const int blk = pl.blk[it.y + s], cq = cc - s * pl.bw;
            y = blk / pl.np;
            j = (blk - y * pl.np) * pl.bw + cq;
            e = blk * 32 + cq;
            return j < an;
        }
        e = ct * kTN + cc;
        y = e / an;
        j = e - y * an;
        return y <= c.hi;
    };
    // this thread's staging row and column
    const int sr = t & (kTM - 1), kr = t >> 7, sc = t & (kTN - 1), kc = t >> 5;
    int x, ab, y, j, e;
    const bool rv = row_of(sr, x, ab), cv = col_of(sc, y, j, e);
    const int a = rv ? ab / an : 0, b = rv ? ab - a * an : 0, eu = rv ? er[mt * kTM + sr] : 0, ev = cv ? ec[e] : 0;
    const double *Qa = Q + a, *Ab = A + (size_t)(rv ? x : 0) * K * an + b, *Aj = A + (size_t)(cv ? y : 0) * K * an + (cv ? j : 0);
    float(*Af)[kTM] = reinterpret_cast<float(*)[kTM]>(As);
    float(*Bf)[kTN] = reinterpret_cast<float(*)[kTN]>(Bs);
    float sum[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) sum[i][q] = 0.f;
    // elements of the tile that are none of the product's (the mask of a tile that timed out is not written)
    uint32_t pend = bits;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int u, v, w;
        if (!row_of(tr + i, u, v)) pend &= ~(15u << (4 * i));
        if (!col_of(tc + i, u, v, w)) pend &= ~(0x1111u << i);
    }
    uint32_t only = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int u, v, w;
        if (!col_of(tc + q, u, v, w)) continue;
        const int eq = ec[w];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if ((pend >> (4 * i + q) & 1u) && fp64_only(er[mt * kTM + tr + i], eq)) only |= 1u << (4 * i + q);
    }
    pend &= ~only;
    const int nch = (K + KT - 1) / KT;
    for (int ch = 0; ch < nch && __syncthreads_or(pend != 0); ++ch) {
        for (int u = kr; u < KT; u += 2) {
            const int k = ch + nch * u;
            Af[u][sr] = (rv && k < K) ? scaled_abs(Qa[(size_t)k * qn] * Ab[(size_t)k * an], eu) : 0.f;
        }
        for (int u = kc; u < KT; u += 8) {
            const int k = ch + nch * u;
            Bf[u][sc] = (cv && k < K) ? scaled_abs(Aj[(size_t)k * an], ev) : 0.f;
        }
        __syncthreads();
        if (pend) {
#pragma unroll 4
            for (int u = 0; u < KT; ++u) {
                const float4 p = *reinterpret_cast<const float4 *>(&Af[u][tr]), q = *reinterpret_cast<const float4 *>(&Bf[u][tc]);
                const float ar[4] = {p.x, p.y, p.z, p.w}, br[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int z = 0; z < 4; ++z) sum[i][z] = fmaf(ar[i], br[z], sum[i][z]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int z = 0; z < 4; ++z)
                    if (sum[i][z] >= kSmall) pend &= ~(1u << (4 * i + z));
        }
    }
    // every term zero: so are the digits' product and the FMAs'
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int z = 0; z < 4; ++z)
            if (sum[i][z] == 0.f) pend &= ~(1u << (4 * i + z));
    pend |= only;
    if (!__syncthreads_or(pend != 0)) return;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = 0.0;
    for (int k0 = 0; k0 < K; k0 += KT) {
        const int kn = min(KT, K - k0);
        for (int u = kr; u < kn; u += 2) As[u][sr] = rv ? Qa[(size_t)(k0 + u) * qn] * Ab[(size_t)(k0 + u) * an] : 0.0;
        for (int u = kc; u < kn; u += 8) Bs[u][sc] = cv ? Aj[(size_t)(k0 + u) * an] : 0.0;
        __syncthreads();
        if (pend)
            for (int u = 0; u < kn; ++u) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (pend >> (4 * i + q) & 1u) acc[i][q] = fma(As[u][tr + i], Bs[u][tc + q], acc[i][q]);
            }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (!(pend >> (4 * i + q) & 1u)) continue;
            if (LIST) {
                int y2, j2, e2;
                col_of(tc + q, y2, j2, e2);
                c.E[((size_t)pl.pair[it.y + (tc + q) / pl.bw] * rx + (mt % pl.tiles_x) * kTM + tr + i) * an + j2] = acc[i][q];
            } else {
                c.E[rt.base + (size_t)(tr + i) * rt.nct * kTN + (size_t)(ct - rt.ct0) * kTN + tc + q] = acc[i][q];
            }
        }
}

static int kpad(int K) { return (K + kBK - 1) / kBK * kBK; }
static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

// [digits][exponents], the row operand's followed by the items' masks
size_t tc_col_bytes(int nr, int an, int K) {
    const size_t ct = ((size_t)nr * an + kTN - 1) / kTN;
    return up256(ct * kDig * kTN * kpad(K) * 2) + up256(sizeof(int) * (size_t)nr * an);
}
size_t tc_row_bytes(long long nrows, int K, long long items) {
    const size_t mt = (size_t)((nrows + kTM - 1) / kTM);
    return up256(mt * kDig * kTM * kpad(K) * 2) + up256(sizeof(int) * mt * kTM) + (size_t)items * kTM * kTN / 8;
}

cudaError_t tc_prep_cols(cudaStream_t st, int nr, int an, int K, const double *A, void *cols) {
    const int Kp = kpad(K), nct = (nr * an + kTN - 1) / kTN;
    int *ec = (int *)((char *)cols + up256((size_t)nct * kDig * kTN * Kp * 2));
    launch_next(k_col_exp, nr, 256, 0, st, an, K, A, ec);
    launch_next(k_col_digits, dim3(nct, (Kp + 127) / 128), 256, 0, st, nr, an, K, Kp, A, ec, (__nv_bfloat16 *)cols);
    return cudaGetLastError();
}

// Row digits and the product kernel; rows_total rows in whole tiles.
template <bool LIST>
static cudaError_t products(cudaStream_t st, const Chunk &c, const PairList &l, size_t ntiles, const CUtensorMap &mb,
                            const double *A, const double *Q, const int *ec, void *rows, int *err) {
    const int Kp = kpad(c.K), nx = c.x1 - c.x0;
    int *er = (int *)((char *)rows + up256(ntiles * kDig * kTM * Kp * 2));
    uint8_t *small = (uint8_t *)er + up256(sizeof(int) * ntiles * kTM);  // a bit an element of the items' tiles
    const long long eb = (long long)nx * ((c.rx() + 31) / 32);
    if (eb <= 1216) launch_next(k_row_exp<16>, dim3(nx, (c.rx() + 31) / 32), 512, 0, st, c, A, Q, er);
    else launch_next(k_row_exp<8>, dim3(nx, (c.rx() + 31) / 32), 256, 0, st, c, A, Q, er);
    const size_t sm = sizeof(double) * 66 * (c.qn + c.an);
    cudaError_t e = cudaFuncSetAttribute(k_row_digits, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    launch_next(k_row_digits, dim3(nx, Kp / 64), 256, sm, st, c, Kp, A, Q, er, (__nv_bfloat16 *)rows);
    CUtensorMap ma;
    if (!make_map(&ma, rows, Kp, (uint64_t)ntiles * kDig * kTM, kTM)) return cudaErrorInvalidValue;
    if ((e = cudaFuncSetAttribute(k_pair_tc<LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem))) return e;
    int dev = 0, nsm = 0;
    if ((e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev))) return e;
    const int nk = Kp / kBK, ks_last = (c.K - (nk - 1) * kBK + 15) / 16;
    launch_next(k_pair_tc<LIST>, (unsigned)std::min<long long>(nsm, c.items), kTcThreads, kTcSmem, st, ma, mb, c, l, nk, ks_last, er,
                                                                                             ec, small, err);
    launch_next(k_pair_mend<LIST>, (unsigned)c.items, 256, 0, st, c, l, A, Q, er, ec, (const uint32_t *)small);
    return cudaGetLastError();
}

cudaError_t tc_products(cudaStream_t st, const Chunk &c, int nr, const double *A, const double *Q, void *cols,
                        void *rows, int *err) {
    const int Kp = kpad(c.K);
    const size_t nct = ((size_t)nr * c.an + kTN - 1) / kTN;
    const int *ec = (const int *)((char *)cols + up256(nct * kDig * kTN * Kp * 2));
    CUtensorMap mb;
    if (!make_map(&mb, cols, Kp, (uint64_t)nct * kDig * kTN, kDig * kTN)) return cudaErrorInvalidValue;
    return products<false>(st, c, PairList{}, (size_t)c.ntiles, mb, A, Q, ec, rows, err);
}

// [digits][block exponents][row exponents]
size_t tc_block_bytes(int nr, int nm, int K) {
    const size_t nb = (size_t)nr * blocks_of(nm);
    return up256(nb * kDig * block_width(nm) * kpad(K) * 2) + up256(nb * 32 * sizeof(int)) + up256(sizeof(int) * (size_t)nr * nm);
}

cudaError_t tc_prep_blocks(cudaStream_t st, int nr, int nm, int K, const double *A, void *cols) {
    const int Kp = kpad(K), np = blocks_of(nm), bw = block_width(nm);
    const size_t nb = (size_t)nr * np;
    int *eb = (int *)((char *)cols + up256(nb * kDig * bw * Kp * 2));
    int *ec = (int *)((char *)eb + up256(nb * 32 * sizeof(int)));
    launch_next(k_col_exp, nr, 256, 0, st, nm, K, A, ec);
    launch_next(k_block_digits, dim3((unsigned)nb, (Kp + 127) / 128), 256, 0, st, nm, np, bw, K, Kp, A, ec, eb, (__nv_bfloat16 *)cols);
    return cudaGetLastError();
}

cudaError_t tc_list_products(cudaStream_t st, const Chunk &c, const PairList &l, int nr, const double *A, const double *Q,
                             void *cols, void *rows, int *err) {
    const int Kp = kpad(c.K);
    const size_t nb = (size_t)nr * l.np;
    const int *eb = (const int *)((char *)cols + up256(nb * kDig * l.bw * Kp * 2));
    CUtensorMap mb;
    if (!make_map(&mb, cols, Kp, (uint64_t)nb * kDig * l.bw, (uint32_t)l.bw)) return cudaErrorInvalidValue;
    return products<true>(st, c, l, (size_t)c.x1 * l.tiles_x, mb, A, Q, eb, rows, err);
}

}  // namespace p64
}  // namespace bsa
