// bsa_list64.cu -- FP64 point sets (Mesher zones and triangles, listed bispectra) through products
// of frequency pairs on the tensor cores (bsa_pair64_tc.cu).
//
// The three terms of a point are elements of E at (|f1|, |f2|), (|f1 + f2|, |f2|) and
// (|f1|, |f1 + f2|).  The points go in batches whose products fit the device; per batch the distinct
// unordered pairs are listed, each multiplied once with the row operand of the frequency that meets
// more partners (a zone line meets its columns and sums), and the point kernel reads its terms from
// the products.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../../include/bsa_gpu.h"
#include "bsa_engine.cuh"
#include "bsa_kernels.cuh"
#include "bsa_pair64.cuh"

namespace bsa {

// Whether a point set goes this way: the point kernel's time against that of the digits and products
// plus the listing of the pairs, from measured rates.  Contraction in ms, point kernel / pair products
// (kept modes nm, K):
//   scattered points (no pair shared): 100, nm 16, K 40: 0.133 / 0.131;  50, 10, 120: 0.092 / 0.087;  200,
//   10, 120: 0.227 / 0.160;  500, 6, 120: 0.183 / 0.227;  200, 6, 300: 0.205 / 0.192;  100, 6, 120: 0.068 /
//   0.088;  1000, 8, 40: 0.168 / 0.291;  500, 3, 300: 0.134 / 0.290;  1000, 4, 400: 0.307 / 0.673;
//   zones of 144 points: nm 8, K 60: 0.057 / 0.076;  3, 600: 0.117 / 0.094;  6, 240: 0.099 / 0.086;  256 points,
//   4, 120: 0.050 / 0.076;  1600, 4, 120: 0.184 / 0.187;  1600, 3, 60: 0.141 / 0.184;  1024, 8, 60: 0.234 / 0.161;
//   1523, 16, 400: 9.46 / 0.58.
bool Engine::list64_wanted(long long npts, int nr) const {
    using namespace p64;
    // the column digits grow with the rows (twice the A rows, modes padded to eights and K to 64): within
    // 32 GB; up to 16 points both are launches and chains over K
    if (K < 24 || npts <= 16 || tc_block_bytes(nr, nme, K) > ((size_t)32 << 30)) return false;
    const double nm = nme, rows = (double)std::min<long long>(nr, 2 * npts) * ((nme * nme + kTM - 1) / kTM) * kTM;
    // a point's chain over K, then the FP64 pipe
    const double point_ms = 0.03 + K * (nme < 8 ? 1.4e-4 : 3.0e-4) + 2.0 * K * nm * nm * nm * (double)npts / (nme < 8 ? 2.0e8 : 4.2e8);
    const double pair_ms = 0.07 + (5.0e-5 + 1.0e-7 * nm * nm * nm) * (double)npts + rows * ((K + 63) / 64 * 64) * 5.0e-9;
    return pair_ms < point_ms;
}

// The points of a list from p0 on.
static PointSrc from(PointSrc q, long long p0) {
    q.ix += p0;
    q.iy += p0;
    q.iz += p0;
    q.f1 += p0;
    q.f2 += p0;
    if (q.w) q.w += p0;
    if (q.zones) {
        q.zid += p0;
        q.zi += p0;
        q.zj += p0;
    }
    if (q.cptr) q.cptr += p0;
    return q;
}

// Third moments (and bispectra) of a point list; rows: the points' A rows on the host (iz < 0: the sum
// reads zero), ps the same on the device.
int Engine::contract_list64(const PointSrc &ps, long long npts, const HostRows &rows, int G, double *bfd, double *brd,
                            Lists64 &lists) {
    using namespace p64;
    const int nr = rows.nr, *ix = rows.ix, *iy = rows.iy, *iz = rows.iz;
    auto &[start, deg, other, pe, xmap, blk, pair, row_of, fill, uniq, items, refs] = lists;
    using Ref = Lists64::Ref;
    deg.assign(nr, 0);
    row_of.assign(nr, 0);
    const int nm = nme, rx = nm * nm, np = blocks_of(nm), bw = block_width(nm), slots = kTN / bw;
    const int tiles_x = (rx + kTM - 1) / kTM;
    const long long nm3 = (long long)rx * nm;
    cudaError_t e;
    // products of a batch: at most 8 GB, and the row digits at most 8 GB (two row operands a point at most)
    const long long rowb = (long long)tc_row_bytes((long long)tiles_x * kTM, K, 0);
    const long long cap = 8LL << 30;
    const long long batch = std::max(1LL, std::min({npts, cap / (24 * nm3), cap / (2 * rowb)}));
    // no room for the column digits, or later for a batch: the point kernel on what is left
    PairPts pp;
    auto rest = [&](long long p0) {
        PointSrc q = from(ps, p0);
        pp.E = nullptr;
        pp.first = p0 == 0;
        const cudaError_t r = launch_bfm_fp64(stream, dA.as<double>(), dQ.as<double>(), K, nm, q, npts - p0, frf(), G,
                                              dPartF.as<double>(), dPartR.as<double>(), bfd ? bfd + (size_t)p0 * nm3 : nullptr,
                                              brd ? brd + (size_t)p0 * nm3 : nullptr, pp);
        return r ? cuda_fail(r, "FP64 point kernel") : BSA_OK;
    };
    if ((e = dFlag.reserve(256)) || (e = cudaMemsetAsync(dFlag.as<int>() + 1, 0, sizeof(int), stream)))
        return cuda_fail(e, "allocating pair products");
    if ((e = dMixB.reserve(tc_block_bytes(nr, nm, K))) == cudaErrorMemoryAllocation) return rest(0);
    if (e) return cuda_fail(e, "allocating pair products");
    if ((e = tc_prep_blocks(stream, nr, nm, K, dA.as<double>(), dMixB.p)))
        return cuda_fail(e, "pair product operands");
    kernels += 2;
    for (long long p0 = 0; p0 < npts; p0 += batch) {
        const int n = (int)std::min(batch, npts - p0);
        // pairs (lo <= hi) bucketed by lo, then by hi; slot 3 p + w is the term that asks for it
        start.assign(nr + 1, 0);
        auto ends = [&](int s, int &a, int &b) {
            const long long p = p0 + s / 3;
            const int w = s % 3;
            a = w == 1 ? iz[p] : ix[p];
            b = w == 2 ? iz[p] : iy[p];
        };
        int a, b;
        for (int s = 0; s < 3 * n; ++s) {
            ends(s, a, b);
            if (a >= 0 && b >= 0) ++start[std::min(a, b) + 1];
        }
        for (int r = 0; r < nr; ++r) start[r + 1] += start[r];
        refs.resize(start[nr]);
        fill.assign(start.begin(), start.end() - 1);
        for (int s = 0; s < 3 * n; ++s) {
            ends(s, a, b);
            if (a >= 0 && b >= 0) refs[fill[std::min(a, b)]++] = Ref{std::max(a, b), s};
        }
        uniq.clear();  // lo << 32 | hi
        pe.assign(3 * (size_t)n, -1);
        std::fill(deg.begin(), deg.end(), 0);
        for (int r = 0; r < nr; ++r) {
            std::sort(refs.begin() + start[r], refs.begin() + start[r + 1],
                      [](const Ref &u, const Ref &v) { return u.hi < v.hi; });
            for (int q = start[r]; q < start[r + 1]; ++q) {
                if (q == start[r] || refs[q].hi != refs[q - 1].hi) {
                    uniq.push_back(((long long)r << 32) | (unsigned)refs[q].hi);
                    ++deg[r];
                    ++deg[refs[q].hi];
                }
                pe[refs[q].slot] = (int)uniq.size() - 1;
            }
        }
        const int nu = (int)uniq.size();
        // row frequency of each pair: the one with more partners; pairs listed by row frequency
        auto row_is_lo = [&](long long k) { return deg[k >> 32] >= deg[(int)(k & 0xffffffff)]; };
        start.assign(nr + 1, 0);
        for (long long k : uniq) ++start[(row_is_lo(k) ? (int)(k >> 32) : (int)(k & 0xffffffff)) + 1];
        xmap.clear();
        for (int r = 0; r < nr; ++r) {
            if (start[r + 1]) {
                row_of[r] = (int)xmap.size();
                xmap.push_back(r);
            }
            start[r + 1] += start[r];
        }
        fill.assign(start.begin(), start.end() - 1);
        blk.resize((size_t)nu * np);
        pair.resize((size_t)nu * np);
        other.resize(nu);  // row frequency of a pair
        for (int q = 0; q < nu; ++q) {
            const int lo = (int)(uniq[q] >> 32), hi = (int)(uniq[q] & 0xffffffff);
            const bool rl = row_is_lo(uniq[q]);
            other[q] = rl ? lo : hi;
            const int at = fill[other[q]]++;
            for (int z = 0; z < np; ++z) {
                blk[(size_t)at * np + z] = (rl ? hi : lo) * np + z;
                pair[(size_t)at * np + z] = q;
            }
        }
        for (int s = 0; s < 3 * n; ++s)
            if (pe[s] >= 0) {
                ends(s, a, b);
                pe[s] = 2 * pe[s] + (other[pe[s]] == a ? 0 : 1);
            }
        items.clear();
        for (int x : xmap)
            for (int t = 0; t < tiles_x; ++t)
                for (int q = start[x] * np; q < start[x + 1] * np; q += slots)
                    items.push_back(make_int4(row_of[x] * tiles_x + t, q, std::min(slots, start[x + 1] * np - q), 0));
        const size_t ib = sizeof(int4) * items.size(), lb = sizeof(int) * blk.size(), xb = sizeof(int) * xmap.size(),
                     pb = sizeof(int) * pe.size();
        e = dMixA.reserve(sizeof(double) * (size_t)nu * nm3);
        if (!e) e = dMshT.reserve(tc_row_bytes((long long)xmap.size() * tiles_x * kTM, K, (long long)items.size()));
        if (!e) e = dMshIdx.reserve(ib + 2 * lb + xb + pb);
        if (e == cudaErrorMemoryAllocation) return rest(p0);
        if (e) return cuda_fail(e, "allocating pair products");
        char *d = (char *)dMshIdx.p;
        int4 *ditems = (int4 *)d;
        int *dblk = (int *)(d + ib), *dpair = (int *)(d + ib + lb), *dx = (int *)(d + ib + 2 * lb), *dpe = (int *)(d + ib + 2 * lb + xb);
        if ((e = cudaMemcpyAsync(ditems, items.data(), ib, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemcpyAsync(dblk, blk.data(), lb, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemcpyAsync(dpair, pair.data(), lb, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemcpyAsync(dx, xmap.data(), xb, cudaMemcpyHostToDevice, stream)) ||
            (e = cudaMemcpyAsync(dpe, pe.data(), pb, cudaMemcpyHostToDevice, stream)))
            return cuda_fail(e, "pair lists");
        h2d += (double)(ib + 2 * lb + xb + pb);
        Chunk c{0, (int)xmap.size(), nm, nm, K, nr - 1, 0, (long long)items.size(), nullptr, dMixA.as<double>(), tiles_x * kTM, dx, wait_test_pair1};
        wait_test_pair1 = 0;  // one launch only
        PairList l{ditems, dblk, dpair, np, bw, tiles_x};
        if ((e = tc_list_products(stream, c, l, nr, dA.as<double>(), dQ.as<double>(), dMixB.p, dMshT.p, dFlag.as<int>() + 1)))
            return cuda_fail(e, "pair product kernel");
        const PointSrc q = from(ps, p0);
        pp.E = dMixA.as<double>();
        pp.pe = dpe;
        pp.first = p0 == 0;
        if ((e = launch_bfm_fp64(stream, dA.as<double>(), dQ.as<double>(), K, nm, q, n, frf(), G, dPartF.as<double>(),
                                 dPartR.as<double>(), bfd ? bfd + (size_t)p0 * nm3 : nullptr,
                                 brd ? brd + (size_t)p0 * nm3 : nullptr, pp)))
            return cuda_fail(e, "FP64 point kernel");
        kernels += 5;
        if (p0 + n < npts && (e = cudaStreamSynchronize(stream))) return cuda_fail(e, "pair products");  // the lists are rewritten
    }
    return BSA_OK;
}

}  // namespace bsa
