// bsa_mlp.cu -- the Mesher's zone-refinement proposer: a small MLP
//   x (din) -> W -> W -> W (ReLU) -> 1 logit,  P(refine) = sigmoid(logit)
// with BF16 weights and FP32 accumulation, trained on the device by its own forward and
// backward kernels: binary cross-entropy (hard or soft targets) with per-sample weights,
// Adam on FP32 master weights, the BF16 copy refreshed after every step.  No counterpart in
// the reference (its Mesher refines by fixed policies); the proposer only chooses which zones
// the plain refinement criterion evaluates at the next lattice level.
//
// Parameter order (flattened, FP32 master / BF16 working copy):
//   W1[W][din] b1[W] W2[W][W] b2[W] W3[W][W] b3[W] w4[W] b4
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bsa_gpu.h"

namespace bsa {
namespace mlp {

constexpr int kMaxNets = 8;

struct Buf {
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t reserve(size_t n) {
        if (n <= bytes && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaSuccess) bytes = n;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <class T> T *as() const { return (T *)p; }
};

struct Net {
    bool used = false;
    int din = 0, W = 0;
    long long np = 0;  // parameters
    long long step = 0;
    Buf master, wbf, grad, m1, m2;                         // parameters, BF16 copy, gradient, Adam moments
    Buf x, y, sw, prob, red, part;         // batch data, probabilities, losses, partial gradients
    int cap = 0;                           // batch capacity
    cudaStream_t st = nullptr;
    long long off_b1() const { return (long long)W * din; }
    long long off_W2() const { return off_b1() + W; }
    long long off_b2() const { return off_W2() + (long long)W * W; }
    long long off_W3() const { return off_b2() + W; }
    long long off_b3() const { return off_W3() + (long long)W * W; }
    long long off_w4() const { return off_b3() + W; }
    long long off_b4() const { return off_w4() + W; }
};

Net g_nets[kMaxNets];
std::string g_err;

int fail(int code, const std::string &msg) {
    g_err = msg;
    return code;
}

// ---------------------------------------------------------------- kernels
// A block takes a tile of samples through every layer in shared memory: activations feature-major
// (lanes over samples, rows padded by one word), the current layer's weights widened to FP32.  Each
// warp owns 8 outputs of a layer and each lane TB / 32 samples, so a weight load is a broadcast and an
// activation load feeds 8 FMAs.  One launch per layer with one sample a block was bound by its global
// loads: 20 000 zones through 13-128-128-128-1 in 1.9 ms, one gradient of 4096 records in 2.2 ms;
// now 0.08 ms and 0.12 ms.
constexpr int kThreads = 512, kWarps = kThreads / 32, kFeat = 128;
constexpr int kLdw = 132;           // floats per weight row: 16-byte aligned broadcasts
constexpr int kTrainTile = 32, kInferTile = 64;

template <int TB>
constexpr size_t act_floats() { return (size_t)kFeat * (TB + 1); }

// Wf[i][o] (transposed, forward) or Wf[o][i] (backward) from Wt[o][i]; zero beyond nin, nout.
__device__ __forceinline__ void stage_w(float *Wf, const __nv_bfloat16 *__restrict__ Wt, int nin, int nout, bool transposed) {
    for (int e = threadIdx.x; e < kFeat * kFeat; e += kThreads) {
        const int o = e >> 7, i = e & 127;
        const float v = (o < nout && i < nin) ? __bfloat162float(Wt[(size_t)o * nin + i]) : 0.f;
        Wf[transposed ? i * kLdw + o : o * kLdw + i] = v;
    }
}

// out[o][s] = relu(bias[o] + sum_i in[i][s] W[o][i]), i in order.
template <int TB>
__device__ __forceinline__ void dense(const float *in, const float *Wf, const __nv_bfloat16 *__restrict__ bias, int nin, int nout,
                                      float *out) {
    constexpr int S = TB / 32, LD = TB + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, o0 = warp * 8;
    float acc[8][S];
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int z = 0; z < S; ++z) acc[q][z] = o0 + q < nout ? __bfloat162float(bias[o0 + q]) : 0.f;
#pragma unroll 4
    for (int i = 0; i < nin; ++i) {
        float a[S];
#pragma unroll
        for (int z = 0; z < S; ++z) a[z] = in[i * LD + lane + 32 * z];
        const float4 w0 = *reinterpret_cast<const float4 *>(Wf + i * kLdw + o0);
        const float4 w1 = *reinterpret_cast<const float4 *>(Wf + i * kLdw + o0 + 4);
        const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int q = 0; q < 8; ++q)
#pragma unroll
            for (int z = 0; z < S; ++z) acc[q][z] = fmaf(a[z], w[q], acc[q][z]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int z = 0; z < S; ++z) out[(o0 + q) * LD + lane + 32 * z] = fmaxf(acc[q][z], 0.f);
}

// dIn[i][s] = sum_o dOut[o][s] W[o][i], zero where the activation mask[i][s] is not positive.
__device__ __forceinline__ void back_act(const float *dOut, const float *Wf, int nout, const float *mask, float *dIn) {
    constexpr int LD = kTrainTile + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i0 = warp * 8;
    float acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.f;
#pragma unroll 4
    for (int o = 0; o < nout; ++o) {
        const float d = dOut[o * LD + lane];
        const float4 w0 = *reinterpret_cast<const float4 *>(Wf + o * kLdw + i0);
        const float4 w1 = *reinterpret_cast<const float4 *>(Wf + o * kLdw + i0 + 4);
        const float w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fmaf(d, w[q], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) dIn[(i0 + q) * LD + lane] = mask[(i0 + q) * LD + lane] > 0.f ? acc[q] : 0.f;
}

// gW[o][i] += sum_s d[o][s] in[i][s], gb[o] += sum_s d[o][s] into the block's own partial.
__device__ __forceinline__ void back_w(const float *d, const float *in, int nin, int nout, float *gW, float *gb) {
    constexpr int LD = kTrainTile + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, o0 = warp * 8;
    float acc[8][4], sb[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        sb[q] = 0.f;
#pragma unroll
        for (int z = 0; z < 4; ++z) acc[q][z] = 0.f;
    }
#pragma unroll 2
    for (int s = 0; s < kTrainTile; ++s) {
        float a[4];
#pragma unroll
        for (int z = 0; z < 4; ++z) a[z] = in[(lane + 32 * z) * LD + s];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float v = d[(o0 + q) * LD + s];
            sb[q] += v;
#pragma unroll
            for (int z = 0; z < 4; ++z) acc[q][z] = fmaf(v, a[z], acc[q][z]);
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        if (o0 + q >= nout) continue;
#pragma unroll
        for (int z = 0; z < 4; ++z)
            if (lane + 32 * z < nin) gW[(size_t)(o0 + q) * nin + lane + 32 * z] += acc[q][z];
        if (lane == 0) gb[o0 + q] += sb[q];
    }
}

struct Layout {
    int din, W;
    long long np, b1, W2, b2, W3, b3, w4, b4;
};

template <int TB>
__device__ __forceinline__ void load_x(float *xs, const float *__restrict__ x, int s0, int n, int din) {
    constexpr int LD = TB + 1;
    for (int e = threadIdx.x; e < TB * din; e += kThreads) {
        const int s = e / din, i = e - s * din;
        xs[i * LD + s] = s0 + s < n ? x[(size_t)(s0 + s) * din + i] : 0.f;
    }
}

template <int TB>
__device__ __forceinline__ float logit_of(const float *z3, int s, const __nv_bfloat16 *__restrict__ w, const Layout &L) {
    float v = __bfloat162float(w[L.b4]);
    for (int k = 0; k < L.W; ++k) v = fmaf(z3[k * (TB + 1) + s], __bfloat162float(w[L.w4 + k]), v);
    return v;
}

// prob[s] = sigmoid(logit) of n samples; a block walks tiles of kInferTile.
__global__ void __launch_bounds__(kThreads, 1) k_mlp_infer(int n, Layout L, const float *__restrict__ x,
                                                           const __nv_bfloat16 *__restrict__ w, float *__restrict__ prob) {
    extern __shared__ __align__(16) float sm[];
    float *Wf = sm, *za = Wf + kFeat * kLdw, *zb = za + act_floats<kInferTile>();
    for (int s0 = blockIdx.x * kInferTile; s0 < n; s0 += gridDim.x * kInferTile) {
        __syncthreads();
        load_x<kInferTile>(za, x, s0, n, L.din);
        stage_w(Wf, w, L.din, L.W, true);
        __syncthreads();
        dense<kInferTile>(za, Wf, w + L.b1, L.din, L.W, zb);
        __syncthreads();
        stage_w(Wf, w + L.W2, L.W, L.W, true);
        __syncthreads();
        dense<kInferTile>(zb, Wf, w + L.b2, L.W, L.W, za);
        __syncthreads();
        stage_w(Wf, w + L.W3, L.W, L.W, true);
        __syncthreads();
        dense<kInferTile>(za, Wf, w + L.b3, L.W, L.W, zb);
        __syncthreads();
        if (threadIdx.x < kInferTile && s0 + (int)threadIdx.x < n)
            prob[s0 + threadIdx.x] = 1.f / (1.f + expf(-logit_of<kInferTile>(zb, threadIdx.x, w, L)));
    }
}

// Weighted binary cross-entropy on the logits, dl = sw (sigmoid(z) - y) / sum(sw), lossv = sw loss /
// sum(sw) (summed on the host), and the block's share of every gradient, added tile after tile into
// part[block][np] (zeroed before the launch).
__global__ void __launch_bounds__(kThreads, 1)
    k_mlp_grad(int n, Layout L, const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ sw,
               float inv_wsum, const __nv_bfloat16 *__restrict__ w, float *__restrict__ lossv, float *__restrict__ part) {
    constexpr int TB = kTrainTile, LD = TB + 1;
    constexpr size_t AF = act_floats<TB>();
    extern __shared__ __align__(16) float sm[];
    __shared__ float dl[TB];
    float *Wf = sm, *xs = Wf + kFeat * kLdw, *z1 = xs + AF, *z2 = z1 + AF, *z3 = z2 + AF, *da = z3 + AF, *db = da + AF;
    float *g = part + (size_t)blockIdx.x * L.np;
    const int W = L.W;
    for (int e = threadIdx.x; e < (int)AF; e += kThreads) xs[e] = 0.f;  // rows past din are read by back_w
    for (int s0 = blockIdx.x * TB; s0 < n; s0 += gridDim.x * TB) {
        __syncthreads();
        load_x<TB>(xs, x, s0, n, L.din);
        stage_w(Wf, w, L.din, W, true);
        __syncthreads();
        dense<TB>(xs, Wf, w + L.b1, L.din, W, z1);
        __syncthreads();
        stage_w(Wf, w + L.W2, W, W, true);
        __syncthreads();
        dense<TB>(z1, Wf, w + L.b2, W, W, z2);
        __syncthreads();
        stage_w(Wf, w + L.W3, W, W, true);
        __syncthreads();
        dense<TB>(z2, Wf, w + L.b3, W, W, z3);
        __syncthreads();
        if (threadIdx.x < TB) {
            const int b = s0 + threadIdx.x;
            float v = 0.f;
            if (b < n) {
                const float zz = logit_of<TB>(z3, threadIdx.x, w, L), p = 1.f / (1.f + expf(-zz));
                // log(1 + exp(-|z|)) + max(z, 0) - y z : the stable form of the cross-entropy
                const float l = log1pf(expf(-fabsf(zz))) + fmaxf(zz, 0.f) - y[b] * zz;
                v = sw[b] * (p - y[b]) * inv_wsum;
                lossv[b] = sw[b] * l * inv_wsum;
            }
            dl[threadIdx.x] = v;
        }
        stage_w(Wf, w + L.W3, W, W, false);
        __syncthreads();
        // output layer: g w4[i] = sum_s dl z3[i][s], g b4 = sum_s dl, d3 = dl w4 where z3 > 0
        for (int i = threadIdx.x; i <= W; i += kThreads) {
            float v = 0.f;
            for (int s = 0; s < TB; ++s) v = i < W ? fmaf(dl[s], z3[i * LD + s], v) : v + dl[s];
            g[i < W ? L.w4 + i : L.b4] += v;
        }
        for (int e = threadIdx.x; e < kFeat * TB; e += kThreads) {
            const int i = e / TB, s = e - i * TB;
            da[i * LD + s] = (i < W && z3[i * LD + s] > 0.f) ? dl[s] * __bfloat162float(w[L.w4 + i]) : 0.f;
        }
        __syncthreads();
        back_w(da, z2, W, W, g + L.W3, g + L.b3);
        back_act(da, Wf, W, z2, db);
        __syncthreads();
        stage_w(Wf, w + L.W2, W, W, false);
        back_w(db, z1, W, W, g + L.W2, g + L.b2);
        __syncthreads();
        back_act(db, Wf, W, z1, da);
        __syncthreads();
        back_w(da, xs, L.din, W, g, g + L.b1);
    }
}

// g[p] = sum of the blocks' partials, block after block.
__global__ void k_grad_sum(long long np, int nblk, const float *__restrict__ part, float *__restrict__ g) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    float s = 0.f;
#pragma unroll 8
    for (int b = 0; b < nblk; ++b) s += part[(size_t)b * np + p];
    g[p] = s;
}

__global__ void k_adam(long long np, float lr, float b1, float b2, float eps, float c1, float c2,
                       float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       __nv_bfloat16 *__restrict__ wbf) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    w[i] = wi;
    wbf[i] = __float2bfloat16_rn(wi);
}

__global__ void k_to_bf16(long long np, const float *__restrict__ w, __nv_bfloat16 *__restrict__ wbf) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < np) wbf[i] = __float2bfloat16_rn(w[i]);
}

// ---------------------------------------------------------------- host helpers
cudaError_t ensure_batch(Net &N, int n) {
    if (n <= N.cap) return cudaSuccess;
    cudaError_t e;
    const size_t f = sizeof(float);
    if ((e = N.x.reserve(f * n * N.din)) || (e = N.y.reserve(f * n)) || (e = N.sw.reserve(f * n)) ||
        (e = N.prob.reserve(f * n)) || (e = N.red.reserve(f * n)))
        return e;
    N.cap = n;
    return cudaSuccess;
}

Layout layout(const Net &N) {
    return Layout{N.din, N.W, N.np, N.off_b1(), N.off_W2(), N.off_b2(), N.off_W3(), N.off_b3(), N.off_w4(), N.off_b4()};
}

// One block per SM walks the tiles.
cudaError_t blocks_for(int n, int tile, int *grid) {
    int dev = 0, nsm = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev))) return e;
    const int tiles = (n + tile - 1) / tile;
    *grid = tiles < nsm ? tiles : nsm;
    return cudaSuccess;
}

// probabilities of the n rows at x (device) into N.prob
cudaError_t forward(Net &N, const float *x, int n) {
    constexpr size_t smem = sizeof(float) * (kFeat * kLdw + 2 * act_floats<kInferTile>());
    cudaError_t e;
    int grid = 0;
    if ((e = blocks_for(n, kInferTile, &grid)) ||
        (e = cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)))
        return e;
    k_mlp_infer<<<grid, kThreads, smem, N.st>>>(n, layout(N), x, N.wbf.as<__nv_bfloat16>(), N.prob.as<float>());
    return cudaGetLastError();
}

// loss + gradient into N.grad for the n rows at x, y, sw (device)
cudaError_t backward(Net &N, const float *x, const float *y, const float *sw, int n, float wsum, float *loss) {
    constexpr size_t smem = sizeof(float) * (kFeat * kLdw + 6 * act_floats<kTrainTile>());
    cudaError_t e;
    int grid = 0;
    if ((e = blocks_for(n, kTrainTile, &grid)) || (e = N.part.reserve(sizeof(float) * (size_t)grid * N.np)) ||
        (e = cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) ||
        (e = cudaMemsetAsync(N.part.p, 0, sizeof(float) * (size_t)grid * N.np, N.st)))
        return e;
    k_mlp_grad<<<grid, kThreads, smem, N.st>>>(n, layout(N), x, y, sw, 1.f / wsum, N.wbf.as<__nv_bfloat16>(),
                                               N.red.as<float>(), N.part.as<float>());
    k_grad_sum<<<(unsigned)((N.np + 255) / 256), 256, 0, N.st>>>(N.np, grid, N.part.as<float>(), N.grad.as<float>());
    if ((e = cudaGetLastError())) return e;
    if (loss) {
        std::vector<float> lv(n);
        if ((e = cudaMemcpyAsync(lv.data(), N.red.p, sizeof(float) * n, cudaMemcpyDeviceToHost, N.st)) ||
            (e = cudaStreamSynchronize(N.st)))
            return e;
        double s = 0.0;
        for (float v : lv) s += v;
        *loss = (float)s;
    }
    return cudaSuccess;
}

Net *get(int h) {
    if (h < 0 || h >= kMaxNets || !g_nets[h].used) return nullptr;
    return &g_nets[h];
}

}  // namespace mlp
}  // namespace bsa

using namespace bsa::mlp;

extern "C" {

int bsa_mlp_create(int din, int width, unsigned long long seed) {
    if (din < 1 || din > 128 || width < 1 || width > 128) return fail(BSA_ERR_ARG, "0 < din, width <= 128");
    int h = -1;
    for (int k = 0; k < kMaxNets; ++k)
        if (!g_nets[k].used) { h = k; break; }
    if (h < 0) return fail(BSA_ERR_STATE, "too many networks");
    Net &N = g_nets[h];
    N = Net();
    N.din = din;
    N.W = width;
    N.np = (long long)width * din + width + 2 * ((long long)width * width + width) + width + 1;
    // He-uniform initialisation from a seeded generator (splitmix64), biases zero
    std::vector<float> p(N.np, 0.f);
    uint64_t s = seed;
    auto rnd = [&]() {
        s += 0x9E3779B97F4A7C15ull;
        uint64_t z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);  // [0, 1)
    };
    auto fill = [&](long long off, long long cnt, int fan_in) {
        const double a = std::sqrt(6.0 / fan_in);
        for (long long i = 0; i < cnt; ++i) p[off + i] = (float)((2.0 * rnd() - 1.0) * a);
    };
    fill(0, (long long)width * din, din);
    fill(N.off_W2(), (long long)width * width, width);
    fill(N.off_W3(), (long long)width * width, width);
    fill(N.off_w4(), width, width);
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&N.st, cudaStreamNonBlocking)) || (e = N.master.reserve(4 * N.np)) ||
        (e = N.wbf.reserve(2 * N.np)) || (e = N.grad.reserve(4 * N.np)) || (e = N.m1.reserve(4 * N.np)) ||
        (e = N.m2.reserve(4 * N.np)))
        return fail(BSA_ERR_CUDA, std::string("MLP allocation: ") + cudaGetErrorString(e));
    if ((e = cudaMemcpyAsync(N.master.p, p.data(), 4 * N.np, cudaMemcpyHostToDevice, N.st)) ||
        (e = cudaMemsetAsync(N.m1.p, 0, 4 * N.np, N.st)) || (e = cudaMemsetAsync(N.m2.p, 0, 4 * N.np, N.st)))
        return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    k_to_bf16<<<(unsigned)((N.np + 255) / 256), 256, 0, N.st>>>(N.np, N.master.as<float>(), N.wbf.as<__nv_bfloat16>());
    if ((e = cudaStreamSynchronize(N.st))) return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    N.used = true;
    return h;
}

int bsa_mlp_destroy(int h) {
    Net *N = get(h);
    if (!N) return BSA_ERR_ARG;
    for (Buf *b : {&N->master, &N->wbf, &N->grad, &N->m1, &N->m2, &N->x, &N->y, &N->sw, &N->prob,
                   &N->red, &N->part})
        b->release();
    if (N->st) cudaStreamDestroy(N->st);
    *N = Net();
    return BSA_OK;
}

long long bsa_mlp_num_params(int h) {
    Net *N = get(h);
    return N ? N->np : BSA_ERR_ARG;
}

// params: FP32 master weights (bf16 == 0) or the BF16 working copy as floats (bf16 != 0)
int bsa_mlp_get_params(int h, float *params, int bf16) {
    Net *N = get(h);
    if (!N || !params) return BSA_ERR_ARG;
    cudaError_t e;
    if (!bf16) {
        if ((e = cudaMemcpyAsync(params, N->master.p, 4 * N->np, cudaMemcpyDeviceToHost, N->st)) ||
            (e = cudaStreamSynchronize(N->st)))
            return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
        return BSA_OK;
    }
    std::vector<__nv_bfloat16> b(N->np);
    if ((e = cudaMemcpyAsync(b.data(), N->wbf.p, 2 * N->np, cudaMemcpyDeviceToHost, N->st)) ||
        (e = cudaStreamSynchronize(N->st)))
        return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    for (long long i = 0; i < N->np; ++i) {
        uint16_t u;
        std::memcpy(&u, &b[i], 2);
        const uint32_t f = (uint32_t)u << 16;
        std::memcpy(&params[i], &f, 4);
    }
    return BSA_OK;
}

int bsa_mlp_set_params(int h, const float *params) {
    Net *N = get(h);
    if (!N || !params) return BSA_ERR_ARG;
    cudaError_t e;
    if ((e = cudaMemcpyAsync(N->master.p, params, 4 * N->np, cudaMemcpyHostToDevice, N->st)))
        return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    k_to_bf16<<<(unsigned)((N->np + 255) / 256), 256, 0, N->st>>>(N->np, N->master.as<float>(),
                                                                  N->wbf.as<__nv_bfloat16>());
    if ((e = cudaStreamSynchronize(N->st))) return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    return BSA_OK;
}

int bsa_mlp_forward(int h, const float *x, int n, float *prob) {
    Net *N = get(h);
    if (!N || !x || !prob || n <= 0) return BSA_ERR_ARG;
    cudaError_t e;
    for (int b0 = 0; b0 < n; b0 += 65536) {
        const int nb = n - b0 < 65536 ? n - b0 : 65536;
        if ((e = ensure_batch(*N, nb)) ||
            (e = cudaMemcpyAsync(N->x.p, x + (size_t)b0 * N->din, 4 * (size_t)nb * N->din, cudaMemcpyHostToDevice,
                                 N->st)))
            return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
        if ((e = forward(*N, N->x.as<float>(), nb)) ||
            (e = cudaMemcpyAsync(prob + b0, N->prob.p, 4 * (size_t)nb, cudaMemcpyDeviceToHost, N->st)) ||
            (e = cudaStreamSynchronize(N->st)))
            return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    }
    return BSA_OK;
}

// Loss and gradient (w.r.t. the BF16 working weights) of the weighted cross-entropy.
int bsa_mlp_gradients(int h, const float *x, const float *y, const float *sw, int n, float *loss, float *grads) {
    Net *N = get(h);
    if (!N || !x || !y || !sw || n <= 0 || n > 65536) return BSA_ERR_ARG;
    double wsum = 0.0;
    for (int b = 0; b < n; ++b) wsum += sw[b];
    if (!(wsum > 0.0)) return fail(BSA_ERR_ARG, "sample weights sum to zero");
    cudaError_t e;
    if ((e = ensure_batch(*N, n)) ||
        (e = cudaMemcpyAsync(N->x.p, x, 4 * (size_t)n * N->din, cudaMemcpyHostToDevice, N->st)) ||
        (e = cudaMemcpyAsync(N->y.p, y, 4 * (size_t)n, cudaMemcpyHostToDevice, N->st)) ||
        (e = cudaMemcpyAsync(N->sw.p, sw, 4 * (size_t)n, cudaMemcpyHostToDevice, N->st)))
        return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    if ((e = backward(*N, N->x.as<float>(), N->y.as<float>(), N->sw.as<float>(), n, (float)wsum, loss)))
        return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    if (grads && ((e = cudaMemcpyAsync(grads, N->grad.p, 4 * N->np, cudaMemcpyDeviceToHost, N->st)) ||
                  (e = cudaStreamSynchronize(N->st))))
        return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    return BSA_OK;
}

// Minibatch Adam over the n samples, `epochs` passes in a seeded order.
int bsa_mlp_train(int h, const float *x, const float *y, const float *sw, int n, int epochs, int batch, float lr,
                  unsigned long long seed, float *loss_out) {
    Net *N = get(h);
    if (!N || !x || !y || !sw || n <= 0 || epochs < 1 || batch < 1 || batch > 65536) return BSA_ERR_ARG;
    std::vector<int> idx(n);
    for (int i = 0; i < n; ++i) idx[i] = i;
    uint64_t s = seed ? seed : 0x2545F4914F6CDD1Dull;
    auto nxt = [&]() {
        s ^= s << 13;
        s ^= s >> 7;
        s ^= s << 17;
        return s;
    };
    std::vector<float> bx((size_t)batch * N->din), by(batch), bw(batch);
    cudaError_t e;
    if ((e = ensure_batch(*N, batch))) return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    float last = 0.f;
    for (int ep = 0; ep < epochs; ++ep) {
        for (int i = n - 1; i > 0; --i) std::swap(idx[i], idx[(int)(nxt() % (uint64_t)(i + 1))]);
        double eloss = 0.0;
        int nb_total = 0;
        for (int b0 = 0; b0 < n; b0 += batch) {
            const int nb = n - b0 < batch ? n - b0 : batch;
            double wsum = 0.0;
            for (int b = 0; b < nb; ++b) {
                const int r = idx[b0 + b];
                std::memcpy(&bx[(size_t)b * N->din], x + (size_t)r * N->din, 4 * N->din);
                by[b] = y[r];
                bw[b] = sw[r];
                wsum += sw[r];
            }
            if (!(wsum > 0.0)) continue;
            if ((e = cudaMemcpyAsync(N->x.p, bx.data(), 4 * (size_t)nb * N->din, cudaMemcpyHostToDevice, N->st)) ||
                (e = cudaMemcpyAsync(N->y.p, by.data(), 4 * (size_t)nb, cudaMemcpyHostToDevice, N->st)) ||
                (e = cudaMemcpyAsync(N->sw.p, bw.data(), 4 * (size_t)nb, cudaMemcpyHostToDevice, N->st)))
                return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
            float l = 0.f;
            if ((e = backward(*N, N->x.as<float>(), N->y.as<float>(), N->sw.as<float>(), nb, (float)wsum, &l)))
                return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
            ++N->step;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.f / (1.f - std::pow(b1, (float)N->step)), c2 = 1.f / (1.f - std::pow(b2, (float)N->step));
            k_adam<<<(unsigned)((N->np + 255) / 256), 256, 0, N->st>>>(N->np, lr, b1, b2, 1e-8f, c1, c2,
                                                                      N->master.as<float>(), N->grad.as<float>(),
                                                                      N->m1.as<float>(), N->m2.as<float>(),
                                                                      N->wbf.as<__nv_bfloat16>());
            if ((e = cudaGetLastError())) return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
            eloss += l;
            ++nb_total;
        }
        last = nb_total ? (float)(eloss / nb_total) : 0.f;
    }
    if ((e = cudaStreamSynchronize(N->st))) return fail(BSA_ERR_CUDA, cudaGetErrorString(e));
    if (loss_out) *loss_out = last;
    return BSA_OK;
}

const char *bsa_mlp_lastError(void) { return g_err.c_str(); }

}  // extern "C"
