// Learned correction of the Jacobi preconditioner: a small multilayer perceptron
// (no counterpart in the reference) with hand-written BF16 inference and
// training kernels, FP32 accumulation.
//
// Layout: layers l = 0..L-1 map n_l -> n_{l+1}; W_l is [n_{l+1}][n_l] row-major,
// b_l [n_{l+1}]; ReLU between layers, linear output. Inputs are standardised with
// (x - mean) / std inside the first layer. Parameters live on the device as an
// FP32 master copy (training, Adam moments beside it) and a BF16 copy used by
// the forward pass; activations are rounded to BF16 between layers, every dot
// product accumulates in FP32.
//
// Kernels: inference of the learned corrections' shape (inputs <= 32, hidden layers of
// 64, one output) on the BF16 tensor cores (k_mlp_forward_mma); other shapes and the
// training pass one thread per sample, the parameters staged in shared memory (all
// threads of a warp read the same weight: broadcast, no bank conflicts). The
// backward pass reduces each weight's per-sample gradient across the warp with
// shuffles, then across the block in shared memory, then into the global FP32
// gradient with one atomic per weight per block.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "hp_gpu.h"
#include "hp_mlp.h"

namespace {

constexpr int kMaxLayers = 6;
constexpr int kMaxWidth = 64;
constexpr int kThreads = 128;

thread_local std::string g_mlp_err;

struct Dims {
    int L;                 // number of affine layers
    int n[kMaxLayers + 1];  // widths n[0] = inputs ... n[L] = outputs
    int woff[kMaxLayers], boff[kMaxLayers];
    int nparam;
};

__device__ __forceinline__ float bf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Forward pass of one sample; acts[l][k] = activation after layer l (BF16-rounded),
// returns outputs in y. params: [W0 b0 W1 b1 ...] (already BF16-rounded floats).
__device__ void forward_one(const Dims &d, const float *p, const float *mean, const float *istd, const float *x,
                            float acts[kMaxLayers + 1][kMaxWidth]) {
    for (int k = 0; k < d.n[0]; ++k) acts[0][k] = bf((x[k] - mean[k]) * istd[k]);
    for (int l = 0; l < d.L; ++l) {
        const float *W = p + d.woff[l], *b = p + d.boff[l];
        const int ni = d.n[l], no = d.n[l + 1];
        for (int o = 0; o < no; ++o) {
            float acc = b[o];
            for (int i = 0; i < ni; ++i) acc += W[o * ni + i] * acts[l][i];
            if (l < d.L - 1) acc = acc > 0.f ? acc : 0.f;
            acts[l + 1][o] = (l < d.L - 1) ? bf(acc) : acc;
        }
    }
}

__global__ void k_mlp_forward(Dims d, const float *__restrict__ pbf, const float *__restrict__ mean,
                              const float *__restrict__ istd, const float *__restrict__ X, int n, float *__restrict__ Y) {
    extern __shared__ float sp[];
    for (int k = threadIdx.x; k < d.nparam; k += blockDim.x) sp[k] = pbf[k];
    __shared__ float sm[kMaxWidth], ss[kMaxWidth];
    for (int k = threadIdx.x; k < d.n[0]; k += blockDim.x) { sm[k] = mean[k]; ss[k] = istd[k]; }
    __syncthreads();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    float acts[kMaxLayers + 1][kMaxWidth];
    forward_one(d, sp, sm, ss, X + (size_t)s * d.n[0], acts);
    for (int o = 0; o < d.n[d.L]; ++o) Y[(size_t)s * d.n[d.L] + o] = acts[d.L][o];
}

// Gradient of 0.5/n * sum_s sum_o mask_o (y_so - t_so)^2 w.r.t. the FP32 master
// parameters (straight-through for the BF16 roundings), accumulated into grad;
// loss accumulated into *loss.
__global__ void k_mlp_backward(Dims d, const float *__restrict__ pbf, const float *__restrict__ mean,
                               const float *__restrict__ istd, const float *__restrict__ X,
                               const float *__restrict__ Tg, const float *__restrict__ mask, int n, float inv_n,
                               float *__restrict__ grad, float *__restrict__ loss) {
    extern __shared__ float sh[];
    float *sp = sh;               // parameters (BF16-rounded)
    float *sg = sh + d.nparam;    // block gradient accumulator
    for (int k = threadIdx.x; k < d.nparam; k += blockDim.x) { sp[k] = pbf[k]; sg[k] = 0.f; }
    __shared__ float sm[kMaxWidth], ss[kMaxWidth], sl;
    for (int k = threadIdx.x; k < d.n[0]; k += blockDim.x) { sm[k] = mean[k]; ss[k] = istd[k]; }
    if (threadIdx.x == 0) sl = 0.f;
    __syncthreads();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const bool act = s < n;
    const int lane = threadIdx.x & 31;
    float acts[kMaxLayers + 1][kMaxWidth];
    float delta[kMaxWidth], prev[kMaxWidth];
    if (act) forward_one(d, sp, sm, ss, X + (size_t)s * d.n[0], acts);
    const int nout = d.n[d.L];
    float l2 = 0.f;
    for (int o = 0; o < nout; ++o) {
        const float e = act ? acts[d.L][o] - Tg[(size_t)s * nout + o] : 0.f;
        l2 += mask[o] * e * e;
        delta[o] = mask[o] * e * inv_n;
    }
    for (int l = d.L - 1; l >= 0; --l) {
        const int ni = d.n[l], no = d.n[l + 1];
        const float *W = sp + d.woff[l];
        // weight and bias gradients: dW[o][i] = delta[o] * acts[l][i]
        for (int o = 0; o < no; ++o) {
            for (int i = 0; i <= ni; ++i) {
                float g = act ? delta[o] * (i < ni ? acts[l][i] : 1.f) : 0.f;
                for (int off = 16; off > 0; off >>= 1) g += __shfl_xor_sync(0xffffffffu, g, off);
                if (lane == 0) atomicAdd(&sg[i < ni ? d.woff[l] + o * ni + i : d.boff[l] + o], g);
            }
        }
        if (l > 0) {
            for (int i = 0; i < ni; ++i) {
                float acc = 0.f;
                for (int o = 0; o < no; ++o) acc += W[o * ni + i] * delta[o];
                prev[i] = acts[l][i] > 0.f ? acc : 0.f;  // ReLU' of the layer that produced acts[l]
            }
            for (int i = 0; i < ni; ++i) delta[i] = prev[i];
        }
    }
    for (int off = 16; off > 0; off >>= 1) l2 += __shfl_xor_sync(0xffffffffu, l2, off);
    if (lane == 0) atomicAdd(&sl, l2);
    __syncthreads();
    for (int k = threadIdx.x; k < d.nparam; k += blockDim.x) atomicAdd(&grad[k], sg[k]);
    if (threadIdx.x == 0) atomicAdd(loss, 0.5f * sl * inv_n);
}

// Forward pass on the BF16 tensor cores (mma.sync.m16n8k16, FP32 accumulation) for the
// shape of the learned corrections: n0 <= 32 inputs, hidden layers of 64, one output.
// A warp takes 32 samples, two fragments of 16: each layer's C fragments (+ bias, ReLU, rounded to
// BF16) are the next layer's A fragments as they sit in the registers (n-tiles 2t and 2t + 1 of
// the output are k-step t of the next product); the weights are the B operands, in fragment order
// (k_round_pack, whenever the weights change) so that a CTA copies them to shared memory as they
// are and one 16-byte load per lane feeds four products; the 64 -> 1 output layer is a dot product
// per sample summed over the four lanes that hold a row. Same arithmetic as forward_one up to the
// order of the FP32 sums. Bound by the issue of the products and of the ReLU and rounding between
// them. Measured on 524,288 samples of 17 inputs, three hidden layers: 138 -> 51 us (61 without the
// copy of the next inputs under the products); before, 16 CTAs an SM each converted and placed all
// weights for 3.5 groups of samples a warp. The products alone take 20 us at this instruction's rate.
constexpr int kMmaW = 64;  // hidden width
constexpr int kFragStep = 4 * 32;  // uint4 of one k-step: [n-tile pair][lane]

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned *>(&v);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
                 "{%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// k-steps of the hidden layers: two for the inputs (K padded to 32), four for each further layer
__host__ __device__ inline int frag_steps(const Dims &d) { return 2 + 4 * (d.L - 2); }

__global__ void __launch_bounds__(128, 3) k_mlp_forward_mma(Dims d, const float *__restrict__ pbf,
                                                            const uint4 *__restrict__ frag,
                                                            const float *__restrict__ mean,
                                                            const float *__restrict__ istd, const float *__restrict__ X,
                                                            int n, float *__restrict__ Y) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int nh = d.L - 1, nfrag = frag_steps(d) * kFragStep;  // hidden layers (each followed by ReLU)
    uint4 *wf = reinterpret_cast<uint4 *>(smraw);
    float *bias = reinterpret_cast<float *>(wf + nfrag);  // [nh][64]
    float *wout = bias + nh * kMmaW;                      // [64], then bout
    float *smean = wout + kMmaW + 1, *sistd = smean + 32;
    const int n0 = d.n[0];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    // the inputs of the warp's next 32 samples, copied while the current ones are computed
    float *xs = sistd + 32 + warp * 32 * n0;
    const long step = (long)gridDim.x * (blockDim.x >> 5) * 32;
    long base = ((long)blockIdx.x * (blockDim.x >> 5) + warp) * 32;
    auto fetch = [&](long b) {
        const long m = ((long)n - b < 32 ? (long)n - b : 32) * n0;
        const float *src = X + (size_t)b * n0;
        for (int k = lane; k < m; k += 32)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(xs + k)),
                         "l"(src + k));
    };
    if (base < n) fetch(base);
    for (int k = threadIdx.x; k < nfrag; k += blockDim.x) wf[k] = frag[k];
    for (int k = threadIdx.x; k < nh * kMmaW; k += blockDim.x) bias[k] = pbf[d.boff[k / kMmaW] + k % kMmaW];
    for (int k = threadIdx.x; k <= kMmaW; k += blockDim.x) wout[k] = pbf[k < kMmaW ? d.woff[nh] + k : d.boff[nh]];
    for (int k = threadIdx.x; k < 32; k += blockDim.x) {
        smean[k] = k < n0 ? mean[k] : 0.f;
        sistd[k] = k < n0 ? istd[k] : 0.f;
    }
    __syncthreads();
    const int nks0 = n0 > 16 ? 2 : 1;  // k-steps of the inputs
    for (; base < n; base += step) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        // layer 0 A fragments: standardised inputs, rounded to BF16, K padded to 32
        unsigned a[2][4][4];
        auto xin = [&](int r, int k) -> float {
            return (base + r < n && k < n0) ? (xs[r * n0 + k] - smean[k]) * sistd[k] : 0.f;
        };
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const int r0 = mt * 16 + g, r1 = r0 + 8;
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                if (ks >= nks0) break;
                const int k = ks * 16 + 2 * t4;
                a[mt][ks][0] = pack_bf16(xin(r0, k), xin(r0, k + 1));
                a[mt][ks][1] = pack_bf16(xin(r1, k), xin(r1, k + 1));
                a[mt][ks][2] = pack_bf16(xin(r0, k + 8), xin(r0, k + 9));
                a[mt][ks][3] = pack_bf16(xin(r1, k + 8), xin(r1, k + 9));
            }
        }
        __syncwarp();
        if (base + step < n) fetch(base + step);
#pragma unroll 1
        for (int l = 0; l < nh; ++l) {
            const float *bl = bias + l * kMmaW;
            float c[2][8][4];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const int col = nt * 8 + 2 * t4;
                const float b0 = bl[col], b1 = bl[col + 1];
#pragma unroll
                for (int mt = 0; mt < 2; ++mt) {
                    c[mt][nt][0] = c[mt][nt][2] = b0;
                    c[mt][nt][1] = c[mt][nt][3] = b1;
                }
            }
            const int nks = l == 0 ? nks0 : 4;
            const uint4 *W = wf + (l == 0 ? 0 : 2 + 4 * (l - 1)) * kFragStep + lane;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                if (ks >= nks) break;
#pragma unroll
                for (int pr = 0; pr < 4; ++pr) {
                    const uint4 w = W[(ks * 4 + pr) * 32];
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        mma_bf16(c[mt][2 * pr], a[mt][ks], w.x, w.y);
                        mma_bf16(c[mt][2 * pr + 1], a[mt][ks], w.z, w.w);
                    }
                }
            }
            // ReLU, BF16: the next layer's A fragments
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    auto rl = [](float v) { return v > 0.f ? v : 0.f; };
                    a[mt][t][0] = pack_bf16(rl(c[mt][2 * t][0]), rl(c[mt][2 * t][1]));
                    a[mt][t][1] = pack_bf16(rl(c[mt][2 * t][2]), rl(c[mt][2 * t][3]));
                    a[mt][t][2] = pack_bf16(rl(c[mt][2 * t + 1][0]), rl(c[mt][2 * t + 1][1]));
                    a[mt][t][3] = pack_bf16(rl(c[mt][2 * t + 1][2]), rl(c[mt][2 * t + 1][3]));
                }
        }
        // output layer 64 -> 1 on the BF16 activations
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            float y0 = 0.f, y1 = 0.f;
#pragma unroll
            for (int t = 0; t < 4; ++t)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = (2 * t + h) * 8 + 2 * t4;
                    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162 *>(&a[mt][t][2 * h]);
                    const __nv_bfloat162 hi = *reinterpret_cast<const __nv_bfloat162 *>(&a[mt][t][2 * h + 1]);
                    y0 += wout[col] * __low2float(lo) + wout[col + 1] * __high2float(lo);
                    y1 += wout[col] * __low2float(hi) + wout[col + 1] * __high2float(hi);
                }
            y0 += __shfl_xor_sync(0xffffffffu, y0, 1);
            y0 += __shfl_xor_sync(0xffffffffu, y0, 2);
            y1 += __shfl_xor_sync(0xffffffffu, y1, 1);
            y1 += __shfl_xor_sync(0xffffffffu, y1, 2);
            if (t4 == 0) {
                const long r0 = base + mt * 16 + g, r1 = r0 + 8;
                if (r0 < n) Y[r0] = wout[kMmaW] + y0;
                if (r1 < n) Y[r1] = wout[kMmaW] + y1;
            }
        }
    }
}

static bool mma_shape(const Dims &d) {
    if (d.L < 2 || d.n[0] > 32 || d.n[d.L] != 1) return false;
    for (int l = 1; l < d.L; ++l)
        if (d.n[l] != kMmaW) return false;
    return true;
}

static size_t mma_smem(const Dims &d) {
    const int nh = d.L - 1;
    return (size_t)frag_steps(d) * kFragStep * 16 + (size_t)nh * kMmaW * 4 + (kMmaW + 1) * 4 + 64 * 4 +
           (size_t)4 * 32 * d.n[0] * 4;
}

// The BF16 forms of the weights, in one launch (a launch of its own for the fragments made a training
// step of a small network 212 -> 220 us): wb, the parameters rounded, and frag (mma_shape, else
// NULL), the hidden layers' weights in B-fragment order: lane (g, t) of n-tile nt, k-step ks holds
// W[8 nt + g][16 ks + 2 t + {0, 1}] and W[8 nt + g][16 ks + 8 + 2 t + {0, 1}] (zero beyond the inputs).
__global__ void k_round_pack(Dims d, const float *__restrict__ w, float *__restrict__ wb, uint4 *__restrict__ frag) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < d.nparam) wb[k] = bf(w[k]);
    if (!frag || k >= frag_steps(d) * kFragStep) return;
    const int lane = k & 31, pr = (k >> 5) & 3, s = k >> 7, g = lane >> 2, t = lane & 3;
    const int l = s < 2 ? 0 : 1 + (s - 2) / 4, ks = s < 2 ? s : (s - 2) % 4, ni = d.n[l];
    unsigned v[4];
    for (int q = 0; q < 4; ++q) {
        const float *row = w + d.woff[l] + ((2 * pr + (q >> 1)) * 8 + g) * ni;
        const int i = ks * 16 + (q & 1) * 8 + 2 * t;
        v[q] = pack_bf16(i < ni ? row[i] : 0.f, i + 1 < ni ? row[i + 1] : 0.f);
    }
    frag[k] = make_uint4(v[0], v[1], v[2], v[3]);
}

__global__ void k_adam(float *w, const float *g, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.f - b1) * gk;
    const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    w[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
}

}  // namespace

struct hp_mlp {
    Dims d;
    float *w = nullptr, *wb = nullptr, *m = nullptr, *v = nullptr, *g = nullptr, *mean = nullptr, *istd = nullptr,
          *loss = nullptr;
    uint4 *frag = nullptr;  // the hidden layers' weights in fragment order (mma_shape)
    int step = 0;
    int nsm = 148;  // of the network's device
};

extern "C" const char *hp_mlp_last_error(void) { return g_mlp_err.c_str(); }

static int merr(int code, const char *m) {
    g_mlp_err = m;
    return code;
}

#define MCK(call)                                                                          \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) return merr(HP_ECUDA, cudaGetErrorString(e_));              \
    } while (0)

// The BF16 forms of the weights after they changed (stream 0).
static void refresh_bf16(hp_mlp *net) {
    const int n = std::max(net->d.nparam, net->frag ? frag_steps(net->d) * kFragStep : 0);
    k_round_pack<<<(n + 127) / 128, 128>>>(net->d, net->w, net->wb, net->frag);
}

extern "C" int hp_mlp_create(int nlayers, const int *widths, unsigned long long seed, hp_mlp **out) {
    if (!widths || !out || nlayers < 1 || nlayers > kMaxLayers) return merr(HP_EINVAL, "bad layer count");
    hp_mlp *net = new hp_mlp();
    int device = 0, nsm = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    if (nsm > 0) net->nsm = nsm;
    Dims &d = net->d;
    d.L = nlayers;
    int off = 0;
    for (int l = 0; l <= nlayers; ++l) {
        if (widths[l] < 1 || widths[l] > kMaxWidth) { delete net; return merr(HP_EINVAL, "width outside [1,64]"); }
        d.n[l] = widths[l];
    }
    for (int l = 0; l < nlayers; ++l) {
        d.woff[l] = off;
        off += d.n[l] * d.n[l + 1];
        d.boff[l] = off;
        off += d.n[l + 1];
    }
    d.nparam = off;
    // He-uniform initialisation from a splitmix64 stream (deterministic)
    std::vector<float> h(off, 0.f);
    unsigned long long z = seed;
    auto next = [&]() {
        z += 0x9E3779B97F4A7C15ull;
        unsigned long long x = z;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        x ^= x >> 31;
        return (double)(x >> 11) * (1.0 / 9007199254740992.0);
    };
    for (int l = 0; l < nlayers; ++l) {
        const float a = std::sqrt(6.0f / d.n[l]) * (l == nlayers - 1 ? 0.1f : 1.0f);
        for (int k = 0; k < d.n[l] * d.n[l + 1]; ++k) h[d.woff[l] + k] = (float)((2.0 * next() - 1.0) * a);
    }
    const size_t B = (size_t)off * 4;
    if (cudaMalloc(&net->w, B) || cudaMalloc(&net->wb, B) || cudaMalloc(&net->m, B) || cudaMalloc(&net->v, B) ||
        cudaMalloc(&net->g, B) || cudaMalloc(&net->mean, kMaxWidth * 4) || cudaMalloc(&net->istd, kMaxWidth * 4) ||
        cudaMalloc(&net->loss, 4) ||
        (mma_shape(d) && cudaMalloc(&net->frag, (size_t)frag_steps(d) * kFragStep * 16))) {
        hp_mlp_destroy(net);
        return merr(HP_ENOMEM, "cudaMalloc failed");
    }
    cudaMemcpy(net->w, h.data(), B, cudaMemcpyHostToDevice);
    cudaMemset(net->m, 0, B);
    cudaMemset(net->v, 0, B);
    std::vector<float> mu(kMaxWidth, 0.f), sd(kMaxWidth, 1.f);
    cudaMemcpy(net->mean, mu.data(), kMaxWidth * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(net->istd, sd.data(), kMaxWidth * 4, cudaMemcpyHostToDevice);
    refresh_bf16(net);
    MCK(cudaDeviceSynchronize());
    *out = net;
    return HP_OK;
}

extern "C" int hp_mlp_destroy(hp_mlp *net) {
    if (!net) return HP_OK;
    for (float *p : {net->w, net->wb, net->m, net->v, net->g, net->mean, net->istd, net->loss})
        if (p) cudaFree(p);
    if (net->frag) cudaFree(net->frag);
    delete net;
    return HP_OK;
}

extern "C" int hp_mlp_nparams(const hp_mlp *net) { return net ? net->d.nparam : HP_EINVAL; }

extern "C" int hp_mlp_set_norm(hp_mlp *net, const float *mean, const float *stdv) {
    if (!net || !mean || !stdv) return merr(HP_EINVAL, "null argument");
    std::vector<float> is(net->d.n[0]);
    for (int k = 0; k < net->d.n[0]; ++k) is[k] = stdv[k] > 0.f ? 1.f / stdv[k] : 1.f;
    MCK(cudaMemcpy(net->mean, mean, net->d.n[0] * 4, cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(net->istd, is.data(), net->d.n[0] * 4, cudaMemcpyHostToDevice));
    return HP_OK;
}

extern "C" int hp_mlp_get_params(const hp_mlp *net, float *host) {
    if (!net || !host) return merr(HP_EINVAL, "null argument");
    MCK(cudaMemcpy(host, net->w, (size_t)net->d.nparam * 4, cudaMemcpyDeviceToHost));
    return HP_OK;
}

extern "C" int hp_mlp_set_params(hp_mlp *net, const float *host) {
    if (!net || !host) return merr(HP_EINVAL, "null argument");
    MCK(cudaMemcpy(net->w, host, (size_t)net->d.nparam * 4, cudaMemcpyHostToDevice));
    refresh_bf16(net);
    MCK(cudaDeviceSynchronize());
    return HP_OK;
}

static size_t fwd_smem(const hp_mlp *net) { return (size_t)net->d.nparam * 4; }

extern "C" int hp_mlp_forward(hp_mlp *net, const float *d_x, int n, float *d_y, void *stream) {
    if (!net || (n > 0 && (!d_x || !d_y)) || n < 0) return merr(HP_EINVAL, "bad argument");
    if (n == 0) return HP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (mma_shape(net->d)) {  // the learned corrections' shape: BF16 tensor cores
        const size_t smm = mma_smem(net->d);
        if (smm > 48 * 1024)
            MCK(cudaFuncSetAttribute(k_mlp_forward_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smm));
        // as many CTAs as are resident: the weights are staged once per CTA
        const long groups = ((long)n + 31) / 32;
        const int blocks = (int)std::min<long>((groups + 3) / 4, 3L * net->nsm);
        k_mlp_forward_mma<<<blocks, 128, smm, st>>>(net->d, net->wb, net->frag, net->mean, net->istd, d_x, n, d_y);
        MCK(cudaGetLastError());
        return HP_OK;
    }
    const size_t sm = fwd_smem(net);
    if (sm > 48 * 1024) MCK(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_mlp_forward<<<(n + kThreads - 1) / kThreads, kThreads, sm, st>>>(net->d, net->wb, net->mean, net->istd, d_x, n,
                                                                       d_y);
    MCK(cudaGetLastError());
    return HP_OK;
}

// Gradient of the masked MSE over n samples into host_grad (FP32, nparam) and the
// loss into *loss; nothing is updated.
static int grad_device(hp_mlp *net, const float *d_x, const float *d_t, const float *mask, int n, cudaStream_t st) {
    const int P = net->d.nparam;
    MCK(cudaMemsetAsync(net->g, 0, (size_t)P * 4, st));
    MCK(cudaMemsetAsync(net->loss, 0, 4, st));
    const size_t sm = (size_t)2 * P * 4;
    MCK(cudaFuncSetAttribute(k_mlp_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_mlp_backward<<<(n + kThreads - 1) / kThreads, kThreads, sm, st>>>(net->d, net->wb, net->mean, net->istd, d_x, d_t,
                                                                        mask, n, 1.f / (float)n, net->g, net->loss);
    MCK(cudaGetLastError());
    return HP_OK;
}

extern "C" int hp_mlp_grad(hp_mlp *net, const float *d_x, const float *d_t, const float *d_mask, int n,
                           float *host_grad, float *loss) {
    if (!net || !d_x || !d_t || !d_mask || n < 1 || !host_grad) return merr(HP_EINVAL, "bad argument");
    int r = grad_device(net, d_x, d_t, d_mask, n, 0);
    if (r) return r;
    MCK(cudaMemcpy(host_grad, net->g, (size_t)net->d.nparam * 4, cudaMemcpyDeviceToHost));
    if (loss) MCK(cudaMemcpy(loss, net->loss, 4, cudaMemcpyDeviceToHost));
    return HP_OK;
}

extern "C" int hp_mlp_train_step(hp_mlp *net, const float *d_x, const float *d_t, const float *d_mask, int n, float lr,
                                 float *loss) {
    if (!net || !d_x || !d_t || !d_mask || n < 1) return merr(HP_EINVAL, "bad argument");
    int r = grad_device(net, d_x, d_t, d_mask, n, 0);
    if (r) return r;
    net->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)net->step), c2 = 1.f - std::pow(b2, (float)net->step);
    const int P = net->d.nparam;
    k_adam<<<(P + 255) / 256, 256>>>(net->w, net->g, net->m, net->v, P, lr, b1, b2, 1e-8f, c1, c2);
    refresh_bf16(net);
    MCK(cudaGetLastError());
    if (loss) MCK(cudaMemcpy(loss, net->loss, 4, cudaMemcpyDeviceToHost));
    return HP_OK;
}

extern "C" int hp_mlp_dims(const hp_mlp *net, int *nin, int *nout) {
    if (!net) return merr(HP_EINVAL, "null network");
    if (nin) *nin = net->d.n[0];
    if (nout) *nout = net->d.n[net->d.L];
    return HP_OK;
}
