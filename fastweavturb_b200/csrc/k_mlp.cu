// k_mlp.cu -- the learned surrogate: a multilayer perceptron n_in -> width x depth (GELU) ->
// n_out whose matrix products run on the tensor cores (BF16 operands, FP32 accumulation), with
// the bias, activation, loss and activation gradient of each product in its epilogue.  FP32
// master weights; BF16 copies (and transposes, for the backward products) are refreshed with
// every update.  No reference counterpart: the surrogate maps generator parameters to the
// statistics the generator produces (the reference only plots those statistics).
//
// Shapes (B = batch padded to a multiple of 64, Kl = layer input width padded to 64):
//   forward   Z_l[B x N_l]  = H_{l-1}[B x K_l] . W_l[N_l x K_l]^T + b_l,  H_l = gelu(Z_l)
//   backward  dH_{l-1}[B x K_l] = dZ_l[B x Np_l] . (W_l^T[K_l x Np_l])^T,  dZ = dH * gelu'(Z)
//             dW_l[N_l x K_l] = dZ_l^T[N_l x B] . (H_{l-1}^T[K_l x B])^T
//
// What bounds it: latency.  At the surrogate's batch of 256 a product is 34 MFLOP, under a
// microsecond of one SM's tensor core, so a step is a chain of dependent launches.  The chain is
// kept short -- pack, one launch per layer forward and back, one for all weight gradients, one for
// the bias gradients, one for Adam and the BF16 copies: 13 launches for depth 4, against 57 with
// the elementwise passes apart (one thread per column summed the bias gradients row by row) --
// and each launch lets the next one start its prologue early (programmatic dependent launch):
// barriers, tensor memory and the weights' tiles, which no kernel of the chain writes, are ready
// when the previous product ends.  Inputs and results cross to the host in one copy each.
// Batch 256, depth 4: 160 us a training step, 760 before; the input gradient of 192 rows 119 us, 628
// before (about 8 us a layer: the wait for the product before, one load latency, the epilogue).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <exception>
#include <string>
#include <vector>

#include "../../include/fwt.h"
#include "fwt_internal.h"
#include "k_gemm_tc.cuh"

namespace fwt {

int gemm_bf16_tc(const void *A, const void *B, float *C, int M, int N, int K, int ldc, int *d_err, cudaStream_t st);

static inline int pad64(int x) { return (x + 63) / 64 * 64; }
static inline unsigned nblk(int64_t n) { return (unsigned)((n + 255) / 256); }

struct MlpLayer {
    int K = 0, Kp = 0, N = 0, Np = 0;   // input/output widths and their 64-padded sizes
    float *W = nullptr, *b = nullptr;   // FP32 master (N x K), (N)
    float *mW = nullptr, *vW = nullptr, *mb = nullptr, *vb = nullptr;
    float *gW = nullptr, *gb = nullptr;
    __nv_bfloat16 *Wh = nullptr;        // N x Kp
    __nv_bfloat16 *Wt = nullptr;        // Kp x Np (transpose)
    float *Z = nullptr;                 // B x N pre-activation (hidden layers)
    __nv_bfloat16 *H = nullptr;         // B x Np activation (input of the next layer)
    __nv_bfloat16 *Ht = nullptr;        // Np x B
    float *dZf = nullptr;               // B x N
    __nv_bfloat16 *dZ = nullptr;        // B x Np
    __nv_bfloat16 *dZt = nullptr;       // N x B
};

}  // namespace fwt

struct fwt_mlp {
    int dev = 0;
    int n_in = 0, width = 0, depth = 0, n_out = 0, bmax = 0;
    std::vector<fwt::MlpLayer> L;
    __nv_bfloat16 *X0 = nullptr, *X0t = nullptr;   // B x 64, 64 x B
    // One exchange buffer with the host, and its mirror there: the loss (FP64), the error flag and a
    // pad, then x (B x n_in; the input gradient replaces it), then from the next 16 bytes on the targets
    // (B x n_out; the forward pass writes its outputs there, 16 bytes a store), then the output weights
    // (n_out).
    // The mirror is ordinary memory: pinning it cost 14-25 ms a network and saved nothing measurable a step.
    unsigned char *io = nullptr;
    std::vector<unsigned char> hmem;
    unsigned char *hio = nullptr;
    int64_t step = 0;
    cudaStream_t st = nullptr;
    std::vector<void *> allocs;

    int *err() const { return (int *)(io + 8); }
    float *x() const { return (float *)(io + 16); }
    size_t t_at(int B) const { return ((size_t)B * n_in + 3) / 4 * 4; }   // floats from x to the targets
    float *t(int B) const { return x() + t_at(B); }
    float *w(int B) const { return t(B) + (size_t)B * n_out; }
};

namespace fwt {

template <typename T>
static int mlp_alloc(fwt_mlp *m, T **p, size_t n)
{
    void *q = nullptr;
    if (cudaMalloc(&q, sizeof(T) * std::max<size_t>(n, 1)) != cudaSuccess) {
        cudaGetLastError();
        return fail(FWT_E_NOMEM, "mlp: device allocation failed");
    }
    cudaMemset(q, 0, sizeof(T) * std::max<size_t>(n, 1));
    m->allocs.push_back(q);
    *p = (T *)q;
    return 0;
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float x)
{
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

constexpr size_t kIoHead = 16;   // bytes of the exchange buffer before x
// Up to this many bytes the forward pass's outputs come with the flag and the inputs before them, in one
// copy through the mirror; beyond, in a copy of their own to the caller's place (64 inputs, 256 outputs, us
// a call, once / apart: 128 rows 90 / 103, 1000 rows 319 / 303, 4096 rows 1110 / 850).
constexpr size_t kIoOnce = 1 << 19;

// X (B x n_in, FP32) -> X0 (Bp x 64 BF16, zero padded) and its transpose
__global__ void mlp_pack_input(const float *__restrict__ X, int B, int Bp, int n_in, __nv_bfloat16 *__restrict__ X0,
                               __nv_bfloat16 *__restrict__ X0t)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Bp * 64) return;
    const int r = i / 64, c = i % 64;
    const float v = (r < B && c < n_in) ? X[(size_t)r * n_in + c] : 0.0f;
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    X0[i] = h;
    X0t[(size_t)c * Bp + r] = h;
}

// What a product's epilogue does with element (r, c) of A . B^T:
enum MlpEpi {
    kHidden = 0,   // Z = . + b; H = gelu(Z) (BF16, zero padded to Np) and H^T
    kOutput,       // Z = . + b
    kLoss,         // y = . + b against the targets: loss = sum w (y - t)^2 / (B n), dZ of the output layer
    kActBack,      // dZ = . * gelu'(Z) for a hidden layer
    kWeight,       // the weight gradient, K wide
    kInput         // the input gradient, n_in wide
};

struct MlpJob {
    const __nv_bfloat16 *A, *Bm;   // M x K, Nb x K (rows beyond Nb count as zero)
    int M, N, K, Nb;
    int epi, b_const;              // b_const: B is not written by the kernels of this step
    int B, Bp, Nl, Np;             // batch, padded batch, the output's width and its padded width
    const float *bias;
    float *Z;                      // B x Nl: written (kHidden, kOutput), read (kActBack)
    __nv_bfloat16 *H, *Ht;         // Bp x Np and Np x Bp (kHidden); dZ and dZ^T (kLoss, kActBack)
    float *F;                      // dZf (kLoss, kActBack), dW (kWeight), dX (kInput)
    const float *T, *w;            // targets and output weights (kLoss)
    double *loss;
};

constexpr int kMlpJobs = 8;       // products of one launch
struct MlpJobs {
    MlpJob j[kMlpJobs];
};

constexpr int kMlpBN = 32, kMlpStages = 4, kMlpThreads = 256;
constexpr size_t kMlpStage = (size_t)(kGemmBM + kMlpBN) * kGemmBK * 2;
constexpr size_t kMlpSmem = kMlpStage * kMlpStages;

// The ring's copies: cp.async group c holds chunk c.  The prologue commits groups 0 .. kMlpStages - 1;
// iteration kc >= 1 refills the stage of chunk kc - 1 and commits group kc - 1 + kMlpStages (empty past the
// last chunk), iteration 0 commits none.  Groups that may still be in flight when iteration kc issues its
// products, so that groups 0 .. kc have landed:
constexpr int ring_pending(int kc) { return kc == 0 ? kMlpStages - 1 : kMlpStages - 2; }
constexpr bool ring_covers(int nk)
{
    int committed = kMlpStages;
    for (int kc = 0; kc < nk; ++kc) {
        if (committed - ring_pending(kc) < kc + 1) return false;
        if (kc > 0 && committed++ != kc - 1 + kMlpStages) return false;   // group c is chunk c
    }
    return true;
}
static_assert(ring_covers(4096), "mlp_gemm_kernel: a chunk is multiplied before its copies have landed");

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in)
{
    const int n = in ? 16 : 0;   // rows beyond the matrix read zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// One 128 x 32 tile of job blockIdx.z per CTA: K in chunks of 64 through a ring of four stages (the
// surrogate's K of 256 is staged whole), cp.async into the no-swizzle K-major layout, four
// tcgen05.mma (M 128, N 32, K 16) per chunk into tensor memory, and the epilogue by eight warps
// (16 columns each) straight from it.  32 columns rather than 256: a layer of 256 x 256 at batch
// 256 spreads over 16 SMs and the epilogue, the longest part, is an eighth as long.  Every wait is
// bounded; on a timeout the CTA sets *err, still frees its tensor memory and returns.
__global__ void __launch_bounds__(kMlpThreads) mlp_gemm_kernel(const __grid_constant__ MlpJobs jobs, int *__restrict__ err)
{
    const MlpJob &J = jobs.j[blockIdx.z];
    const int m0 = blockIdx.x * kGemmBM, n0 = blockIdx.y * kMlpBN;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (m0 >= J.M || n0 >= J.N) {
        // the next kernel may rely on this one's wait for all that came before
        asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bar[kMlpStages];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bar);
    const int K = J.K, nk = K / kGemmBK;
    auto load_a = [&](int kc) {
        const uint32_t s = s0 + (uint32_t)(kc % kMlpStages) * (uint32_t)kMlpStage;
        for (int i = tid; i < kGemmBM * 8; i += kMlpThreads) {
            const int r = i >> 3, k8 = i & 7;
            const bool in = m0 + r < J.M;
            cp_async16(s + core_off(r, k8, kGemmBM), J.A + (size_t)(in ? m0 + r : 0) * K + kc * kGemmBK + k8 * 8, in);
        }
    };
    auto load_b = [&](int kc) {
        const uint32_t s = s0 + (uint32_t)(kc % kMlpStages) * (uint32_t)kMlpStage + kGemmBM * kGemmBK * 2;
        for (int i = tid; i < kMlpBN * 8; i += kMlpThreads) {
            const int r = i >> 3, k8 = i & 7;
            const bool in = n0 + r < J.Nb;
            cp_async16(s + core_off(r, k8, kMlpBN), J.Bm + (size_t)(in ? n0 + r : 0) * K + kc * kGemmBK + k8 * 8, in);
        }
    };
    if (warp == 0) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&tmem_base);
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(kMlpBN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid < kMlpStages)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * (uint32_t)tid) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const int pre = min(nk, kMlpStages);
    if (J.b_const)
        for (int kc = 0; kc < pre; ++kc) load_b(kc);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int kc = 0; kc < kMlpStages; ++kc) {   // one group per stage, empty ones included
        if (kc < pre) {
            if (!J.b_const) load_b(kc);
            load_a(kc);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = umma_idesc_bf16(kGemmBM, kMlpBN);
    // The epilogue's own operands, read while the product runs: warps w and w + 4 take accumulator
    // lanes 32 (w & 3) .. + 31, 16 columns each.
    const int row = m0 + (warp & 3) * 32 + lane, c0 = n0 + 16 * (warp >> 2);
    const bool in_b = row < (J.epi == kWeight ? J.M : J.B);
    const int nc = in_b ? max(0, min(16, J.Nl - c0)) : 0;   // this thread's columns inside the result
    const size_t at = (size_t)row * J.Nl + c0;
    const bool vec = nc == 16 && (J.Nl & 3) == 0;           // its 16 values start on 16 bytes, as every result does
    float e0[16], e1[16], e2[16];   // bias or Z; targets; output weights
#pragma unroll
    for (int i = 0; i < 16; ++i) e0[i] = e1[i] = e2[i] = 0.0f;
    if (J.epi == kActBack) {
        if (vec) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float4 *>(e0 + 4 * i) = *reinterpret_cast<const float4 *>(J.Z + at + 4 * i);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < nc) e0[i] = J.Z[at + i];
        }
    } else if (J.epi <= kLoss) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < nc) e0[i] = J.bias[c0 + i];
        if (J.epi == kLoss) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < nc) {
                    e1[i] = J.T[at + i];
                    e2[i] = J.w[c0 + i];
                }
        }
    }
    bool ok = true;
    for (int kc = 0; kc < nk && ok; ++kc) {
        if (kc == 0) asm volatile("cp.async.wait_group %0;" ::"n"(ring_pending(0)) : "memory");
        else asm volatile("cp.async.wait_group %0;" ::"n"(ring_pending(1)) : "memory");
        // the MMA reads shared memory through the async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = s0 + (uint32_t)(kc % kMlpStages) * (uint32_t)kMlpStage, sb = sa + kGemmBM * kGemmBK * 2;
#pragma unroll
            for (int kk = 0; kk < kGemmBK / 16; ++kk) {
                // K = 16 covers the core matrices 2kk and 2kk+1 along K
                const uint64_t da = umma_smem_desc(sa + (uint32_t)(2 * kk * kGemmBM * 16), kGemmBM * 16, 128);
                const uint64_t db = umma_smem_desc(sb + (uint32_t)(2 * kk * kMlpBN * 16), kMlpBN * 16, 128);
                const uint32_t acc = (kc > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             bar0 + 8u * (uint32_t)(kc % kMlpStages))
                         : "memory");
        }
        // refill the stage of the chunk before, once its products have read it
        const int nx = kc - 1 + kMlpStages;
        if (kc > 0 && nx < nk) {
            ok = gemm_mbar_wait(bar0 + 8u * (uint32_t)((kc - 1) % kMlpStages), (uint32_t)((kc - 1) / kMlpStages) & 1u);
            ok = __syncthreads_and(ok) != 0;
            if (ok) {
                load_b(nx);
                load_a(nx);
            }
        }
        if (kc > 0) asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (ok) {
        ok = gemm_mbar_wait(bar0 + 8u * (uint32_t)((nk - 1) % kMlpStages), (uint32_t)((nk - 1) / kMlpStages) & 1u);
        ok = __syncthreads_and(ok) != 0;
    }
    if (!ok) {
        if (tid == 0) atomicOr(err, 1);
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float v[16];
        {
            uint32_t u[16];
            const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(16 * (warp >> 2));
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];"
                : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
                  "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
        }
        double l = 0.0;
        float *keep = J.F;   // the FP32 values kept: B x Nl (kWeight: M x Nl)
        if (J.epi <= kOutput) {
            keep = J.Z;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += e0[i];
        } else if (J.epi == kActBack) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = v[i] * gelu_d(e0[i]);
        } else if (J.epi == kLoss) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float d = (v[i] + e0[i]) - e1[i];
                if (i < nc) l += (double)e2[i] * d * d / ((double)J.B * J.Nl);
                v[i] = 2.0f * e2[i] * d / ((float)J.B * (float)J.Nl);
            }
        }
        if (vec) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float4 *>(keep + at + 4 * i) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < nc) keep[at + i] = v[i];
        }
        if (row < J.M && (J.epi == kHidden || J.epi == kLoss || J.epi == kActBack)) {
            // a BF16 matrix for the next product, zero padded, and its transpose
            __align__(16) __nv_bfloat16 h[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float o = J.epi == kHidden ? gelu(v[i]) : v[i];
                h[i] = __float2bfloat16_rn(i < nc ? o : 0.0f);
            }
            if (c0 < J.Np) {   // Np is a multiple of 64: all 16 columns are inside or none
                uint4 *out = reinterpret_cast<uint4 *>(J.H + (size_t)row * J.Np + c0);
                out[0] = *reinterpret_cast<const uint4 *>(h);
                out[1] = *reinterpret_cast<const uint4 *>(h + 8);
            }
            const int nt = (J.epi == kHidden ? J.Np : J.Nl) - c0;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < nt) J.Ht[(size_t)(c0 + i) * J.Bp + row] = h[i];
        }
        if (J.epi == kLoss) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0 && l != 0.0) atomicAdd(J.loss, l);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kMlpBN));
}

// Per-layer arguments of the bias gradients and of Adam.
struct MlpParam {
    float *W, *mW, *vW, *gW, *b, *mb, *vb, *gb;
    __nv_bfloat16 *Wh, *Wt;
    const float *dZf;
    int N, K, Kp, Np;
};
struct MlpParams {
    MlpParam l[kMlpJobs];
};

// db = column sums of dZ (FP64 sums, fixed order): a block takes 32 columns of layer blockIdx.y, a
// warp every eighth row.
__global__ void __launch_bounds__(256) mlp_bias_grad(const __grid_constant__ MlpParams P, int B)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const MlpParam &L = P.l[blockIdx.y];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    __shared__ double part[8][32];
    double s = 0.0;
    if (c < L.N) {
#pragma unroll 4
        for (int r = warp; r < B; r += 8) s += L.dZf[(size_t)r * L.N + c];
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && c < L.N) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += part[i][lane];
        L.gb[c] = (float)t;
    }
}

__device__ __forceinline__ float adam_step(float *p, const float *g, float *m1, float *m2, int i, float lr, float b1,
                                           float b2, float c1, float c2, float eps)
{
    const float gi = g[i];
    const float a = b1 * m1[i] + (1.0f - b1) * gi, v = b2 * m2[i] + (1.0f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = v;
    const float q = p[i] - lr * (a / c1) / (sqrtf(v / c2) + eps);
    p[i] = q;
    return q;
}

// Adam on every weight and bias of the layers, and the weights' BF16 copies; nothing when a product
// of the step timed out (*err).
__global__ void __launch_bounds__(256) mlp_adam(const __grid_constant__ MlpParams P, float lr, float b1, float b2, float c1,
                                                float c2, float eps, const int *__restrict__ err)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const MlpParam &L = P.l[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x, n = L.N * L.K;
    if (*err != 0) return;
    if (i < n) {
        const __nv_bfloat16 h =
            __float2bfloat16_rn(adam_step(L.W, L.gW, L.mW, L.vW, i, lr, b1, b2, c1, c2, eps));
        const int r = i / L.K, k = i % L.K;
        L.Wh[(size_t)r * L.Kp + k] = h;
        L.Wt[(size_t)k * L.Np + r] = h;
    } else if (i < n + L.N) {
        adam_step(L.b, L.gb, L.mb, L.vb, i - n, lr, b1, b2, c1, c2, eps);
    }
}

// BF16 copies of W: Wh (N x Kp, zero padded) and Wt (Kp x Np)
__global__ void mlp_refresh(const float *__restrict__ W, int N, int K, int Kp, int Np, __nv_bfloat16 *__restrict__ Wh,
                            __nv_bfloat16 *__restrict__ Wt)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Np * Kp) return;
    const int n = i / Kp, k = i % Kp;
    const __nv_bfloat16 v = __float2bfloat16_rn((n < N && k < K) ? W[(size_t)n * K + k] : 0.0f);
    if (n < N) Wh[(size_t)n * Kp + k] = v;
    Wt[(size_t)k * Np + n] = v;
}

static int mlp_refresh_all(fwt_mlp *m)
{
    for (auto &l : m->L)
        mlp_refresh<<<nblk((int64_t)l.Np * l.Kp), 256, 0, m->st>>>(l.W, l.N, l.K, l.Kp, l.Np, l.Wh, l.Wt);
    FWT_CUDA(cudaGetLastError());
    return 0;
}

// Launch with the programmatic dependence on the kernel before it in the stream (every kernel of the
// chain waits for it with griddepcontrol.wait before it touches what that kernel writes).
template <typename K, typename... Args>
static int mlp_launch(fwt_mlp *m, K kernel, dim3 grid, int threads, size_t smem, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = m->st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FWT_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    return 0;
}

static int mlp_products(fwt_mlp *m, const MlpJob *j, int n)
{
    for (int o = 0; o < n; o += kMlpJobs) {
        MlpJobs jobs = {};
        int M = 0, N = 0;
        const int c = std::min(kMlpJobs, n - o);
        for (int i = 0; i < c; ++i) {
            jobs.j[i] = j[o + i];
            M = std::max(M, j[o + i].M);
            N = std::max(N, j[o + i].N);
        }
        const dim3 grid((unsigned)((M + kGemmBM - 1) / kGemmBM), (unsigned)((N + kMlpBN - 1) / kMlpBN), (unsigned)c);
        FWT_TRY(mlp_launch(m, mlp_gemm_kernel, grid, kMlpThreads, kMlpSmem, jobs, m->err()));
    }
    return 0;
}

// Forward pass of the batch in the exchange buffer; the output layer's values go to the targets'
// place, or (loss) to the loss and its gradient.
static int mlp_forward(fwt_mlp *m, int B, bool loss)
{
    const int Bp = pad64(B);
    FWT_TRY(mlp_launch(m, mlp_pack_input, dim3(nblk((int64_t)Bp * 64)), 256, 0, (const float *)m->x(), B, Bp, m->n_in, m->X0,
                       m->X0t));
    const __nv_bfloat16 *Hin = m->X0;
    for (size_t li = 0; li < m->L.size(); ++li) {
        MlpLayer &l = m->L[li];
        const bool last = li + 1 == m->L.size();
        MlpJob j = {};
        j.A = Hin;
        j.Bm = l.Wh;
        j.M = Bp;
        j.N = l.N;
        j.Nb = l.N;
        j.K = l.Kp;
        j.b_const = 1;
        j.B = B;
        j.Bp = Bp;
        j.Nl = l.N;
        j.Np = l.Np;
        j.bias = l.b;
        if (!last) {
            j.epi = kHidden;
            j.N = l.Np;   // the padding of H is written too
            j.Z = l.Z;
            j.H = l.H;
            j.Ht = l.Ht;
        } else if (!loss) {
            j.epi = kOutput;
            j.Z = m->t(B);
        } else {
            j.epi = kLoss;
            j.N = l.Np;
            j.H = l.dZ;
            j.Ht = l.dZt;
            j.F = l.dZf;
            j.T = m->t(B);
            j.w = m->w(B);
            j.loss = (double *)m->io;
        }
        FWT_TRY(mlp_products(m, &j, 1));
        Hin = l.H;
    }
    return 0;
}

static void mlp_param_list(fwt_mlp *m, size_t o, int c, MlpParams &P)
{
    P = {};
    for (int i = 0; i < c; ++i) {
        MlpLayer &l = m->L[o + i];
        P.l[i] = {l.W, l.mW, l.vW, l.gW, l.b, l.mb, l.vb, l.gb, l.Wh, l.Wt, l.dZf, l.N, l.K, l.Kp, l.Np};
    }
}

// After mlp_forward(loss): the gradients of the weighted MSE w.r.t. the inputs (in the inputs' place)
// and, if params, every parameter (into l.gW, l.gb).
static int mlp_backward(fwt_mlp *m, int B, bool params, bool inputs)
{
    const int Bp = pad64(B);
    for (int li = (int)m->L.size() - 1; li > 0 || (li == 0 && inputs); --li) {
        MlpLayer &l = m->L[li];
        // dH_prev = dZ . W  (M = Bp, N = Kp, K = Np)
        MlpJob j = {};
        j.A = l.dZ;
        j.Bm = l.Wt;
        j.M = Bp;
        j.N = j.Nb = l.Kp;
        j.K = l.Np;
        j.b_const = 1;
        j.B = B;
        j.Bp = Bp;
        if (li == 0) {
            j.epi = kInput;
            j.Nl = m->n_in;
            j.F = m->x();
        } else {
            MlpLayer &p = m->L[li - 1];
            j.epi = kActBack;
            j.Nl = p.N;
            j.Np = p.Np;
            j.Z = p.Z;
            j.H = p.dZ;
            j.Ht = p.dZt;
            j.F = p.dZf;
        }
        FWT_TRY(mlp_products(m, &j, 1));
    }
    if (!params) return 0;
    // dW = dZ^T . Hprev  (M = N_l, N = Kp, K = Bp), every layer in one launch
    std::vector<MlpJob> jobs;
    for (size_t li = 0; li < m->L.size(); ++li) {
        MlpLayer &l = m->L[li];
        MlpJob j = {};
        j.A = l.dZt;
        j.Bm = li > 0 ? m->L[li - 1].Ht : m->X0t;
        j.M = l.N;
        j.N = j.Nb = l.Kp;
        j.K = Bp;
        j.epi = kWeight;
        j.B = B;
        j.Nl = l.K;
        j.F = l.gW;
        jobs.push_back(j);
    }
    FWT_TRY(mlp_products(m, jobs.data(), (int)jobs.size()));
    for (size_t o = 0; o < m->L.size(); o += kMlpJobs) {
        const int c = (int)std::min<size_t>(kMlpJobs, m->L.size() - o);
        MlpParams P;
        mlp_param_list(m, o, c, P);
        int N = 0;
        for (int i = 0; i < c; ++i) N = std::max(N, P.l[i].N);
        FWT_TRY(mlp_launch(m, mlp_bias_grad, dim3((unsigned)((N + 31) / 32), (unsigned)c), 256, 0, P, B));
    }
    return 0;
}

// The inputs, targets and output weights (1 where w_out is null) of a batch to the device, with the
// loss and the error flag zeroed: one copy.
static int mlp_upload(fwt_mlp *m, const float *x, const float *t, const float *w_out, int B)
{
    std::memset(m->hio, 0, kIoHead);
    float *h = (float *)(m->hio + kIoHead);
    std::memcpy(h, x, sizeof(float) * (size_t)B * m->n_in);
    size_t n = (size_t)B * m->n_in;
    if (t) {
        n = m->t_at(B);
        std::memcpy(h + n, t, sizeof(float) * (size_t)B * m->n_out);
        n += (size_t)B * m->n_out;
        for (int i = 0; i < m->n_out; ++i) h[n + i] = w_out ? w_out[i] : 1.0f;
        n += m->n_out;
    }
    FWT_CUDA(cudaMemcpyAsync(m->io, m->hio, kIoHead + sizeof(float) * n, cudaMemcpyHostToDevice, m->st));
    return 0;
}

// The head of the exchange buffer and `floats` values after it, in the mirror; waits.
static int mlp_download(fwt_mlp *m, size_t floats)
{
    FWT_CUDA(cudaMemcpyAsync(m->hio, m->io, kIoHead + sizeof(float) * floats, cudaMemcpyDeviceToHost, m->st));
    FWT_CUDA(cudaStreamSynchronize(m->st));
    int herr = 0;
    std::memcpy(&herr, m->hio + 8, sizeof(int));
    if (herr) return fail(FWT_E_TIMEOUT, "mlp: tensor-core product's wait ran out");
    return 0;
}

}  // namespace fwt

using namespace fwt;

extern "C" {

int fwt_gemm_bf16(const void *dA, const void *dB, float *dC, int M, int N, int K, int ldc, void *stream)
{
    if (!dA || !dB || !dC || ldc < N) return fail(FWT_E_ARG, "gemm: null operand or ldc < N");
    int *d_err = nullptr;
    if (cudaMalloc(&d_err, sizeof(int)) != cudaSuccess) return fail(FWT_E_NOMEM, "gemm: error flag allocation");
    cudaStream_t st = (cudaStream_t)stream;
    cudaMemsetAsync(d_err, 0, sizeof(int), st);
    int rc = gemm_bf16_tc(dA, dB, dC, M, N, K, ldc, d_err, st);
    int herr = 0;
    if (rc == 0) {
        cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) rc = fail(FWT_E_CUDA, "gemm: kernel failed");
        else if (herr) rc = fail(FWT_E_TIMEOUT, "gemm: tensor-core wait ran out");
    }
    cudaFree(d_err);
    return rc;
}

int fwt_mlp_create(int device, int n_in, int width, int depth, int n_out, int batch_max, uint64_t seed, fwt_mlp **out)
{
    if (!out || n_in < 1 || n_in > 64 || width < 16 || width > 256 || width % 16 || depth < 1 || n_out < 1 ||
        n_out > 256 || batch_max < 1)
        return fail(FWT_E_ARG, "mlp: n_in 1..64, width 16..256 (multiple of 16), depth >= 1, n_out 1..256");
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return fail(FWT_E_CUDA, "mlp: no such device");
    fwt_mlp *m = new fwt_mlp();
    m->dev = device;
    m->n_in = n_in;
    m->width = width;
    m->depth = depth;
    m->n_out = n_out;
    m->bmax = pad64(batch_max);
    const int Bp = m->bmax;
    int rc = 0;
    auto try_ = [&](int r) {
        if (rc == 0 && r != 0) rc = r;
    };
    if (cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking) != cudaSuccess) rc = fail(FWT_E_CUDA, "mlp: stream");
    // widths: n_in -> width (depth times) -> n_out
    std::vector<int> w = {n_in};
    for (int i = 0; i < depth; ++i) w.push_back(width);
    w.push_back(n_out);
    uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto urand = [&]() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (double)(s >> 11) * (1.0 / 9007199254740992.0);
    };
    for (size_t i = 0; i + 1 < w.size() && rc == 0; ++i) {
        MlpLayer l;
        l.K = w[i];
        l.Kp = pad64(l.K);
        l.N = w[i + 1];
        l.Np = pad64(l.N);
        try_(mlp_alloc(m, &l.W, (size_t)l.N * l.K));
        try_(mlp_alloc(m, &l.b, l.N));
        try_(mlp_alloc(m, &l.mW, (size_t)l.N * l.K));
        try_(mlp_alloc(m, &l.vW, (size_t)l.N * l.K));
        try_(mlp_alloc(m, &l.mb, l.N));
        try_(mlp_alloc(m, &l.vb, l.N));
        try_(mlp_alloc(m, &l.gW, (size_t)l.N * l.K));
        try_(mlp_alloc(m, &l.gb, l.N));
        try_(mlp_alloc(m, &l.Wh, (size_t)l.N * l.Kp));
        try_(mlp_alloc(m, &l.Wt, (size_t)l.Kp * l.Np));
        try_(mlp_alloc(m, &l.Z, (size_t)Bp * l.N));
        try_(mlp_alloc(m, &l.H, (size_t)Bp * l.Np));
        try_(mlp_alloc(m, &l.Ht, (size_t)l.Np * Bp));
        try_(mlp_alloc(m, &l.dZf, (size_t)Bp * l.N));
        try_(mlp_alloc(m, &l.dZ, (size_t)Bp * l.Np));
        try_(mlp_alloc(m, &l.dZt, (size_t)l.N * Bp));
        if (rc) break;
        // uniform +-sqrt(6 / (fan_in + fan_out)), zero biases
        std::vector<float> hw((size_t)l.N * l.K);
        const double a = std::sqrt(6.0 / (l.K + l.N));
        for (auto &v : hw) v = (float)((2.0 * urand() - 1.0) * a);
        if (cudaMemcpy(l.W, hw.data(), sizeof(float) * hw.size(), cudaMemcpyHostToDevice) != cudaSuccess)
            rc = fail(FWT_E_CUDA, "mlp: weight upload");
        m->L.push_back(l);
    }
    try_(mlp_alloc(m, &m->X0, (size_t)Bp * 64));
    try_(mlp_alloc(m, &m->X0t, (size_t)64 * Bp));
    // (Bp x n_in is a multiple of four floats: no batch needs more)
    const size_t io_bytes = kIoHead + sizeof(float) * ((size_t)Bp * (n_in + n_out) + n_out);
    try_(mlp_alloc(m, &m->io, io_bytes));
    if (rc == 0) {   // a failed device allocation leaves no reason to ask the host for as much
        try {
            m->hmem.resize(io_bytes);
        } catch (const std::exception &) {
            rc = fail(FWT_E_NOMEM, "mlp: host allocation failed");
        }
        m->hio = m->hmem.data();
    }
    if (rc == 0 && cudaFuncSetAttribute(mlp_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMlpSmem) != cudaSuccess)
        rc = fail(FWT_E_CUDA, "mlp: kernel attribute");
    if (rc == 0) rc = mlp_refresh_all(m);
    if (rc == 0 && cudaStreamSynchronize(m->st) != cudaSuccess) rc = fail(FWT_E_CUDA, "mlp: set-up failed");
    if (rc) {
        fwt_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return 0;
}

int fwt_mlp_destroy(fwt_mlp *m)
{
    if (!m) return 0;
    cudaSetDevice(m->dev);
    if (m->st) cudaStreamSynchronize(m->st);
    for (void *p : m->allocs) cudaFree(p);
    if (m->st) cudaStreamDestroy(m->st);
    delete m;
    return 0;
}

int fwt_mlp_nparams(fwt_mlp *m, int64_t *n)
{
    if (!m || !n) return fail(FWT_E_ARG, "mlp: null argument");
    int64_t t = 0;
    for (auto &l : m->L) t += (int64_t)l.N * l.K + l.N;
    *n = t;
    return 0;
}

// parameters flattened layer by layer: W_l (N x K, row-major) then b_l
int fwt_mlp_get_params(fwt_mlp *m, float *host)
{
    if (!m || !host) return fail(FWT_E_ARG, "mlp: null argument");
    cudaSetDevice(m->dev);
    for (auto &l : m->L) {
        FWT_CUDA(cudaMemcpyAsync(host, l.W, sizeof(float) * l.N * l.K, cudaMemcpyDeviceToHost, m->st));
        host += (size_t)l.N * l.K;
        FWT_CUDA(cudaMemcpyAsync(host, l.b, sizeof(float) * l.N, cudaMemcpyDeviceToHost, m->st));
        host += l.N;
    }
    FWT_CUDA(cudaStreamSynchronize(m->st));
    return 0;
}

int fwt_mlp_set_params(fwt_mlp *m, const float *host)
{
    if (!m || !host) return fail(FWT_E_ARG, "mlp: null argument");
    cudaSetDevice(m->dev);
    for (auto &l : m->L) {
        FWT_CUDA(cudaMemcpyAsync(l.W, host, sizeof(float) * l.N * l.K, cudaMemcpyHostToDevice, m->st));
        host += (size_t)l.N * l.K;
        FWT_CUDA(cudaMemcpyAsync(l.b, host, sizeof(float) * l.N, cudaMemcpyHostToDevice, m->st));
        host += l.N;
    }
    FWT_TRY(mlp_refresh_all(m));
    FWT_CUDA(cudaStreamSynchronize(m->st));
    return 0;
}

// y (batch x n_out, host) = mlp(x (batch x n_in, host))
int fwt_mlp_forward(fwt_mlp *m, const float *x, int batch, float *y)
{
    if (!m || !x || !y || batch < 1 || batch > m->bmax) return fail(FWT_E_ARG, "mlp: batch outside 1..batch_max");
    cudaSetDevice(m->dev);
    FWT_TRY(mlp_upload(m, x, nullptr, nullptr, batch));
    FWT_TRY(mlp_forward(m, batch, false));
    const size_t nx = m->t_at(batch), ny = (size_t)batch * m->n_out;
    if (sizeof(float) * (nx + ny) > kIoOnce) {
        FWT_CUDA(cudaMemcpyAsync(y, m->t(batch), sizeof(float) * ny, cudaMemcpyDeviceToHost, m->st));
        return mlp_download(m, 0);
    }
    FWT_TRY(mlp_download(m, nx + ny));
    std::memcpy(y, m->hio + kIoHead + sizeof(float) * nx, sizeof(float) * ny);
    return 0;
}

// loss and its gradients: grad_params (nparams, layout of fwt_mlp_get_params) and grad_x
// (batch x n_in); either may be NULL.  w_out: n_out output weights or NULL (all 1).
int fwt_mlp_loss_grad(fwt_mlp *m, const float *x, const float *t, const float *w_out, int batch, double *loss,
                      float *grad_params, float *grad_x)
{
    if (!m || !x || !t || batch < 1 || batch > m->bmax) return fail(FWT_E_ARG, "mlp: batch outside 1..batch_max");
    cudaSetDevice(m->dev);
    FWT_TRY(mlp_upload(m, x, t, w_out, batch));
    FWT_TRY(mlp_forward(m, batch, true));
    FWT_TRY(mlp_backward(m, batch, grad_params != nullptr, grad_x != nullptr));
    if (grad_params) {
        float *h = grad_params;
        for (auto &l : m->L) {
            FWT_CUDA(cudaMemcpyAsync(h, l.gW, sizeof(float) * l.N * l.K, cudaMemcpyDeviceToHost, m->st));
            h += (size_t)l.N * l.K;
            FWT_CUDA(cudaMemcpyAsync(h, l.gb, sizeof(float) * l.N, cudaMemcpyDeviceToHost, m->st));
            h += l.N;
        }
    }
    const size_t nx = grad_x ? (size_t)batch * m->n_in : 0;
    FWT_TRY(mlp_download(m, nx));
    if (loss) std::memcpy(loss, m->hio, sizeof(double));
    if (grad_x) std::memcpy(grad_x, m->hio + kIoHead, sizeof(float) * nx);
    return 0;
}

// one Adam step (beta1 0.9, beta2 0.999, eps 1e-8) on the weighted MSE of a batch
int fwt_mlp_train_step(fwt_mlp *m, const float *x, const float *t, const float *w_out, int batch, float lr,
                       double *loss)
{
    if (!m || !x || !t || batch < 1 || batch > m->bmax) return fail(FWT_E_ARG, "mlp: batch outside 1..batch_max");
    cudaSetDevice(m->dev);
    FWT_TRY(mlp_upload(m, x, t, w_out, batch));
    FWT_TRY(mlp_forward(m, batch, true));
    FWT_TRY(mlp_backward(m, batch, true, false));
    const int64_t step = m->step + 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - (float)std::pow(0.9, (double)step), c2 = 1.0f - (float)std::pow(0.999, (double)step);
    for (size_t o = 0; o < m->L.size(); o += kMlpJobs) {
        const int c = (int)std::min<size_t>(kMlpJobs, m->L.size() - o);
        MlpParams P;
        mlp_param_list(m, o, c, P);
        int64_t n = 0;
        for (int i = 0; i < c; ++i) n = std::max<int64_t>(n, (int64_t)P.l[i].N * P.l[i].K + P.l[i].N);
        FWT_TRY(mlp_launch(m, mlp_adam, dim3(nblk(n), (unsigned)c), 256, 0, P, lr, b1, b2, c1, c2, 1e-8f,
                           (const int *)m->err()));
    }
    FWT_TRY(mlp_download(m, 0));   // a step that timed out left the weights as they were
    m->step = step;
    if (loss) std::memcpy(loss, m->hio, sizeof(double));
    return 0;
}

}  // extern "C"
