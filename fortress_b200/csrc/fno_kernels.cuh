// fno_kernels.cuh -- kernels of the learned initial guess (Fourier neural
// operator): a batched strided GEMM with FP32 accumulation (the weight
// operand may be stored in BF16), bias + GELU, their backward passes, channel
// sums, the MSE loss and Adam with BF16 weight copies.  Every dense piece of
// the network (pointwise channel mixing, the truncated DFT onto the retained
// modes, the per-mode channel mixing) is expressed as this GEMM.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fno {

__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ float ldf(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// C[b](i,j) = alpha * sum_k A[b](i,k) B[b](k,j) + beta * C[b](i,j)
// element (i,k) of A[b] at A + b*sAb + i*sAi + k*sAk, likewise B and C.
// 64x64 output tile per block, 16-wide K slices, 256 threads x (4x4).
template <typename TA>
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, float alpha, const TA* __restrict__ A,
                                              long long sAb, long long sAi, long long sAk, const float* __restrict__ B,
                                              long long sBb, long long sBk, long long sBj, float beta, float* C,
                                              long long sCb, long long sCi, long long sCj) {
    __shared__ float As[16][68];
    __shared__ float Bs[16][68];
    const long long b = blockIdx.z;
    const int i0 = blockIdx.y * 64, j0 = blockIdx.x * 64;
    A += b * sAb;
    B += b * sBb;
    C += b * sCb;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r][q] = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int e = threadIdx.x; e < 1024; e += 256) {
            // A tile: 64 rows x 16 k; choose the walk that keeps the
            // contiguous index fastest across threads
            int ii, kk;
            if (sAk == 1) { kk = e % 16; ii = e / 16; } else { ii = e % 64; kk = e / 64; }
            const int i = i0 + ii, k = k0 + kk;
            As[kk][ii] = (i < M && k < K) ? ldf(A + i * sAi + k * sAk) : 0.f;
            int jj, kb;
            if (sBj == 1) { jj = e % 64; kb = e / 64; } else { kb = e % 16; jj = e / 16; }
            const int j = j0 + jj, kq = k0 + kb;
            Bs[kb][jj] = (j < N && kq < K) ? B[kq * sBk + j * sBj] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            float a[4], bb[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r] = As[kk][ty * 4 + r];
#pragma unroll
            for (int q = 0; q < 4; ++q) bb[q] = Bs[kk][tx * 4 + q];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[r][q] = fmaf(a[r], bb[q], acc[r][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = i0 + ty * 4 + r, j = j0 + tx * 4 + q;
            if (i < M && j < N) {
                float* c = C + i * sCi + j * sCj;
                *c = beta == 0.f ? alpha * acc[r][q] : alpha * acc[r][q] + beta * *c;
            }
        }
}

__device__ __forceinline__ float gelu_f(float x) {
    const float c = 0.7978845608028654f;  // sqrt(2/pi)
    return 0.5f * x * (1.f + tanhf(c * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float gelu_g(float x) {
    const float c = 0.7978845608028654f;
    const float u = c * (x + 0.044715f * x * x * x);
    const float t = tanhf(u);
    return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * c * (1.f + 3.f * 0.044715f * x * x);
}

// z[b,c,s] += bias[c]; h = act(z) (act 1: GELU, 0: identity).  vec: four
// values per access (16-byte aligned rows, S a multiple of 4).
__global__ void k_bias_act(float* z, float* h, const float* bias, long long C, long long S, long long n, int act, int vec) {
    const long long step = (long long)gridDim.x * blockDim.x, t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (vec) {
        for (long long t = t0; t < n / 4; t += step) {
            const float b = bias ? bias[(4 * t / S) % C] : 0.f;
            float4 v = ((const float4*)z)[t];
            v.x += b; v.y += b; v.z += b; v.w += b;
            ((float4*)z)[t] = v;
            if (h) {
                if (act) v = make_float4(gelu_f(v.x), gelu_f(v.y), gelu_f(v.z), gelu_f(v.w));
                ((float4*)h)[t] = v;
            }
        }
        return;
    }
    for (long long t = t0; t < n; t += step) {
        const long long c = (t / S) % C;
        const float v = z[t] + (bias ? bias[c] : 0.f);
        z[t] = v;
        if (h) h[t] = act ? gelu_f(v) : v;
    }
}

__global__ void k_act_bwd(float* dz, const float* dh, const float* z, long long n, int vec) {
    const long long step = (long long)gridDim.x * blockDim.x, t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (vec) {
        for (long long t = t0; t < n / 4; t += step) {
            const float4 d = ((const float4*)dh)[t], v = ((const float4*)z)[t];
            ((float4*)dz)[t] = make_float4(d.x * gelu_g(v.x), d.y * gelu_g(v.y), d.z * gelu_g(v.z), d.w * gelu_g(v.w));
        }
        return;
    }
    for (long long t = t0; t < n; t += step) dz[t] = dh[t] * gelu_g(z[t]);
}

// out[c] = beta*out[c] + sum_{b,s} x[b,c,s] in a fixed order, in FP64.
//
// S == 1 (the per-chunk weight-gradient partials): 32 channels per block,
// eight threads each walk every eighth b with reads coalesced across channels
// (1024 weights x 128 chunks: one thread per weight took 15 us, most of it one
// load after the other).
__global__ void __launch_bounds__(256) k_channel_sum_rows(float* out, const float* x, long long B, long long C, float beta) {
    __shared__ double red[8][33];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const long long c = (long long)blockIdx.x * 32 + lane;
    double acc = 0.0;
    if (c < C) {
#pragma unroll 4
        for (long long b = g; b < B; b += 8) acc += x[b * C + c];
    }
    red[g][lane] = acc;
    __syncthreads();
    if (g == 0 && c < C) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) s += red[q][lane];
        out[c] = beta * out[c] + (float)s;
    }
}

// Otherwise one cluster of eight blocks per channel, an eighth of s each: a
// layer has 32 channels, and one block per channel left most of the GPU idle
// (32 channels of 2^18 points: 33 -> 9 us).
constexpr int kSumBlocks = 8;
__global__ void __cluster_dims__(kSumBlocks, 1, 1) __launch_bounds__(256)
k_channel_sum(float* out, const float* x, long long B, long long C, long long S, float beta) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const long long c = blockIdx.x / kSumBlocks;
    const long long per = ((S + kSumBlocks - 1) / kSumBlocks + 3) / 4 * 4;
    const long long s0 = per * rank < S ? per * rank : S, s1 = s0 + per < S ? s0 + per : S;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    for (long long b = 0; b < B; ++b) {
        const float* row = x + (b * C + c) * S;
        if (((uintptr_t)row & 15) == 0) {          // s0 is a multiple of 4
            const long long v1 = s0 + (s1 - s0) / 4 * 4;
#pragma unroll 4
            for (long long s = s0 + 4 * threadIdx.x; s < v1; s += 1024) {
                const float4 v = *(const float4*)(row + s);
                a[0] += v.x; a[1] += v.y; a[2] += v.z; a[3] += v.w;
            }
            for (long long s = v1 + threadIdx.x; s < s1; s += 256) a[0] += row[s];
        } else {
#pragma unroll 4
            for (long long s = s0 + threadIdx.x; s < s1; s += 256) a[0] += row[s];
        }
    }
    __shared__ double red[256];
    red[threadIdx.x] = (a[0] + a[1]) + (a[2] + a[3]);
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    cl.sync();
    if (rank == 0 && threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < kSumBlocks; ++q) s += *cl.map_shared_rank(red, q);
        out[c] = beta * out[c] + (float)s;
    }
    cl.sync();          // no block leaves while its sum is read
}

__global__ void k_axpy(float* y, const float* x, float a, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        y[t] += a * x[t];
}

// per-block partial sums of (out-target)^2; dout = 2 (out-target)/n
__global__ void k_mse(const float* out, const float* tgt, float* dout, double* part, long long n) {
    double acc = 0.0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const float d = out[t] - tgt[t];
        acc += (double)d * d;
        if (dout) dout[t] = 2.f * d / (float)n;
    }
    __shared__ double red[256];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_sum_parts(const double* part, int n, double scale, double* out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < n; ++i) s += part[i];
        *out = s * scale;
    }
}

// Adam on the FP32 master weights; wb receives the BF16 copy the GEMMs read.
__global__ void k_adam(float* w, __nv_bfloat16* wb, const float* g, float* m, float* v, long long n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const float gg = g[t];
        const float mm = b1 * m[t] + (1.f - b1) * gg;
        const float vv = b2 * v[t] + (1.f - b2) * gg * gg;
        m[t] = mm;
        v[t] = vv;
        const float upd = lr * (mm / c1) / (sqrtf(vv / c2) + eps);
        w[t] -= upd;
        if (wb) wb[t] = __float2bfloat16(w[t]);
    }
}

__global__ void k_to_bf16(const float* x, __nv_bfloat16* y, long long n) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        y[t] = __float2bfloat16(x[t]);
}

// Real block form of the per-mode complex channel mixing G = R H:
//   Rbig[mode] = [[Rr, -Ri], [Ri, Rr]]   (2O x 2C), R stored [mode][O][C]
__global__ void k_rbig_build(const float* rr, const float* ri, __nv_bfloat16* rb, long long nmodes, int O, int C) {
    const long long n = nmodes * 4LL * O * C;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const long long mode = t / (4LL * O * C);
        const int e = (int)(t % (4LL * O * C));
        const int row = e / (2 * C), col = e % (2 * C);
        const int po = row / O, o = row % O, pc = col / C, c = col % C;
        const long long src = (mode * O + o) * C + c;
        float v;
        if (po == pc) v = rr[src];
        else v = (po == 0) ? -ri[src] : ri[src];
        rb[t] = __float2bfloat16(v);
    }
}

// Gradient of the block form folded back: dRr = d00 + d11, dRi = d10 - d01.
__global__ void k_rbig_fold(const float* drb, float* drr, float* dri, long long nmodes, int O, int C) {
    const long long n = nmodes * (long long)O * C;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const long long mode = t / ((long long)O * C);
        const int o = (int)((t / C) % O), c = (int)(t % C);
        const float* d = drb + mode * 4LL * O * C;
        const float d00 = d[(long long)o * 2 * C + c], d01 = d[(long long)o * 2 * C + C + c];
        const float d10 = d[(long long)(O + o) * 2 * C + c], d11 = d[(long long)(O + o) * 2 * C + C + c];
        drr[t] = d00 + d11;
        dri[t] = d10 - d01;
    }
}

// ------------------------------------------------- tensor-core dense layer
// z[m][n] = sum_k W(m,k) x[k][n] + bias[m],  h = GELU(z) or z,  for the
// pointwise channel mixes (M, K <= 128 channels, n over all B*N*N points).
// W(m,k) = W[m*K+k] (or W[k*M+m] when transposed), BF16; x is FP32 and is
// rounded to BF16 on its way into shared memory; accumulation is FP32 in
// tensor memory.  The points are the tile's rows and the M output channels its
// columns: a layer has 6 to 128 channels and 10^5 points, so every row of the
// 128-row accumulator is a point, and a warp stores 32 adjacent points of
// one channel at a time.  A CTA (4 warps) is persistent over tiles of 128
// points; W and the tensor memory are set up once:
//   - all threads stage the x tile (point-major 8x8 core matrices, no swizzle);
//   - thread 0 issues one tcgen05.mma (kind::f16, M = 128, N = channels, K =
//     16) per 16 channels and commits to an mbarrier;
//   - each thread reads its point's accumulators with tcgen05.ld, adds the
//     bias, applies GELU and stores.
// Bound by reading x and writing z and h; several CTAs per SM overlap each
// other's phases.  32 -> 32 channels of 2^18 points: 35 -> 20 us (3.4 TB/s) against
// one CTA per 128 columns with the channels as rows, three quarters of which
// were padding.
// The mbarrier wait is bounded; on expiry the CTA sets *err, stores nothing
// more and frees its tensor memory.
namespace tc {
constexpr int TP = 128;      // points per tile (accumulator rows)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (no swizzle): start, leading and stride
// byte offsets in 16-byte units, version 1 at bits 46-47.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor: F32 accumulator, BF16 A and B, A point-major (bit
// 15), B K-major, N = np, M = TP.
__device__ __forceinline__ uint32_t idesc_bf16(int np) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)(np >> 3) << 17) | ((uint32_t)(TP >> 4) << 24);
}
// channels of a layer in tensor memory: accumulator columns, allocated columns
__host__ __device__ __forceinline__ int dense_np(int M) { return (M + 15) / 16 * 16; }
__host__ __device__ __forceinline__ int dense_cols(int M) { const int np = dense_np(M); return np <= 32 ? 32 : np <= 64 ? 64 : 128; }
__host__ __device__ __forceinline__ size_t dense_smem(int M, int K) {
    const int KP = (K + 15) / 16 * 16;
    return 1024 + (size_t)KP * TP * 2 + (size_t)KP * dense_np(M) * 2;
}
}  // namespace tc

__global__ void __launch_bounds__(128)
k_dense_tc(const __nv_bfloat16* __restrict__ W, int transw, const float* __restrict__ x, const float* __restrict__ bias,
           float* __restrict__ z, float* __restrict__ h, int M, int K, long long BS, int act, int* err) {
    using namespace tc;
    extern __shared__ __align__(1024) unsigned char smraw[];
    const int KP = (K + 15) / 16 * 16, NP = dense_np(M), cols = dense_cols(M);
    // 1024-byte aligned operand tiles
    const uint32_t base = smem_u32(smraw);
    const uint32_t pad = (1024u - (base & 1023u)) & 1023u;
    unsigned char* sA = smraw + pad;                          // KP x TP bf16, point-major cores
    unsigned char* sB = sA + (size_t)KP * TP * 2;             // NP x KP bf16, K-major cores
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ uint32_t tmem_slot;
    __shared__ float sbias[128];
    const int tid = threadIdx.x, warp = tid >> 5;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar)), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    sbias[tid] = (bias && tid < M) ? bias[tid] : 0.f;
    // W: element (m, k) -> core (k/8, m/8), row m%8, column k%8
    for (int e = tid; e < NP * KP; e += 128) {
        const int m = e / KP, k = e - (e / KP) * KP;
        __nv_bfloat16 v = __float2bfloat16(0.f);
        if (m < M && k < K) v = transw ? W[(size_t)k * M + m] : W[(size_t)m * K + k];
        const int off = (((k >> 3) * (NP / 8) + (m >> 3)) << 7) + ((m & 7) << 4) + ((k & 7) << 1);
        *(__nv_bfloat16*)(sB + off) = v;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const bool rows16 = (BS & 3) == 0 && ((uintptr_t)x & 15) == 0;
    const long long ntiles = (BS + TP - 1) / TP;
    uint32_t phase = 0;
    bool ok = true;
    for (long long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const long long n0 = tile * TP;
        // x: eight consecutive points of one k -> 16 bytes of core (k/8, p/8), row k%8
#pragma unroll 4
        for (int e = tid; e < KP * (TP / 8); e += 128) {
            const int k = e / (TP / 8), g = e % (TP / 8);
            const long long n = n0 + g * 8;
            float f[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = 0.f;
            if (k < K) {
                const float* src = x + (size_t)k * BS + n;
                if (rows16 && n + 8 <= BS) {
                    const float4 a = *(const float4*)src, b = *(const float4*)(src + 4);
                    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) f[j] = (n + j < BS) ? src[j] : 0.f;
                }
            }
            __nv_bfloat162 p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
            *(uint4*)(sA + ((((k >> 3) * (TP / 8) + g) << 7) + ((k & 7) << 4))) = *(uint4*)p;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (tid == 0) {
            const uint32_t idesc = idesc_bf16(NP);
            for (int s = 0; s < KP / 16; ++s) {
                // point-major A: k groups TP/8 cores apart, 8-point groups 128 B apart
                const uint64_t da = sdesc(smem_u32(sA) + s * 2 * (TP / 8) * 128, (TP / 8) * 128, 128);
                // K-major B: k groups NP/8 cores apart, 8-channel groups 128 B apart
                const uint64_t db = sdesc(smem_u32(sB) + s * 2 * (NP / 8) * 128, (NP / 8) * 128, 128);
                const uint32_t acc = s > 0 ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                smem_u32(&mbar)));
        }
        // bounded wait for the accumulator
        uint32_t done = 0;
        for (long long it = 0; it < (1LL << 22) && !done; ++it) {
            asm volatile(
                "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                "selp.b32 %0, 1, 0, P1;\n\t}\n"
                : "=r"(done)
                : "r"(smem_u32(&mbar)), "r"(phase));
        }
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        ok = __syncthreads_and((int)done) != 0;
        if (!ok) break;
        const long long n = n0 + tid;            // this thread's point
        for (int cb = 0; cb < NP; cb += 16) {
            uint32_t r[16];
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)cb;
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (n < BS) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (cb + j < M) {
                        const float v = __uint_as_float(r[j]) + sbias[cb + j];
                        const size_t at = (size_t)(cb + j) * BS + n;
                        if (z) z[at] = v;
                        if (h) h[at] = act ? gelu_f(v) : v;
                    }
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (!ok && tid == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

}  // namespace fno
