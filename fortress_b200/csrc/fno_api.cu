// fno_api.cu -- C ABI of the learned guess's kernels (include/fno.h).
#include <math.h>

#include <algorithm>
#include <string>

#include "../../include/fgpe.h"
#include "../../include/fno.h"
#include "fgpe_error.h"
#include "fno_gemm_tc.cuh"
#include "fno_kernels.cuh"

extern "C" {

static int fno_ck(cudaError_t e) {
    if (e != cudaSuccess) { fgpe::set_last_error(cudaGetErrorString(e)); return FGPE_E_CUDA; }
    return FGPE_OK;
}
static unsigned fno_grid(long long n) { long long g = (n + 255) / 256; return (unsigned)std::min<long long>(g, 148LL * 32); }

int fno_gemm(int batch, int M, int N, int K, float alpha, const void* A, int a_bf16, long long sAb, long long sAi,
             long long sAk, const float* B, long long sBb, long long sBk, long long sBj, float beta, float* C,
             long long sCb, long long sCi, long long sCj, void* stream) {
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return FGPE_E_ARG;
    if (batch > 65535) return FGPE_E_ARG;
    dim3 grid((N + 63) / 64, (M + 63) / 64, batch);
    cudaStream_t st = (cudaStream_t)stream;
    if (a_bf16)
        fno::k_gemm<__nv_bfloat16><<<grid, 256, 0, st>>>(M, N, K, alpha, (const __nv_bfloat16*)A, sAb, sAi, sAk, B, sBb,
                                                         sBk, sBj, beta, C, sCb, sCi, sCj);
    else
        fno::k_gemm<float><<<grid, 256, 0, st>>>(M, N, K, alpha, (const float*)A, sAb, sAi, sAk, B, sBb, sBk, sBj, beta, C,
                                                 sCb, sCi, sCj);
    return fno_ck(cudaGetLastError());
}

}  // extern "C"

// Tensor-core variant of fno_gemm (fno_gemm_tc.cuh).  When A is shared by
// every batch entry and B is not, the product is taken transposed (C^T =
// B^T A^T) so that the shared operand becomes B and the entries fold into one
// tall GEMM; the tile width GN is the smallest of 16..256 that covers N.
// CTAs per SM: as many as the shared memory (about 227 KB) and the 512 TMEM
// columns hold, at most four; CTAs beyond those resident wait their turn.
template <int GN, int PAIR> constexpr int gemm_tc_per_sm() {
    const int by_smem = (int)((227 * 1024) / (fno::gtc::smem_bytes<GN, PAIR>() + 3 * 1024));
    const int by_tmem = 512 / fno::gtc::tmem_cols<GN, PAIR>();
    return std::min(4, std::min(by_smem, by_tmem));
}

template <typename TA, int GN, int PAIR> static int gemm_tc_launch(const fno::GemmTc& g, cudaStream_t st) {
    static bool attr_set[64] = {false};
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return FGPE_E_ARG;
    const size_t smem = fno::gtc::smem_bytes<GN, PAIR>();
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(fno::k_gemm_tc<TA, GN, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fno_ck(e);
        attr_set[dev] = true;
    }
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long rows = g.fold ? (long long)g.batch * g.M : (long long)g.M;
    const long long tiles = (rows + fno::gtc::TM - 1) / fno::gtc::TM * ((g.N + GN - 1) / GN) * (g.fold ? 1 : g.batch);
    const long long grid = std::min<long long>(tiles, (long long)gemm_tc_per_sm<GN, PAIR>() * nsm);
    fno::k_gemm_tc<TA, GN, PAIR><<<(unsigned)grid, 128, smem, st>>>(g);
    return fno_ck(cudaGetLastError());
}

template <typename TA> static int gemm_tc_width(const fno::GemmTc& g, cudaStream_t st) {
    if (g.N <= 16) return gemm_tc_launch<TA, 16, fno::PAIR_NONE>(g, st);
    if (g.N <= 32) return gemm_tc_launch<TA, 32, fno::PAIR_NONE>(g, st);
    if (g.N <= 64) return gemm_tc_launch<TA, 64, fno::PAIR_NONE>(g, st);
    if (g.N <= 128) return gemm_tc_launch<TA, 128, fno::PAIR_NONE>(g, st);
    return gemm_tc_launch<TA, 256, fno::PAIR_NONE>(g, st);
}
// Pairs take tiles of up to 64 columns (two accumulators, 128 of the 512
// tensor-memory columns, so that four CTAs fit an SM).
template <int PAIR> static int gemm_tc_pair_width(const fno::GemmTc& g, cudaStream_t st) {
    if (g.N <= 16) return gemm_tc_launch<float, 16, PAIR>(g, st);
    if (g.N <= 32) return gemm_tc_launch<float, 32, PAIR>(g, st);
    return gemm_tc_launch<float, 64, PAIR>(g, st);
}

// Checks, the transposed form for a shared left operand, and the float4
// forms, for one product (A1 = B1 = C1 = null) or a pair.
static int gemm_tc_args(int batch, int M, int N, int K, float alpha, const void* A, const void* A1, int a_bf16, long long sAb,
                        long long sAi, long long sAk, const float* B, const float* B1, long long sBb, long long sBk,
                        long long sBj, float beta, float* C, float* C1, long long sCb, long long sCi, long long sCj,
                        int* err_dev, fno::GemmTc* out) {
    if (!A || !B || !C || !err_dev) { fgpe::set_last_error("null argument"); return FGPE_E_ARG; }
    if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) { fgpe::set_last_error("empty GEMM"); return FGPE_E_ARG; }
    if (sAb < 0 || sAi < 0 || sAk < 0 || sBb < 0 || sBk < 0 || sBj < 0 || sCb < 0 || sCi < 0 || sCj < 0) {
        fgpe::set_last_error("negative stride");
        return FGPE_E_ARG;
    }
    fno::GemmTc g{M, N, K, batch, 0, alpha, beta, A, sAb, sAi, sAk, B, sBb, sBk, sBj, C, sCb, sCi, sCj, err_dev, 0, 0, 0,
                  A1, B1, C1, nullptr, nullptr, 1, 1, 0};
    if (batch > 1 && sAb == 0 && sBb != 0 && !a_bf16) {
        // C^T = B^T A^T: the shared A becomes the B operand
        g = fno::GemmTc{N, M, K, batch, 0, alpha, beta, B, sBb, sBj, sBk, (const float*)A, 0, sAk, sAi,
                        C, sCb, sCj, sCi, err_dev, 0, 0, 0, B1, (const float*)A1, C1, nullptr, nullptr, 1, 1, 0};
    }
    g.fold = batch > 1 && g.sBb == 0;
    // float4 operand reads where the unit-stride runs start on 16-byte boundaries
    const bool a16 = (((uintptr_t)g.A | (uintptr_t)g.A1) & 15) == 0, b16 = (((uintptr_t)g.B | (uintptr_t)g.B1) & 15) == 0;
    g.avec = !a_bf16 && a16 && g.sAk == 1 && g.sAi % 4 == 0 && g.sAb % 4 == 0;
    if (b16 && g.sBb % 4 == 0) {
        if (g.sBj == 1 && g.sBk % 4 == 0) g.bvec = 1;
        else if (g.sBk == 1 && g.sBj % 4 == 0) g.bvec = 2;
    }
    g.cvec = (((uintptr_t)g.C | (uintptr_t)g.C1) & 15) == 0 && g.sCj == 1 && g.sCi % 4 == 0 && g.sCb % 4 == 0;
    *out = g;
    return FGPE_OK;
}

extern "C" {

int fno_gemm_tc(int batch, int M, int N, int K, float alpha, const void* A, int a_bf16, long long sAb, long long sAi,
                long long sAk, const float* B, long long sBb, long long sBk, long long sBj, float beta, float* C,
                long long sCb, long long sCi, long long sCj, int* err_dev, void* stream) {
    fno::GemmTc g;
    const int rc = gemm_tc_args(batch, M, N, K, alpha, A, nullptr, a_bf16, sAb, sAi, sAk, B, nullptr, sBb, sBk, sBj, beta, C,
                                nullptr, sCb, sCi, sCj, err_dev, &g);
    if (rc) return rc;
    const cudaStream_t st = (cudaStream_t)stream;
    return a_bf16 ? gemm_tc_width<__nv_bfloat16>(g, st) : gemm_tc_width<float>(g, st);
}

int fno_gemm_tc2(int batch, int M, int N, int K, float alpha, const float* A0, const float* A1, long long sAb, long long sAi,
                 long long sAk, const float* B0, const float* B1, long long sBb, long long sBk, long long sBj, float beta,
                 float* C0, float* C1, long long sCb, long long sCi, long long sCj, int* err_dev, void* stream) {
    if (!A1 || !B1 || !C1) { fgpe::set_last_error("null argument"); return FGPE_E_ARG; }
    fno::GemmTc g;
    const int rc = gemm_tc_args(batch, M, N, K, alpha, A0, A1, 0, sAb, sAi, sAk, B0, B1, sBb, sBk, sBj, beta, C0, C1, sCb, sCi,
                                sCj, err_dev, &g);
    if (rc) return rc;
    const cudaStream_t st = (cudaStream_t)stream;
    if (C0 == C1) return gemm_tc_pair_width<fno::PAIR_SUM>(g, st);
    if (g.A == g.A1) return gemm_tc_pair_width<fno::PAIR_SPLIT>(g, st);
    // a shared B that is the batched operand of a batch of one: not folded, so
    // one launch a product
    if (batch == 1 && sAb == 0 && sBb != 0 && B0 == B1) {
        const int rc0 = fno_gemm_tc(batch, M, N, K, alpha, A0, 0, sAb, sAi, sAk, B0, sBb, sBk, sBj, beta, C0, sCb, sCi, sCj,
                                    err_dev, stream);
        return rc0 ? rc0 : fno_gemm_tc(batch, M, N, K, alpha, A1, 0, sAb, sAi, sAk, B1, sBb, sBk, sBj, beta, C1, sCb, sCi, sCj,
                                       err_dev, stream);
    }
    fgpe::set_last_error("a pair of products shares its output, or its batched operand");
    return FGPE_E_ARG;
}
int fno_gemm_tc2_act(int batch, int M, int N, int K, float alpha, const float* A0, const float* A1, long long sAb, long long sAi,
                     long long sAk, const float* B0, const float* B1, long long sBb, long long sBk, long long sBj, float beta,
                     float* C, long long sCb, long long sCi, long long sCj, const float* bias, long long nch, long long S,
                     int act, float* H, int* err_dev, void* stream) {
    if (!A1 || !B1 || !H) { fgpe::set_last_error("null argument"); return FGPE_E_ARG; }
    if (nch <= 0 || S <= 0) { fgpe::set_last_error("empty channels"); return FGPE_E_ARG; }
    fno::GemmTc g;
    const int rc = gemm_tc_args(batch, M, N, K, alpha, A0, A1, 0, sAb, sAi, sAk, B0, B1, sBb, sBk, sBj, beta, C, C, sCb, sCi,
                                sCj, err_dev, &g);
    if (rc) return rc;
    g.bias = bias; g.H = H; g.nch = nch; g.S = S; g.act = act;
    g.cvec = g.cvec && ((uintptr_t)H & 15) == 0;
    return gemm_tc_pair_width<fno::PAIR_SUM>(g, (cudaStream_t)stream);
}

int fno_bias_act(float* z, float* h, const float* bias, long long C, long long S, long long n, int act, void* stream) {
    const int vec = S % 4 == 0 && n % 4 == 0 && (((uintptr_t)z | (uintptr_t)h) & 15) == 0;
    fno::k_bias_act<<<fno_grid(vec ? n / 4 : n), 256, 0, (cudaStream_t)stream>>>(z, h, bias, C, S, n, act, vec);
    return fno_ck(cudaGetLastError());
}

int fno_act_bwd(float* dz, const float* dh, const float* z, long long n, void* stream) {
    const int vec = n % 4 == 0 && (((uintptr_t)dz | (uintptr_t)dh | (uintptr_t)z) & 15) == 0;
    fno::k_act_bwd<<<fno_grid(vec ? n / 4 : n), 256, 0, (cudaStream_t)stream>>>(dz, dh, z, n, vec);
    return fno_ck(cudaGetLastError());
}

int fno_channel_sum(float* out, const float* x, long long B, long long C, long long S, float beta, void* stream) {
    if (S == 1)
        fno::k_channel_sum_rows<<<(unsigned)((C + 31) / 32), 256, 0, (cudaStream_t)stream>>>(out, x, B, C, beta);
    else
        fno::k_channel_sum<<<(unsigned)C * fno::kSumBlocks, 256, 0, (cudaStream_t)stream>>>(out, x, B, C, S, beta);
    return fno_ck(cudaGetLastError());
}

int fno_axpy(float* y, const float* x, float a, long long n, void* stream) {
    fno::k_axpy<<<fno_grid(n), 256, 0, (cudaStream_t)stream>>>(y, x, a, n);
    return fno_ck(cudaGetLastError());
}

int fno_mse(const float* out, const float* target, float* dout, double* loss_dev, double* scratch, long long n,
            void* stream) {
    fno::k_mse<<<256, 256, 0, (cudaStream_t)stream>>>(out, target, dout, scratch, n);
    fno::k_sum_parts<<<1, 32, 0, (cudaStream_t)stream>>>(scratch, 256, 1.0 / (double)n, loss_dev);
    return fno_ck(cudaGetLastError());
}

int fno_adam(float* w, void* w_bf16, const float* g, float* m, float* v, long long n, float lr, float beta1,
             float beta2, float eps, int t, void* stream) {
    const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
    fno::k_adam<<<fno_grid(n), 256, 0, (cudaStream_t)stream>>>(w, (__nv_bfloat16*)w_bf16, g, m, v, n, lr, beta1, beta2,
                                                              eps, c1, c2);
    return fno_ck(cudaGetLastError());
}

int fno_to_bf16(const float* x, void* y, long long n, void* stream) {
    fno::k_to_bf16<<<fno_grid(n), 256, 0, (cudaStream_t)stream>>>(x, (__nv_bfloat16*)y, n);
    return fno_ck(cudaGetLastError());
}

int fno_dense_tc(const void* w_bf16, int transpose_w, const float* x, const float* bias, float* z, float* h, int M,
                 int K, long long n, int act, int* err_dev, void* stream) {
    if (!w_bf16 || !x || !err_dev || (!z && !h)) { fgpe::set_last_error("null argument"); return FGPE_E_ARG; }
    if (M < 1 || M > 128 || K < 1 || K > 128 || n < 1) {
        fgpe::set_last_error("dense layer needs 1 <= M <= 128 output and 1 <= K <= 128 input channels");
        return FGPE_E_ARG;
    }
    const size_t smem = fno::tc::dense_smem(M, K);
    static bool attr_set[64] = {false};
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(fno::k_dense_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)fno::tc::dense_smem(128, 128));
        if (e != cudaSuccess) return fno_ck(e);
        attr_set[dev] = true;
    }
    // CTAs per SM: the tensor memory's 512 columns, shared memory, eight at most
    const int fit = (int)std::min<size_t>(std::min(8, 512 / fno::tc::dense_cols(M)), (220 * 1024) / (smem + 2048));
    const long long tiles = (n + fno::tc::TP - 1) / fno::tc::TP;
    const unsigned grid = (unsigned)std::min<long long>(tiles, (long long)nsm * fit);
    fno::k_dense_tc<<<grid, 128, smem, (cudaStream_t)stream>>>(
        (const __nv_bfloat16*)w_bf16, transpose_w, x, bias, z, h, M, K, n, act, err_dev);
    return fno_ck(cudaGetLastError());
}

int fno_rbig_build(const float* rr, const float* ri, void* rbig, long long nmodes, int O, int C, void* stream) {
    if (nmodes <= 0 || O <= 0 || C <= 0) return FGPE_E_ARG;
    fno::k_rbig_build<<<fno_grid(nmodes * 4LL * O * C), 256, 0, (cudaStream_t)stream>>>(rr, ri, (__nv_bfloat16*)rbig,
                                                                                        nmodes, O, C);
    return fno_ck(cudaGetLastError());
}

int fno_rbig_fold(const float* drbig, float* drr, float* dri, long long nmodes, int O, int C, void* stream) {
    if (nmodes <= 0 || O <= 0 || C <= 0) return FGPE_E_ARG;
    fno::k_rbig_fold<<<fno_grid(nmodes * (long long)O * C), 256, 0, (cudaStream_t)stream>>>(drbig, drr, dri, nmodes, O, C);
    return fno_ck(cudaGetLastError());
}

}  // extern "C"
