// Learned form (MG_FORM_MLP), training side: a 4 -> 64 -> 64 -> 64 -> 6
// network (activation silu_p, mg_mlp_common.cuh) learns the correction that
// the DMD Gauss-Hermite smearing (ff_dmd_I.cpp:178-259) adds to the unsmeared
// spline values of phi, rho and their r / alpha derivatives.  Inputs (r, w_i,
// w_j, species pair) with w = alpha^-1/2; outputs (phi, rho, dphi/dr,
// drho/dr, dphi/dalpha, drho/dalpha) of the pair exponent
// alpha = alpha_i alpha_j / (alpha_i + alpha_j), minus their unsmeared values.
//
// Everything runs in this library's own kernels:
//   * k_mlp_labels  -- training samples drawn from a counter-based hash RNG,
//     labelled by the FP64 quadrature of the loaded tables minus the FP64
//     unsmeared spline values;
//   * k_mlp_train   -- one 64-row tile per CTA: forward and backward with
//     BF16 tensor-core MMAs (mma.sync m16n8k16, FP32 accumulation), weight
//     gradients written as per-CTA partials;
//   * k_mlp_adam    -- sums the partials, Adam with a cosine learning rate,
//     refreshes the BF16 weight copy.
// Deployment inside force_calc is mg_mlp_tc.cu (tcgen05 tensor cores, TMEM
// accumulators).
// Species pairs: code 0 = (0,0), 1 = the unordered cross pair, 2 = (1,1); the
// cross code uses one network for (0,1) and (1,0), which needs rho_AB =
// rho_BA (true for the potentials this form is trained on).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_bf16.h>

#include "mg_reduce.cuh"
#include "mg_launch.cuh"
#include "mg_dmd_common.cuh"
#include "mg_mlp_common.cuh"

namespace mg {
namespace {

using namespace mlp;

constexpr int kRows = 64;       // rows per tile
constexpr int kMlpThreads = 128;

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Warp-tiled product out(m, n) = sum_k A(m, k) B(k, n) over M x N x K (multiples
// of 16, 8, 16).  A and B are accessors returning bf16; out receives FP32.
// The warps of the CTA split the 16x8 output tiles.
template <int M, int N, int K, class FA, class FB, class FO>
__device__ __forceinline__ void cta_gemm(const FA& A, const FB& B, const FO& out)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nwarps = blockDim.x >> 5;
    constexpr int TN = N / 8, NTILE = (M / 16) * TN;
    for (int tile = warp; tile < NTILE; tile += nwarps) {
        const int m0 = (tile / TN) * 16, n0 = (tile % TN) * 8;
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k0 = 0; k0 < K; k0 += 16) {
            uint32_t a[4], b[2];
            a[0] = pack2(A(m0 + g, k0 + 2 * t), A(m0 + g, k0 + 2 * t + 1));
            a[1] = pack2(A(m0 + g + 8, k0 + 2 * t), A(m0 + g + 8, k0 + 2 * t + 1));
            a[2] = pack2(A(m0 + g, k0 + 2 * t + 8), A(m0 + g, k0 + 2 * t + 9));
            a[3] = pack2(A(m0 + g + 8, k0 + 2 * t + 8), A(m0 + g + 8, k0 + 2 * t + 9));
            b[0] = pack2(B(k0 + 2 * t, n0 + g), B(k0 + 2 * t + 1, n0 + g));
            b[1] = pack2(B(k0 + 2 * t + 8, n0 + g), B(k0 + 2 * t + 9, n0 + g));
            mma16816(c, a, b);
        }
        out(m0 + g, n0 + 2 * t, c[0]);
        out(m0 + g, n0 + 2 * t + 1, c[1]);
        out(m0 + g + 8, n0 + 2 * t, c[2]);
        out(m0 + g + 8, n0 + 2 * t + 1, c[3]);
    }
}


// shared-memory image of one tile's forward state
struct Tile {
    __nv_bfloat16 x[kRows][16];
    __nv_bfloat16 h[3][kRows][H];
    float z[3][kRows][H];
    float y[kRows][8];
    __nv_bfloat16 w1[16][H], w2[H][H], w3[H][H], w4[H][8];
    float b1[H], b2[H], b3[H], b4[8];
};

// the weights, BF16 for the MMAs, biases FP32
__device__ void load_weights(Tile& T, const __nv_bfloat16* __restrict__ wbf, const float* __restrict__ par)
{
    for (int k = threadIdx.x; k < 16 * H; k += blockDim.x) (&T.w1[0][0])[k] = wbf[OW1 + k];
    for (int k = threadIdx.x; k < H * H; k += blockDim.x) {
        (&T.w2[0][0])[k] = wbf[OW2 + k];
        (&T.w3[0][0])[k] = wbf[OW3 + k];
    }
    for (int k = threadIdx.x; k < H * 8; k += blockDim.x) (&T.w4[0][0])[k] = wbf[OW4 + k];
    for (int k = threadIdx.x; k < H; k += blockDim.x) {
        T.b1[k] = par[OB1 + k];
        T.b2[k] = par[OB2 + k];
        T.b3[k] = par[OB3 + k];
    }
    if (threadIdx.x < 8) T.b4[threadIdx.x] = par[OB4 + threadIdx.x];
}

// forward pass of the tile (T.x filled); leaves z, h and y in shared memory
__device__ void forward(Tile& T, int act)
{
    cta_gemm<kRows, H, 16>([&](int m, int k) { return T.x[m][k]; }, [&](int k, int n) { return T.w1[k][n]; },
                           [&](int m, int n, float v) { T.z[0][m][n] = v + T.b1[n]; });
    __syncthreads();
    for (int e = threadIdx.x; e < kRows * H; e += blockDim.x) (&T.h[0][0][0])[e] = __float2bfloat16(act_rt(act, e & (H - 1), (&T.z[0][0][0])[e]));
    __syncthreads();
    cta_gemm<kRows, H, H>([&](int m, int k) { return T.h[0][m][k]; }, [&](int k, int n) { return T.w2[k][n]; },
                          [&](int m, int n, float v) { T.z[1][m][n] = v + T.b2[n]; });
    __syncthreads();
    for (int e = threadIdx.x; e < kRows * H; e += blockDim.x) (&T.h[1][0][0])[e] = __float2bfloat16(act_rt(act, e & (H - 1), (&T.z[1][0][0])[e]));
    __syncthreads();
    cta_gemm<kRows, H, H>([&](int m, int k) { return T.h[1][m][k]; }, [&](int k, int n) { return T.w3[k][n]; },
                          [&](int m, int n, float v) { T.z[2][m][n] = v + T.b3[n]; });
    __syncthreads();
    for (int e = threadIdx.x; e < kRows * H; e += blockDim.x) (&T.h[2][0][0])[e] = __float2bfloat16(act_rt(act, e & (H - 1), (&T.z[2][0][0])[e]));
    __syncthreads();
    cta_gemm<kRows, 8, H>([&](int m, int k) { return T.h[2][m][k]; }, [&](int k, int n) { return T.w4[k][n]; },
                          [&](int m, int n, float v) { T.y[m][n] = v + T.b4[n]; });
    __syncthreads();
}

// ---- training set -----------------------------------------------------------
// Sample k: r ~ U[r_lo, r_hi], w_i, w_j ~ U[w_lo, w_hi], code uniform over the
// species pairs; labels = FP64 quadrature (outputs of smear() for the ordered
// pair (a, b) = (0,0), (1,0), (1,1)) minus the unsmeared spline values at r.
__global__ void k_mlp_labels(Dev d, MlpBox box, unsigned long long seed, int n, float* __restrict__ X,
                             float* __restrict__ Y)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    unsigned long long h = mix64(seed ^ (0x1000000ull * (unsigned long long)k));
    double r = box.r_lo + (box.r_hi - box.r_lo) * u01(h);
    int ncode = d.nt == 1 ? 1 : 3;
    int code = (int)(mix64(h + 3) % (unsigned long long)ncode);
    int a = code == 0 ? 0 : 1, b = code == 2 ? 1 : 0;
    // (w_i, w_j) redrawn (at most 16 times) until the pair exponent lies where
    // the quadrature is defined, alpha_min < alpha < alpha_max; the network is
    // never evaluated outside that range, so zero labels there would only put a
    // step into the fitted function
    double wi = 0, wj = 0, alpha = 0;
    for (int t = 0; t < 16; t++) {
        wi = box.w_lo + (box.w_hi - box.w_lo) * u01(mix64(h + 4 + 2 * t));
        wj = box.w_lo + (box.w_hi - box.w_lo) * u01(mix64(h + 5 + 2 * t));
        double ai = 1.0 / (wi * wi), aj = 1.0 / (wj * wj);
        alpha = (ai * aj) / (ai + aj);
        if (d.alpha_min < alpha && alpha < d.alpha_max) break;
    }
    double r_inv = 1.0 / r, rsq = r * r;
    double g0 = 0, gdr = 0, gda = 0, f0 = 0, fdr = 0, fda = 0;
    if (!smear<true, true, 0>(d, b * d.nt + a, comp_idx(a, b), r, r_inv, rsq, alpha, g0, gdr, gda, f0, fdr, fda))
        g0 = gdr = gda = f0 = fdr = fda = 0.0;
    double base[6];
    base_f64(d, b * d.nt + a, comp_idx(a, b), r, base);
    X[4 * (size_t)k + 0] = (float)r;
    X[4 * (size_t)k + 1] = (float)wi;
    X[4 * (size_t)k + 2] = (float)wj;
    X[4 * (size_t)k + 3] = (float)code;
    // label: the smearing correction (quadrature minus the unsmeared values)
    float* y = Y + 6 * (size_t)k;
    y[0] = (float)(f0 - base[0]);
    y[1] = (float)(g0 - base[1]);
    y[2] = (float)(fdr - base[2]);
    y[3] = (float)(gdr - base[3]);
    y[4] = (float)(fda - base[4]);
    y[5] = (float)(gda - base[5]);
}

// Sums of the labels and of their squares per output, one row of 12 doubles per
// block (the caller adds the rows): the standardisation needs 96 bytes a block
// instead of the whole label array on the host.
__global__ void __launch_bounds__(256) k_mlp_label_sums(const float* __restrict__ Y, int n, double* __restrict__ out)
{
    __shared__ double sh[8][12];
    double v[12];
#pragma unroll
    for (int q = 0; q < 12; q++) v[q] = 0.0;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const float2* y = reinterpret_cast<const float2*>(Y + 6 * k);
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const float2 p = y[u];
            v[2 * u] += (double)p.x;
            v[2 * u + 1] += (double)p.y;
            v[6 + 2 * u] += (double)p.x * (double)p.x;
            v[7 + 2 * u] += (double)p.y * (double)p.y;
        }
    }
#pragma unroll
    for (int q = 0; q < 12; q++) {
        const double s = warp_sum(v[q]);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][q] = s;
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        double s = 0.0;
        for (int w = 0; w < 8; w++) s += sh[w][threadIdx.x];
        out[(size_t)blockIdx.x * 12 + threadIdx.x] = s;
    }
}

// ---- one training step --------------------------------------------------------
// CTA c takes rows idx = hash(seed, step, c*64 + r) % n of the training set,
// or rows [c*64, c*64+64) of the given batch when `fixed` is set (gradient
// checks).  Loss = mean over rows and outputs of the squared error of the
// standardised outputs.
//
// What bounds it: latency -- a step has one 64-row tile per CTA (64 CTAs for
// 4096 rows), ten dependent small products and a barrier between each.  So the
// tile is spread over 16 warps that each own the same two 16x8 output tiles of
// every 64x64 product (the pre-activations z stay in registers from the forward
// to the backward pass and the activations are applied in the product's
// epilogue), fragments come from padded rows by ldmatrix (conflict-free, the
// transposed operands by its .trans form), and two further warps sum the bias
// gradients beside the products.  With 4 warps, element loads of the fragments
// (up to 8-way bank conflicts) and separate passes over z a step took 73 us; now
// 14 us alone, and 14.4 us with its Adam kernel when the two overlap their starts
// (83 before).  The products, their order of accumulation and every rounding are the
// same, so the gradients are the same bits (compared with that kernel's at 64, 192
// and 12864 rows, all three activations; the loss is summed in another order).
constexpr int kTrainWarps = 16, kTrainThreads = (kTrainWarps + 2) * 32;
constexpr int HP = H + 8;  // row pitch: 8 rows of 16 bytes fall into different banks

struct TrainTile {
    __nv_bfloat16 x[kRows][24], dy[kRows][24];
    __nv_bfloat16 h[3][kRows][HP], dz[kRows][HP];
    __nv_bfloat16 w1[16][HP], w2[H][HP], w3[H][HP], w4[H][8];
    float zf[kRows][HP];
    float y[kRows][8], tgt[kRows][8];
    float b[3][H], b4[8], loss[4];
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const __nv_bfloat16* p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// Two neighbouring 16x8 tiles (columns n0 and n0 + 8) of A B over K in steps of
// 16.  A is stored [m][k] (AT: [k][m]), B [k][n] (BN: [n][k]), pitches lda, ldb.
template <bool AT, bool BN, int K>
__device__ __forceinline__ void warp_gemm2(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int m0, int n0,
                                           float (&c)[2][4])
{
    const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) c[j][q] = 0.f;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 16) {
        uint32_t a[4], b[4];
        if (AT) ldsm4t(a, A + (k0 + (mat >> 1) * 8 + r) * lda + m0 + (mat & 1) * 8);
        else ldsm4(a, A + (m0 + (mat & 1) * 8 + r) * lda + k0 + (mat >> 1) * 8);
        if (BN) ldsm4(b, B + (n0 + (mat >> 1) * 8 + r) * ldb + k0 + (mat & 1) * 8);
        else ldsm4t(b, B + (k0 + (mat & 1) * 8 + r) * ldb + n0 + (mat >> 1) * 8);
        const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
        mma16816(c[0], a, b0);
        mma16816(c[1], a, b1);
    }
}

// one 16x8 tile with B stored [k][n] in rows of 8 (pitch ldb)
template <bool AT, int K>
__device__ __forceinline__ void warp_gemm8(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int m0, float (&c)[4])
{
    const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
#pragma unroll
    for (int q = 0; q < 4; q++) c[q] = 0.f;
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += 32) {
        uint32_t a[4], b[4];
        ldsm4t(b, B + (k0 + mat * 8 + r) * ldb);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int k = k0 + 16 * u;
            if (AT) ldsm4t(a, A + (k + (mat >> 1) * 8 + r) * lda + m0 + (mat & 1) * 8);
            else ldsm4(a, A + (m0 + (mat & 1) * 8 + r) * lda + k + (mat >> 1) * 8);
            const uint32_t bb[2] = {b[2 * u], b[2 * u + 1]};
            mma16816(c, a, bb);
        }
    }
}

__device__ __forceinline__ void load_w(__nv_bfloat16* dst, const __nv_bfloat16* src, int rows, int first, int k)
{
    // 16-byte piece k - first of a [rows][64] matrix, into rows of pitch HP
    const int e = k - first;
    if (e >= 0 && e < rows * 8)
        *reinterpret_cast<uint4*>(dst + (e >> 3) * HP + (e & 7) * 8) = *reinterpret_cast<const uint4*>(src + e * 8);
}

__global__ void __launch_bounds__(kTrainThreads) k_mlp_train(MlpState S, const float* X, const float* Y, int n, int batch,
                                                             unsigned long long seed, int step, int fixed)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TrainTile& T = *reinterpret_cast<TrainTile*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // (before dep_wait: a tile's rows depend on nothing a step writes, and until the
    // wait only this CTA's shared memory is written; the run's first step is launched
    // plainly, when X and Y are complete)
    dep_start();
    // 8 threads per row: one takes the inputs, six a target each
    if (tid < kRows * 8) {
        const int r = tid >> 3, part = tid & 7;
        const long long row = (long long)blockIdx.x * kRows + r;
        const long long idx = fixed ? row : (long long)(mix64(seed ^ (0x10000000000ull * (unsigned long long)(step + 1)) ^
                                                              (unsigned long long)row) %
                                                        (unsigned long long)n);
        if (part == 0) {
            float in[4];
            net_inputs(S.box, X[4 * idx], X[4 * idx + 1], X[4 * idx + 2], (int)X[4 * idx + 3], in);
            uint4* xr = reinterpret_cast<uint4*>(T.x[r]);
            xr[0] = make_uint4(pack2f(in[0], in[1]), pack2f(in[2], in[3]), 0u, 0u);
            xr[1] = make_uint4(0u, 0u, 0u, 0u);
        } else if (part < 7) {
            const int q = part - 1;
            T.tgt[r][q] = (Y[6 * idx + q] - S.out_mean[q]) / S.out_scale[q];
        } else
            reinterpret_cast<uint4*>(T.dy[r])[1] = make_uint4(0u, 0u, 0u, 0u);
    }
    dep_wait();  // the previous step's weights
    for (int k = tid; k < 1216; k += kTrainThreads) {
        load_w(&T.w1[0][0], S.wbf + OW1, 16, 0, k);
        load_w(&T.w2[0][0], S.wbf + OW2, H, 128, k);
        load_w(&T.w3[0][0], S.wbf + OW3, H, 640, k);
        if (k >= 1152) reinterpret_cast<uint4*>(&T.w4[0][0])[k - 1152] = reinterpret_cast<const uint4*>(S.wbf + OW4)[k - 1152];
    }
    if (tid < H) {
        T.b[0][tid] = S.par[OB1 + tid];
        T.b[1][tid] = S.par[OB2 + tid];
        T.b[2][tid] = S.par[OB3 + tid];
        if (tid < 8) T.b4[tid] = S.par[OB4 + tid];
    }
    __syncthreads();
    const bool gw = warp < kTrainWarps;
    const int m0 = (warp >> 2) * 16, n0 = (warp & 3) * 16;
    float z[3][2][4], c[2][4];
    // forward: z = h W + b in registers, h in shared memory
#pragma unroll
    for (int l = 0; l < 3; l++) {
        if (gw) {
            if (l == 0) warp_gemm2<false, false, 16>(&T.x[0][0], 24, &T.w1[0][0], HP, m0, n0, c);
            else warp_gemm2<false, false, H>(&T.h[l - 1][0][0], HP, l == 1 ? &T.w2[0][0] : &T.w3[0][0], HP, m0, n0, c);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int col = n0 + 8 * j + 2 * t;
#pragma unroll
                for (int q = 0; q < 4; q++) z[l][j][q] = c[j][q] + T.b[l][col + (q & 1)];
#pragma unroll
                for (int u = 0; u < 2; u++)
                    *reinterpret_cast<uint32_t*>(&T.h[l][m0 + g + 8 * u][col]) =
                        pack2f(act_rt(S.act, col, z[l][j][2 * u]), act_rt(S.act, col + 1, z[l][j][2 * u + 1]));
            }
        }
        __syncthreads();
    }
    float* gp = S.gpart + (size_t)blockIdx.x * NPART;
    const float inv = 2.0f / ((float)batch * 6.0f);
    // output layer, dL/dy (BF16 for the products, FP32 for the bias gradient), loss
    if (warp < 4) {
        float o[4], sum = 0.f;
        warp_gemm8<false, H>(&T.h[2][0][0], HP, &T.w4[0][0], 8, warp * 16, o);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int r = warp * 16 + g + 8 * u;
            float v[2] = {0.f, 0.f};
            if (t < 3) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float diff = o[2 * u + e] + T.b4[2 * t + e] - T.tgt[r][2 * t + e];
                    v[e] = inv * diff;
                    sum += diff * diff / ((float)batch * 6.0f);
                }
            }
            *reinterpret_cast<uint32_t*>(&T.dy[r][2 * t]) = pack2f(v[0], v[1]);
            *reinterpret_cast<float2*>(&T.y[r][2 * t]) = make_float2(v[0], v[1]);
        }
        sum = warp_sumf(sum);
        if (lane == 0) T.loss[warp] = sum;
    }
    __syncthreads();
    // layer 4: dh3 = dy W4^T (its K of 16 is 8 outputs and zeros); dW4 = h3^T dy, db4 = sum dy
    auto put_dz = [&]() {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int col = n0 + 8 * j + 2 * t;
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const float v0 = c[j][2 * u], v1 = c[j][2 * u + 1];
                *reinterpret_cast<float2*>(&T.zf[m0 + g + 8 * u][col]) = make_float2(v0, v1);
                *reinterpret_cast<uint32_t*>(&T.dz[m0 + g + 8 * u][col]) = pack2f(v0, v1);
            }
        }
    };
    auto times_dact = [&](int l) {
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int q = 0; q < 4; q++)
                c[j][q] = c[j][q] * dact_rt(S.act, n0 + 8 * j + 2 * t + (q & 1), z[l][j][q]);
    };
    if (gw) {
        uint32_t a[4], b[4];
        const int mat = lane >> 3, r = lane & 7;
        ldsm4(a, &T.dy[m0 + (mat & 1) * 8 + r][(mat >> 1) * 8]);
        ldsm4(b, &T.w4[n0 + (mat & 1) * 8 + r][0]);
        const uint32_t b0[2] = {b[0], 0u}, b1[2] = {b[1], 0u};
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) c[j][q] = 0.f;
        mma16816(c[0], a, b0);
        mma16816(c[1], a, b1);
        times_dact(2);
        put_dz();
        if (warp < 4) {
            float o[4];
            warp_gemm8<true, kRows>(&T.h[2][0][0], HP, &T.dy[0][0], 24, warp * 16, o);
#pragma unroll
            for (int u = 0; u < 2; u++)
                *reinterpret_cast<float2*>(&gp[OW4 + (warp * 16 + g + 8 * u) * 8 + 2 * t]) = make_float2(o[2 * u], o[2 * u + 1]);
        }
    } else if (warp == kTrainWarps && lane < 8) {
        float s = 0.f;
#pragma unroll 16
        for (int r = 0; r < kRows; r++) s += T.y[r][lane];
        gp[OB4 + lane] = s;
    }
    __syncthreads();
    // layers 3, 2, 1: zf and dz hold dL/dz_l
#pragma unroll
    for (int l = 2; l >= 0; l--) {
        const int ow = l == 2 ? OW3 : (l == 1 ? OW2 : OW1), ob = l == 2 ? OB3 : (l == 1 ? OB2 : OB1);
        if (gw) {
            if (l > 0 || warp < 4) {
                float w[2][4];
                if (l > 0) warp_gemm2<true, false, kRows>(&T.h[l > 0 ? l - 1 : 0][0][0], HP, &T.dz[0][0], HP, m0, n0, w);
                else warp_gemm2<true, false, kRows>(&T.x[0][0], 24, &T.dz[0][0], HP, 0, n0, w);
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int u = 0; u < 2; u++)
                        *reinterpret_cast<float2*>(&gp[ow + ((l > 0 ? m0 : 0) + g + 8 * u) * H + n0 + 8 * j + 2 * t]) =
                            make_float2(w[j][2 * u], w[j][2 * u + 1]);
            }
            if (l > 0) {
                warp_gemm2<false, true, H>(&T.dz[0][0], HP, l == 2 ? &T.w3[0][0] : &T.w2[0][0], HP, m0, n0, c);
                times_dact(l - 1);
            }
        } else {
            const int col = tid - kTrainWarps * 32;
            float s = 0.f;
#pragma unroll 16
            for (int r = 0; r < kRows; r++) s += T.zf[r][col];
            gp[ob + col] = s;
        }
        if (l > 0) {
            __syncthreads();
            if (gw) put_dz();
            __syncthreads();
        }
    }
    if (tid == 0) gp[OLOSS] = (T.loss[0] + T.loss[1]) + (T.loss[2] + T.loss[3]);
}

// Sum of the per-CTA partial gradients; Adam (Kingma & Ba 2015) with a cosine
// learning rate; BF16 copy of the weights.  With lr == 0 only the summed
// gradient is written (gradient checks).  Small blocks, so that the reads of the
// partials spread over all SMs.
constexpr int kAdamThreads = 64;
__global__ void __launch_bounds__(kAdamThreads) k_mlp_adam(MlpState S, int nblocks, int step, int total_steps, float lr0, float* __restrict__ grad_out,
                           float* __restrict__ loss_hist)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    dep_start();  // (the next step waits for this kernel before it reads weights or writes partials)
    if (p > NPARAM) return;  // (every block has threads that go on and wait)
    dep_wait();  // this step's partial gradients
    float g = 0.f;
#pragma unroll 16
    for (int c = 0; c < nblocks; c++) g += S.gpart[(size_t)c * NPART + p];
    if (p == NPARAM) {
        if (loss_hist) loss_hist[step] = g;
        return;
    }
    if (grad_out) grad_out[p] = g;
    if (lr0 <= 0.f) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float lr = 0.5f * lr0 * (1.0f + cospif((float)step / (float)total_steps));
    float m = b1 * S.m[p] + (1.f - b1) * g;
    float v = b2 * S.v[p] + (1.f - b2) * g * g;
    S.m[p] = m;
    S.v[p] = v;
    float mh = m / (1.f - powf(b1, (float)(step + 1)));
    float vh = v / (1.f - powf(b2, (float)(step + 1)));
    float w = S.par[p] - lr * mh / (sqrtf(vh) + eps);
    S.par[p] = w;
    S.wbf[p] = __float2bfloat16(w);
}

// Evaluate the network on n raw inputs (r, w_i, w_j, code); y receives its
// outputs in physical units: the smearing corrections of (phi, rho, dphi/dr,
// drho/dr, dphi/dalpha, drho/dalpha).
__global__ void __launch_bounds__(kMlpThreads) k_mlp_eval(MlpState S, const float* __restrict__ X, int n,
                                                          float* __restrict__ Y)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Tile& T = *reinterpret_cast<Tile*>(smem_raw);
    load_weights(T, S.wbf, S.par);
    for (long long t0 = (long long)blockIdx.x * kRows; t0 < n; t0 += (long long)gridDim.x * kRows) {
        __syncthreads();
        for (int r = threadIdx.x; r < kRows; r += blockDim.x) {
            long long k = t0 + r;
            float in[4] = {0, 0, 0, 0};
            if (k < n) net_inputs(S.box, X[4 * k], X[4 * k + 1], X[4 * k + 2], (int)X[4 * k + 3], in);
            for (int q = 0; q < 16; q++) T.x[r][q] = __float2bfloat16(q < 4 ? in[q] : 0.f);
        }
        __syncthreads();
        forward(T, S.act);
        for (int e = threadIdx.x; e < kRows * 6; e += blockDim.x) {
            int r = e / 6, q = e % 6;
            long long k = t0 + r;
            if (k < n) Y[6 * k + q] = T.y[r][q] * S.out_scale[q] + S.out_mean[q];
        }
    }
}

}  // namespace

size_t mlp_smem_bytes() { return sizeof(Tile); }
int mlp_nparam() { return NPARAM; }
int mlp_npart() { return NPART; }

cudaError_t launch_mlp_labels(const Dev& d, const MlpBox& box, unsigned long long seed, int n, float* X, float* Y,
                              cudaStream_t st)
{
    k_mlp_labels<<<div_up(n, 128), 128, 0, st>>>(d, box, seed, n, X, Y);
    return cudaGetLastError();
}

int mlp_label_sum_rows(int n) { return std::min(div_up(n, 256), 2 * num_sms()); }

cudaError_t launch_mlp_label_sums(const float* Y, int n, double* out, cudaStream_t st)
{
    k_mlp_label_sums<<<mlp_label_sum_rows(n), 256, 0, st>>>(Y, n, out);
    return cudaGetLastError();
}

cudaError_t launch_mlp_train_step(const MlpState& S, const float* X, const float* Y, int n, int batch,
                                  unsigned long long seed, int step, int total, float lr, int fixed, float* grad_out,
                                  float* loss_hist, cudaStream_t st)
{
    constexpr size_t sm = sizeof(TrainTile);
    const int nb = batch / kRows;
    cudaError_t e;
    if (step == 0 || fixed) {
        // the first step of a run is a plain launch: k_mlp_train reads X and Y before
        // its wait, so it must not start before the work that fills them is complete;
        // behind it only steps follow, and those write neither
        e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
        k_mlp_train<<<nb, kTrainThreads, sm, st>>>(S, X, Y, n, batch, seed, step, fixed);
        e = cudaGetLastError();
    } else
        e = launch_dep(k_mlp_train, nb, kTrainThreads, sm, st, S, X, Y, n, batch, seed, step, fixed);
    if (e != cudaSuccess) return e;
    e = launch_dep(k_mlp_adam, div_up(NPARAM + 1, kAdamThreads), kAdamThreads, 0, st, S, nb, step, total, lr, grad_out,
                   loss_hist);
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_mlp_eval(const MlpState& S, const float* X, int n, float* Y, cudaStream_t st)
{
    size_t sm = sizeof(Tile);
    cudaFuncSetAttribute(k_mlp_eval, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    int grid = div_up(n, kRows);
    if (grid > num_sms() * 4) grid = num_sms() * 4;
    k_mlp_eval<<<grid, kMlpThreads, sm, st>>>(S, X, n, Y);
    return cudaGetLastError();
}

}  // namespace mg
