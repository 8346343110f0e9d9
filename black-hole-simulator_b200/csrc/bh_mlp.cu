// bh_mlp.cu -- the learned con2prim initial guess: a 6 -> 64 -> 64 -> 2
// network (tanh hidden layers) mapping scale-free features of a cell's
// conserved state to y0 = log(xi / D) and y1 = log W (xi = rho h W^2, the
// unknown of conserved::ctop's Newton iteration, conserved.cpp:170-187).
// Inference reads BF16 weights and accumulates in FP32; training keeps FP32
// master weights, evaluates the forward pass with their BF16 roundings (the
// weights inference will see), back-propagates in FP32 and takes Adam steps.
// The solver's own FP64 con2prim produces the training pairs and still
// decides every cell: the guess only moves Newton's starting point.
//
// Parameters, FP32, one flat array (and its BF16 copy), in this order:
//   W1 [64][6], b1 [64], W2 [64][64], b2 [64], W3 [2][64], b3 [2]
// followed by 12 floats of feature normalisation (mean[6], 1/std[6]).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <math.h>
#include "bhgpu.h"
#include "bh_tc.cuh"

namespace {

constexpr int NI = 6, NH = 64, NO = 2;
constexpr int OW1 = 0, OB1 = OW1 + NH * NI, OW2 = OB1 + NH, OB2 = OW2 + NH * NH, OW3 = OB2 + NH,
              OB3 = OW3 + NO * NH, NPAR = OB3 + NO, ONORM = NPAR;
static_assert(NPAR == BH_MLP_NPARAM, "parameter count");
constexpr int TPB = 128;

inline cudaStream_t S(void* s) { return (cudaStream_t)s; }
inline int launched() { return cudaGetLastError() == cudaSuccess ? BH_OK : BH_ECUDA; }

// features of cell q from the con2prim preamble pre [5][n] and r
__device__ inline void features(const double* pre, const double* r, int64_t n, int64_t q, float x[NI]) {
    double p5[5] = {pre[q], pre[n + q], pre[2 * n + q], pre[3 * n + q], pre[4 * n + q]};
    bh_tc::features(p5, r[q], x);
}

__device__ inline float bf(__nv_bfloat16 v) { return __bfloat162float(v); }

// inference: xi0 = D exp(y0); NaN where a feature is not finite
__global__ void k_guess(const __nv_bfloat16* wb, const float* norm, const double* pre, const double* r, int64_t n,
                        double* xi0) {
    int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    float x[NI], h1[NH], h2[NH], y[NO];
    features(pre, r, n, q, x);
    bool ok = true;
    for (int i = 0; i < NI; i++) ok &= isfinite(x[i]);
    if (!ok) { xi0[q] = NAN; return; }
    float xn[NI];
    for (int i = 0; i < NI; i++) xn[i] = (x[i] - norm[i]) * norm[NI + i];
    for (int j = 0; j < NH; j++) {
        float a = bf(wb[OB1 + j]);
        for (int i = 0; i < NI; i++) a += bf(wb[OW1 + j * NI + i]) * xn[i];
        h1[j] = tanhf(a);
    }
    for (int j = 0; j < NH; j++) {
        float a = bf(wb[OB2 + j]);
        for (int i = 0; i < NH; i++) a += bf(wb[OW2 + j * NH + i]) * h1[i];
        h2[j] = tanhf(a);
    }
    for (int o = 0; o < NO; o++) {
        float a = bf(wb[OB3 + o]);
        for (int i = 0; i < NH; i++) a += bf(wb[OW3 + o * NH + i]) * h2[i];
        y[o] = a;
    }
    xi0[q] = pre[q] * exp((double)y[0]);
}

// training: forward with the BF16 roundings of the FP32 weights, loss
// L = mean over cells of sum_o (y_o - t_o)^2, and its gradient.  A CTA takes
// tiles of TR_C cells and keeps a tile's activations and deltas in shared
// memory, so the three 64 x 64 contractions (layer 2 forward, its
// back-propagation, the weight gradient) and the gradient's sum over the
// tile's cells never leave the SM; its sums over all its tiles go out once,
// as one partial gradient per CTA.
//   Bound: latency (a batch is one tile per CTA: features, then three short
// FP32 contractions; 0.2 GFLOP and 0.6 MB for 8192 cells).  64 cells x 4
// threads: a thread holds 16 outputs of one cell, the weights broadcast from
// shared memory as float4.  Each cell's forward and backward sums keep the
// order i = 0 .. 63 of the inference kernel; the gradient is a sum over the
// tile, then over the CTAs, which rounds less than one long sum.
constexpr int TR_C = 64, TR_T = 256, TR_P = TR_C + 1;   // cells, threads, row pitch (no bank conflicts)
static_assert(TR_T == 4 * TR_C && NH == 64 && TR_C == NH, "4 threads per cell, 16 outputs each; 4 x 4 gradient tiles");
struct TrainSmem {
    alignas(16) float w1t[NI][NH];    // W1 transposed, FP32 values of the BF16 weights
    alignas(16) float w2t[NH][NH];    // W2 transposed (forward)
    alignas(16) float w2[NH][NH];     // W2 (backward)
    float b1[NH], b2[NH], w3[NO][NH], b3[NO], norm[2 * NI];
    float xn[NI][TR_P], h1[NH][TR_P], h2[NH][TR_P], g2[NH][TR_P], d1[NH][TR_P], dy[NO][TR_P];
    float red[TR_T / 32];
};
// the gradients other than W2's, in this order: W1, b1, b2, W3, b3
constexpr int NSMALL = NH * NI + NH + NH + NO * NH + NO;

// o[q] = a[q] + sum_i w[i][16 part + q] x[i][c], i ascending
template <int K>
__device__ inline void contract16(float* a, const float (*w)[NH], const float (*x)[TR_P], int part, int c) {
#pragma unroll 8
    for (int i = 0; i < K; i++) {
        const float v = x[i][c];
        const float4* wi = reinterpret_cast<const float4*>(&w[i][16 * part]);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 m = wi[q];
            a[4 * q] += m.x * v; a[4 * q + 1] += m.y * v; a[4 * q + 2] += m.z * v; a[4 * q + 3] += m.w * v;
        }
    }
}

__global__ void __launch_bounds__(TR_T) k_train(const __nv_bfloat16* wb, const float* norm, const double* pre,
                                               const double* r, const float* target, int64_t n, float* lossp,
                                               float* gradp) {
    extern __shared__ __align__(16) unsigned char smem[];
    TrainSmem& s = *reinterpret_cast<TrainSmem*>(smem);
    const int t = threadIdx.x, c = t % TR_C, part = t / TR_C;
    for (int e = t; e < NH * NI; e += TR_T) s.w1t[e % NI][e / NI] = bf(wb[OW1 + e]);
    for (int e = t; e < NH * NH; e += TR_T) {
        const float v = bf(wb[OW2 + e]);
        s.w2[e / NH][e % NH] = v;
        s.w2t[e % NH][e / NH] = v;
    }
    if (t < NH) { s.b1[t] = bf(wb[OB1 + t]); s.b2[t] = bf(wb[OB2 + t]); }
    if (t < NO * NH) s.w3[t / NH][t % NH] = bf(wb[OW3 + t]);
    if (t < NO) s.b3[t] = bf(wb[OB3 + t]);
    if (t < 2 * NI) s.norm[t] = norm[t];
    float g[16], gs[3], l = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; q++) g[q] = 0.0f;
    gs[0] = gs[1] = gs[2] = 0.0f;
    const int j0 = 4 * (t / 16), i0 = t % 16;   // W2's gradient: rows j0..j0+3, columns i0 + 16 q
    const int64_t ntile = (n + TR_C - 1) / TR_C;
    for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int64_t q0 = tile * TR_C + c;
        const bool in = q0 < n;
        __syncthreads();   // weights staged; the previous tile's reads are done
        // features: x0, x5 | x1 | x2, x3 | x4 by the cell's four threads
        double p5[5] = {1.0, 1.0, 1.0, 1.0, 1.0}, rr = 1.0;
        if (in) {
            for (int v = 0; v < 5; v++) p5[v] = pre[v * n + q0];
            rr = r[q0];
        }
        auto put = [&](int i, float x) { s.xn[i][c] = in ? (x - s.norm[i]) * s.norm[NI + i] : 0.0f; };
        if (part == 0) { put(0, bh_tc::feature<0>(p5, rr)); put(5, bh_tc::feature<5>(p5, rr)); }
        else if (part == 1) put(1, bh_tc::feature<1>(p5, rr));
        else if (part == 2) { put(2, bh_tc::feature<2>(p5, rr)); put(3, bh_tc::feature<3>(p5, rr)); }
        else put(4, bh_tc::feature<4>(p5, rr));
        __syncthreads();
        float a[16];
#pragma unroll
        for (int q = 0; q < 16; q++) a[q] = s.b1[16 * part + q];
        contract16<NI>(a, s.w1t, s.xn, part, c);
#pragma unroll
        for (int q = 0; q < 16; q++) s.h1[16 * part + q][c] = tanhf(a[q]);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; q++) a[q] = s.b2[16 * part + q];
        contract16<NH>(a, s.w2t, s.h1, part, c);
#pragma unroll
        for (int q = 0; q < 16; q++) s.h2[16 * part + q][c] = tanhf(a[q]);
        __syncthreads();
        if (part < NO) {
            float y = s.b3[part], d = 0.0f;
#pragma unroll 16
            for (int i = 0; i < NH; i++) y += s.w3[part][i] * s.h2[i][c];
            if (in) {
                const float e = y - target[part * n + q0];
                l += e * e;
                d = 2.0f * e / (float)n;
            }
            s.dy[part][c] = d;   // (0 past the batch's end: no contribution below)
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const int i = 16 * part + q;
            float v = 0.0f;
            for (int o = 0; o < NO; o++) v += s.w3[o][i] * s.dy[o][c];
            const float h = s.h2[i][c];
            s.g2[i][c] = v * (1.0f - h * h);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; q++) a[q] = 0.0f;
        contract16<NH>(a, s.w2, s.g2, part, c);
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float h = s.h1[16 * part + q][c];
            s.d1[16 * part + q][c] = a[q] * (1.0f - h * h);
        }
        // W2's gradient: 4 x 4 outputs per thread over the tile's cells
#pragma unroll 4
        for (int k = 0; k < TR_C; k++) {
            float dj[4], hi[4];
#pragma unroll
            for (int q = 0; q < 4; q++) { dj[q] = s.g2[j0 + q][k]; hi[q] = s.h1[i0 + 16 * q][k]; }
#pragma unroll
            for (int q = 0; q < 16; q++) g[q] += dj[q / 4] * hi[q % 4];
        }
        __syncthreads();   // d1 written
#pragma unroll
        for (int u = 0; u < 3; u++) {
            int e = t + u * TR_T;
            if (e >= NSMALL) break;
            const float *dl, *ac = nullptr;   // delta row and activation row (none for a bias)
            if (e < NH * NI) { dl = s.d1[e / NI]; ac = s.xn[e % NI]; }
            else if ((e -= NH * NI) < NH) dl = s.d1[e];
            else if ((e -= NH) < NH) dl = s.g2[e];
            else if ((e -= NH) < NO * NH) { dl = s.dy[e / NH]; ac = s.h2[e % NH]; }
            else dl = s.dy[e - NO * NH];
            float v = 0.0f;
            if (ac) {
#pragma unroll 8
                for (int k = 0; k < TR_C; k++) v += dl[k] * ac[k];
            } else {
#pragma unroll 8
                for (int k = 0; k < TR_C; k++) v += dl[k];
            }
            gs[u] += v;
        }
    }
    float* gp = gradp + (int64_t)blockIdx.x * NPAR;
#pragma unroll
    for (int q = 0; q < 16; q++) gp[OW2 + (j0 + q / 4) * NH + i0 + 16 * (q % 4)] = g[q];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const int e = t + u * TR_T;
        if (e >= NSMALL) break;
        // W1 and b1 lie before W2, b2, W3 and b3 after it
        gp[e < NH * NI + NH ? OW1 + e : OB2 + e - (NH * NI + NH)] = gs[u];
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((t & 31) == 0) s.red[t >> 5] = l;
    __syncthreads();
    if (t == 0) {
        l = 0.0f;
        for (int w = 0; w < TR_T / 32; w++) l += s.red[w];
        lossp[blockIdx.x] = l;
    }
}
static_assert(OB1 == OW1 + NH * NI && OW2 == OB1 + NH && OW3 == OB2 + NH && OB3 == OW3 + NO * NH, "parameter order");

// the CTAs' partial gradients summed (8 slices of them per output, then the
// slices in order), and with lr > 0 the Adam step (Kingma & Ba 2015) on the
// FP32 master weights and their BF16 copy; output NPAR is the loss
constexpr int RD_O = 32, RD_S = 8;
__global__ void __launch_bounds__(RD_O* RD_S) k_train_reduce(const float* lossp, const float* gradp, int np,
                                                            float* grad, float* loss_out, float* w, float* m,
                                                            float* v, __nv_bfloat16* wb, float lr, float b1, float b2,
                                                            float eps, float c1, float c2) {
    __shared__ float red[RD_S][RD_O];
    const int o = threadIdx.x % RD_O, sl = threadIdx.x / RD_O, t = blockIdx.x * RD_O + o;
    float a = 0.0f;
    if (t < NPAR) {
#pragma unroll 4
        for (int p = sl; p < np; p += RD_S) a += gradp[(int64_t)p * NPAR + t];
    } else if (t == NPAR) {
        for (int p = sl; p < np; p += RD_S) a += lossp[p];
    }
    red[sl][o] = a;
    __syncthreads();
    if (sl != 0 || t > NPAR) return;
    float gi = red[0][o];
    for (int q = 1; q < RD_S; q++) gi += red[q][o];
    if (t == NPAR) {
        if (loss_out) *loss_out = gi;
        return;
    }
    grad[t] = gi;
    if (!(lr > 0.0f)) return;
    float mi = b1 * m[t] + (1.0f - b1) * gi;
    float vi = b2 * v[t] + (1.0f - b2) * gi * gi;
    m[t] = mi; v[t] = vi;
    w[t] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    wb[t] = __float2bfloat16_rn(w[t]);
}
__global__ void k_to_bf16(const float* w, __nv_bfloat16* wb) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < NPAR) wb[t] = __float2bfloat16_rn(w[t]);
}

// the bounded wait of the tensor-core kernels on an mbarrier that nothing
// arrives on: it must give up and report, never hang
__global__ void k_wait_selftest(int32_t* err) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) bh_tc::mbar_init(&bar);
    __syncthreads();
    bool ok = bh_tc::mbar_wait(&bar, 0);
    if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicOr(err, BH_ERR_TIMEOUT);
}

}  // namespace

extern "C" {

int bh_wait_selftest(int32_t* err, void* stream) {
    if (!err) return BH_EINVAL;
    k_wait_selftest<<<1, 32, 0, S(stream)>>>(err);
    return launched();
}

int bh_mlp_sync_bf16(bh_mlp* m, void* stream) {
    if (!m || !m->w || !m->wb) return BH_EINVAL;
    k_to_bf16<<<(NPAR + 255) / 256, 256, 0, S(stream)>>>(m->w, (__nv_bfloat16*)m->wb);
    return launched();
}

int bh_mlp_guess(const bh_mlp* m, const double* pre, const double* r, int64_t n, double* xi0, void* stream) {
    if (!m || !m->wb || !pre || !r || !xi0 || n < 0) return BH_EINVAL;
    if (n == 0) return BH_OK;
    k_guess<<<(unsigned)((n + TPB - 1) / TPB), TPB, 0, S(stream)>>>((const __nv_bfloat16*)m->wb, m->w + ONORM, pre,
                                                                  r, n, xi0);
    return launched();
}

int bh_mlp_train_step(bh_mlp* m, const double* pre, const double* r, const float* target, int64_t n, float lr,
                      float* scratch, float* loss_out, void* stream) {
    if (!m || !m->w || !m->wb || !m->adam_m || !m->adam_v || !pre || !r || !target || !scratch || n <= 0)
        return BH_EINVAL;
    cudaStream_t st = S(stream);
    // a CTA per tile up to two per SM (their shared memory), which then walk
    // the rest: at most 2 x SMs partial gradients whatever the batch
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem)) !=
            cudaSuccess)
        return BH_ECUDA;
    const int64_t ntile = (n + TR_C - 1) / TR_C;
    const int np = (int)(ntile < 2 * (int64_t)sms ? ntile : 2 * (int64_t)sms);
    // scratch: the loss partials, the gradient partials, the gradient; with
    // one partial (a batch of up to 64 cells, whose scratch may hold no
    // more) the CTA writes the gradient in place
    float* grad = scratch + (4 * NH + NI + NO + 1) * n;
    float* lossp = scratch;
    float* gradp = np == 1 ? grad : scratch + np;
    const __nv_bfloat16* wb = (const __nv_bfloat16*)m->wb;
    k_train<<<np, TR_T, sizeof(TrainSmem), st>>>(wb, m->w + ONORM, pre, r, target, n, lossp, gradp);
    const float b1 = 0.9f, b2 = 0.999f;
    float c1 = 1.0f, c2 = 1.0f;
    if (lr > 0.0f) {
        m->step += 1;
        c1 = 1.0f - powf(b1, (float)m->step);
        c2 = 1.0f - powf(b2, (float)m->step);
    }
    k_train_reduce<<<(NPAR + 1 + RD_O - 1) / RD_O, RD_O * RD_S, 0, st>>>(lossp, gradp, np, grad, loss_out, m->w,
                                                                        m->adam_m, m->adam_v,
                                                                        (__nv_bfloat16*)m->wb, lr, b1, b2, 1e-8f, c1,
                                                                        c2);
    return launched();
}

}  // extern "C"
