/*
 * k_mlp.cu -- the MGFM seed surrogate: a 12-64-64-64-2 tanh MLP that predicts the
 * star pressure and velocity of the two-material Riemann problem solved by
 * MPM::MGFM (mpm.cpp:882-926), used as the Newton starting guess in place of the
 * reference's max(p_l, p_r) (mpm.cpp:893).  The pressure output is a log
 * correction to a closed-form two-shock baseline (mgfm_baseline below); the
 * velocity output is trained with a small weight and does not enter the seed.  The plain Newton solve stays the
 * fallback and the final check: a seeded solve that does not reach |f| <= tol within
 * the iteration cap is redone from the plain seed, and a problem without a
 * positive root (f(1e-8) < 0) goes straight to the plain solve.
 *
 * Everything here is project code: feature construction, forward pass (BF16
 * weights, FP32 accumulation), backward pass and Adam, all on the device.
 *
 * Parameter layout (FP32 master copy, n = 9282):
 *   W1[64][12] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] W4[2][64] b4[2]
 * followed by the fixed feature/target normalisation (NORM = 28 floats):
 *   mean_x[12] std_x[12] mean_y[2] std_y[2]
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/pgdg.h"
#include "pgdg_dev.cuh"

namespace pgdg {

constexpr int NI = 12, NH = 64, NO = 2;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NI, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NH * NH, OFF_W4 = OFF_B3 + NH, OFF_B4 = OFF_W4 + NO * NH,
              NPARAM = OFF_B4 + NO;
constexpr int NNORM = 2 * NI + 2 * NO;

/* ------------------------------------------------------------------ */
/* features of one Riemann problem                                    */
/* ------------------------------------------------------------------ */
/* Closed-form baseline p_b of the star pressure: the acoustic estimate
 * p_ac = (Z_r p_l + Z_l p_r + Z_l Z_r (u_l - u_r)) / (Z_l + Z_r), Z = sqrt(gamma (p + p_inf) rho),
 * then one linearised step of the two-shock relation with the shock speeds W
 * (mpm.cpp:908, glbfunc.h:314-337) frozen at max(p_ac, 1e-8).  For weak waves
 * the error is far below the Newton tolerance; the network corrects strong ones. */
__host__ __device__ inline double mgfm_baseline(double ul, double ur, double pl, double pr, double rl, double rr,
                                                double gl, double il, double gr, double ir) {
  const double Zl = sqrt(gl * (pl + il) * rl), Zr = sqrt(gr * (pr + ir) * rr);
  double p0 = (Zr * pl + Zl * pr + Zl * Zr * (ul - ur)) / (Zl + Zr);
  if (!(p0 > 1e-8)) p0 = 1e-8;
  const double Wl = sqrt(0.5 * rl * ((gl + 1.) * p0 + (gl - 1.) * pl + 2. * gl * il));
  const double Wr = sqrt(0.5 * rr * ((gr + 1.) * p0 + (gr - 1.) * pr + 2. * gr * ir));
  const double yl = drcp(Wl), yr = drcp(Wr);
  double pt = (ddiv_by(pl, Wl, yl) + ddiv_by(pr, Wr, yr) + (ul - ur)) / (yl + yr);
  if (!(pt > 1e-8)) pt = 1e-8;
  return pt;
}

/* Scale-free description of a problem (FP32 transcendentals; the baseline in
 * FP64):
 *   x0,x1  log((p + p_inf)/P0) left/right, P0 the larger effective pressure
 *   x2     log(rho_l / rho_r)
 *   x3     (u_l - u_r) / a0, a0 = sqrt(P0 / sqrt(rho_l rho_r)), clamped to +-20
 *   x4     log(p_b / p_l)          x11  log(p_b / p_r)
 *   x5,x6  gamma left/right        x7,x8  p_inf / P0 left/right
 *   x9,x10 log(p / P0) left/right
 * The network's first output y predicts log(p* / p_b) / sc with the strength
 * scale sc = s^2 / (1 + s^2), s = |x4| + |x11|: the correction vanishes for
 * weak waves, where the baseline is already far inside the Newton tolerance. */
__host__ __device__ inline void mgfm_features(const double* q, double gl, double il, double gr, double ir, float* x,
                                              double* pb_out, float* sc_out) {
  double ul = q[0], ur = q[1], pl = q[2], pr = q[3], rl = q[4], rr = q[5];
  if (pl < 1e-10) pl = 1e-10;
  if (pr < 1e-10) pr = 1e-10;
  if (rl < 1e-10) rl = 1e-10;
  if (rr < 1e-10) rr = 1e-10;
  const double Pl = pl + il, Pr = pr + ir;
  const double P0 = Pl > Pr ? Pl : Pr;
  const float a0 = sqrtf((float)P0 / sqrtf((float)rl * (float)rr));
  const float du = (float)(ul - ur) / a0;
  const double pb = mgfm_baseline(ul, ur, pl, pr, rl, rr, gl, il, gr, ir);
  const double y0 = drcp(P0); /* six quotients by P0 */
  const float lbl = logf((float)(pb / pl)), lbr = logf((float)(pb / pr));
  const float sv = fabsf(lbl) + fabsf(lbr);
  x[0] = logf((float)ddiv_by(Pl, P0, y0));
  x[1] = logf((float)ddiv_by(Pr, P0, y0));
  x[2] = logf((float)(rl / rr));
  x[3] = du > 20.f ? 20.f : (du < -20.f ? -20.f : du);
  x[4] = lbl;
  x[5] = (float)gl;
  x[6] = (float)gr;
  x[7] = (float)ddiv_by(il, P0, y0);
  x[8] = (float)ddiv_by(ir, P0, y0);
  x[9] = logf((float)(ddiv_by(pl, P0, y0) + 1e-30));
  x[10] = logf((float)(ddiv_by(pr, P0, y0) + 1e-30));
  x[11] = lbr;
  *pb_out = pb;
  *sc_out = sv * sv / (1.f + sv * sv);
}

__global__ void k_features(const double* in6, const int8_t* mat2, const double* gam, const double* pinf, float* X,
                           int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int s = mat2[2 * i], s1 = mat2[2 * i + 1];
    double pb;
    float sc, x[NI];
    mgfm_features(in6 + 6 * i, gam[s], pinf[s], gam[s1], pinf[s1], x, &pb, &sc);
    for (int k = 0; k < NI; k++) X[i * NI + k] = x[k];
  }
}

/* ------------------------------------------------------------------ */
/* forward pass: one thread per sample, weights (BF16-rounded) in smem */
/* ------------------------------------------------------------------ */
template <bool BF16>
__device__ __forceinline__ float wq(float w) {
  if (BF16) return __bfloat162float(__float2bfloat16_rn(w));
  return w;
}

/* stage the parameters in shared memory, weights rounded to BF16 when asked */
template <bool BF16>
__device__ __forceinline__ void load_params(const float* __restrict__ params, float* w) {
  for (int k = threadIdx.x; k < NPARAM; k += blockDim.x) {
    bool isb = (k >= OFF_B1 && k < OFF_W2) || (k >= OFF_B2 && k < OFF_W3) || (k >= OFF_B3 && k < OFF_W4) || k >= OFF_B4;
    w[k] = isb ? params[k] : wq<BF16>(params[k]);
  }
  for (int k = threadIdx.x; k < NNORM; k += blockDim.x) w[NPARAM + k] = params[NPARAM + k];
  __syncthreads();
}

/* one sample through the network (normalised input xn); the loops are fully
 * unrolled so the activations stay in registers */
template <int NOUT>
__device__ __forceinline__ void mlp_eval(const float* w, const float* xn, float* y) {
  float h[NH], g[NH];
#pragma unroll
  for (int j = 0; j < NH; j++) {
    float a = w[OFF_B1 + j];
#pragma unroll
    for (int k = 0; k < NI; k++) a = fmaf(w[OFF_W1 + j * NI + k], xn[k], a);
    h[j] = tanhf(a);
  }
#pragma unroll
  for (int j = 0; j < NH; j++) {
    float a = w[OFF_B2 + j];
#pragma unroll
    for (int k = 0; k < NH; k++) a = fmaf(w[OFF_W2 + j * NH + k], h[k], a);
    g[j] = tanhf(a);
  }
#pragma unroll
  for (int j = 0; j < NH; j++) {
    float a = w[OFF_B3 + j];
#pragma unroll
    for (int k = 0; k < NH; k++) a = fmaf(w[OFF_W3 + j * NH + k], g[k], a);
    h[j] = tanhf(a);
  }
#pragma unroll
  for (int o = 0; o < NOUT; o++) {
    float a = w[OFF_B4 + o];
#pragma unroll
    for (int k = 0; k < NH; k++) a = fmaf(w[OFF_W4 + o * NH + k], h[k], a);
    y[o] = a;
  }
}

/* Y[n][2] (normalised outputs) from raw features X */
template <bool BF16>
__global__ void __launch_bounds__(128) k_mlp_forward(const float* __restrict__ params, const float* __restrict__ X,
                                                     float* __restrict__ Y, int64_t n,
                                                     const unsigned long long* __restrict__ dn) {
  if (dn && (int64_t)*dn < n) n = (int64_t)*dn; /* live count of a batch sized for capacity */
  __shared__ __align__(16) float w[NPARAM + NNORM];
  load_params<BF16>(params, w);
  const float* mx = w + NPARAM;
  const float* sx = mx + NI;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float xn[NI], y[NO];
#pragma unroll
    for (int k = 0; k < NI; k++) xn[k] = (X[i * NI + k] - mx[k]) / sx[k];
    mlp_eval<NO>(w, xn, y);
    Y[i * NO + 0] = y[0];
    Y[i * NO + 1] = y[1];
  }
}

/* ------------------------------------------------------------------ */
/* backward pass                                                      */
/* ------------------------------------------------------------------ */
/* Loss and gradient of a batch in one kernel.  A block of 256 threads takes tiles of
 * 32 samples: forward, output gradient and backward passes run on activations that
 * stay in shared memory (feature-major, each layer's gradient replacing its
 * activations), and the weight gradients are summed in registers over the block's
 * tiles, then written once as that block's partial; k_grad_sum adds the partials in a
 * fixed order.  FP32 throughout, each activation and each back-propagated value summed
 * in index order.  A thread owns 4 x 2 (layers) or 4 x 4 (weight gradients) results, two
 * shared-memory loads for 8 or 16 multiply-adds, which is what bounds a tile; rows are
 * padded so that the float4 of eight lanes fall into different banks (36 floats of samples,
 * 68 of weights).  8192 samples: 24 us and 4 us for the sum, 54 us a call with the
 * launches and the copy to the host; as separate passes over stored activations, a block
 * per weight row reading them uncoalesced, the call took 1.74 ms.  Its 0.46 GFLOP would
 * take 6 us at the FP32 rate; a tile is a chain of ten short phases, and 256 tiles are
 * 1.7 a multiprocessor. */
constexpr int GT = 32, GS = GT + 4, GW = NH + 4; /* samples of a tile, strides of activations and weights */
constexpr int GRAD_BLOCKS = 2 * 152;             /* two blocks per SM are resident */
struct GradSmem {
  float w1[NH * NI], w2[NH * GW], w3[NH * GW], w4[NO * NH];
  float b1[NH], b2[NH], b3[NH], b4[4], norm[NNORM];
  float x[NI * GS], a1[NH * GS], a2[NH * GS], a3[NH * GS], dz4[4 * GS];
  double loss[2];
};
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}
/* out[j][i] = tanh(b[j] + sum_k w[j][k] in[k][i]) for four j and two i; samples beyond the batch get 0 */
template <int K, int WS>
__device__ __forceinline__ void grad_layer(const float* w, const float* b, const float* in, float* out, int j0, int i0,
                                           int live) {
  float a[4][2];
#pragma unroll
  for (int r = 0; r < 4; r++) a[r][0] = a[r][1] = b[j0 + r];
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 wr[4];
#pragma unroll
    for (int r = 0; r < 4; r++) wr[r] = *(const float4*)(w + (j0 + r) * WS + k);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const float2 h = *(const float2*)(in + (k + c) * GS + i0);
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float wk = c == 0 ? wr[r].x : c == 1 ? wr[r].y : c == 2 ? wr[r].z : wr[r].w;
        a[r][0] = fmaf(wk, h.x, a[r][0]);
        a[r][1] = fmaf(wk, h.y, a[r][1]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; r++)
    *(float2*)(out + (j0 + r) * GS + i0) =
        make_float2(i0 < live ? tanhf(a[r][0]) : 0.f, i0 + 1 < live ? tanhf(a[r][1]) : 0.f);
}
/* s[k][i] = sum_j dz[j][i] w[j][k] for four k and two i */
template <int J, int WS>
__device__ __forceinline__ void grad_back(const float* w, const float* dz, int k0, int i0, float (&s)[4][2]) {
#pragma unroll
  for (int r = 0; r < 4; r++) s[r][0] = s[r][1] = 0.f;
#pragma unroll 8
  for (int j = 0; j < J; j++) {
    const float4 wr = *(const float4*)(w + j * WS + k0);
    const float2 d = *(const float2*)(dz + j * GS + i0);
    const float wk[4] = {wr.x, wr.y, wr.z, wr.w};
#pragma unroll
    for (int r = 0; r < 4; r++) {
      s[r][0] = fmaf(d.x, wk[r], s[r][0]);
      s[r][1] = fmaf(d.y, wk[r], s[r][1]);
    }
  }
}
/* a = s (1 - a^2), 0 for samples beyond the batch */
__device__ __forceinline__ void grad_act(float* a, int k0, int i0, int live, const float (&s)[4][2]) {
#pragma unroll
  for (int r = 0; r < 4; r++) {
    float2* p = (float2*)(a + (k0 + r) * GS + i0);
    const float2 v = *p;
    *p = make_float2(i0 < live ? s[r][0] * (1.f - v.x * v.x) : 0.f, i0 + 1 < live ? s[r][1] * (1.f - v.y * v.y) : 0.f);
  }
}
/* g[r][c] += sum_i dz[j0 + r][i] a[k0 + 16 c][i] (rows 16 apart: neighbouring lanes read neighbouring rows) */
__device__ __forceinline__ void grad_w(const float* dz, const float* a, int j0, int k0, float (&g)[4][4]) {
#pragma unroll 2
  for (int i = 0; i < GT; i += 4) {
    float4 d[4], v[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      d[r] = *(const float4*)(dz + (j0 + r) * GS + i);
      v[r] = *(const float4*)(a + (k0 + 16 * r) * GS + i);
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) g[r][c] = dot4(d[r], v[c], g[r][c]);
  }
}
__device__ __forceinline__ float row_sum(const float* dz, int j, float s) {
  const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
  for (int i = 0; i < GT; i += 4) s = dot4(*(const float4*)(dz + j * GS + i), one, s);
  return s;
}
template <bool BF16>
__global__ void __launch_bounds__(256, 2)
    k_mlp_grad(const float* __restrict__ params, const float* __restrict__ X, const float* __restrict__ T,
               float* __restrict__ part, double* __restrict__ lpart, int64_t n) {
  extern __shared__ __align__(16) unsigned char grad_smem[];
  GradSmem& s = *reinterpret_cast<GradSmem*>(grad_smem);
  const int t = threadIdx.x;
  for (int e = t; e < NH * NI; e += 256) s.w1[e] = wq<BF16>(params[OFF_W1 + e]);
  for (int e = t; e < NH * NH; e += 256) {
    const int at = (e / NH) * GW + e % NH;
    s.w2[at] = wq<BF16>(params[OFF_W2 + e]);
    s.w3[at] = wq<BF16>(params[OFF_W3 + e]);
  }
  if (t < NO * NH) s.w4[t] = wq<BF16>(params[OFF_W4 + t]);
  if (t < NH) {
    s.b1[t] = params[OFF_B1 + t];
    s.b2[t] = params[OFF_B2 + t];
    s.b3[t] = params[OFF_B3 + t];
  }
  if (t < NO) s.b4[t] = params[OFF_B4 + t];
  if (t < NNORM) s.norm[t] = params[NPARAM + t];
  const float *mx = s.norm, *sx = mx + NI, *my = sx + NI, *sy = my + NO;

  const int q0 = (t >> 4) * 4, i0 = (t & 15) * 2; /* layers: four features, two samples */
  const int j1 = t >> 2, k1 = (t & 3) * 3;        /* first layer's weights: one row, three columns */
  float g2[4][4] = {}, g3[4][4] = {}, g1[3] = {}, g4 = 0.f, gb[3] = {}, gb4 = 0.f;
  double loss = 0.0;
  const int64_t tiles = (n + GT - 1) / GT;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t base = tile * GT;
    const int live = (int)min((int64_t)GT, n - base);
    __syncthreads(); /* the parameters; the tile before */
    for (int e = t; e < GT * NI; e += 256) {
      const int i = e / NI, k = e % NI;
      s.x[k * GS + i] = i < live ? (X[base * NI + e] - mx[k]) / sx[k] : 0.f;
    }
    __syncthreads();
    grad_layer<NI, NI>(s.w1, s.b1, s.x, s.a1, q0, i0, live);
    __syncthreads();
    grad_layer<NH, GW>(s.w2, s.b2, s.a1, s.a2, q0, i0, live);
    __syncthreads();
    grad_layer<NH, GW>(s.w3, s.b3, s.a2, s.a3, q0, i0, live);
    __syncthreads();
    if (t < NO * GT) {
      const int o = t / GT, i = t % GT;
      float y = s.b4[o];
#pragma unroll 16
      for (int k = 0; k < NH; k++) y = fmaf(s.w4[o * NH + k], s.a3[k * GS + i], y);
      float dz = 0.f;
      if (i < live) {
        const float d = y - (T[(base + i) * NO + o] - my[o]) / sy[o];
        dz = 2.f * d / (float)(n * NO);
        loss += (double)d * d;
      }
      s.dz4[o * GS + i] = dz;
    }
    __syncthreads();
    float b[4][2];
    if (t < NO * NH) {
      const float *d = s.dz4 + (t / NH) * GS, *a = s.a3 + (t % NH) * GS;
#pragma unroll
      for (int i = 0; i < GT; i += 4) g4 = dot4(*(const float4*)(d + i), *(const float4*)(a + i), g4);
    } else if (t < NO * NH + NO) {
      gb4 = row_sum(s.dz4, t - NO * NH, gb4);
    }
    grad_back<NO, NH>(s.w4, s.dz4, q0, i0, b);
    __syncthreads();
    grad_act(s.a3, q0, i0, live, b);
    __syncthreads();
    grad_w(s.a3, s.a2, q0, t & 15, g3);
    if (t < NH) gb[2] = row_sum(s.a3, t, gb[2]);
    grad_back<NH, GW>(s.w3, s.a3, q0, i0, b);
    __syncthreads();
    grad_act(s.a2, q0, i0, live, b);
    __syncthreads();
    grad_w(s.a2, s.a1, q0, t & 15, g2);
    if (t < NH) gb[1] = row_sum(s.a2, t, gb[1]);
    grad_back<NH, GW>(s.w2, s.a2, q0, i0, b);
    __syncthreads();
    grad_act(s.a1, q0, i0, live, b);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < GT; i += 4) {
      const float4 d = *(const float4*)(s.a1 + j1 * GS + i);
#pragma unroll
      for (int c = 0; c < 3; c++) g1[c] = dot4(d, *(const float4*)(s.x + (k1 + c) * GS + i), g1[c]);
    }
    if (t < NH) gb[0] = row_sum(s.a1, t, gb[0]);
  }
  float* g = part + (int64_t)blockIdx.x * NPARAM;
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      g[OFF_W2 + (q0 + r) * NH + (t & 15) + 16 * c] = g2[r][c];
      g[OFF_W3 + (q0 + r) * NH + (t & 15) + 16 * c] = g3[r][c];
    }
#pragma unroll
  for (int c = 0; c < 3; c++) g[OFF_W1 + j1 * NI + k1 + c] = g1[c];
  if (t < NO * NH) g[OFF_W4 + t] = g4;
  else if (t < NO * NH + NO) g[OFF_B4 + t - NO * NH] = gb4;
  if (t < NH) {
    g[OFF_B1 + t] = gb[0];
    g[OFF_B2 + t] = gb[1];
    g[OFF_B3 + t] = gb[2];
  }
  if (t < NO * GT) {
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if ((t & 31) == 0) s.loss[t / 32] = loss;
  }
  __syncthreads();
  if (t == 0) lpart[blockIdx.x] = s.loss[0] + s.loss[1];
}

/* The partials of nb blocks added: 32 parameters by 8 shares of the blocks per block,
 * the loss by the first block's first thread row. */
__global__ void __launch_bounds__(256) k_grad_sum(const float* __restrict__ part, const double* __restrict__ lpart,
                                                  int nb, float* __restrict__ g, double* __restrict__ loss) {
  __shared__ float red[8][32];
  const int x = threadIdx.x, y = threadIdx.y, k = blockIdx.x * 32 + x;
  float s = 0.f;
  if (k < NPARAM)
#pragma unroll 8
    for (int b = y; b < nb; b += 8) s += part[(int64_t)b * NPARAM + k];
  red[y][x] = s;
  __syncthreads();
  if (y == 0 && k < NPARAM)
    g[k] = ((red[0][x] + red[1][x]) + (red[2][x] + red[3][x])) + ((red[4][x] + red[5][x]) + (red[6][x] + red[7][x]));
  if (blockIdx.x == 0 && y == 1) {
    double l = 0.0;
    for (int b = x; b < nb; b += 32) l += lpart[b];
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (x == 0) *loss = l;
  }
}

__global__ void k_adam(float* p, const float* g, float* m, float* v, int np, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
    float gk = g[k];
    float mk = b1 * m[k] + (1 - b1) * gk;
    float vk = b2 * v[k] + (1 - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    p[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
  }
}

/* ------------------------------------------------------------------ */
/* seeded MGFM                                                        */
/* ------------------------------------------------------------------ */
/* f(p) of the two-shock relation at p (mpm.cpp:908) */
__device__ __forceinline__ double mgfm_f(double ul, double ur, double pl, double pr, double rhol, double rhor,
                                         double gl, double pinfl, double gr, double pinfr, double p) {
  double Wl = wl_cal(rhol, pl, p, gl, pinfl);
  double Wr = wl_cal(rhor, pr, p, gr, pinfr);
  return ul - ur - (p - pl) / Wl - (p - pr) / Wr;
}

/* the seed from the baseline, the strength scale and the network output; an
 * output far outside the training range that overflows the exponential gives
 * -1, the plain seed */
__device__ __forceinline__ double seed_value(double pb, float sc, float y0, float my0, float sy0) {
  const double ps = pb * (double)expf(sc * (y0 * sy0 + my0));
  if (!isfinite(ps)) return -1.0;
  return ps > 1e-8 ? ps : 1e-8;
}

/* Seeds of a batch: features, network and seed p_b exp(sc y) in one pass per
 * problem; -1 (plain solve) for a problem without a positive root, f(1e-8) < 0,
 * evaluated with the clamps of the MGFM variant (mpm.cpp:886-893). */
template <bool BF16>
__global__ void __launch_bounds__(128) k_seed(const float* __restrict__ params, const double* __restrict__ in6,
                                              const int8_t* __restrict__ mat2, const double* __restrict__ gam,
                                              const double* __restrict__ pinf, int variant, double* __restrict__ seed,
                                              int64_t n) {
  __shared__ __align__(16) float w[NPARAM + NNORM];
  load_params<BF16>(params, w);
  const float* mx = w + NPARAM;
  const float* sx = mx + NI;
  const float my0 = w[NPARAM + 2 * NI], sy0 = w[NPARAM + 2 * NI + NO];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* q = in6 + 6 * i;
    const int s = mat2[2 * i], s1 = mat2[2 * i + 1];
    const double gl = gam[s], il = pinf[s], gr = gam[s1], ir = pinf[s1];
    double pl = q[2], pr = q[3], rl = q[4], rr = q[5];
    if (variant == 0) {
      pl = amax1(pl, 1e-10);
      pr = amax1(pr, 1e-10);
      rl = amax1(rl, 1e-10);
      rr = amax1(rr, 1e-10);
    } else {
      if (pl < 0) pl = 0;
      if (pr < 0) pr = 0;
    }
    if (mgfm_f(q[0], q[1], pl, pr, rl, rr, gl, il, gr, ir, 1e-8) < 0) {
      seed[i] = -1.0;
      continue;
    }
    double pb;
    float sc, xn[NI], y[1];
    mgfm_features(q, gl, il, gr, ir, xn, &pb, &sc);
#pragma unroll
    for (int k = 0; k < NI; k++) xn[k] = (xn[k] - mx[k]) / sx[k];
    mlp_eval<1>(w, xn, y);
    seed[i] = seed_value(pb, sc, y[0], my0, sy0);
  }
}

/* first half of the split seed path: features, baseline and strength scale
 * of each problem (pb < 0 marks a problem without a positive root) */
__global__ void k_seed_features(const double* __restrict__ in6, const int8_t* __restrict__ mat2,
                                const double* __restrict__ gam, const double* __restrict__ pinf, int variant,
                                float* __restrict__ X, double* __restrict__ pb_out, float* __restrict__ sc_out,
                                int64_t n, const unsigned long long* __restrict__ dn) {
  if (dn && (int64_t)*dn < n) n = (int64_t)*dn;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* q = in6 + 6 * i;
    const int s = mat2[2 * i], s1 = mat2[2 * i + 1];
    const double gl = gam[s], il = pinf[s], gr = gam[s1], ir = pinf[s1];
    double pl = q[2], pr = q[3], rl = q[4], rr = q[5];
    if (variant == 0) {
      pl = amax1(pl, 1e-10);
      pr = amax1(pr, 1e-10);
      rl = amax1(rl, 1e-10);
      rr = amax1(rr, 1e-10);
    } else {
      if (pl < 0) pl = 0;
      if (pr < 0) pr = 0;
    }
    if (mgfm_f(q[0], q[1], pl, pr, rl, rr, gl, il, gr, ir, 1e-8) < 0) {
      pb_out[i] = -1.0;
      continue;
    }
    double pb;
    float sc, x[NI];
    mgfm_features(q, gl, il, gr, ir, x, &pb, &sc);
    for (int k = 0; k < NI; k++) X[i * NI + k] = x[k];
    pb_out[i] = pb;
    sc_out[i] = sc;
  }
}

/* partition of a seeded batch by the existence of a positive root (pb > 0):
 * flag[i] = 1 for a problem with a root */
__global__ void k_root_flag(const double* __restrict__ pb, unsigned long long* __restrict__ flag, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flag[i] = pb[i] > 0 ? 1ull : 0ull;
}
/* order: problems with a root first, then the others, each in input order;
 * pos is the exclusive prefix of the flags, nroot_p their total */
__global__ void k_root_perm(const unsigned long long* __restrict__ pos, const unsigned long long* __restrict__ nroot_p,
                            int32_t* __restrict__ perm, int64_t n) {
  const int64_t nroot = (int64_t)*nroot_p;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = (int64_t)pos[i];
    const bool root = (i + 1 < n ? (int64_t)pos[i + 1] : nroot) > p;
    perm[root ? p : nroot + (i - p)] = (int32_t)i;
  }
}

/* Threads per block of the FP64 kernels of the batched solve of n problems.  An
 * FP64 instruction occupies a quarter of an SM for 64 cycles a warp, so the time of a
 * batch that is resident at once is the largest number of warps on any quarter, and
 * blocks of 64 spread it evenly; a larger batch wants all 2048 threads of an SM,
 * which the capped grid reaches with blocks of 256 (1000 problems: 86 us with 64,
 * 130 with 256; 65537: 235 and 257; 2^22: 13.1 ms and 11.8).  A stage of a run knows
 * its room, not its size, and its problems are few and come first, so it takes 64. */
inline int newton_threads(int64_t n, bool stage = false) { return stage || n <= 152 * 1024 ? 64 : 256; }

/* Newton from the seed (or the plain seed when seed is NULL or the entry is
 * negative); a seeded solve that has not converged at the cap is redone from
 * the plain seed, and its iterations are counted together */
__global__ void k_mgfm_seeded(const double* __restrict__ in6, const int8_t* __restrict__ mat2,
                              const double* __restrict__ gam, const double* __restrict__ pinf, int variant,
                              const double* __restrict__ seed, double* __restrict__ out3, int32_t* __restrict__ iters,
                              int64_t n, unsigned long long* stats, const float* __restrict__ Y,
                              const float* __restrict__ sc, const float* __restrict__ params,
                              const int32_t* __restrict__ perm, const int* __restrict__ yerr,
                              const unsigned long long* __restrict__ dn) {
  if (dn && (int64_t)*dn < n) n = (int64_t)*dn;
  unsigned long long nit = 0, nmax = 0, ncall = 0;
  /* a tensor-core forward pass that gave up leaves Y unset: every problem then
   * starts from the plain seed (the reference's), so results stay valid */
  if (yerr && *yerr) Y = nullptr;
  const float my0 = params ? params[NPARAM + 2 * NI] : 0.f, sy0 = params ? params[NPARAM + 2 * NI + NO] : 1.f;
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = perm ? (int64_t)perm[j] : j;
    const double* q = in6 + 6 * i;
    int s = mat2[2 * i], s1 = mat2[2 * i + 1];
    double o[3];
    int it = 0;
    /* seed: given, or (split path) formed from the baseline in seed[], the
     * scale and the network output */
    double sd = seed ? seed[i] : -1.0;
    if (Y && sd > 0) sd = seed_value(sd, sc[i], Y[i * NO], my0, sy0);
    else if (seed && !Y && yerr) sd = -1.0;
    bool done = false;
    if (sd > 0) {
      it = mgfm(q[0], q[1], q[2], q[3], q[4], q[5], gam[s], pinf[s], gam[s1], pinf[s1], variant, sd, o);
      /* a seeded solve is kept only when it converged to finite values (a
       * non-finite iterate fails the tolerance test and would leave the loop
       * early); otherwise the problem is solved again from the plain seed */
      done = it < 50 && isfinite(o[0]) && isfinite(o[1]) && isfinite(o[2]);
    }
    if (!done) it += mgfm(q[0], q[1], q[2], q[3], q[4], q[5], gam[s], pinf[s], gam[s1], pinf[s1], variant, -1.0, o,
                           seed && sd <= 0 ? 1 : 0);
    out3[3 * i + 0] = o[0];
    out3[3 * i + 1] = o[1];
    out3[3 * i + 2] = o[2];
    if (iters) iters[i] = it;
    ncall++;
    nit += it;
    if (it >= 50) nmax++;
  }
  if (stats && ncall) {
    atomicAdd(&stats[0], ncall);
    atomicAdd(&stats[1], nit);
    if (nmax) atomicAdd(&stats[2], nmax);
  }
}

}  // namespace pgdg

/* ---------------------------------------------------------------------- */
/* host side                                                              */
/* ---------------------------------------------------------------------- */
using namespace pgdg;

struct pgdg_mlp {
  int bf16 = 1;
  int tc = 0;           /* forward passes on the tensor cores (BF16 activations) */
  int* d_tcerr = nullptr;
  float* d_params = nullptr; /* NPARAM + NNORM */
  float *d_m = nullptr, *d_v = nullptr;
  float* d_g = nullptr; /* NPARAM gradients, then the sum of squares (a double) */
  double* loss() const { return (double*)(d_g + NPARAM); }
  int64_t step = 0;
  /* gradients: the blocks' partial sums, of a fixed size whatever the batch */
  float* g_part = nullptr;
  double* l_part = nullptr;
  PartScratch part;         /* root partition of batched solves */
  double* seeds = nullptr; /* per-problem seeds (or baselines) of batched solves */
  float* sc = nullptr;     /* per-problem strength scale of the split seed path */
  float *Xb = nullptr, *Yb = nullptr; /* features and network outputs of batched solves */
  int64_t seeds_cap = 0;
  int reserve_seeds(int64_t n) {
    if (n <= seeds_cap) return PGDG_OK;
    void** bufs[] = {(void**)&seeds, (void**)&sc, (void**)&Xb, (void**)&Yb};
    const size_t w[] = {sizeof(double), sizeof(float), sizeof(float) * NI, sizeof(float) * NO};
    seeds_cap = 0;
    for (int k = 0; k < 4; k++) {
      if (*bufs[k]) cudaFree(*bufs[k]);
      *bufs[k] = nullptr;
      if (cudaMalloc(bufs[k], w[k] * (size_t)n) != cudaSuccess) return PGDG_ENOMEM;
    }
    seeds_cap = n;
    return PGDG_OK;
  }
  int reserve_grad() {
    if (!g_part && cudaMalloc((void**)&g_part, sizeof(float) * NPARAM * GRAD_BLOCKS) != cudaSuccess) return PGDG_ENOMEM;
    if (!l_part && cudaMalloc((void**)&l_part, sizeof(double) * GRAD_BLOCKS) != cudaSuccess) return PGDG_ENOMEM;
    return PGDG_OK;
  }
  ~pgdg_mlp() {
    float* bufs[] = {d_params, d_m, d_v, d_g, g_part};
    for (float* b : bufs)
      if (b) cudaFree(b);
    if (l_part) cudaFree(l_part);
    if (seeds) cudaFree(seeds);
    if (sc) cudaFree(sc);
    if (Xb) cudaFree(Xb);
    if (Yb) cudaFree(Yb);
    if (d_tcerr) cudaFree(d_tcerr);
    part.release();
  }
};

namespace {
inline int g_for(int64_t n, int b) {
  int64_t g = (n + b - 1) / b;
  if (g > 152 * 16) g = 152 * 16;
  return g < 1 ? 1 : (int)g;
}
void forward(pgdg_mlp* m, const float* X, float* Y, int64_t n, cudaStream_t st,
             const unsigned long long* dn = nullptr) {
  if (m->tc) {
    /* the flag reports this forward pass only */
    cudaMemsetAsync(m->d_tcerr, 0, sizeof(int), st);
    mlp_tc_forward(m->d_params, X, Y, n, m->d_tcerr, st, dn);
    return;
  }
  if (m->bf16) k_mlp_forward<true><<<g_for(n, 128), 128, 0, st>>>(m->d_params, X, Y, n, dn);
  else k_mlp_forward<false><<<g_for(n, 128), 128, 0, st>>>(m->d_params, X, Y, n, dn);
}
void seed_launch(pgdg_mlp* m, const double* in6, const int8_t* mat2, const double* gam, const double* pinf,
                 int variant, double* seed, int64_t n, cudaStream_t st) {
  if (m->bf16) k_seed<true><<<g_for(n, 128), 128, 0, st>>>(m->d_params, in6, mat2, gam, pinf, variant, seed, n);
  else k_seed<false><<<g_for(n, 128), 128, 0, st>>>(m->d_params, in6, mat2, gam, pinf, variant, seed, n);
}
/* gradient of the mean squared error of the normalised outputs, and its sum of squares, into m->d_g */
template <bool BF16>
cudaError_t gradients(pgdg_mlp* m, const float* X, const float* T, int64_t n, cudaStream_t st) {
  const cudaError_t e =
      cudaFuncSetAttribute(k_mlp_grad<BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem));
  if (e != cudaSuccess) return e;
  const int64_t tiles = (n + GT - 1) / GT;
  const int nb = tiles < 1 ? 1 : tiles > GRAD_BLOCKS ? GRAD_BLOCKS : (int)tiles;
  k_mlp_grad<BF16><<<nb, 256, sizeof(GradSmem), st>>>(m->d_params, X, T, m->g_part, m->l_part, n);
  k_grad_sum<<<(NPARAM + 31) / 32, dim3(32, 8), 0, st>>>(m->g_part, m->l_part, nb, m->d_g, m->loss());
  return cudaGetLastError();
}
int gradients(pgdg_mlp* m, const float* X, const float* T, int64_t n, cudaStream_t st) {
  const int rc = m->reserve_grad();
  if (rc) return rc;
  return (m->bf16 ? gradients<true>(m, X, T, n, st) : gradients<false>(m, X, T, n, st)) == cudaSuccess ? PGDG_OK
                                                                                                       : PGDG_ECUDA;
}
}  // namespace

extern "C" {

int pgdg_surrogate_create(int bf16, pgdg_mlp** out) {
  int dev = 0;
  if (cudaGetDeviceCount(&dev) != cudaSuccess || dev < 1) return PGDG_ECUDA;
  if (bf16 < 0 || bf16 > 2) return PGDG_EINVAL;
  pgdg_mlp* m = new pgdg_mlp();
  m->bf16 = bf16 ? 1 : 0;
  m->tc = bf16 == 2 ? 1 : 0;
  if (cudaMalloc((void**)&m->d_tcerr, sizeof(int)) != cudaSuccess) {
    delete m;
    return PGDG_ENOMEM;
  }
  cudaMemset(m->d_tcerr, 0, sizeof(int));
  const size_t np = NPARAM + NNORM;
  if (cudaMalloc((void**)&m->d_params, sizeof(float) * np) != cudaSuccess ||
      cudaMalloc((void**)&m->d_m, sizeof(float) * NPARAM) != cudaSuccess ||
      cudaMalloc((void**)&m->d_v, sizeof(float) * NPARAM) != cudaSuccess ||
      cudaMalloc((void**)&m->d_g, sizeof(float) * NPARAM + sizeof(double)) != cudaSuccess) {
    delete m;
    return PGDG_ENOMEM;
  }
  cudaMemset(m->d_params, 0, sizeof(float) * np);
  cudaMemset(m->d_m, 0, sizeof(float) * NPARAM);
  cudaMemset(m->d_v, 0, sizeof(float) * NPARAM);
  *out = m;
  return PGDG_OK;
}
int pgdg_surrogate_destroy(pgdg_mlp* m) {
  delete m;
  return PGDG_OK;
}
int pgdg_surrogate_num_params(void) { return NPARAM + NNORM; }
/* host arrays of NPARAM + NNORM floats */
int pgdg_surrogate_set_params(pgdg_mlp* m, const float* params) {
  return cudaMemcpy(m->d_params, params, sizeof(float) * (NPARAM + NNORM), cudaMemcpyHostToDevice) == cudaSuccess
             ? PGDG_OK : PGDG_ECUDA;
}
int pgdg_surrogate_get_params(pgdg_mlp* m, float* params) {
  return cudaMemcpy(params, m->d_params, sizeof(float) * (NPARAM + NNORM), cudaMemcpyDeviceToHost) == cudaSuccess
             ? PGDG_OK : PGDG_ECUDA;
}
/* device pointers: in6 [n][6], mat2 [n][2], gam/pinf [nmat] -> X [n][12] */
int pgdg_surrogate_features(const double* in6, const int8_t* mat2, const double* gam, const double* pinf,
                            float* X, int64_t n) {
  if (n <= 0) return PGDG_OK;
  k_features<<<g_for(n, 256), 256>>>(in6, mat2, gam, pinf, X, n);
  return cudaGetLastError() == cudaSuccess ? PGDG_OK : PGDG_ECUDA;
}
/* device pointers: X [n][12] raw features -> Y [n][2] normalised outputs */
int pgdg_surrogate_forward(pgdg_mlp* m, const float* X, float* Y, int64_t n) {
  if (n <= 0) return PGDG_OK;
  forward(m, X, Y, n, 0);
  if (cudaGetLastError() != cudaSuccess) return PGDG_ECUDA;
  if (m->tc) {
    int e = 0;
    if (cudaMemcpy(&e, m->d_tcerr, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return PGDG_ECUDA;
    if (e) return PGDG_ETIMEOUT;
  }
  return PGDG_OK;
}
/* gradient of the loss 1/(2n) sum |Y - normalise(T)|^2 ... returned to the host
 * (NPARAM floats) together with the loss */
int pgdg_surrogate_gradients(pgdg_mlp* m, const float* X, const float* T, int64_t n, float* grad_host,
                             double* loss) {
  int rc = gradients(m, X, T, n, 0);
  if (rc) return rc;
  /* gradient and loss in one copy */
  unsigned char out[sizeof(float) * NPARAM + sizeof(double)];
  if (cudaMemcpy(out, m->d_g, sizeof(out), cudaMemcpyDeviceToHost) != cudaSuccess) return PGDG_ECUDA;
  double l;
  memcpy(&l, out + sizeof(float) * NPARAM, sizeof(l));
  if (loss) *loss = l / (double)(n * NO);
  if (grad_host) memcpy(grad_host, out, sizeof(float) * NPARAM);
  return PGDG_OK;
}
/* one Adam step on a batch (device pointers) */
int pgdg_surrogate_train_step(pgdg_mlp* m, const float* X, const float* T, int64_t n, float lr, double* loss) {
  int rc = gradients(m, X, T, n, 0);
  if (rc) return rc;
  m->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  float c1 = 1.f - powf(b1, (float)m->step), c2 = 1.f - powf(b2, (float)m->step);
  k_adam<<<g_for(NPARAM, 256), 256>>>(m->d_params, m->d_g, m->d_m, m->d_v, NPARAM, lr, b1, b2, 1e-8f, c1, c2);
  if (loss) {
    double l = 0;
    cudaMemcpy(&l, m->loss(), sizeof(double), cudaMemcpyDeviceToHost);
    *loss = l / (double)(n * NO);
  }
  return cudaGetLastError() == cudaSuccess ? PGDG_OK : PGDG_ECUDA;
}

/* batched MGFM (mpm.cpp:882-926) on device buffers; net == NULL: the reference's
 * plain seed; otherwise the surrogate seed with the plain solve as fallback */
int pgdg_mgfm_batched(const pgdg_mlp* net, const double* in6, const int8_t* mat2, const double* gam,
                      const double* pinf, int nmat, int variant, double* out3, int32_t* iters, int64_t n) {
  if (n < 0 || !in6 || !mat2 || !gam || !pinf || !out3 || nmat < 1) return PGDG_EINVAL;
  if (n == 0) return PGDG_OK;
  /* the partition scratch is the network's; plain solves need none */
  return mgfm_seeded_run((void*)net, in6, mat2, gam, pinf, variant, out3, iters, n, nullptr,
                         net ? &const_cast<pgdg_mlp*>(net)->part : nullptr, 0, nullptr);
}

/* Seeds of pgdg_mgfm_batched_noalloc: a file-scope device array, so the call
 * itself never allocates (see the declaration for which callers need that).
 * Its address is looked up once per device. */
static __device__ __align__(256) double g_noalloc_seeds[PGDG_MGFM_NOALLOC_MAX];

int pgdg_mgfm_batched_noalloc(const pgdg_mlp* net, const double* in6, const int8_t* mat2, const double* gam,
                              const double* pinf, int nmat, int variant, double* out3, int32_t* iters, int64_t n) {
  if (n < 0 || !in6 || !mat2 || !gam || !pinf || !out3 || nmat < 1) return PGDG_EINVAL;
  if (n > PGDG_MGFM_NOALLOC_MAX) return PGDG_EOVERFLOW;
  if (net && net->tc) return PGDG_EINVAL; /* its seeds come from the SIMT network only */
  if (n == 0) return PGDG_OK;
  const double* sd = nullptr;
  if (net) {
    constexpr int MAXDEV = 64;
    static double* seeds_of[MAXDEV] = {};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAXDEV) return PGDG_ECUDA;
    double* seeds = nullptr;
    {
      std::lock_guard<std::mutex> lk(mu);
      if (!seeds_of[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_seeds) != cudaSuccess || !p) return PGDG_ECUDA;
        seeds_of[dev] = static_cast<double*>(p);
      }
      seeds = seeds_of[dev];
    }
    seed_launch(const_cast<pgdg_mlp*>(net), in6, mat2, gam, pinf, variant, seeds, n, 0);
    sd = seeds;
  }
  k_mgfm_seeded<<<g_for(n, newton_threads(n)), newton_threads(n)>>>(in6, mat2, gam, pinf, variant, sd, out3, iters, n, nullptr, nullptr, nullptr,
                                        nullptr, nullptr, nullptr, nullptr);
  return cudaGetLastError() == cudaSuccess ? PGDG_OK : PGDG_ECUDA;
}

}  // extern "C"

namespace pgdg {
int PartScratch::reserve(int64_t n) {
  if (n <= cap) return PGDG_OK;
  if (pos) cudaFree(pos);
  if (blk) cudaFree(blk);
  if (perm) cudaFree(perm);
  if (dn) cudaFree(dn);
  pos = blk = dn = nullptr;
  perm = nullptr;
  cap = 0;
  if (cudaMalloc((void**)&pos, sizeof(unsigned long long) * (size_t)(n + 1)) != cudaSuccess ||
      cudaMalloc((void**)&blk, sizeof(unsigned long long) * (size_t)(n / 2048 + 2)) != cudaSuccess ||
      cudaMalloc((void**)&perm, sizeof(int32_t) * (size_t)n) != cudaSuccess ||
      cudaMalloc((void**)&dn, sizeof(unsigned long long)) != cudaSuccess)
    return PGDG_ENOMEM;
  cap = n;
  return PGDG_OK;
}
void PartScratch::release() {
  if (pos) cudaFree(pos);
  if (blk) cudaFree(blk);
  if (perm) cudaFree(perm);
  if (dn) cudaFree(dn);
  pos = blk = dn = nullptr;
  perm = nullptr;
  cap = 0;
}

int mgfm_seeded_reserve(void* netv, int64_t n) {
  return netv ? static_cast<pgdg_mlp*>(netv)->reserve_seeds(n) : PGDG_OK;
}

int mgfm_seeded_run(void* netv, const double* in6, const int8_t* mat2, const double* gam, const double* pinf,
                    int variant, double* out3, int32_t* iters, int64_t n, unsigned long long* stats,
                    PartScratch* ps, cudaStream_t st, const unsigned long long* dn) {
  if (n <= 0) return PGDG_OK;
  if (n > INT32_MAX) return PGDG_EINVAL;
  pgdg_mlp* m = static_cast<pgdg_mlp*>(netv);
  const double* sd = nullptr;
  const int nt = newton_threads(n, dn != nullptr);
  if (m) {
    /* split seed path: features and baseline, the network, then Newton with the
     * seed formed per problem (same arithmetic as the fused k_seed) */
    const int rc = m->reserve_seeds(n);
    if (rc) return rc;
    k_seed_features<<<g_for(n, nt), nt, 0, st>>>(in6, mat2, gam, pinf, variant, m->Xb, m->seeds, m->sc, n, dn);
    forward(m, m->Xb, m->Yb, n, st, dn);
    sd = m->seeds;
  }
  /* A problem without a root takes about as long as one with a root from the plain
   * seed (mgfm replays its descent), so plain solves are one launch: 2^22 problems
   * 17.3 -> 11.8 ms, 65537 problems 495 -> 235 us.  Seeded, it takes about six
   * iterations and the others two, and a batch is sorted, problems with a root
   * first: 2^22 problems 10.9 -> 5.9 ms; at 65537 217 us sorted and 242 unsorted, at
   * 1000 111 and 103.  A stage of a run (dn) is not sorted: nearly all its problems
   * have a root. */
  const bool sorted = m && ps && !dn && n > 16384;
  if (!sorted) {
    k_mgfm_seeded<<<g_for(n, nt), nt, 0, st>>>(in6, mat2, gam, pinf, variant, sd, out3, iters, n, stats,
                                                 m ? m->Yb : nullptr, m ? m->sc : nullptr, m ? m->d_params : nullptr,
                                                 nullptr, m && m->tc ? m->d_tcerr : nullptr, dn);
    return cudaGetLastError() == cudaSuccess ? PGDG_OK : PGDG_ECUDA;
  }
  const int rc = ps->reserve(n);
  if (rc) return rc;
  const unsigned long long nn = (unsigned long long)n;
  cudaMemcpyAsync(ps->dn, &nn, sizeof(nn), cudaMemcpyHostToDevice, st);
  k_root_flag<<<g_for(n, 256), 256, 0, st>>>(sd, ps->pos, n);
  scan_u64(ps->pos, ps->blk, ps->dn, n, st);
  k_root_perm<<<g_for(n, 256), 256, 0, st>>>(ps->pos, ps->blk + (n + 2047) / 2048, ps->perm, n);
  k_mgfm_seeded<<<g_for(n, nt), nt, 0, st>>>(in6, mat2, gam, pinf, variant, sd, out3, iters, n, stats,
                                               m->Yb, m->sc, m->d_params, ps->perm, m->tc ? m->d_tcerr : nullptr, nullptr);
  return cudaGetLastError() == cudaSuccess ? PGDG_OK : PGDG_ECUDA;
}
}  // namespace pgdg
