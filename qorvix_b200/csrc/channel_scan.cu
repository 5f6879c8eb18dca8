// Recurrences whose decay is a vector over the key channels, with or without the delta rule's removal term:
//
//   S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T,      y_t = S_t^T q_t * q_scale
//
// per request and head, S [dk x dv] float32 in the request's state slot, both first terms reading the old state.
// Without removal (au, u null) this is gated linear attention's S_t = diag(w_t) S_(t-1) + k_t v_t^T.
//
// qv_channel_gates    per-channel factors from a low-rank pre-activation: z = W2 f(x1) + b, then
//                       POW_SIGMOID      sigmoid(z)^p                  (a decay with temperature 1/p)
//                       EXP_NEG_SIGMOID  exp(-p * sigmoid(z))          (a decay bounded below by exp(-p))
//                       EXP_NEG_SOFTPLUS exp(-rate_c * softplus(z))    (a step size times a rate per channel)
//                       LINEAR           z                             (a pre-activation for a later kernel)
//                     f the identity or tanh.
// qv_unit_keys        u = k / sqrt(sum(k^2) + eps) per head and au = sigmoid(a + bias) * u.
// qv_channel_scan     the recurrence.  The columns of S are independent of one another: a few lanes own a column, each a run of
//                     its rows in registers, so u^T S and S^T q are short sums in a fixed order; the warps of a CTA share the
//                     tokens' vectors, which arrive in shared memory by cp.async a chunk ahead.  Only u^T S lies on the chain
//                     from token to token.
// qv_head_norm_gate   the unit norm per head (RMS over a head's values) with weight, gate (sigmoid or SiLU, behind the norm)
//                     and a fixed factor that follows a scan.
//
// Everything is float32: the inputs are column slices of float32 products (row strides given), the state, the
// factors and all sums.  The order of every sum depends on the sizes alone, so a token's result does not depend
// on how its request was cut into steps or on what else is in the batch.
#include "common.cuh"
#include "per_device.h"
#include "portion_rounds.h"

#define GATE_POW_SIGMOID 0
#define GATE_EXP_NEG_SIGMOID 1
#define GATE_EXP_NEG_SOFTPLUS 2
#define GATE_LINEAR 3

// x1 [T, R] (row stride ld_x), W2 transposed [R, N] float32, bias [N] or null -> out [T, N] (row stride ld_out).
// A CTA takes CG_TOKENS tokens and CG_CHANNELS channels, so that an entry of W2 is read once for all of its tokens; the sum over r
// is cut into four quarters (r ascending in each, by four groups of threads) that are added in order, so that a step of
// few tokens still has many loads in flight and the order of a sum depends on R alone.
// Portions take 16 tokens a CTA and, where R is a multiple of 16, read a token's row four entries at a time (one shared-memory read a
// multiply-add: 47 us for 1,531 tokens x 64 x 2,048, which now take the tiles below; 38 so).  The order of a sum is the same.
struct CgForm { int kind; float p; const float* rate; };
__device__ __forceinline__ float cg_gate(float zz, const CgForm& f, int c) {
  if (f.kind == GATE_POW_SIGMOID) return expf(f.p * (fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)))));             // log sigmoid(z)
  if (f.kind == GATE_EXP_NEG_SIGMOID) return expf(-f.p * (1.0f / (1.0f + expf(-zz))));
  if (f.kind == GATE_EXP_NEG_SOFTPLUS) return expf(-f.rate[c] * (fmaxf(zz, 0.f) + log1pf(expf(-fabsf(zz)))));  // softplus(z)
  return zz;
}

#define CG_CHANNELS 64
template <int CG_TOKENS>
__global__ void __launch_bounds__(4 * CG_CHANNELS) channel_gates_kernel(float* __restrict__ out, int ld_out, const float* __restrict__ x1,
                                                                       int ld_x, const float* __restrict__ w2t,
                                                                       const float* __restrict__ bias, int T, int N, int R,
                                                                       int pre_tanh, CgForm form) {
  extern __shared__ __align__(16) float cg_smem[]; // [CG_TOKENS][R] the tokens' low-rank rows, then [4][CG_TOKENS][CG_CHANNELS] partial sums
  float* xs = cg_smem;
  float* part = cg_smem + CG_TOKENS * R;
  pdl_wait();
  pdl_launch_dependents();
  const int t0 = blockIdx.x * CG_TOKENS;
  const int nt = min(CG_TOKENS, T - t0);
  for (int i = threadIdx.x; i < CG_TOKENS * R; i += blockDim.x) {
    const int j = i / R, r = i % R;
    float v = 0.f;
    if (j < nt) {
      v = x1[(size_t)(t0 + j) * ld_x + r];
      if (pre_tanh) v = tanhf(v);
    }
    xs[i] = v;
  }
  __syncthreads();
  const int cq = threadIdx.x / CG_CHANNELS, cl = threadIdx.x % CG_CHANNELS;
  const int c = blockIdx.y * CG_CHANNELS + cl;
  const int rq = (R + 3) / 4;
  const int r_lo = cq * rq, r_hi = min(R, r_lo + rq);
  float z[CG_TOKENS];
#pragma unroll
  for (int j = 0; j < CG_TOKENS; ++j) z[j] = 0.f;
  if (c < N && (R & 15) == 0) {
#pragma unroll 2
    for (int r = r_lo; r < r_hi; r += 4) {
      float wv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) wv[k] = w2t[(size_t)(r + k) * N + c];
#pragma unroll
      for (int j = 0; j < CG_TOKENS; ++j) {
        const float4 x = *(const float4*)(xs + j * R + r);
        z[j] = fmaf(x.x, wv[0], z[j]);
        z[j] = fmaf(x.y, wv[1], z[j]);
        z[j] = fmaf(x.z, wv[2], z[j]);
        z[j] = fmaf(x.w, wv[3], z[j]);
      }
    }
  } else if (c < N) {
#pragma unroll 8
    for (int r = r_lo; r < r_hi; ++r) {
      const float wv = w2t[(size_t)r * N + c];
#pragma unroll
      for (int j = 0; j < CG_TOKENS; ++j) z[j] = fmaf(xs[j * R + r], wv, z[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < CG_TOKENS; ++j) part[(cq * CG_TOKENS + j) * CG_CHANNELS + cl] = z[j];
  __syncthreads();
  if (c >= N) return;
  const float bc = bias ? bias[c] : 0.f;
  for (int j = cq; j < nt; j += 4) {               // the four groups share the tokens' last step
    float zz = part[j * CG_CHANNELS + cl];
#pragma unroll
    for (int q = 1; q < 4; ++q) zz += part[(q * CG_TOKENS + j) * CG_CHANNELS + cl];
    zz += bc;
    out[(size_t)(t0 + j) * ld_out + c] = cg_gate(zz, form, c);
  }
}

// Portions of many tokens with ranks in whole 16s: a tile of 64 tokens x 64 channels a CTA, 8 x 4 of them a thread, whose sums stay in registers (the
// kernel above has a multiply-add for each entry of x it reads, and meets in shared memory): 1,531 tokens x 64 x 2,048 with softplus 37 us
// above, 28 here (without a function 30 and 21; see qv_channel_gates_tiles); bound by the multiply-adds and the gates' functions.  The same sums in the same order: four quarters of a row, added in
// order.
#define CT_TOKENS 64
#define CT_MAX_RANK 128
__global__ void __launch_bounds__(128, 5) channel_gates_tile_kernel(float* __restrict__ out, int ld_out, const float* __restrict__ x1, int ld_x,
                                                                 const float* __restrict__ w2t, const float* __restrict__ bias, int T, int N, int R,
                                                                 int pre_tanh, CgForm form) {
  extern __shared__ __align__(16) float cg_smem[];   // [64 tokens][R + 4], [R][64 channels]
  const int ldx = R + 4;
  float* xs = cg_smem;
  float* wsm = xs + CT_TOKENS * ldx;
  const int tid = threadIdx.x, c0 = blockIdx.y * CG_CHANNELS, t0 = blockIdx.x * CT_TOKENS;
  pdl_wait();
  pdl_launch_dependents();
  if (N % 4 == 0 && ((uintptr_t)w2t & 15) == 0 && c0 + CG_CHANNELS <= N) {
#pragma unroll 8
    for (int i = tid * 4; i < R * CG_CHANNELS; i += 512) *(float4*)(wsm + i) = *(const float4*)(w2t + (size_t)(i / CG_CHANNELS) * N + c0 + i % CG_CHANNELS);
  } else {
#pragma unroll 8
    for (int i = tid; i < R * CG_CHANNELS; i += 128) {
      const int r = i / CG_CHANNELS, c = c0 + i % CG_CHANNELS;
      wsm[i] = c < N ? w2t[(size_t)r * N + c] : 0.f;
    }
  }
  for (int r = tid & 31; r < R; r += 32) {           // a token a warp
    const float* xp = x1 + (size_t)t0 * ld_x + r;
#pragma unroll 16
    for (int j = tid >> 5; j < CT_TOKENS; j += 4) {
      float v = t0 + j < T ? xp[(size_t)j * ld_x] : 0.f;
      if (pre_tanh) v = tanhf(v);
      xs[j * ldx + r] = v;
    }
  }
  __syncthreads();
  const int cl = (tid & 15) * 4, tl = (tid >> 4) * 8;
  float z[8][4] = {};
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    float part[8][4] = {};
#pragma unroll 1
    for (int r = q * (R >> 2); r < (q + 1) * (R >> 2); r += 4) {
      float w[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float4 v = *(const float4*)(wsm + (r + k) * CG_CHANNELS + cl);
        w[k][0] = v.x; w[k][1] = v.y; w[k][2] = v.z; w[k][3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 x = *(const float4*)(xs + (tl + j) * ldx + r);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          part[j][c] = fmaf(x.x, w[0][c], part[j][c]);
          part[j][c] = fmaf(x.y, w[1][c], part[j][c]);
          part[j][c] = fmaf(x.z, w[2][c], part[j][c]);
          part[j][c] = fmaf(x.w, w[3][c], part[j][c]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) z[j][c] += part[j][c];
  }
  // the gates' functions in a loop over the tile in shared memory: written out for a thread's 32 sums they are more code than the
  // instruction cache holds
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) *(float4*)(cg_smem + (tl + j) * (CG_CHANNELS + 4) + cl) = make_float4(z[j][0], z[j][1], z[j][2], z[j][3]);
  __syncthreads();
  const int c = c0 + (tid & 63);
  if (c >= N) return;
  const float bc = bias ? bias[c] : 0.f;
  const int last = T - t0 < CT_TOKENS ? T - t0 : CT_TOKENS;
  float* o = out + (size_t)t0 * ld_out + c;
#pragma unroll 2
  for (int j = tid >> 6; j < last; j += 2) o[(size_t)j * ld_out] = cg_gate(cg_smem[j * (CG_CHANNELS + 4) + (tid & 63)] + bc, form, c);
}

// Whether the tiles take a portion: ranks in whole 16s that fit, and tiles enough to hide their loads and functions behind one another: a tile
// has four times the work in a row that a CTA of the other kernel has.  us with the other kernel and with the tiles (rows in L2): 64 tiles of
// rank 64 5.2 and 9.7 with softplus (without a function 4.7 and 6.9); 256 tiles 12.7 and 11.6 (11.2 and 8.4), of rank 16 6.9 and 7.9
// (5.5 and 4.8); 320 of rank 32 0.99 of the other kernel's time; 512 of rank 16 12.3 and 12.6; 1,024 of rank 64 43 and 28 (38 and 21).
extern "C" int qv_channel_gates_tiles(int T, int N, int R, int kind) {
  const long long tiles = (long long)((T + CT_TOKENS - 1) / CT_TOKENS) * ((N + CG_CHANNELS - 1) / CG_CHANNELS);
  return T >= 256 && R % 16 == 0 && R <= CT_MAX_RANK && tiles >= (kind == GATE_LINEAR ? 256 : R >= 32 ? 320 : 640);
}

// rate [N] float32: the factor per channel of GATE_EXP_NEG_SOFTPLUS (null for the other kinds).
extern "C" int qv_channel_gates(float* out, int ld_out, const float* x1, int ld_x, const float* w2t, const float* bias, int T, int N,
                                int R, int pre_tanh, int kind, float p, const float* rate, void* stream) {
  if (T <= 0 || N <= 0) return 0;
  const size_t smem8 = ((size_t)8 * R + 4 * 8 * CG_CHANNELS) * sizeof(float);
  if (R <= 0 || smem8 > 48 * 1024) return QV_ERR_UNSUPPORTED;
  const int tokens = T >= 256 && 2 * smem8 <= 48 * 1024 ? 16 : 8;
  const size_t smem = tokens == 16 ? 2 * smem8 : smem8;
  if (kind < GATE_POW_SIGMOID || kind > GATE_LINEAR || (kind == GATE_EXP_NEG_SOFTPLUS && rate == nullptr)) return QV_ERR_UNSUPPORTED;
  const int by = (N + CG_CHANNELS - 1) / CG_CHANNELS;
  if (by > 65535) return QV_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  const CgForm form = {kind, p, rate};
  if (qv_channel_gates_tiles(T, N, R, kind)) {
    static PerDevice allowed;
    const int rc = qv_allow_smem(channel_gates_tile_kernel, (CT_TOKENS * (CT_MAX_RANK + 4) + CT_MAX_RANK * CG_CHANNELS) * 4, allowed);
    if (rc) return rc;
    return qv_launch(channel_gates_tile_kernel, dim3((T + CT_TOKENS - 1) / CT_TOKENS, by), dim3(128),
                     (size_t)(CT_TOKENS * (R + 4) + R * CG_CHANNELS) * 4 + (R < 48 ? CT_TOKENS * (CG_CHANNELS + 4) * 4 : 0), st, out, ld_out, x1, ld_x, w2t, bias, T, N, R, pre_tanh, form);
  }
  const int per = 65535 * tokens;
  for (int done = 0; done < T; done += per) {
    const int rows = T - done < per ? T - done : per;
    const int rc = qv_launch(tokens == 16 ? channel_gates_kernel<16> : channel_gates_kernel<8>, dim3((rows + tokens - 1) / tokens, by), dim3(4 * CG_CHANNELS), smem, st,
                             out + (size_t)done * ld_out, ld_out, x1 + (size_t)done * ld_x, ld_x, w2t, bias, rows, N, R, pre_tanh, form);
    if (rc) return rc;
  }
  return 0;
}

// k, a [T, H * n] float32 (row strides) -> u, au [T, H * n] dense.  One warp per (token, head).
__global__ void __launch_bounds__(128) unit_keys_kernel(float* __restrict__ u, float* __restrict__ au, const float* __restrict__ k, int ld_k,
                                                       const float* __restrict__ a, int ld_a, const float* __restrict__ a_bias, int H, int n,
                                                       float eps) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= H) return;
  const float* kr = k + (size_t)t * ld_k + (size_t)h * n;
  const float* ar = a + (size_t)t * ld_a + (size_t)h * n;
  float ss = 0.f;
  for (int i = lane; i < n; i += 32) ss = fmaf(kr[i], kr[i], ss);
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss + eps);
  const size_t o = ((size_t)t * H + h) * n;
  for (int i = lane; i < n; i += 32) {
    const float uu = kr[i] * inv;
    const float z = ar[i] + (a_bias ? a_bias[(size_t)h * n + i] : 0.f);
    u[o + i] = uu;
    au[o + i] = uu * (1.0f / (1.0f + expf(-z)));
  }
}

extern "C" int qv_unit_keys(float* u, float* au, const float* k, int ld_k, const float* a, int ld_a, const float* a_bias, int T, int H,
                            int n, float eps, void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || n <= 0) return QV_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  for (int done = 0; done < T; done += 65535) {
    const int rows = T - done < 65535 ? T - done : 65535;
    const int rc = qv_launch(unit_keys_kernel, dim3(rows, (H + 3) / 4), dim3(128), 0, st, u + (size_t)done * H * n,
                             au + (size_t)done * H * n, k + (size_t)done * ld_k, ld_k, a + (size_t)done * ld_a, ld_a, a_bias, H, n, eps);
    if (rc) return rc;
  }
  return 0;
}

// The operands of the delta rule whose removal reads the decayed state,
//   S' = diag(g) S,  S = S' + k (beta (v - S'^T k))^T = diag(g) S - (beta k) ((g * k)^T S) + (beta k) v^T,
// in the scan's terms: w = g, u = g * k, au = beta k and the written key beta k, with k and q unit vectors per head
// (x / sqrt(sum x^2 + eps)) and q times q_scale.  q, k [T, G * n] float32 (row strides; head h reads group h / (H / G)),
// b [T, H] the pre-activation of beta = sigmoid(b), g [T, H * n] -> qh, kb, ug dense [T, H * n].  One warp per (token, head).
__global__ void __launch_bounds__(128) delta_operands_kernel(float* __restrict__ qh, float* __restrict__ kb, float* __restrict__ ug,
                                                            const float* __restrict__ q, int ld_q, const float* __restrict__ k, int ld_k,
                                                            const float* __restrict__ b, int ld_b, const float* __restrict__ g, int ld_g,
                                                            int H, int G, int n, float eps, float q_scale) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= H) return;
  const int grp = h / (H / G);
  const float* qr = q + (size_t)t * ld_q + (size_t)grp * n;
  const float* kr = k + (size_t)t * ld_k + (size_t)grp * n;
  const float* gr = g + (size_t)t * ld_g + (size_t)h * n;
  float sq = 0.f, sk = 0.f;
  for (int i = lane; i < n; i += 32) { sq = fmaf(qr[i], qr[i], sq); sk = fmaf(kr[i], kr[i], sk); }
  sq = warp_sum(sq);
  sk = warp_sum(sk);
  const float iq = q_scale / sqrtf(sq + eps), ik = 1.0f / sqrtf(sk + eps);
  const float beta = 1.0f / (1.0f + expf(-b[(size_t)t * ld_b + h]));
  const size_t o = ((size_t)t * H + h) * n;
  for (int i = lane; i < n; i += 32) {
    const float kk = kr[i] * ik;
    qh[o + i] = qr[i] * iq;
    kb[o + i] = beta * kk;
    ug[o + i] = gr[i] * kk;
  }
}

extern "C" int qv_delta_operands(float* qh, float* kb, float* ug, const float* q, int ld_q, const float* k, int ld_k, const float* b,
                                 int ld_b, const float* g, int ld_g, int T, int H, int G, int n, float eps, float q_scale, void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || n <= 0) return QV_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  for (int done = 0; done < T; done += 65535) {
    const int rows = T - done < 65535 ? T - done : 65535;
    const size_t o = (size_t)done * H * n;
    const int rc = qv_launch(delta_operands_kernel, dim3(rows, (H + 3) / 4), dim3(128), 0, st, qh + o, kb + o, ug + o,
                             q + (size_t)done * ld_q, ld_q, k + (size_t)done * ld_k, ld_k, b + (size_t)done * ld_b, ld_b,
                             g + (size_t)done * ld_g, ld_g, H, G, n, eps, q_scale);
    if (rc) return rc;
  }
  return 0;
}

// ---------------------------------------------------------------- the scan
// A column of S belongs to LPC lanes that hold CS_ROWS rows each (rows lic * CS_ROWS ..), so LPC = 1, 2, 4, 8, 16 serves key
// sizes up to 16, 32, 64, 128, 256; a warp holds 32 / LPC columns, a CTA four times that.  (Eight rows a lane and the next
// token's vectors fetched into registers ahead were measured and were slower: more shuffles and more registers.)  The sums over a column's rows
// are CS_ROWS multiply-adds a lane (four partial sums, a fixed order) and log2(LPC) shuffles.  The tokens' vectors arrive in
// shared memory by cp.async, a chunk of tokens ahead of the warps that work through them, and are read 16 bytes at a time.
// The state of a request is kept in the order of the registers ([head][warp tile][row of the lane][lane]), so that it is read and
// written in whole lines; rows and columns beyond the sizes hold zeros.
#define CS_WARPS 4
#define CS_ROWS 16
#define CS_PAD 20           // floats a lane's rows take in a stage: 16 and 4 of padding, so that 16-byte reads of the LPC lanes miss one another's banks

struct ChannelScanArgs {
  float* out; int ld_out;                 // [T, H * dv]
  const float* q; int ld_q;               // [T, H * dk] ...
  const float* k; int ld_k;
  const float* v; int ld_v;               // [T, H * dv]
  const float* w; int ld_w;               // decay per key channel
  const float* au; int ld_au;             // removal: a * u and u, or null
  const float* u; int ld_u;
  float q_scale;
  float* state; long long slot_stride;    // per slot: [H][tiles][CS_ROWS][32]
  const int* seg_q_start; const int* seg_slot;
  int H, dk, dv;
};

// 4 or 16 bytes, or as many zero bytes where `valid` is false
__device__ __forceinline__ void cs_cp4(float* dst, const float* src, bool valid) {
  const int bytes = valid ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cs_cp16(float* dst, const float* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ float cs_sum4(const float* p) { return (p[0] + p[1]) + (p[2] + p[3]); }

// `chunk` tokens a stage, two stages.  vec4: every vector starts on 16 bytes and dk is a multiple of 4 (16-byte copies).
template <int LPC, bool REMOVAL>
__global__ void __launch_bounds__(32 * CS_WARPS) channel_scan_kernel(ChannelScanArgs a, int chunk, int vec4) {
  extern __shared__ __align__(16) float cs_ring[];
  constexpr int NV = REMOVAL ? 5 : 3;
  constexpr int CPW = 32 / LPC, CTA_COLS = CS_WARPS * CPW, NTH = 32 * CS_WARPS;
  constexpr int VEC = CS_PAD * LPC;                // floats a vector takes in a stage
  constexpr int ROW = NV * VEC + CTA_COLS;         // floats a token takes
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lic = lane % LPC, cw = lane / LPC;
  const int dk = a.dk, dv = a.dv;
  const int cta_col0 = blockIdx.z * CTA_COLS;
  const int col = cta_col0 + warp * CPW + cw;
  const int tiles = (dv + CPW - 1) / CPW;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  const int tile = blockIdx.z * CS_WARPS + warp;
  const bool active = tile < tiles;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + ((size_t)h * tiles + tile) * (CS_ROWS * 32) + lane;
  float S[CS_ROWS];
#pragma unroll
  for (int i = 0; i < CS_ROWS; ++i) S[i] = active ? st[i * 32] : 0.f;
  const size_t hk = (size_t)h * dk, hv = (size_t)h * dv;
  const float* srcs[5] = {a.w + hk, a.k + hk, a.q + hk, REMOVAL ? a.au + hk : nullptr, REMOVAL ? a.u + hk : nullptr};
  const int lds[5] = {a.ld_w, a.ld_k, a.ld_q, a.ld_au, a.ld_u};
  auto issue = [&](int c) {
    float* base = cs_ring + (size_t)(c & 1) * chunk * ROW;
    const int j0 = c * chunk, nt = min(chunk, len - j0);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (vec4) {
        constexpr int PER = CS_ROWS * LPC / 4;       // 16-byte pieces a vector (padding rows included)
        for (int i = tid; i < nt * PER; i += NTH) {
          const int j = i / PER, r = (i % PER) * 4;
          cs_cp16(base + j * ROW + v * VEC + r + (r / CS_ROWS) * (CS_PAD - CS_ROWS), srcs[v] + (size_t)(q0 + j0 + j) * lds[v] + r, r < dk);
        }
      } else {
        constexpr int PER = CS_ROWS * LPC;
        for (int i = tid; i < nt * PER; i += NTH) {
          const int j = i / PER, r = i % PER;
          cs_cp4(base + j * ROW + v * VEC + r + (r / CS_ROWS) * (CS_PAD - CS_ROWS), srcs[v] + (size_t)(q0 + j0 + j) * lds[v] + r, r < dk);
        }
      }
    }
    for (int i = tid; i < nt * CTA_COLS; i += NTH) {
      const int j = i / CTA_COLS, cc = i % CTA_COLS;
      cs_cp4(base + j * ROW + NV * VEC + cc, a.v + (size_t)(q0 + j0 + j) * a.ld_v + hv + cta_col0 + cc, cta_col0 + cc < dv);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int nchunks = (len + chunk - 1) / chunk;
  if (nchunks > 0) issue(0);
  for (int c = 0; c < nchunks; ++c) {
    if (c + 1 < nchunks) {
      issue(c + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int j0 = c * chunk, nt = min(chunk, len - j0);
    if (active) {
#pragma unroll(REMOVAL ? 2 : 4)
      for (int j = 0; j < nt; ++j) {
        const float* d = cs_ring + ((size_t)(c & 1) * chunk + j) * ROW;
        const float4* pw = (const float4*)(d + lic * CS_PAD);
        const float4* pk = (const float4*)(d + VEC + lic * CS_PAD);
        const float4* pq = (const float4*)(d + 2 * VEC + lic * CS_PAD);
        const float vv = d[NV * VEC + warp * CPW + cw];
        float dd = 0.f;
        if (REMOVAL) {
          const float4* pu = (const float4*)(d + 4 * VEC + lic * CS_PAD);
          float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < CS_ROWS / 4; ++i) {
            const float4 u4 = pu[i];
            p[0] = fmaf(u4.x, S[4 * i], p[0]); p[1] = fmaf(u4.y, S[4 * i + 1], p[1]);
            p[2] = fmaf(u4.z, S[4 * i + 2], p[2]); p[3] = fmaf(u4.w, S[4 * i + 3], p[3]);
          }
          dd = cs_sum4(p);
#pragma unroll
          for (int o = LPC / 2; o > 0; o >>= 1) dd += __shfl_xor_sync(0xffffffffu, dd, o);
        }
        float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < CS_ROWS / 4; ++i) {
          const float4 w4 = pw[i], k4 = pk[i], q4 = pq[i];
          float n0 = fmaf(k4.x, vv, w4.x * S[4 * i]), n1 = fmaf(k4.y, vv, w4.y * S[4 * i + 1]);
          float n2 = fmaf(k4.z, vv, w4.z * S[4 * i + 2]), n3 = fmaf(k4.w, vv, w4.w * S[4 * i + 3]);
          if (REMOVAL) {
            const float4 a4 = ((const float4*)(d + 3 * VEC + lic * CS_PAD))[i];
            n0 = fmaf(-a4.x, dd, n0); n1 = fmaf(-a4.y, dd, n1); n2 = fmaf(-a4.z, dd, n2); n3 = fmaf(-a4.w, dd, n3);
          }
          S[4 * i] = n0; S[4 * i + 1] = n1; S[4 * i + 2] = n2; S[4 * i + 3] = n3;
          y[0] = fmaf(q4.x, n0, y[0]); y[1] = fmaf(q4.y, n1, y[1]); y[2] = fmaf(q4.z, n2, y[2]); y[3] = fmaf(q4.w, n3, y[3]);
        }
        float yy = cs_sum4(y);
#pragma unroll
        for (int o = LPC / 2; o > 0; o >>= 1) yy += __shfl_xor_sync(0xffffffffu, yy, o);
        if (lic == 0 && col < dv) a.out[(size_t)(q0 + j0 + j) * a.ld_out + hv + col] = yy * a.q_scale;
      }
    }
    __syncthreads();
  }
  pdl_launch_dependents();
  if (!active) return;
#pragma unroll
  for (int i = 0; i < CS_ROWS; ++i) st[i * 32] = S[i];
}

// A launch that starts only when the kernel before it has ended.  For portions the scan is a long kernel of few CTAs that wants an
// SM each: launched ahead (programmatic dependent launch) its CTAs are placed while the kernel before it still fills the SMs, several
// on one SM, and the scan of a 2,048-token prompt was measured to take 1.6 to 2 times as long.
template <typename... KArgs, typename... Args>
static inline int cs_launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  return (int)cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

static inline int cs_lanes_per_column(int dk) { return dk <= 16 ? 1 : dk <= 32 ? 2 : dk <= 64 ? 4 : dk <= 128 ? 8 : 16; }

extern "C" long long qv_channel_scan_state_floats(int H, int dk, int dv) {
  const int cpw = 32 / cs_lanes_per_column(dk);
  return (long long)H * ((dv + cpw - 1) / cpw) * CS_ROWS * 32;
}

// max_q_len: the longest segment of the step (how many tokens a stage of the ring holds follows from it).
extern "C" int qv_channel_scan(float* out, int ld_out, const float* q, int ld_q, const float* k, int ld_k, const float* v, int ld_v,
                               const float* w, int ld_w, const float* au, int ld_au, const float* u, int ld_u, float q_scale,
                               float* state, long long slot_stride, const int* seg_q_start, const int* seg_slot, int S, int max_q_len,
                               int H, int dk, int dv, void* stream) {
  if (S <= 0) return 0;
  if (H <= 0 || dk <= 0 || dv <= 0 || H > 65535 || (au == nullptr) != (u == nullptr)) return QV_ERR_UNSUPPORTED;
  if (dk > 256) return QV_ERR_TOO_LARGE;
  ChannelScanArgs a;
  a.out = out; a.ld_out = ld_out; a.q = q; a.ld_q = ld_q; a.k = k; a.ld_k = ld_k; a.v = v; a.ld_v = ld_v; a.w = w; a.ld_w = ld_w;
  a.au = au; a.ld_au = ld_au; a.u = u; a.ld_u = ld_u; a.q_scale = q_scale; a.state = state; a.slot_stride = slot_stride;
  a.seg_q_start = seg_q_start; a.seg_slot = seg_slot; a.H = H; a.dk = dk; a.dv = dv;
  const int lpc = cs_lanes_per_column(dk);
  const int cta_cols = CS_WARPS * 32 / lpc;
  const int ctas = (dv + cta_cols - 1) / cta_cols;
  if (ctas > 65535) return QV_ERR_TOO_LARGE;
  dim3 grid(S, H, ctas), block(32 * CS_WARPS);
  cudaStream_t st = (cudaStream_t)stream;
  const bool rem = au != nullptr;
  const int row = (rem ? 5 : 3) * CS_PAD * lpc + cta_cols;
  int chunk = max_q_len < 1 ? 1 : (max_q_len > 16 ? 16 : max_q_len);
  while (chunk > 1 && (size_t)2 * chunk * row * sizeof(float) > 64 * 1024) chunk >>= 1;
  const size_t smem = (size_t)2 * chunk * row * sizeof(float);
  auto aligned = [](const float* p, int ld) { return p == nullptr || (((uintptr_t)p & 15) == 0 && ld % 4 == 0); };
  const bool long_rows = max_q_len >= 16;
  const int vec4 = dk % 4 == 0 && aligned(q, ld_q) && aligned(k, ld_k) && aligned(w, ld_w) && aligned(au, ld_au) && aligned(u, ld_u);
#define CS_LAUNCH(LPC_)                                                                                                  \
  do {                                                                                                                   \
    if (rem) {                                                                                                           \
      cudaFuncSetAttribute(channel_scan_kernel<LPC_, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);     \
      if (long_rows) return cs_launch_after(channel_scan_kernel<LPC_, true>, grid, block, smem, st, a, chunk, vec4);     \
      return qv_launch(channel_scan_kernel<LPC_, true>, grid, block, smem, st, a, chunk, vec4);                          \
    }                                                                                                                    \
    cudaFuncSetAttribute(channel_scan_kernel<LPC_, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);      \
    if (long_rows) return cs_launch_after(channel_scan_kernel<LPC_, false>, grid, block, smem, st, a, chunk, vec4);      \
    return qv_launch(channel_scan_kernel<LPC_, false>, grid, block, smem, st, a, chunk, vec4);                           \
  } while (0)
  if (lpc == 1) CS_LAUNCH(1);
  if (lpc == 2) CS_LAUNCH(2);
  if (lpc == 4) CS_LAUNCH(4);
  if (lpc == 8) CS_LAUNCH(8);
  CS_LAUNCH(16);
#undef CS_LAUNCH
}

// ---------------------------------------------------------------- delta rule on the decayed state: sixteen tokens at a time
// With S_0 the state ahead of a block of up to 16 tokens, P_t the product of the decays of the block's tokens up to t (per channel) and
// kb = beta k, the recurrence S_t = diag(g_t) S_(t-1) + kb_t e_t^T, e_t = v_t - S_(t-1)^T (g_t k_t), y_t = S_t^T q_t unrolls to
//   e_t   = v_t - S_0^T (P_t k_t) - sum_(l < t) A_tl e_l        A_tl = sum_c k_t (g_(l+1) .. g_t) kb_l
//   y_t   = S_0^T (P_t q_t) + sum_(l <= t) B_tl e_l             B_tl = sum_c q_t (g_(l+1) .. g_t) kb_l
//   S_end = diag(P_end) S_0 + sum_l (g_(l+1) .. g_end kb_l) e_l^T
// and, the triangular system solved ahead for both of its right sides (X = P k, column by column, and v), to
//   X'_t  = P_t k_t - sum_(l < t) A_tl X'_l        v'_t = v_t - sum_(l < t) A_tl v'_l
//   X''_t = P_t q_t - sum_(l <= t) B_tl X'_l       v''_t = sum_(l <= t) B_tl v'_l
//   e_t   = v'_t - S_0^T X'_t,                     y_t = v''_t + S_0^T X''_t
// so that all but the products with S_0 and the update is worked out for all blocks at once, and a block costs its recurrence two products
// and two barriers.  Only products of decays (each at most one) occur, no quotients.
//   delta_block_operands_kernel   a CTA per (block, head): everything that does not depend on the state, float32, the triangular system's sums float64
//   delta_blocks_kernel           the recurrence: a CTA owns 16 value columns of a (segment, head), a warp 16 of the keys
// The products with S_0 and of the update are mma.sync on both sides' three bfloat16 terms (the six products that count for 24 bits; the
// large one's sum apart from the small ones', which the tensor cores would cut off), sums over the keys' slices in float32.
// 1,531 tokens of 16 heads of 128 x 128: 607 us token by token, 460 with four tokens at a time and float32 multiply-adds, and
// 168 here (operands 65, recurrence 103; operands 58 with the triangular system's sums in float32, which left portions of 16 to 100 tokens
// further off float64 than four tokens at a time had; 61 and 139 with operands of float32 that every CTA split again, read straight to
// registers).
// Blocks are counted from the start of a request's portion, so cuts agree to rounding (the 32-bit path takes channel_scan_kernel).
#define CD_BLOCK 16
#define CD_COLS 16
#define CD_OP_THREADS 256
#define CD_ITEMS 96
struct ChannelDeltaArgs {
  float* out; int ld_out;                 // [T, H * dv]
  const float *q, *k, *v, *b, *g; int ld_q, ld_k, ld_v, ld_b, ld_g;
  float* ws;                              // [slots][H][cd_slot_floats]: the round's blocks
  float* state; long long slot_stride;    // as ChannelScanArgs
  const int* seg_q_start; const int* seg_slot;
  int H, G, dk, dv, dkp, dvp;             // dkp, dvp: in whole 16s
  float eps, q_scale;
  PortionRound<CD_ITEMS> round;           // some blocks of some segments, a slot of the workspace each
};
// A block's floats: X', X'' and W = (g_(l+1) .. g_end) kb_l in three bfloat16 terms, as the products' operands lie in the lanes, P_end;
// then per tile of 16 columns v' and v'' ([16 tokens][16 columns] each).
__host__ __device__ inline size_t cd_slot_floats(int dkp, int dvp) { return (size_t)73 * dkp + 32 * (size_t)dvp; }
__device__ __forceinline__ float* cd_slot(const ChannelDeltaArgs& a, int slot, int h) {
  return a.ws + ((size_t)slot * a.H + h) * cd_slot_floats(a.dkp, a.dvp);
}
// x and y as three bfloat16 terms each (x in the lower half of a word)
__device__ __forceinline__ void cd_split3(float x, float y, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  uint32_t t[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    t[i] = *(const uint32_t*)&h;
    x -= __low2float(h);
    y -= __high2float(h);
  }
  t0 = t[0]; t1 = t[1]; t2 = t[2];
}

// grid (slots, heads).  Bound by its multiply-adds and the reads of shared memory beside them.
__global__ void __launch_bounds__(CD_OP_THREADS, 3) delta_block_operands_kernel(const __grid_constant__ ChannelDeltaArgs a) {
  extern __shared__ __align__(16) float cd_smem[];
  pdl_wait();
  pdl_launch_dependents();
  int first = 0;                                     // whose slot this is
  for (int last = a.round.items - 1; first < last;) {
    const int mid = (first + last + 1) >> 1;
    if (a.round.item[mid].slot <= (int)blockIdx.x) first = mid;
    else last = mid - 1;
  }
  const PortionItem& it = a.round.item[first];
  const int s = it.seg, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0, j0 = (it.first + (int)blockIdx.x - it.slot) * CD_BLOCK;
  if (j0 >= len) return;
  const int nb = len - j0 < CD_BLOCK ? len - j0 : CD_BLOCK;
  const int dk = a.dk, dkp = a.dkp, ld = dkp + 4;
  float* qs = cd_smem;                               // [16][ld] unit vectors, q times q_scale
  float* ks = qs + CD_BLOCK * ld;
  float* gs = ks + CD_BLOCK * ld;
  double* As = (double*)(gs + CD_BLOCK * ld);        // [16][16]
  double* Bs = As + CD_BLOCK * CD_BLOCK;             // [16][16]
  float* beta = (float*)(Bs + CD_BLOCK * CD_BLOCK);  // [16]
  const int grp = h / (a.H / a.G);
  // two tokens a warp; beyond the segment: keys and queries zero, decays one
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = warp * 2 + i;
    const bool in = t < nb;
    const size_t row = (size_t)(q0 + j0 + (in ? t : 0));
    const float* qr = a.q + row * a.ld_q + (size_t)grp * dk;
    const float* kr = a.k + row * a.ld_k + (size_t)grp * dk;
    const float* gr = a.g + row * a.ld_g + (size_t)h * dk;
    float qv[8], kv[8], gv[8], sq = 0.f, sk = 0.f;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int c = lane + 32 * x;
      const bool ok = in && c < dk;
      qv[x] = ok ? qr[c] : 0.f;
      kv[x] = ok ? kr[c] : 0.f;
      gv[x] = ok ? gr[c] : 1.f;
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) { sq = fmaf(qv[x], qv[x], sq); sk = fmaf(kv[x], kv[x], sk); }
    const float iq = a.q_scale / sqrtf(warp_sum(sq) + a.eps), ik = 1.0f / sqrtf(warp_sum(sk) + a.eps);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const int c = lane + 32 * x;
      if (c < dkp) {
        qs[t * ld + c] = qv[x] * iq;
        ks[t * ld + c] = kv[x] * ik;
        gs[t * ld + c] = gv[x];
      }
    }
    if (lane == 0) beta[t] = in ? 1.0f / (1.0f + expf(-a.b[row * a.ld_b + h])) : 0.f;
  }
  __syncthreads();
  // columns l and 15 - l of A and B a warp, four channels a lane and pass: 17 tokens' steps for every warp
#pragma unroll 1
  for (int i = 0; i < 2; ++i) {
    const int l = i ? CD_BLOCK - 1 - warp : warp;
    float sum[2 * CD_BLOCK] = {};                    // A_tl, then B_tl
    for (int c = lane * 4; c < dkp; c += 128) {
      const float bl = beta[l];
      float4 kd = *(const float4*)(ks + l * ld + c);
      kd.x *= bl; kd.y *= bl; kd.z *= bl; kd.w *= bl;
#pragma unroll
      for (int t = 0; t < CD_BLOCK; ++t) {
        if (t < l) continue;
        const float4 q4 = *(const float4*)(qs + t * ld + c);
        if (t > l) {
          const float4 g4 = *(const float4*)(gs + t * ld + c), k4 = *(const float4*)(ks + t * ld + c);
          kd.x *= g4.x; kd.y *= g4.y; kd.z *= g4.z; kd.w *= g4.w;
          sum[t] += fmaf(k4.x, kd.x, k4.y * kd.y) + fmaf(k4.z, kd.z, k4.w * kd.w);
        }
        sum[CD_BLOCK + t] += fmaf(q4.x, kd.x, q4.y * kd.y) + fmaf(q4.z, kd.z, q4.w * kd.w);
      }
    }
    // 32 sums over 32 lanes: a lane ends with its own
#pragma unroll
    for (int half = 16; half > 0; half >>= 1)
#pragma unroll
      for (int x = 0; x < half; ++x) {
        const bool up = lane & half;
        const float send = up ? sum[x] : sum[x + half], keep = up ? sum[x + half] : sum[x];
        sum[x] = keep + __shfl_xor_sync(0xffffffffu, send, half);
      }
    (lane < CD_BLOCK ? As : Bs)[(lane & 15) * CD_BLOCK + l] = sum[0];
  }
  __syncthreads();
  float* ws = cd_slot(a, blockIdx.x, h);
  uint32_t *X1 = (uint32_t*)ws, *X2 = X1 + 24 * dkp, *Wf = X2 + 24 * dkp;
  float *Pe = ws + 72 * dkp, *Vs = Pe + dkp;
  for (int col = tid; col < dkp + a.dvp; col += CD_OP_THREADS) {     // (whole warps: dkp and dvp are multiples of 16, and half warps stay together)
    const bool key = col < dkp;
    // the system's sums in float64 (16 products of numbers of 24 bits in a row, where a block of four had four), their results in float32
    double xd[CD_BLOCK];
    float y[CD_BLOCK];
    if (key) {
      float decay = 1.f;
#pragma unroll
      for (int t = 0; t < CD_BLOCK; ++t) {
        decay *= gs[t * ld + col];
        xd[t] = decay * ks[t * ld + col];
      }
      Pe[col] = decay;
    } else {
      const int cv = col - dkp;
      const float* vr = a.v + (size_t)(q0 + j0) * a.ld_v + (size_t)h * a.dv + cv;
#pragma unroll
      for (int t = 0; t < CD_BLOCK; ++t) xd[t] = t < nb && cv < a.dv ? vr[(size_t)t * a.ld_v] : 0.f;
    }
#pragma unroll
    for (int t = 0; t < CD_BLOCK; ++t) {
      double sum = xd[t];
#pragma unroll
      for (int l2 = 0; l2 + 1 < t; l2 += 2) {
        const double2 A2 = *(const double2*)(As + t * CD_BLOCK + l2);
        sum = fma(-A2.y, xd[l2 + 1], fma(-A2.x, xd[l2], sum));
      }
      if (t & 1) sum = fma(-As[t * CD_BLOCK + t - 1], xd[t - 1], sum);
      xd[t] = t < nb ? (float)sum : 0.f;
    }
    float P = 1.f;
#pragma unroll
    for (int t = 0; t < CD_BLOCK; ++t) {
      double sum = 0.0;
#pragma unroll
      for (int l2 = 0; l2 + 1 <= t; l2 += 2) {
        const double2 B2 = *(const double2*)(Bs + t * CD_BLOCK + l2);
        sum = fma(B2.y, xd[l2 + 1], fma(B2.x, xd[l2], sum));
      }
      if (!(t & 1)) sum = fma(Bs[t * CD_BLOCK + t], xd[t], sum);
      if (key) {
        P *= gs[t * ld + col];
        sum = t < nb ? fma((double)P, (double)qs[t * ld + col], -sum) : 0.0;
      }
      y[t] = (float)sum;
    }
    if (key) {
      // X' and X'' as the products' first operand: lane (t % 8) 4 + (key % 8) / 2 holds, a term, the words of {t, t + 8} x {key, key + 8}, a word
      // an even key and the next one.  Of two neighbouring keys the even one's thread makes the words of tokens 0..7, the other 8..15.
      const int odd = col & 1, lane0 = (col & 7) >> 1, reg = odd + 2 * ((col >> 3) & 1);
      uint32_t* dst = X1 + (size_t)(col >> 4) * 384 + lane0 * 4 + reg;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const float z0 = m ? y[t] : (float)xd[t], z8 = m ? y[t + 8] : (float)xd[t + 8];
          const float other = __shfl_xor_sync(3u << (lane & 30), odd ? z0 : z8, 1);
          uint32_t w0, w1, w2;
          cd_split3(odd ? other : z0, odd ? z8 : other, w0, w1, w2);
          uint32_t* d = dst + m * 24 * dkp + t * 16;
          d[0] = w0; d[128] = w1; d[256] = w2;
        }
      }
      // W as the update's second operand: lane (key % 8) 4 + t4 holds, a term, {tokens 2 t4, 2 t4 + 1; 2 t4 + 8, 2 t4 + 9} of key and of key + 8
      float f = 1.f;
#pragma unroll
      for (int t = CD_BLOCK - 1; t >= 0; --t) {
        y[t] = f * (beta[t] * ks[t * ld + col]);
        f *= gs[t * ld + col];
      }
      uint32_t* wd = Wf + (size_t)(col >> 4) * 384 + (col & 7) * 16 + 2 * ((col >> 3) & 1);
#pragma unroll
      for (int t4 = 0; t4 < 4; ++t4) {
        uint32_t w[2][3];
        cd_split3(y[2 * t4], y[2 * t4 + 1], w[0][0], w[0][1], w[0][2]);
        cd_split3(y[2 * t4 + 8], y[2 * t4 + 9], w[1][0], w[1][1], w[1][2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) *(uint2*)(wd + i * 128 + t4 * 4) = make_uint2(w[0][i], w[1][i]);
      }
    } else {
      const int cv = col - dkp;
#pragma unroll
      for (int t = 0; t < CD_BLOCK; ++t) {
        Vs[(cv >> 4) * 512 + t * 16 + (cv & 15)] = (float)xd[t];
        Vs[(cv >> 4) * 512 + 256 + t * 16 + (cv & 15)] = y[t];
      }
    }
  }
}

__device__ __forceinline__ void cd_mma(float* c, const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cd_ldsm4(uint32_t (&r)[4], const void* p) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
// c = a b of three terms each, as three sums
struct CdSums { float hi[4], lo[4], lo2[4]; };
__device__ __forceinline__ void cd_product(CdSums& c, const uint32_t (&a)[3][4], const uint32_t (&b0)[3], const uint32_t (&b1)[3]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) c.hi[i] = c.lo[i] = c.lo2[i] = 0.f;
  cd_mma(c.lo, a[0], b0[1], b1[1]);
  cd_mma(c.lo2, a[2], b0[0], b1[0]);
  cd_mma(c.hi, a[0], b0[0], b1[0]);
  cd_mma(c.lo, a[1], b0[0], b1[0]);
  cd_mma(c.lo2, a[0], b0[2], b1[2]);
  cd_mma(c.lo2, a[1], b0[1], b1[1]);
}
__device__ __forceinline__ float cd_sum(const CdSums& c, int i) { return c.hi[i] + (c.lo[i] + c.lo2[i]); }
__device__ __forceinline__ void cd_words(uint32_t (&a)[3][4], const uint4* p) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint4 w = p[i * 32];
    a[i][0] = w.x; a[i][1] = w.y; a[i][2] = w.z; a[i][3] = w.w;
  }
}

// grid (items, heads, column tiles); NS warps, a slice of 16 keys each, S^T in registers as the accumulators of the update (value columns x
// keys), which are the second operand of X S_0.  A block: the slices' shares of X' S_0 into shared memory, a barrier, their sums e (and y of
// the block ahead), a barrier, the update; X'' S_0 is formed between the two, where the tensor cores have nothing else to do, and summed a
// block later.  The operands arrive STAGES - 1 blocks ahead (cp.async).  Bound by that chain: two barriers, three rounds through shared memory,
// two products of three terms a side and the splits between them.
template <int NS> struct CdShape {
  static constexpr int LD = NS == 16 ? 20 : 24;      // 24: the writes of a half warp hit every bank once; 16 slices of that are too much
  static constexpr int STAGES = NS == 16 ? 2 : 4;
  static constexpr int RED = NS * CD_BLOCK * LD;     // floats
  __host__ __device__ static int stage_floats(int dkp) { return 73 * dkp + 512; }
  __host__ __device__ static int bytes(int dkp) { return (STAGES * stage_floats(dkp) + 2 * RED) * 4 + 3 * CD_COLS * CD_BLOCK * 2; }
};
template <int NS>
__global__ void __launch_bounds__(32 * NS, 1) delta_blocks_kernel(const __grid_constant__ ChannelDeltaArgs a) {
  typedef CdShape<NS> Sh;
  constexpr int THREADS = 32 * NS, STAGES = Sh::STAGES, LD = Sh::LD;
  constexpr int EACH = THREADS >= 256 ? 1 : 256 / THREADS;           // of the 16 x 16 sums, a thread's
  constexpr int PER_ROW = CD_COLS / EACH;            // threads a row
  extern __shared__ __align__(16) float cd_smem[];
  pdl_wait();
  const PortionItem& it = a.round.item[blockIdx.x];
  const int s = it.seg, h = blockIdx.y, col0 = blockIdx.z * CD_COLS, block0 = it.first;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g8 = lane >> 2, t4 = lane & 3;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  const int dk = a.dk, dv = a.dv, dkp = a.dkp, stage_floats = Sh::stage_floats(dkp);
  float* red = cd_smem + STAGES * stage_floats;      // [NS][16][LD] of e
  float* red2 = red + Sh::RED;                       // of y
  bf16* eT = (bf16*)(red2 + Sh::RED);                // [term][column][token], 16-byte halves of a row swapped in every other four columns
  const int lpc = dk <= 16 ? 1 : dk <= 32 ? 2 : dk <= 64 ? 4 : dk <= 128 ? 8 : 16, cpt = 32 / lpc, tiles = (dv + cpt - 1) / cpt;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + (size_t)h * tiles * 512;
  const int k0 = warp * 16;
  const bool holds = k0 < dkp;
  auto at = [&](int nt, int i) -> float* {           // where S^T's entry lies in the state (channel_scan_kernel's layout; rows from dk on: zeros), or null
    const int k = k0 + nt * 8 + 2 * t4 + (i & 1), col = col0 + g8 + (i >> 1) * 8;
    return k < 16 * lpc && col < tiles * cpt ? st + (size_t)(col / cpt) * 512 + (k & 15) * 32 + (col % cpt) * lpc + (k >> 4) : nullptr;
  };
  const int all = (len + CD_BLOCK - 1) / CD_BLOCK - block0, nblocks = all < it.count ? all : it.count;
  if (nblocks <= 0) return;
  const size_t stride = (size_t)a.H * cd_slot_floats(dkp, a.dvp);
  const float* ws = cd_slot(a, it.slot, h);
  const int pieces = 73 * dkp / 4;
  auto issue = [&](int blk) {
    if (blk < nblocks) {
      float* d = cd_smem + (blk % STAGES) * stage_floats;
      const float* src = ws + (size_t)blk * stride;
#pragma unroll
      for (int i = 0; i < 10; ++i)                   // (73 * 16 NS floats are 9.1 pieces a thread)
        if (tid + i * THREADS < pieces) cs_cp16(d + (tid + i * THREADS) * 4, src + (tid + i * THREADS) * 4, true);
      if (tid < 128) cs_cp16(d + 73 * dkp + tid * 4, src + 73 * dkp + blockIdx.z * 512 + tid * 4, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) issue(i);
  float S[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* p = at(nt, i);
      S[nt][i] = p && k0 + nt * 8 + 2 * t4 + (i & 1) < dk ? *p : 0.f;
    }
  const int orow = (tid / PER_ROW) & 15, ocol = (tid % PER_ROW) * EACH;      // the sums this thread forms
  const bool sums_e = tid < 256, sums_y = THREADS > 256 ? tid >= 256 : true;
  float v2[EACH] = {};                               // v'' of the block ahead
  float* yp = a.out + (size_t)(q0 + block0 * CD_BLOCK + orow) * a.ld_out + (size_t)h * dv + col0 + ocol;
  const size_t ystep = (size_t)CD_BLOCK * a.ld_out;
  const int yleft = len - block0 * CD_BLOCK - orow, ycols = dv - col0 - ocol;
  for (int i = tid; i < 2 * Sh::RED; i += THREADS) red[i] = 0.f;             // (slices that dk does not reach add nothing)
  auto finish = [&](int blk) {                       // y of a block, from the shares in red2
    if (!sums_y) return;
    float sum[EACH] = {};
#pragma unroll
    for (int sl = 0; sl < NS; ++sl)
#pragma unroll
      for (int i = 0; i < EACH; ++i) sum[i] += red2[(sl * CD_BLOCK + orow) * LD + ocol + i];
    if (blk * CD_BLOCK < yleft) {
#pragma unroll
      for (int i = 0; i < EACH; ++i)
        if (i < ycols) yp[i] = v2[i] + sum[i];
    }
    yp += ystep;
  };
  asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
  __syncthreads();                                   // block 0 is in place
  for (int blk = 0; blk < nblocks; ++blk) {
    const float* d = cd_smem + (blk % STAGES) * stage_floats;
    const uint4* words = (const uint4*)d + warp * 96 + lane;
    uint32_t b0[2][3], b1[2][3];                     // S_0: [column tile][term]
    CdSums c2[2];
    float v1[EACH];
#pragma unroll
    for (int i = 0; i < EACH; ++i) v1[i] = d[73 * dkp + orow * 16 + ocol + i];
    if (holds) {
      uint32_t x[3][4];
      cd_words(x, words);
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        cd_split3(S[0][2 * nb], S[0][2 * nb + 1], b0[nb][0], b0[nb][1], b0[nb][2]);
        cd_split3(S[1][2 * nb], S[1][2 * nb + 1], b1[nb][0], b1[nb][1], b1[nb][2]);
      }
      CdSums c[2];
      cd_product(c[0], x, b0[0], b1[0]);
      cd_product(c[1], x, b0[1], b1[1]);
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        float* r = red + (warp * CD_BLOCK + g8) * LD + nb * 8 + 2 * t4;
        *(float2*)r = make_float2(cd_sum(c[nb], 0), cd_sum(c[nb], 1));
        *(float2*)(r + 8 * LD) = make_float2(cd_sum(c[nb], 2), cd_sum(c[nb], 3));
      }
    }
    __syncthreads();                                 // the shares of e, and of y of the block ahead, are in place; eT and that block's operands have been read
    if (sums_e) {
      float sum[EACH] = {};
#pragma unroll
      for (int sl = 0; sl < NS; ++sl)
#pragma unroll
        for (int i = 0; i < EACH; ++i) sum[i] += red[(sl * CD_BLOCK + orow) * LD + ocol + i];
#pragma unroll
      for (int i = 0; i < EACH; ++i) {
        float e = v1[i] - sum[i];
        bf16* to = eT + (ocol + i) * CD_BLOCK + (orow ^ (((ocol + i) >> 2) & 1) * 8);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const bf16 term = __float2bfloat16_rn(e);
          to[x * CD_COLS * CD_BLOCK] = term;
          e -= __bfloat162float(term);
        }
      }
    }
    if (holds) {
      uint32_t x[3][4];
      cd_words(x, words + 6 * dkp);
      cd_product(c2[0], x, b0[0], b1[0]);
      cd_product(c2[1], x, b0[1], b1[1]);
    }
    if (blk) finish(blk - 1);
#pragma unroll
    for (int i = 0; i < EACH; ++i) v2[i] = d[73 * dkp + 256 + orow * 16 + ocol + i];
    issue(blk + STAGES - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                 // e is in place, and the next block's operands; the shares have been read
    if (holds) {
      uint32_t e[3][4], w[3][4];                     // e^T: columns g8, g8 + 8; tokens 2 t4, 2 t4 + 1 and 8 further
#pragma unroll
      for (int x = 0; x < 3; ++x) cd_ldsm4(e[x], eT + x * CD_COLS * CD_BLOCK + (lane & 15) * CD_BLOCK + (((lane >> 4) ^ ((lane >> 2) & 1)) * 8));
      cd_words(w, words + 12 * dkp);
      CdSums c[2];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const uint32_t w0[3] = {w[0][2 * nt], w[1][2 * nt], w[2][2 * nt]}, w1[3] = {w[0][2 * nt + 1], w[1][2 * nt + 1], w[2][2 * nt + 1]};
        cd_product(c[nt], e, w0, w1);
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float2 P = *(const float2*)(d + 72 * dkp + k0 + nt * 8 + 2 * t4);
#pragma unroll
        for (int i = 0; i < 4; ++i) S[nt][i] = fmaf(i & 1 ? P.y : P.x, S[nt][i], cd_sum(c[nt], i));
      }
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) {
        float* r = red2 + (warp * CD_BLOCK + g8) * LD + nb * 8 + 2 * t4;
        *(float2*)r = make_float2(cd_sum(c2[nb], 0), cd_sum(c2[nb], 1));
        *(float2*)(r + 8 * LD) = make_float2(cd_sum(c2[nb], 2), cd_sum(c2[nb], 3));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  finish(nblocks - 1);
  pdl_launch_dependents();
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* p = at(nt, i);
      if (p) *p = S[nt][i];
    }
}

template <int NS>
static int launch_delta_blocks(const ChannelDeltaArgs& a, dim3 grid, cudaStream_t st) {
  static PerDevice allowed;
  const int rc = qv_allow_smem(delta_blocks_kernel<NS>, CdShape<NS>::bytes(16 * NS), allowed);
  if (rc) return rc;
  const int smem = CdShape<NS>::bytes(a.dkp);
  return cs_launch_after(delta_blocks_kernel<NS>, grid, dim3(32 * NS), (size_t)smem, st, a);
}

// What qv_channel_delta takes beside its operands, in floats: for lead_tokens that go token by token, and for segs segments of max_rest tokens each
// (where they are not alike: of their mean number of blocks) in blocks, of which as many at a time as CD_ROOM floats hold.
#define CD_ROOM ((size_t)48 << 20)
#define CD_FEW 16                          // blocks of a segment that are worth a round of launches
static inline size_t cd_slot_all_heads(int H, int dk, int dv) { return H * cd_slot_floats((dk + 15) / 16 * 16, (dv + 15) / 16 * 16); }
static inline size_t cd_room_slots(int H, int dk, int dv) {
  const size_t fit = CD_ROOM / cd_slot_all_heads(H, dk, dv);
  return fit ? fit : 1;
}
extern "C" long long qv_channel_delta_workspace_floats(int lead_tokens, int segs, int max_rest, int H, int dk, int dv) {
  const size_t blocks = segs > 0 && max_rest > 0 ? (size_t)((max_rest + CD_BLOCK - 1) / CD_BLOCK) * segs : 0, fit = cd_room_slots(H, dk, dv);
  return (long long)((size_t)lead_tokens * H * 3 * dk + cd_slot_all_heads(H, dk, dv) * (blocks < fit ? blocks : fit));
}

// The recurrence over a step's segments: q, k [T, G * dk] float32 (row strides) as the convolutions leave them, b [T, H] the pre-activation of
// beta, g [T, H * dk] the decays, v [T, H * dv].  The first S_lead segments (T_lead tokens, the longest of them max_lead) go token by token, the
// others (lens [S], host) in blocks, for which dk is a multiple of 4, at most 256.  workspace: qv_channel_delta_workspace_floats, ws_floats of
// them, 16-byte aligned.  *launches: how many kernels were launched.
extern "C" int qv_channel_delta(float* out, int ld_out, const float* q, int ld_q, const float* k, int ld_k, const float* v, int ld_v,
                                const float* b, int ld_b, const float* g, int ld_g, float eps, float q_scale, float* state,
                                long long slot_stride, const int* seg_q_start, const int* seg_slot, int S, int T, int S_lead,
                                int T_lead, int max_lead, const int* lens, int H, int G, int dk, int dv, float* workspace, long long ws_floats,
                                int* launches, void* stream) {
  *launches = 0;
  if (S <= 0 || T <= 0) return 0;
  if (H <= 0 || G <= 0 || H % G || dk <= 0 || dv <= 0 || H > 65535 || S_lead < 0 || S_lead > S || T_lead < 0 || T_lead > T) return QV_ERR_UNSUPPORTED;
  if (S_lead < S && (dk % 4 || !lens || ((uintptr_t)workspace & 15))) return QV_ERR_UNSUPPORTED;
  if (dk > 256) return QV_ERR_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  if (S_lead > 0) {
    const size_t n = (size_t)T_lead * H * dk;
    float *qh = workspace, *kb = qh + n, *ug = kb + n;
    int rc = qv_delta_operands(qh, kb, ug, q, ld_q, k, ld_k, b, ld_b, g, ld_g, T_lead, H, G, dk, eps, q_scale, stream);
    if (rc) return rc;
    rc = qv_channel_scan(out, ld_out, qh, H * dk, kb, H * dk, v, ld_v, g, ld_g, kb, H * dk, ug, H * dk, 1.0f, state, slot_stride, seg_q_start,
                         seg_slot, S_lead, max_lead, H, dk, dv, stream);
    *launches += 2;
    if (rc || S_lead == S) return rc;
    workspace += 3 * n;
    ws_floats -= 3 * n;
  }
  ChannelDeltaArgs a;
  a.out = out; a.ld_out = ld_out; a.q = q; a.k = k; a.v = v; a.b = b; a.g = g; a.ld_q = ld_q; a.ld_k = ld_k; a.ld_v = ld_v; a.ld_b = ld_b; a.ld_g = ld_g;
  a.ws = workspace; a.state = state; a.slot_stride = slot_stride; a.seg_q_start = seg_q_start + S_lead; a.seg_slot = seg_slot + S_lead;
  a.H = H; a.G = G; a.dk = dk; a.dv = dv; a.dkp = (dk + 15) / 16 * 16; a.dvp = (dv + 15) / 16 * 16; a.eps = eps; a.q_scale = q_scale;
  const int col_tiles = a.dvp / CD_COLS;
  if (col_tiles > 65535) return QV_ERR_TOO_LARGE;
  const int smem = (3 * CD_BLOCK * (a.dkp + 4) + 4 * CD_BLOCK * CD_BLOCK + CD_BLOCK) * 4;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(delta_block_operands_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
  }
  try {
    PortionRounds rounds(lens + S_lead, S - S_lead, CD_BLOCK, 0, cd_room_slots(H, dk, dv), CD_FEW);
    if (ws_floats < (long long)(rounds.slots() * cd_slot_all_heads(H, dk, dv))) return QV_ERR_UNSUPPORTED;
    while (rounds.next(a.round)) {
      int rc = qv_launch(delta_block_operands_kernel, dim3(a.round.slots, H), dim3(CD_OP_THREADS), (size_t)smem, st, a);
      if (rc) return rc;
      const dim3 grid(a.round.items, H, col_tiles);
      rc = dk <= 64 ? launch_delta_blocks<4>(a, grid, st) : dk <= 128 ? launch_delta_blocks<8>(a, grid, st) : launch_delta_blocks<16>(a, grid, st);
      if (rc) return rc;
      *launches += 2;
    }
  } catch (...) {
    return QV_ERR_TOO_LARGE;
  }
  return 0;
}

// ---------------------------------------------------------------- unit norm per head, weight, gate, factor
// y [T, H * dv] float32 -> out[t, h, i] = y / sqrt(mean_i(y^2) + eps) * w[h * dv + i] * gate(g[t, h * dv + i]) * factor,
// gate 0: sigmoid, 1: SiLU; g float32 (row stride ld_g).  One warp per (token, head); the sum's order follows dv alone.
template <typename T>
__global__ void __launch_bounds__(128) head_norm_gate_kernel(T* __restrict__ out, int ld_out, const float* __restrict__ y, int ld_y,
                                                            const float* __restrict__ g, int ld_g, const float* __restrict__ w, int H,
                                                            int dv, float eps, int gate, float factor) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= H) return;
  const float* yr = y + (size_t)t * ld_y + (size_t)h * dv;
  const float* gr = g + (size_t)t * ld_g + (size_t)h * dv;
  const float* wr = w + (size_t)h * dv;
  T* o = out + (size_t)t * ld_out + (size_t)h * dv;
  float ss = 0.f;
  for (int i = lane; i < dv; i += 32) ss = fmaf(yr[i], yr[i], ss);
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss / (float)dv + eps);
  for (int i = lane; i < dv; i += 32) {
    const float z = gr[i];
    const float sg = 1.0f / (1.0f + expf(-z));
    const float gv = gate == 1 ? z * sg : sg;
    o[i] = from_f<T>(yr[i] * inv * wr[i] * gv * factor);
  }
}

// The same for heads of 4 to 512 values in whole pieces of four, 16-byte accesses, each value read once (a lane holds Q pieces).
// 1,531 tokens of 16 heads of 128: 14.1 us with one element a lane and two reads, 9.1 now.
template <typename T, int Q>
__global__ void __launch_bounds__(128) head_norm_gate_vec_kernel(T* __restrict__ out, int ld_out, const float* __restrict__ y, int ld_y,
                                                                const float* __restrict__ g, int ld_g, const float* __restrict__ w, int H,
                                                                int dv, float eps, int gate, float factor) {
  struct alignas(4 * sizeof(T)) Pack { T v[4]; };
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= H) return;
  const float4* yr = (const float4*)(y + (size_t)t * ld_y + (size_t)h * dv);
  const float4* gr = (const float4*)(g + (size_t)t * ld_g + (size_t)h * dv);
  const float4* wr = (const float4*)(w + (size_t)h * dv);
  Pack* o = (Pack*)(out + (size_t)t * ld_out + (size_t)h * dv);
  float4 yv[Q], gv[Q], wv[Q];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int p = lane + 32 * i;
    yv[i] = gv[i] = wv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (4 * p < dv) { yv[i] = yr[p]; gv[i] = gr[p]; wv[i] = wr[p]; }
  }
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    ss = fmaf(yv[i].x, yv[i].x, ss); ss = fmaf(yv[i].y, yv[i].y, ss);
    ss = fmaf(yv[i].z, yv[i].z, ss); ss = fmaf(yv[i].w, yv[i].w, ss);
  }
  const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dv + eps);
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int p = lane + 32 * i;
    if (4 * p >= dv) break;
    const float yy[4] = {yv[i].x, yv[i].y, yv[i].z, yv[i].w}, zz[4] = {gv[i].x, gv[i].y, gv[i].z, gv[i].w},
                ww[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
    Pack r;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float sg = 1.0f / (1.0f + expf(-zz[k]));
      r.v[k] = from_f<T>(yy[k] * inv * ww[k] * (gate == 1 ? zz[k] * sg : sg) * factor);
    }
    o[p] = r;
  }
}

extern "C" int qv_head_norm_gate(void* out, int ld_out, const float* y, int ld_y, const float* g, int ld_g, const float* w, int T, int H,
                                 int dv, float eps, int gate, float factor, int out_dt, void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || dv <= 0 || (gate != 0 && gate != 1)) return QV_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t esz = out_dt == QV_DT_F32 ? 4 : 2;
  const bool vec = dv % 4 == 0 && dv <= 512 && ld_out % 4 == 0 && ld_y % 4 == 0 && ld_g % 4 == 0 &&
                   (((uintptr_t)y | (uintptr_t)g | (uintptr_t)w) & 15) == 0 && ((uintptr_t)out & (4 * esz - 1)) == 0;
  for (int done = 0; done < T; done += 65535) {
    const int rows = T - done < 65535 ? T - done : 65535;
    int rc = QV_ERR_UNSUPPORTED;
    if (vec) {
#define HNG(TT, QQ)                                                                                                              \
  rc = qv_launch(head_norm_gate_vec_kernel<TT, QQ>, dim3(rows, (H + 3) / 4), dim3(128), 0, st,                                    \
                 (TT*)((char*)out + (size_t)done * ld_out * esz), ld_out, y + (size_t)done * ld_y, ld_y, g + (size_t)done * ld_g, ld_g, w, H, \
                 dv, eps, gate, factor)
      QV_DISPATCH_DT(out_dt, TT, if (dv <= 128) HNG(TT, 1); else if (dv <= 256) HNG(TT, 2); else HNG(TT, 4));
#undef HNG
      if (rc) return rc;
      continue;
    }
    QV_DISPATCH_DT(out_dt, TT,
                   rc = qv_launch(head_norm_gate_kernel<TT>, dim3(rows, (H + 3) / 4), dim3(128), 0, st,
                                  (TT*)((char*)out + (size_t)done * ld_out * esz), ld_out, y + (size_t)done * ld_y, ld_y,
                                  g + (size_t)done * ld_g, ld_g, w, H, dv, eps, gate, factor));
    if (rc) return rc;
  }
  return 0;
}
