// Recurrent mixers' kernels: a per-request state of fixed size carried from token to token.
//
// qv_conv_state     short causal convolution per channel with optional bias, optional SiLU and optionally the input
//                   added to the result, the last taps-1 inputs of a request kept as state so that a portion continues
//                   where the last one ended.
// qv_linear_scan    S_t = a_t S_(t-1) + b_t k_t v_t^T;  y_t = S_t^T q_t  per head, S in float32, in two kinds:
//                     GATED_MAX  exponential gates stabilised by a running maximum (matrix-memory LSTM):
//                                log i = cap tanh((gi + bi)/cap), log f = logsigmoid(cap tanh((gf + bf)/cap)),
//                                m_t = max(log f + m_(t-1), log i), a = exp(log f + m_(t-1) - m_t), b = exp(log i - m_t),
//                                n_t = a n_(t-1) + b k_t,  y_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + 1e-6)
//                     DECAY      selective state space with a scalar decay per head:
//                                dt = softplus(g + bias), a = exp(-exp(A_log) dt), b = dt, y_t = S_t^T q_t + D v_t
// qv_gated_group_norm  the unit norm (RMS over equal parts of a row) with weight and gate that follows a scan.
//
// All state arithmetic, gates, decays and norms are float32; q, k and v are read in the compute type.
#include "common.cuh"
#include "per_device.h"
#include "portion_rounds.h"

#define CONV_MAX_TAPS 16
#define CONV_CHUNK 16

// in/out: [T, channels] with row strides and types of their own; w [channels, taps] (last column: the current token),
// bias [channels] or null; tail [slots][(taps-1) * channels] float32, oldest input first.  act 1: SiLU of the sum, 0: the sum
// as it is; add_input 1: the current input is added to the result (out = in + conv(in), after the activation).
// grid (segments, channel tiles, time chunks).  MT: the most taps this instance takes (its arrays stay in registers).
template <typename TI, typename TO, int MT>
__global__ void __launch_bounds__(128) conv_state_kernel(TO* __restrict__ out, int ld_out, const TI* __restrict__ in, int ld_in,
                                                         const float* __restrict__ w, const float* __restrict__ bias,
                                                         float* __restrict__ tail, long long slot_stride,
                                                         const int* __restrict__ seg_q_start, const int* __restrict__ seg_slot,
                                                         int channels, int taps, int act, int add_input) {
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x;
  const int c = blockIdx.y * 128 + threadIdx.x;
  const int q0 = seg_q_start[s], len = seg_q_start[s + 1] - q0;
  const int j0 = blockIdx.z * CONV_CHUNK;
  if (c >= channels || j0 >= len) return;
  const int j1 = j0 + CONV_CHUNK < len ? j0 + CONV_CHUNK : len;
  float* tl = tail + (size_t)seg_slot[s] * slot_stride;
  float curs[CONV_CHUNK];                        // the chunk's inputs, all loads in flight before the first is used
#pragma unroll
  for (int jj = 0; jj < CONV_CHUNK; ++jj) curs[jj] = j0 + jj < j1 ? to_f(in[(size_t)(q0 + j0 + jj) * ld_in + c]) : 0.f;
  float wt[MT], win[MT];
  // win[i]: the input taps - 1 - i places ahead of the token in turn; a chunk is at least as long as the longest filter reaches
  // back, so only the first chunk reads the state
#pragma unroll
  for (int i = 0; i < MT; ++i) {
    wt[i] = i < taps ? w[(size_t)c * taps + i] : 0.f;
    win[i] = 0.f;
    if (i < taps - 1) {
      const int idx = j0 - (taps - 1) + i;
      win[i] = idx >= 0 ? to_f(in[(size_t)(q0 + idx) * ld_in + c]) : tl[(size_t)(taps - 1 + idx) * channels + c];
    }
  }
  if (blockIdx.z == 0) {
    // the state after this segment: its last taps - 1 inputs, or, of a segment shorter than that, what is left of the old state
    // ahead of its own inputs.  Written now from values in registers (only this thread reads or writes these entries).
#pragma unroll
    for (int i = 0; i < MT - 1; ++i) {
      if (i < taps - 1) {
        const int idx = len - (taps - 1) + i;             // place in the segment; below zero: entry len + i of the old state
        float v = 0.f;
        if (idx < 0) {
#pragma unroll
          for (int k = 0; k < MT - 1; ++k)
            if (k == len + i) v = win[k];
        } else if (idx < CONV_CHUNK) {
#pragma unroll
          for (int k = 0; k < CONV_CHUNK; ++k)
            if (k == idx) v = curs[k];
        } else {
          v = to_f(in[(size_t)(q0 + idx) * ld_in + c]);
        }
        tl[(size_t)i * channels + c] = v;
      }
    }
  }
  const float b = bias ? bias[c] : 0.f;
#pragma unroll
  for (int jj = 0; jj < CONV_CHUNK; ++jj) {
    if (j0 + jj >= j1) break;
    const float cur = curs[jj];
    float acc = b;
#pragma unroll
    for (int i = 0; i < MT - 1; ++i) {
      if (i < taps - 1) acc = fmaf(wt[i], win[i], acc);
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      if (i == taps - 1) acc = fmaf(wt[i], cur, acc);
    }
#pragma unroll
    for (int i = 0; i < MT - 1; ++i) {
      if (i < taps - 2) win[i] = win[i + 1];
      else if (i == taps - 2) win[i] = cur;
    }
    if (act) acc = acc / (1.0f + expf(-acc));
    if (add_input) acc += cur;
    out[(size_t)(q0 + j0 + jj) * ld_out + c] = from_f<TO>(acc);
  }
}

// Portions: four neighbouring channels a thread, so that a warp's access is 512 (float32) or 256 bytes of a row; the same sums.  1,943 tokens of 4,352
// channels in bfloat16: 31 us with a channel a thread, 22 here; 1,531 of 4,096 in float32 22 and 15: bound by the SiLUs'
// exponentials and divisions and by the reads.  From 16 tokens on, for filters of 2 to 4 taps (longer ones would not leave the chunk's inputs
// in registers).
template <typename T> struct ConvPack { T v[4]; };
template <> struct alignas(16) ConvPack<float> { float v[4]; };
template <> struct alignas(8) ConvPack<bf16> { bf16 v[4]; };
#define CONV_VEC_CHUNK 8
template <typename TI, typename TO, int TAPS>
__global__ void __launch_bounds__(128) conv_state_vec_kernel(TO* __restrict__ out, int ld_out, const TI* __restrict__ in, int ld_in,
                                                             const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ tail,
                                                             long long slot_stride, const int* __restrict__ seg_q_start,
                                                             const int* __restrict__ seg_slot, int channels, int act, int add_input) {
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x;
  const int c = (blockIdx.y * 128 + threadIdx.x) * 4;
  const int q0 = seg_q_start[s], len = seg_q_start[s + 1] - q0;
  const int j0 = blockIdx.z * CONV_VEC_CHUNK;
  if (c >= channels || j0 >= len) return;
  const int n = len - j0 < CONV_VEC_CHUNK ? len - j0 : CONV_VEC_CHUNK;
  float* tl = tail + (size_t)seg_slot[s] * slot_stride;
  const TI* ip = in + (size_t)q0 * ld_in + c;
  ConvPack<TI> cur[CONV_VEC_CHUNK] = {};                 // the chunk's inputs, all loads in flight before the first is used
#pragma unroll
  for (int j = 0; j < CONV_VEC_CHUNK; ++j)
    if (j < n) cur[j] = *(const ConvPack<TI>*)(ip + (size_t)(j0 + j) * ld_in);
  float wt[TAPS][4], win[TAPS - 1][4], b[4];         // win[i]: the input TAPS - 1 - i places ahead of the token in turn
#pragma unroll
  for (int i = 0; i < TAPS - 1; ++i) {
    const int idx = j0 - (TAPS - 1) + i;
    if (idx >= 0) {
      const ConvPack<TI> p = *(const ConvPack<TI>*)(ip + (size_t)idx * ld_in);
#pragma unroll
      for (int k = 0; k < 4; ++k) win[i][k] = to_f(p.v[k]);
    } else {
      const float4 p = *(const float4*)(tl + (size_t)(TAPS - 1 + idx) * channels + c);
      win[i][0] = p.x; win[i][1] = p.y; win[i][2] = p.z; win[i][3] = p.w;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    b[k] = bias ? bias[c + k] : 0.f;
#pragma unroll
    for (int i = 0; i < TAPS; ++i) wt[i][k] = w[(size_t)(c + k) * TAPS + i];
  }
  if (j0 == 0) {
    // the state after this segment: its last TAPS - 1 inputs, or, of a segment shorter than that, what is left of the old state ahead of its
    // own inputs (only this thread reads or writes these entries)
#pragma unroll
    for (int i = 0; i < TAPS - 1; ++i) {
      const int idx = len - (TAPS - 1) + i;          // place in the segment; below zero: entry len + i of the old state
      float4 v;
      if (idx >= 0) {
        const ConvPack<TI> p = *(const ConvPack<TI>*)(ip + (size_t)idx * ld_in);
        v = make_float4(to_f(p.v[0]), to_f(p.v[1]), to_f(p.v[2]), to_f(p.v[3]));
      } else {
        v = *(const float4*)(tl + (size_t)(len + i) * channels + c);           // (an entry behind those written so far)
      }
      *(float4*)(tl + (size_t)i * channels + c) = v;
    }
  }
  TO* op = out + (size_t)(q0 + j0) * ld_out + c;
#pragma unroll
  for (int j = 0; j < CONV_VEC_CHUNK; ++j) {
    if (j >= n) break;
    ConvPack<TO> o;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float x = to_f(cur[j].v[k]);
      float acc = b[k];
#pragma unroll
      for (int i = 0; i < TAPS - 1; ++i) acc = fmaf(wt[i][k], win[i][k], acc);
      acc = fmaf(wt[TAPS - 1][k], x, acc);
#pragma unroll
      for (int i = 0; i < TAPS - 1; ++i) win[i][k] = i < TAPS - 2 ? win[i + 1][k] : x;
      if (act) acc = acc / (1.0f + expf(-acc));
      if (add_input) acc += x;
      o.v[k] = from_f<TO>(acc);
    }
    *(ConvPack<TO>*)(op + (size_t)j * ld_out) = o;
  }
}

extern "C" int qv_conv_state(void* out, int ld_out, const void* in, int ld_in, const float* w, const float* bias, float* tail,
                             long long slot_stride, const int* seg_q_start, const int* seg_slot, int S, int max_q_len,
                             int channels, int taps, int in_dt, int out_dt, int act, int add_input, void* stream) {
  if (S <= 0 || channels <= 0) return 0;
  if (taps < 1 || taps > CONV_MAX_TAPS) return QV_ERR_UNSUPPORTED;
  const int chunks = max_q_len > 0 ? (max_q_len + CONV_CHUNK - 1) / CONV_CHUNK : 1;
  if (chunks > 65535 || (channels + 127) / 128 > 65535) return QV_ERR_TOO_LARGE;
  dim3 grid(S, (channels + 127) / 128, chunks);
  const bool vec = max_q_len >= CONV_CHUNK && max_q_len <= 65535 * CONV_VEC_CHUNK && taps >= 2 && taps <= 4 && channels % 4 == 0 && ld_in % 4 == 0 && ld_out % 4 == 0 && slot_stride % 4 == 0 &&
                   ((uintptr_t)tail & 15) == 0 && ((uintptr_t)in & (in_dt == QV_DT_F32 ? 15 : 7)) == 0 &&
                   ((uintptr_t)out & (out_dt == QV_DT_F32 ? 15 : 7)) == 0;
  const int vchunks = (max_q_len + CONV_VEC_CHUNK - 1) / CONV_VEC_CHUNK;
  const dim3 vgrid(S, (channels / 4 + 127) / 128, vchunks);
#define LAUNCH_CONV_VEC(TI, TO, TAPS)                                                                                          \
  return qv_launch(conv_state_vec_kernel<TI, TO, TAPS>, vgrid, dim3(128), 0, (cudaStream_t)stream, (TO*)out, ld_out,           \
                   (const TI*)in, ld_in, w, bias, tail, slot_stride, seg_q_start, seg_slot, channels, act, add_input)
#define LAUNCH_CONV(TI, TO)                                                                                                    \
  do {                                                                                                                         \
    if (vec && taps == 2) LAUNCH_CONV_VEC(TI, TO, 2);                                                                          \
    if (vec && taps == 3) LAUNCH_CONV_VEC(TI, TO, 3);                                                                          \
    if (vec) LAUNCH_CONV_VEC(TI, TO, 4);                                                                                       \
    if (taps <= 4)                                                                                                             \
      return qv_launch(conv_state_kernel<TI, TO, 4>, grid, dim3(128), 0, (cudaStream_t)stream, (TO*)out, ld_out, (const TI*)in, \
                       ld_in, w, bias, tail, slot_stride, seg_q_start, seg_slot, channels, taps, act, add_input);              \
    return qv_launch(conv_state_kernel<TI, TO, CONV_MAX_TAPS>, grid, dim3(128), 0, (cudaStream_t)stream, (TO*)out, ld_out,     \
                     (const TI*)in, ld_in, w, bias, tail, slot_stride, seg_q_start, seg_slot, channels, taps, act, add_input); \
  } while (0)
  if (in_dt == QV_DT_F32 && out_dt == QV_DT_F32) LAUNCH_CONV(float, float);
  if (in_dt == QV_DT_BF16 && out_dt == QV_DT_BF16) LAUNCH_CONV(bf16, bf16);
  if (in_dt == QV_DT_F32 && out_dt == QV_DT_BF16) LAUNCH_CONV(float, bf16);
  if (in_dt == QV_DT_BF16 && out_dt == QV_DT_F32) LAUNCH_CONV(bf16, float);
#undef LAUNCH_CONV
#undef LAUNCH_CONV_VEC
  return QV_ERR_UNSUPPORTED;
}

// ---------------------------------------------------------------- the scan
#define SCAN_VT 32          // value columns per block (one per lane)
#define SCAN_WARPS 8        // the key rows are dealt to the warps
#define SCAN_GATED_MAX 0
#define SCAN_DECAY 1

struct ScanArgs {
  float* out; int ld_out;                 // [T, H * dv] float32
  const void* q; int ld_q; int q_group;   // head h reads columns (h / q_group) * dk ... of q and of k
  const void* k; int ld_k;
  const void* v; int ld_v;                // head h reads columns h * dv ...
  const float* g1; int ld_g1;             // [T, >= H]: input-gate pre-activation | step pre-activation
  const float* g2; int ld_g2;             // [T, >= H]: forget-gate pre-activation (GATED_MAX)
  const float* p1; const float* p2; const float* p3;   // per head: bi | dt bias;  bf | A_log;  - | D
  float cap; float q_scale;
  float* state; long long slot_stride;    // per slot: [H][tiles][dk * 32 (+ dk + 1 for GATED_MAX)]
  const int* seg_q_start; const int* seg_slot;
  int H, dk, dv;
  int chunk_from;                         // segments of at least this many tokens are linear_scan_chunk_kernel's (INT_MAX: none),
  int parallel_from;                      // of at least this many lp_states_kernel's and lp_outputs_kernel's
};

__host__ __device__ inline int scan_tile_floats(int kind, int dk, int vt = SCAN_VT) { return dk * vt + (kind == SCAN_GATED_MAX ? dk + 1 : 0); }
// Value columns a CTA owns: 32, or 16 for key sizes of 129..256, where a thread would else keep 32 rows (more than
// its registers hold) and wide heads give few CTAs.  A function of the key size alone: the state's layout follows it.
static inline int scan_vt(int dk) { return (dk > 128 && dk <= 256) ? 16 : 32; }

template <typename T, int KIND>
__global__ void __launch_bounds__(SCAN_VT * SCAN_WARPS) linear_scan_kernel(ScanArgs a) {
  extern __shared__ float sm[];
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, tile = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dk = a.dk, dv = a.dv;
  const int tiles = (dv + SCAN_VT - 1) / SCAN_VT;
  float* S = sm;                           // [dk][32]
  float* qs = S + (size_t)dk * SCAN_VT;    // [dk]
  float* ks = qs + dk;                     // [dk]
  float* ns = ks + dk;                     // [dk] (GATED_MAX)
  float* red = ns + dk;                    // [SCAN_WARPS][32]
  float* sc = red + SCAN_WARPS * SCAN_VT;  // [2]: n . q, spare
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  if (len >= a.chunk_from) return;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + ((size_t)h * tiles + tile) * scan_tile_floats(KIND, dk);
  for (int i = threadIdx.x; i < dk * SCAN_VT; i += blockDim.x) S[i] = st[i];
  float m = 0.f;
  if (KIND == SCAN_GATED_MAX) {
    for (int i = threadIdx.x; i < dk; i += blockDim.x) ns[i] = st[dk * SCAN_VT + i];
    m = st[dk * SCAN_VT + dk];
  }
  const int col = tile * SCAN_VT + lane;
  const bool live = col < dv;
  const T* qb = (const T*)a.q + (size_t)(h / a.q_group) * dk;
  const T* kb = (const T*)a.k + (size_t)(h / a.q_group) * dk;
  const T* vb = (const T*)a.v + (size_t)h * dv;
  const float b1 = a.p1 ? a.p1[h] : 0.f, b2 = a.p2 ? a.p2[h] : 0.f, b3 = a.p3 ? a.p3[h] : 0.f;
  __syncthreads();
  for (int j = 0; j < len; ++j) {
    const size_t t = (size_t)(q0 + j);
    for (int i = threadIdx.x; i < dk; i += blockDim.x) {
      qs[i] = to_f(qb[t * a.ld_q + i]) * a.q_scale;
      ks[i] = to_f(kb[t * a.ld_k + i]);
    }
    const float vv = live ? to_f(vb[t * a.ld_v + col]) : 0.f;
    float keep, take;
    if (KIND == SCAN_GATED_MAX) {
      const float li = a.cap * tanhf((a.g1[t * a.ld_g1 + h] + b1) / a.cap);
      const float zf = a.cap * tanhf((a.g2[t * a.ld_g2 + h] + b2) / a.cap);
      const float lf = fminf(zf, 0.f) - log1pf(expf(-fabsf(zf)));          // log sigmoid
      const float m_new = fmaxf(lf + m, li);
      keep = expf(lf + m - m_new);
      take = expf(li - m_new);
      m = m_new;
    } else {
      const float z = a.g1[t * a.ld_g1 + h] + b1;
      const float dt = z > 20.f ? z : log1pf(expf(z));                      // softplus
      keep = expf(-expf(b2) * dt);
      take = dt;
    }
    __syncthreads();                       // qs, ks are in place; red of the last token has been read
    if (KIND == SCAN_GATED_MAX && warp == 0) {
      float dot = 0.f;
      for (int i = lane; i < dk; i += 32) {
        const float n = keep * ns[i] + take * ks[i];
        ns[i] = n;
        dot = fmaf(n, qs[i], dot);
      }
      dot = warp_sum(dot);
      if (lane == 0) sc[0] = dot;
    }
    float acc = 0.f;
    const float tv = take * vv;
    for (int i = warp; i < dk; i += SCAN_WARPS) {
      const float sv = fmaf(keep, S[i * SCAN_VT + lane], tv * ks[i]);
      S[i * SCAN_VT + lane] = sv;
      acc = fmaf(sv, qs[i], acc);
    }
    red[warp * SCAN_VT + lane] = acc;
    __syncthreads();
    if (warp == 0 && live) {
      float y = 0.f;
#pragma unroll
      for (int w = 0; w < SCAN_WARPS; ++w) y += red[w * SCAN_VT + lane];
      if (KIND == SCAN_GATED_MAX) y = y / (fmaxf(fabsf(sc[0]), expf(-m)) + 1e-6f);
      else y = fmaf(b3, vv, y);
      a.out[t * a.ld_out + (size_t)h * dv + col] = y;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < dk * SCAN_VT; i += blockDim.x) st[i] = S[i];
  if (KIND == SCAN_GATED_MAX) {
    for (int i = threadIdx.x; i < dk; i += blockDim.x) st[dk * SCAN_VT + i] = ns[i];
    if (threadIdx.x == 0) st[dk * SCAN_VT + dk] = m;
  }
}

// The same recurrence with the state in registers (key sizes up to 8 * RPT rows: a thread keeps RPT rows of its value
// column) and tokens taken four at a time: their inputs are fetched together, the block meets twice per four tokens
// instead of twice per token, and each of the first four warps sums one token's partial outputs.  Arithmetic and
// summation order are those of linear_scan_kernel; the state's layout in memory is the same.
#define SCAN_TB 4
#define SCAN_CH 256      // tokens whose gates are worked out together (one a thread)
// ASYNC: the rows of q and k start on 16 bytes, and the next four tokens' rows are copied into the other of two
// buffers by cp.async while the present four are worked on (else plain loads ahead of the work).
template <typename T, int KIND, int RPT, bool ASYNC, int VT>
__global__ void __launch_bounds__(SCAN_VT * SCAN_WARPS) linear_scan_reg_kernel(ScanArgs a) {
  extern __shared__ __align__(16) float sm[];
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, tile = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dk = a.dk, dv = a.dv;
  constexpr int RS = 32 / VT;                       // row groups a warp: with 16 columns a tile, the lanes' halves take alternate rows
  const int cl = lane % VT, rsub = lane / VT;
  const int tiles = (dv + VT - 1) / VT;
  const int rowpad = (dk + 7) & ~7;                // a token's row in the buffers (elements): whole 16-byte pieces
  T* raw = (T*)sm;                                 // [2 buffers][q, k][TB][rowpad] as stored (the scale of q is applied to the sums)
  float* ns = sm + (4 * SCAN_TB * rowpad * sizeof(T) + 3) / 4;   // [dk]
  float* red = ns + dk;                            // [TB][SCAN_WARPS][32]
  float* sc = red + SCAN_TB * SCAN_WARPS * SCAN_VT;  // [TB]
  float* gk = sc + SCAN_TB;                        // [SCAN_CH] keep factors of the tokens in work
  float* gt = gk + SCAN_CH;                        // [SCAN_CH] take factors
  float* ge = gt + SCAN_CH;                        // [SCAN_CH] exp(-m) (GATED_MAX)
  float* gm = ge + SCAN_CH;                        // [SCAN_CH] scratch of the running maximum
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  if (len >= a.chunk_from) return;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + ((size_t)h * tiles + tile) * scan_tile_floats(KIND, dk, VT);
  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int k = warp * RS + rsub + SCAN_WARPS * RS * i;
    S[i] = k < dk ? st[k * VT + cl] : 0.f;
  }
  float m = 0.f;
  if (KIND == SCAN_GATED_MAX) {
    for (int i = threadIdx.x; i < dk; i += blockDim.x) ns[i] = st[dk * VT + i];
    m = st[dk * VT + dk];
  }
  const int col = tile * VT + cl;
  const bool live = col < dv;
  const T* qb = (const T*)a.q + (size_t)(h / a.q_group) * dk;
  const T* kb = (const T*)a.k + (size_t)(h / a.q_group) * dk;
  const T* vb = (const T*)a.v + (size_t)h * dv;
  const float b1 = a.p1 ? a.p1[h] : 0.f, b2 = a.p2 ? a.p2[h] : 0.f, b3 = a.p3 ? a.p3[h] : 0.f;
  const float rate = KIND == SCAN_DECAY ? expf(b2) : 0.f;
  auto issue = [&](int buf, int j0) {
    const int nb = len - j0 < SCAN_TB ? len - j0 : SCAN_TB;
    const int pieces = dk * (int)sizeof(T) / 16, per = 16 / (int)sizeof(T);
    T* dst = raw + (size_t)buf * 2 * SCAN_TB * rowpad;
    for (int c = threadIdx.x; c < 2 * nb * pieces; c += blockDim.x) {
      const int which = c / (nb * pieces), rem = c - which * nb * pieces, tt = rem / pieces, pc = rem - tt * pieces;
      const T* src = (which ? kb + (size_t)(q0 + j0 + tt) * a.ld_k : qb + (size_t)(q0 + j0 + tt) * a.ld_q) + pc * per;
      const unsigned sa = (unsigned)__cvta_generic_to_shared(dst + (which * SCAN_TB + tt) * rowpad + pc * per);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (ASYNC) issue(0, 0);
  // Gates are worked out for 256 tokens at a time, one token a thread, and kept in shared memory: the transcendental
  // functions then lie off the path from one token to the next.  Only the running maximum is a chain (thread 0).
  for (int c0 = 0; c0 < len; c0 += SCAN_CH) {
    const int nch = len - c0 < SCAN_CH ? len - c0 : SCAN_CH;
    __syncthreads();                         // the gates of the last 256 tokens have been used
    if ((int)threadIdx.x < nch) {
      const size_t t = (size_t)(q0 + c0 + threadIdx.x);
      if (KIND == SCAN_GATED_MAX) {
        const float zf = a.cap * tanhf((a.g2[t * a.ld_g2 + h] + b2) / a.cap);
        gk[threadIdx.x] = fminf(zf, 0.f) - log1pf(expf(-fabsf(zf)));          // log forget gate
        gt[threadIdx.x] = a.cap * tanhf((a.g1[t * a.ld_g1 + h] + b1) / a.cap);  // log input gate
      } else {
        const float z = a.g1[t * a.ld_g1 + h] + b1;
        const float dt = z > 20.f ? z : log1pf(expf(z));
        gk[threadIdx.x] = expf(-rate * dt);
        gt[threadIdx.x] = dt;
      }
    }
    if (KIND == SCAN_GATED_MAX) {
      __syncthreads();
      if (threadIdx.x == 0) {
        float mm = m;
        for (int j = 0; j < nch; ++j) {
          const float m_new = fmaxf(gk[j] + mm, gt[j]);
          gm[j] = mm;                          // the maximum before this token
          ge[j] = m_new;                       // and after it
          mm = m_new;
        }
      }
      __syncthreads();
      m = ge[nch - 1];
      __syncthreads();                       // everyone has the maximum before its place is used for exp(-m)
      if ((int)threadIdx.x < nch) {
        const float lf = gk[threadIdx.x], li = gt[threadIdx.x], mp = gm[threadIdx.x], mc = ge[threadIdx.x];
        gk[threadIdx.x] = expf(lf + mp - mc);
        gt[threadIdx.x] = expf(li - mc);
        ge[threadIdx.x] = expf(-mc);
      }
    }
    __syncthreads();
  for (int j0 = c0; j0 < c0 + nch; j0 += SCAN_TB) {
    const int nb = c0 + nch - j0 < SCAN_TB ? c0 + nch - j0 : SCAN_TB;
    const size_t t0 = (size_t)(q0 + j0);
    const int buf = (j0 / SCAN_TB) & 1;
    const T* qs = raw + (size_t)buf * 2 * SCAN_TB * rowpad;
    const T* ks = qs + SCAN_TB * rowpad;
    if (ASYNC) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
      T* wq = raw + (size_t)buf * 2 * SCAN_TB * rowpad;
      for (int c = threadIdx.x; c < nb * dk; c += blockDim.x) {
        const int tt = c / dk, i = c - tt * dk;
        wq[tt * rowpad + i] = qb[(t0 + tt) * a.ld_q + i];
        wq[(SCAN_TB + tt) * rowpad + i] = kb[(t0 + tt) * a.ld_k + i];
      }
    }
    float vv[SCAN_TB], keep[SCAN_TB], take[SCAN_TB], mt[SCAN_TB];
#pragma unroll
    for (int tt = 0; tt < SCAN_TB; ++tt) {
      vv[tt] = 0.f; keep[tt] = 1.f; take[tt] = 0.f; mt[tt] = 1.f;
      if (tt < nb) {
        vv[tt] = live ? to_f(vb[(t0 + tt) * a.ld_v + col]) : 0.f;
        keep[tt] = gk[j0 - c0 + tt];
        take[tt] = gt[j0 - c0 + tt];
        if (KIND == SCAN_GATED_MAX) mt[tt] = ge[j0 - c0 + tt];          // exp(-m) after the token
      }
    }
    __syncthreads();                       // the four tokens' q and k are in place; red and sc of the last four have been read
    if (ASYNC && j0 + SCAN_TB < len) issue(buf ^ 1, j0 + SCAN_TB);
    if (KIND == SCAN_GATED_MAX && warp == 0) {
      for (int tt = 0; tt < nb; ++tt) {
        float dot = 0.f;
        for (int i = lane; i < dk; i += 32) {
          const float n = keep[tt] * ns[i] + take[tt] * to_f(ks[tt * rowpad + i]);
          ns[i] = n;
          dot = fmaf(n, to_f(qs[tt * rowpad + i]), dot);
        }
        dot = warp_sum(dot);
        if (lane == 0) sc[tt] = dot * a.q_scale;
      }
    }
#pragma unroll
    for (int tt = 0; tt < SCAN_TB; ++tt) {
      if (tt < nb) {
        float acc = 0.f;
        const float tv = take[tt] * vv[tt];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int k = warp * RS + rsub + SCAN_WARPS * RS * i;
          if (k < dk) {
            S[i] = fmaf(keep[tt], S[i], tv * to_f(ks[tt * rowpad + k]));
            acc = fmaf(S[i], to_f(qs[tt * rowpad + k]), acc);
          }
        }
        red[(tt * SCAN_WARPS + warp) * SCAN_VT + lane] = acc;
      }
    }
    __syncthreads();
    if (warp < nb && live && rsub == 0) {
      const int tt = warp;
      float y = 0.f;
#pragma unroll
      for (int w = 0; w < SCAN_WARPS; ++w)
#pragma unroll
        for (int g = 0; g < RS; ++g) y += red[(tt * SCAN_WARPS + w) * SCAN_VT + g * VT + cl];
      y *= a.q_scale;
      // vv and mt of token tt, which this thread holds at a compile-time index only: pick without indexing registers
      float v_tt = vv[0], m_tt = mt[0];
#pragma unroll
      for (int x = 1; x < SCAN_TB; ++x) if (x == tt) { v_tt = vv[x]; m_tt = mt[x]; }
      if (KIND == SCAN_GATED_MAX) y = y / (fmaxf(fabsf(sc[tt]), m_tt) + 1e-6f);
      else y = fmaf(b3, v_tt, y);
      a.out[(t0 + tt) * a.ld_out + (size_t)h * dv + col] = y;
    }
  }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int k = warp * RS + rsub + SCAN_WARPS * RS * i;
    if (k < dk) st[k * VT + cl] = S[i];
  }
  if (KIND == SCAN_GATED_MAX) {
    for (int i = threadIdx.x; i < dk; i += blockDim.x) st[dk * VT + i] = ns[i];
    if (threadIdx.x == 0) st[dk * VT + dk] = m;
  }
}

// ---------------------------------------------------------------- portions: tokens in chunks, on the tensor cores (bfloat16 q, k, v)
// Within a chunk of 64 tokens, with the decays' running logarithm F_t (from the chunk's start), the running maximum m_t and S_0 the state
// ahead of the chunk:
//   y_t   = A_t S_0^T q_t + sum_{j <= t} W_tj v_j        W_tj = exp(G_t + H_j) b_j (q_t . k_j),  A_t = exp(G_t + m_0)
//   S_end = A_63 S_0 + sum_j (c_j v_j) k_j^T             c_j  = exp(G_63 + H_j) b_j
// GATED_MAX: G_t = F_t - m_t, H_j = log i_j - F_j, b_j = 1, m_t = F_t + max(m_0, max_{j <= t} H_j), and n . q is n_0's share plus the rows'
// sums of W.  DECAY: G_t = F_t, H_j = -F_j, b_j = dt_j, m_0 = 0.  Every exponent is <= 0; F, m, G and H are kept in float64, so that the
// difference of two long sums is as good as a short one; for W, G and H are kept as pairs of float32.
// All four products are mma.sync with float32 sums whose one operand holds bfloat16 values as they are stored (q, k, v) and whose other
// is a float32 quantity (state, W, c v) in three bfloat16 terms that hold its 24 bits: what was float32 in the token-by-token kernel is
// as exact here.
// A CTA owns a (segment, head, tile of VT value columns) and keeps its state in registers as S^T: a warp has 16 columns and a slice of
// 16 NK key rows, laid out so that the accumulators of the update are, term by term, the second operand of S^T q without any exchange.
// Products with S_0 are split over the key slices, so the slices' sums meet in shared memory.  Eight warps hold the state (first S^T q,
// then the update), eight form W and W v (then the sums and the output); one of these, whose part of W is empty, works out the next chunk's
// gates; the next chunk's
// q, k, v arrive by cp.async (a bulk copy a row takes its issuing warp 50 clocks, three times what the chunk may take): a chunk is two stretches between CTA barriers.  n . q is formed like a value column's.
// The tensor cores cut the sums' low bits off as they add; so long sums are taken in short runs that are added in float32, a term's small
// parts apart from its large one, and the update apart from the state.
// What bounds it: a chunk's chain of products and the two barriers (a prompt has only heads x tiles CTAs); mma.sync issues a product in
// some 8 clocks a scheduler.  2,048 tokens of 4 heads of 256 x 512: 2,573 us token by token, 175 in chunks; portions of 777, 583 and
// 583 tokens of 64 heads of 128 x 64: 897 and 80 us (90 with an exponential for every entry of W).
#define LC_C 64
__device__ __forceinline__ void lc_ldsm4(uint32_t* r, const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void lc_ldsm4t(uint32_t* r, const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void lc_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from zero.
__device__ __forceinline__ void lc_mma0(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void lc_mma(bool first, float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if (first) lc_mma0(c, a, b0, b1);
  else lc_mma(c, a, b0, b1);
}
// x and y as three bfloat16 terms each (x in the lower half of a word)
__device__ __forceinline__ void lc_split3(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    t[i] = *(const uint32_t*)&h;
    x -= __low2float(h);
    y -= __high2float(h);
  }
}

__device__ __forceinline__ void lc_cp16(void* dst, const void* src, bool live) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ float2 lc_pair(double x) {
  const float hi = (float)x;
  return make_float2(hi, (float)(x - (double)hi));
}
// exp(x + y) of two such numbers whose sum is small beside them (Knuth's two-sum: what the first sum's rounding dropped)
__device__ __forceinline__ float lc_exp_sum(float2 x, float2 y) {
  const float s = x.x + y.x, b = s - x.x;
  const float e = (x.x - (s - b)) + (y.x - b);
  return expf(s + (e + (x.y + y.y)));
}

struct LcGates {                           // what a chunk's gates amount to
  float2 G[LC_C], H[LC_C];                           // a number and what rounding it to float32 left over
  float b[LC_C], A[LC_C], c[LC_C], em[LC_C];         // em: exp(-m_t)
  float R[3][LC_C], E[LC_C];                         // blocks of 16 tokens, M_i the largest H in block i: exp(G_t + M_i) for t behind it, b_j exp(H_j - M)
  float A_end, m_end, pad[2];
};
#define LC_GATE_WARP 9                     // of the eight that form W: its 16 x 32 tokens lie above the diagonal
#define LC_BATCH 512                       // tokens whose gates' logarithms are worked out together, by all threads

template <int VT, int NK> struct LcShape {
  static constexpr int SLICES = VT == 16 ? 8 : 4;    // key slices; warps = slices x (VT / 16)
  static constexpr int DKP = SLICES * 16 * NK;
  static constexpr int LDQ = DKP + 8, LDV = VT + 8, LDR = VT + 8;
  static constexpr int STAGE = 2 * LC_C * LDQ * 2;                                     // bytes: q and k of a chunk
  static constexpr int RED = (SLICES + 2) * LC_C * LDR * 4;                            // the slices' sums, and W v's two
  static constexpr int V = LC_C * LDV * 2;
  static constexpr int BYTES = 2 * STAGE + RED + 5 * V + 2 * (int)sizeof(LcGates) + LC_C * 2 * 4 + SLICES * LC_C * 4 + 2 * LC_BATCH * 4 + 2 * DKP * 4;
};

#define LC_THREADS 512
// A segment's share (one head, one tile of value columns) token by token, from the state as the step found it: for values that are infinite
// or NaN.  Within a chunk the weights of later tokens are set to zero, which does not keep their infinities out of earlier tokens' sums;
// here a token sees its own and earlier ones only.  Slow (some microseconds a token), and apart from the chunks' loop, which it would
// cost registers (2,048 tokens of 4 heads of 256 x 512: 271 us a layer with the chunk's own sums formed once more in place, 264 so).
// n0: n ahead of the first token, n_parts sums of n_ld entries.
template <int KIND, int VT, int THREADS>
__device__ __noinline__ void lc_token_by_token(const ScanArgs& a, const float* n0, int n_parts, int n_ld, int s, int q0, int len, int h, int tile,
                                               float* S) {
  constexpr int PARTS = THREADS / VT;
  const int dk = a.dk, tid = threadIdx.x, col = tid % VT, part = tid / VT;
  float* qs = S + dk * VT;                           // S [dk][VT]
  float* ks = qs + dk;
  float* ns = ks + dk;
  float* sums = ns + dk;                             // [PARTS][VT]
  float* sc = sums + THREADS;                     // n . q
  const int tiles = (a.dv + VT - 1) / VT;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + ((size_t)h * tiles + tile) * scan_tile_floats(KIND, dk, VT);
  for (int i = tid; i < dk * VT; i += THREADS) S[i] = st[i];
  float m = 0.f;
  if (KIND == SCAN_GATED_MAX) {
    for (int i = tid; i < dk; i += THREADS) {
      float n = 0.f;
      for (int p = 0; p < n_parts; ++p) n += n0[(size_t)p * n_ld + i];
      ns[i] = n;
    }
    m = st[dk * VT + dk];
  }
  const bool live = tile * VT + col < a.dv;
  const float b1 = a.p1 ? a.p1[h] : 0.f, b2 = a.p2 ? a.p2[h] : 0.f, b3 = a.p3 ? a.p3[h] : 0.f;
  for (int j = 0; j < len; ++j) {
    const size_t t = (size_t)(q0 + j);
    for (int i = tid; i < dk; i += THREADS) {
      qs[i] = to_f(((const bf16*)a.q)[t * a.ld_q + (size_t)(h / a.q_group) * dk + i]) * a.q_scale;
      ks[i] = to_f(((const bf16*)a.k)[t * a.ld_k + (size_t)(h / a.q_group) * dk + i]);
    }
    const float v = live ? to_f(((const bf16*)a.v)[t * a.ld_v + (size_t)h * a.dv + tile * VT + col]) : 0.f;
    float keep, take;
    if (KIND == SCAN_GATED_MAX) {
      const float li = a.cap * tanhf((a.g1[t * a.ld_g1 + h] + b1) / a.cap), zf = a.cap * tanhf((a.g2[t * a.ld_g2 + h] + b2) / a.cap);
      const float lf = fminf(zf, 0.f) - log1pf(expf(-fabsf(zf)));
      const float m_new = fmaxf(lf + m, li);
      keep = expf(lf + m - m_new);
      take = expf(li - m_new);
      m = m_new;
    } else {
      const float z = a.g1[t * a.ld_g1 + h] + b1;
      take = z > 20.f ? z : log1pf(expf(z));
      keep = expf(-expf(b2) * take);
    }
    __syncthreads();                                 // q and k are in place; the last token's sums have been read
    if (KIND == SCAN_GATED_MAX && tid < 32) {
      float dot = 0.f;
      for (int i = tid; i < dk; i += 32) {
        const float n = keep * ns[i] + take * ks[i];
        ns[i] = n;
        dot = fmaf(n, qs[i], dot);
      }
      dot = warp_sum(dot);
      if (tid == 0) *sc = dot;
    }
    float acc = 0.f;
    for (int i = part; i < dk; i += PARTS) {
      const float x = fmaf(keep, S[i * VT + col], take * v * ks[i]);
      S[i * VT + col] = x;
      acc = fmaf(x, qs[i], acc);
    }
    sums[part * VT + col] = acc;
    __syncthreads();
    if (part == 0 && live) {
      float y = 0.f;
      for (int i = 0; i < PARTS; ++i) y += sums[i * VT + col];
      y = KIND == SCAN_GATED_MAX ? y / (fmaxf(fabsf(*sc), expf(-m)) + 1e-6f) : fmaf(b3, v, y);
      a.out[t * a.ld_out + (size_t)h * a.dv + tile * VT + col] = y;
    }
  }
  __syncthreads();
  for (int i = tid; i < dk * VT; i += THREADS) st[i] = S[i];
  if (KIND == SCAN_GATED_MAX) {
    for (int i = tid; i < dk; i += THREADS) st[dk * VT + i] = ns[i];
    if (tid == 0) st[dk * VT + dk] = m;
  }
  __syncthreads();
}

template <int KIND, int VT, int NK>
__global__ void __launch_bounds__(LC_THREADS, 1) linear_scan_chunk_kernel(const __grid_constant__ ScanArgs a) {
  typedef LcShape<VT, NK> Sh;
  constexpr int SLICES = Sh::SLICES, DKP = Sh::DKP, LDQ = Sh::LDQ, LDV = Sh::LDV, LDR = Sh::LDR;
  extern __shared__ __align__(16) unsigned char lc_smem[];
  unsigned char* stages = lc_smem;                                   // [2][q | k]
  float* red = (float*)(lc_smem + 2 * Sh::STAGE);                    // [SLICES + 2][64][LDR]
  bf16* vbuf = (bf16*)(lc_smem + 2 * Sh::STAGE + Sh::RED);           // [2][64][LDV]
  bf16* vs = vbuf + 2 * LC_C * LDV;                                  // [3][64][LDV] terms of c_j v_j
  LcGates* gates = (LcGates*)(vs + 3 * LC_C * LDV);                  // [2]
  float* rowsum = (float*)(gates + 2);                               // [64][2]
  float* nq = rowsum + LC_C * 2;                                     // [SLICES][64] the slices' shares of A_t n_0 . q_t
  float* lfb = nq + SLICES * LC_C;                                   // [LC_BATCH] log of the decay
  float* lib = lfb + LC_BATCH;                                       // [LC_BATCH] log of the input gate | step size
  float* ns = lib + LC_BATCH;                                        // [2][DKP] n as two sums (GATED_MAX)
  pdl_wait();
  pdl_launch_dependents();
  const int s = blockIdx.x, h = blockIdx.y, tile = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  if (len < a.chunk_from || len >= a.parallel_from) return;
  const int dk = a.dk, dv = a.dv;
  const int tiles = (dv + VT - 1) / VT;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + ((size_t)h * tiles + tile) * scan_tile_floats(KIND, dk, VT);
  const bf16* qb = (const bf16*)a.q + (size_t)(h / a.q_group) * dk;
  const bf16* kb = (const bf16*)a.k + (size_t)(h / a.q_group) * dk;
  const bf16* vb = (const bf16*)a.v + (size_t)h * dv + tile * VT;
  const int nchunks = (len + LC_C - 1) / LC_C;
  const int slice = warp % SLICES, half = (warp / SLICES) * 16;      // of the state's warps: key rows, value columns
  const int k0 = slice * 16 * NK;
  const int g8 = lane >> 2, t4 = lane & 3, mi = lane >> 3, r8 = lane & 7;

  // chunk c's q, k, v (zeros beyond the segment and beyond dk): a thread copies the same 16 bytes of every few rows
  constexpr int PQ = DKP / 8, PV = VT / 8, RSTEP = LC_THREADS / PQ;
  const int qrow = tid / PQ, qpc = tid % PQ, vrow = tid / PV, vpc = tid % PV;
  const bf16* qp = qb + (size_t)(q0 + qrow) * a.ld_q + qpc * 8;
  const bf16* kp = kb + (size_t)(q0 + qrow) * a.ld_k + qpc * 8;
  const bf16* vp = vb + (size_t)(q0 + vrow) * a.ld_v + vpc * 8;
  const bool q_in = qpc * 8 < dk, v_in = vrow < LC_C && tile * VT + vpc * 8 < dv;
  auto issue = [&](int c) {
    bf16* qs = (bf16*)(stages + (c & 1) * Sh::STAGE) + qrow * LDQ + qpc * 8;
    const int left = len - c * LC_C;
#pragma unroll
    for (int i = 0; i < LC_C / RSTEP; ++i) {
      const bool live = q_in && qrow + i * RSTEP < left;
      lc_cp16(qs + i * RSTEP * LDQ, live ? qp + (size_t)(i * RSTEP) * a.ld_q : (const bf16*)a.q, live);
      lc_cp16(qs + (LC_C + i * RSTEP) * LDQ, live ? kp + (size_t)(i * RSTEP) * a.ld_k : (const bf16*)a.k, live);
    }
    if (vrow < LC_C) {
      const bool live = v_in && vrow < left;
      lc_cp16(vbuf + ((c & 1) * LC_C + vrow) * LDV + vpc * 8, live ? vp : (const bf16*)a.v, live);
    }
    qp += (size_t)LC_C * a.ld_q;
    kp += (size_t)LC_C * a.ld_k;
    vp += (size_t)LC_C * a.ld_v;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the gates of chunk c, by one warp: two neighbouring tokens a lane, sums and maxima by scans over the warp
  const float b1 = a.p1 ? a.p1[h] : 0.f, b2 = a.p2 ? a.p2[h] : 0.f, b3 = a.p3 ? a.p3[h] : 0.f;
  const float rate = KIND == SCAN_DECAY ? expf(b2) : 0.f;
  double m_run = 0.0;
  if (KIND == SCAN_GATED_MAX) m_run = (double)st[dk * VT + dk];
  // the logarithms of a batch of tokens' gates, a token a thread
  auto work_logs = [&](int first) {
    for (int i = tid; i < LC_BATCH && first + i < len; i += LC_THREADS) {
      const size_t row = (size_t)(q0 + first + i);
      if (KIND == SCAN_GATED_MAX) {
        const float zf = a.cap * tanhf((a.g2[row * a.ld_g2 + h] + b2) / a.cap);
        lfb[i] = fminf(zf, 0.f) - log1pf(expf(-fabsf(zf)));
        lib[i] = a.cap * tanhf((a.g1[row * a.ld_g1 + h] + b1) / a.cap);
      } else {
        const float z = a.g1[row * a.ld_g1 + h] + b1;
        lib[i] = z > 20.f ? z : log1pf(expf(z));
      }
    }
  };
  auto work_gates = [&](int c) {
    LcGates& gt = gates[c & 1];
    double lf[2], li[2];
    float bb[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = c * LC_C + 2 * lane + i, tb = t % LC_BATCH;
      lf[i] = 0.0; li[i] = -1e30; bb[i] = KIND == SCAN_DECAY ? 0.f : 1.f;      // a token beyond the segment: keeps all, adds nothing
      if (t < len) {
        if (KIND == SCAN_GATED_MAX) {
          lf[i] = (double)lfb[tb];
          li[i] = (double)lib[tb];
        } else {
          bb[i] = lib[tb];
          lf[i] = -(double)rate * (double)bb[i];
        }
      }
    }
    double sum = lf[0] + lf[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    const double sum_ahead = __shfl_up_sync(0xffffffffu, sum, 1);
    double F[2], Hh[2], G[2], m[2] = {0.0, 0.0};
    F[1] = sum;
    F[0] = (lane ? sum_ahead : 0.0) + lf[0];         // (not sum - lf[1]: a token's gates say nothing about the token ahead of it)
    if (KIND == SCAN_GATED_MAX) {
      Hh[0] = li[0] - F[0]; Hh[1] = li[1] - F[1];
      double mx = fmax(Hh[0], Hh[1]);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, mx, o);
        if (lane >= o) mx = fmax(mx, up);
      }
      const double ahead = __shfl_up_sync(0xffffffffu, mx, 1);
      const double before = lane ? fmax(m_run, ahead) : m_run;
      m[0] = F[0] + fmax(before, Hh[0]);
      m[1] = F[1] + fmax(m_run, mx);
      G[0] = F[0] - m[0]; G[1] = F[1] - m[1];
    } else {
      Hh[0] = -F[0]; Hh[1] = -F[1];
      G[0] = F[0]; G[1] = F[1];
    }
    const double G_end = __shfl_sync(0xffffffffu, G[1], 31), m_end = __shfl_sync(0xffffffffu, m[1], 31);
    const float c0 = expf((float)(G_end + Hh[0])) * bb[0], c1 = expf((float)(G_end + Hh[1])) * bb[1];
    double M = fmax(Hh[0], Hh[1]);                   // of the 16 tokens of eight lanes
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) M = fmax(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double Mi = __shfl_sync(0xffffffffu, M, 8 * i);
      if (lane >= 8 * i + 8) *(float2*)(gt.R[i] + 2 * lane) = make_float2(expf((float)(G[0] + Mi)), expf((float)(G[1] + Mi)));
    }
    *(float2*)(gt.E + 2 * lane) = make_float2(expf((float)(Hh[0] - M)) * bb[0], expf((float)(Hh[1] - M)) * bb[1]);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      gt.G[t] = lc_pair(G[i]);
      gt.H[t] = lc_pair(Hh[i]);
      gt.b[t] = bb[i];
      gt.A[t] = expf((float)(G[i] + m_run));
      gt.c[t] = i ? c1 : c0;
      gt.em[t] = KIND == SCAN_GATED_MAX ? expf((float)-m[i]) : 1.f;
    }
    if (lane == 0) { gt.A_end = expf((float)(G_end + m_run)); gt.m_end = (float)m_end; }
    m_run = m_end;
  };

  issue(0);
  work_logs(0);
  __syncthreads();
  if (warp == LC_GATE_WARP) work_gates(0);
  // n . q is formed like one more value column's; n itself is summed by the warps of W, which have time for it (as a product of 16 rows of
  // which one counts it was half as many again as the state's own in half of these warps: 195 us where this takes 175)
  const bool has_n = KIND == SCAN_GATED_MAX && half == 0;
  if (KIND == SCAN_GATED_MAX)
    for (int i = tid; i < 2 * DKP; i += LC_THREADS) ns[i] = i < dk ? st[dk * VT + i] : 0.f;
  float sT[2 * NK][4];                               // S^T: value columns half + g8 (+ 8), key rows k0 + 8 nt + 2 t4 (+ 1)
  if (warp < 8) {
#pragma unroll
    for (int nt = 0; nt < 2 * NK; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = k0 + nt * 8 + 2 * t4 + (i & 1), col = half + g8 + (i >> 1) * 8;
        sT[nt][i] = k < dk ? st[k * VT + col] : 0.f;
      }
  }

  uint32_t odd = 0;                                  // bits 15 and 31: a value of this thread's had an exponent of all ones
  int any_odd = 0;                                   // some thread's had
  for (int c = 0; c < nchunks; ++c) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                 // chunk c and its gates are in place; everyone is done with chunk c - 1
    if (c + 1 < nchunks) issue(c + 1);
    const bf16* qs = (const bf16*)(stages + (c & 1) * Sh::STAGE);
    const bf16* ks = qs + LC_C * LDQ;
    const bf16* vc = vbuf + (c & 1) * LC_C * LDV;
    const LcGates& gt = gates[c & 1];
    if (warp < 8) {
      // c_j v_j in three terms, for the update
      for (int i = tid; i < LC_C * VT / 2; i += 256) {
        const int t = i / (VT / 2), cc = (i - t * (VT / 2)) * 2;
        const float cj = gt.c[t];
        odd |= (*(const uint32_t*)(vc + t * LDV + cc) & 0x7fff7fffu) + 0x00800080u;
        uint32_t w[3];
        lc_split3(cj * to_f(vc[t * LDV + cc]), cj * to_f(vc[t * LDV + cc + 1]), w);
#pragma unroll
        for (int x = 0; x < 3; ++x) *(uint32_t*)(vs + (x * LC_C + t) * LDV + cc) = w[x];
      }
      // this slice's share of A_t q_t S_0
      uint32_t b0[NK][2][3], b1t[NK][2][3];          // [key step][column tile][term]
#pragma unroll
      for (int kk = 0; kk < NK; ++kk)
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          lc_split3(sT[2 * kk][2 * nb], sT[2 * kk][2 * nb + 1], b0[kk][nb]);
          lc_split3(sT[2 * kk + 1][2 * nb], sT[2 * kk + 1][2 * nb + 1], b1t[kk][nb]);
        }
      uint32_t n0[NK][3], n1[NK][3];                 // n's: column 0 of a tile of eight
      if (has_n) {
#pragma unroll
        for (int kk = 0; kk < NK; ++kk) {
          const float* np = ns + k0 + kk * 16 + 2 * t4;
          lc_split3(g8 ? 0.f : np[0] + np[DKP], g8 ? 0.f : np[1] + np[DKP + 1], n0[kk]);
          lc_split3(g8 ? 0.f : np[8] + np[DKP + 8], g8 ? 0.f : np[9] + np[DKP + 9], n1[kk]);
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float hi[2][4] = {}, lo[2][4] = {}, nh[4] = {}, nl[4] = {};
#pragma unroll
        for (int kk = 0; kk < NK; ++kk) {
          uint32_t af[4];
          lc_ldsm4(af, qs + (m * 16 + (mi & 1) * 8 + r8) * LDQ + k0 + kk * 16 + (mi >> 1) * 8);
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) {
            lc_mma(lo[nb], af, b0[kk][nb][2], b1t[kk][nb][2]);
            lc_mma(hi[nb], af, b0[kk][nb][0], b1t[kk][nb][0]);
            lc_mma(lo[nb], af, b0[kk][nb][1], b1t[kk][nb][1]);
          }
          if (has_n) {
            lc_mma(nl, af, n0[kk][2], n1[kk][2]);
            lc_mma(nh, af, n0[kk][0], n1[kk][0]);
            lc_mma(nl, af, n0[kk][1], n1[kk][1]);
          }
        }
        const float a_lo = gt.A[m * 16 + g8], a_hi = gt.A[m * 16 + g8 + 8];
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          float* d = red + ((size_t)slice * LC_C + m * 16 + g8) * LDR + half + nb * 8 + 2 * t4;
          *(float2*)d = make_float2(a_lo * (hi[nb][0] + lo[nb][0]), a_lo * (hi[nb][1] + lo[nb][1]));
          *(float2*)(d + 8 * LDR) = make_float2(a_hi * (hi[nb][2] + lo[nb][2]), a_hi * (hi[nb][3] + lo[nb][3]));
        }
        if (has_n && t4 == 0) {
          nq[slice * LC_C + m * 16 + g8] = a_lo * (nh[0] + nl[0]);
          nq[slice * LC_C + m * 16 + g8 + 8] = a_hi * (nh[2] + nl[2]);
        }
      }
    } else {
      if (warp == LC_GATE_WARP && c + 1 < nchunks) work_gates(c + 1);
      // W = q k^T of 16 tokens x 32 tokens, decayed, and its product with v: two blocks of 16 x 16, nothing of what lies above the diagonal.  On the
      // diagonal an exponential an entry; a block below it takes a factor a row and a factor a column (G_t + M and H_j - M are <= 0 for M the
      // largest H of tokens all ahead of t)
      const int mt = (warp - 8) >> 1, j0 = (warp & 1) * 32, below = mt - 2 * (warp & 1);         // blocks left of the diagonal's: `below` of the two
      float hi[VT / 8][4] = {}, lo[VT / 8][4] = {};
      float rs[2] = {0.f, 0.f};
      if (j0 <= mt * 16 + 15) {
        float w[4][4] = {};
#pragma unroll
        for (int k4 = 0; k4 < DKP; k4 += 64) {       // runs of four products, added up in float32
          float part[4][4] = {};
#pragma unroll
          for (int kk = k4; kk < k4 + 64; kk += 16) {
            uint32_t af[4], bq[4];
            lc_ldsm4(af, qs + (mt * 16 + (mi & 1) * 8 + r8) * LDQ + kk + (mi >> 1) * 8);
#pragma unroll
            for (int pr = 0; pr < 2; ++pr) {
              if (pr > below) break;
              lc_ldsm4(bq, ks + (j0 + pr * 16 + (mi >> 1) * 8 + r8) * LDQ + kk + (mi & 1) * 8);
              lc_mma(part[2 * pr], af, bq[0], bq[1]);
              lc_mma(part[2 * pr + 1], af, bq[2], bq[3]);
            }
          }
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int x = 0; x < 4; ++x) w[nt][x] += part[nt][x];
        }
#pragma unroll
        for (int pr = 0; pr < 2; ++pr) {
          if (pr > below) break;
          if (pr < below) {
            const float* Rb = gt.R[2 * (warp & 1) + pr] + mt * 16 + g8;
            const float R[2] = {Rb[0], Rb[8]};
#pragma unroll
            for (int h8 = 0; h8 < 2; ++h8) {
              const float2 E = *(const float2*)(gt.E + j0 + pr * 16 + h8 * 8 + 2 * t4);
              float* f = w[2 * pr + h8];
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                f[2 * r] *= R[r] * E.x;
                f[2 * r + 1] *= R[r] * E.y;
                rs[r] += f[2 * r] + f[2 * r + 1];
              }
            }
          } else {
            const float2 Gt[2] = {gt.G[mt * 16 + g8], gt.G[mt * 16 + g8 + 8]};
#pragma unroll
            for (int h8 = 0; h8 < 2; ++h8)
#pragma unroll
              for (int jj = 0; jj < 2; ++jj) {
                const int jr = h8 * 8 + 2 * t4 + jj;
                const float2 Hj = gt.H[mt * 16 + jr];
                const float bj = KIND == SCAN_DECAY ? gt.b[mt * 16 + jr] : 1.f;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  const float f = jr <= g8 + r * 8 ? w[2 * pr + h8][2 * r + jj] * (lc_exp_sum(Gt[r], Hj) * bj) : 0.f;
                  w[2 * pr + h8][2 * r + jj] = f;
                  rs[r] += f;
                }
              }
          }
        }
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          if (kk > below) break;
          uint32_t t0[3], t1[3], t2[3], t3[3];
          lc_split3(w[2 * kk][0], w[2 * kk][1], t0);
          lc_split3(w[2 * kk][2], w[2 * kk][3], t1);
          lc_split3(w[2 * kk + 1][0], w[2 * kk + 1][1], t2);
          lc_split3(w[2 * kk + 1][2], w[2 * kk + 1][3], t3);
#pragma unroll
          for (int nb = 0; nb < VT / 16; ++nb) {
            uint32_t bv[4];
            lc_ldsm4t(bv, vc + (j0 + kk * 16 + (mi & 1) * 8 + r8) * LDV + nb * 16 + (mi >> 1) * 8);
#pragma unroll
            for (int x = 2; x >= 0; --x) {
              const uint32_t af[4] = {t0[x], t1[x], t2[x], t3[x]};
              lc_mma(x ? lo[2 * nb] : hi[2 * nb], af, bv[0], bv[1]);
              lc_mma(x ? lo[2 * nb + 1] : hi[2 * nb + 1], af, bv[2], bv[3]);
            }
          }
        }
      }
      if (KIND == SCAN_GATED_MAX) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          rs[x] += __shfl_xor_sync(0xffffffffu, rs[x], 1);
          rs[x] += __shfl_xor_sync(0xffffffffu, rs[x], 2);
          if (t4 == 0) rowsum[(mt * 16 + g8 + x * 8) * 2 + (warp & 1)] = rs[x];
        }
      }
#pragma unroll
      for (int nb = 0; nb < VT / 8; ++nb) {
        float* d = red + ((size_t)(SLICES + (warp & 1)) * LC_C + mt * 16 + g8) * LDR + nb * 8 + 2 * t4;
        *(float2*)d = make_float2(hi[nb][0] + lo[nb][0], hi[nb][1] + lo[nb][1]);
        *(float2*)(d + 8 * LDR) = make_float2(hi[nb][2] + lo[nb][2], hi[nb][3] + lo[nb][3]);
      }
    }
    any_odd |= __syncthreads_or(odd & 0x80008000u);  // the terms of c v and all sums are in place
    if (warp < 8) {
      float up[2 * NK][4] = {}, lo[2 * NK][4] = {};
#pragma unroll
      for (int kk = 0; kk < LC_C; kk += 16) {
        uint32_t af[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) lc_ldsm4t(af[x], vs + (x * LC_C + kk + (mi >> 1) * 8 + r8) * LDV + half + (mi & 1) * 8);
#pragma unroll
        for (int nb = 0; nb < NK; ++nb) {
          uint32_t bk[4];
          lc_ldsm4t(bk, ks + (kk + (mi & 1) * 8 + r8) * LDQ + k0 + nb * 16 + (mi >> 1) * 8);
#pragma unroll
          for (int x = 2; x >= 0; --x) {
            lc_mma(x ? lo[2 * nb] : up[2 * nb], af[x], bk[0], bk[1]);
            lc_mma(x ? lo[2 * nb + 1] : up[2 * nb + 1], af[x], bk[2], bk[3]);
          }
        }
      }
      const float ae = gt.A_end;
#pragma unroll
      for (int nt = 0; nt < 2 * NK; ++nt)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          sT[nt][x] = fmaf(ae, sT[nt][x], up[nt][x] + lo[nt][x]);
        }
    } else {
      if (KIND == SCAN_GATED_MAX && ((tid - 256) & 127) * 2 < DKP) {         // n: two key rows and half the tokens a thread
        const int kr = ((tid - 256) & 127) * 2, jb = (tid - 256) >> 7 ? 32 : 0;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 c4 = *(const float4*)(gt.c + jb + j);
          const float cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const __nv_bfloat162 kv = *(const __nv_bfloat162*)(ks + (jb + j + u) * LDQ + kr);
            a0 = fmaf(cc[u], __low2float(kv), a0);
            a1 = fmaf(cc[u], __high2float(kv), a1);
          }
        }
        float* np = ns + (jb ? DKP : 0) + kr;
        np[0] = fmaf(gt.A_end, np[0], a0);
        np[1] = fmaf(gt.A_end, np[1], a1);
      }
      for (int i = tid - 256; i < LC_C * VT / 4; i += 256) {
        const int t = i / (VT / 4), cc = (i - t * (VT / 4)) * 4;
        if (c * LC_C + t >= len || tile * VT + cc >= dv) continue;
        float4 y = *(const float4*)(red + (size_t)t * LDR + cc);
#pragma unroll
        for (int sl = 1; sl < SLICES + 2; ++sl) {
          const float4 z = *(const float4*)(red + ((size_t)sl * LC_C + t) * LDR + cc);
          y.x += z.x; y.y += z.y; y.z += z.z; y.w += z.w;
        }
        y.x *= a.q_scale; y.y *= a.q_scale; y.z *= a.q_scale; y.w *= a.q_scale;
        if (KIND == SCAN_GATED_MAX) {
          float dot = rowsum[2 * t] + rowsum[2 * t + 1];
#pragma unroll
          for (int sl = 0; sl < SLICES; ++sl) dot += nq[sl * LC_C + t];
          dot *= a.q_scale;
          const float den = fmaxf(fabsf(dot), gt.em[t]) + 1e-6f;
          y.x /= den; y.y /= den; y.z /= den; y.w /= den;
        } else {
          const bf16* vr = vc + t * LDV + cc;
          y.x = fmaf(b3, to_f(vr[0]), y.x); y.y = fmaf(b3, to_f(vr[1]), y.y); y.z = fmaf(b3, to_f(vr[2]), y.z); y.w = fmaf(b3, to_f(vr[3]), y.w);
        }
        *(float4*)(a.out + (size_t)(q0 + c * LC_C + t) * a.ld_out + (size_t)h * dv + tile * VT + cc) = y;
      }
    }
    // the logarithms of the batch that begins with chunk c + 2 (the present one's last gates were worked out ahead of the barrier)
    if ((c + 2) % (LC_BATCH / LC_C) == 0) work_logs((c + 2) * LC_C);
  }
  if (any_odd) {
    __syncthreads();                                 // all are done with shared memory and with their outputs
    return lc_token_by_token<KIND, VT, LC_THREADS>(a, st + dk * VT, 1, 0, s, q0, len, h, tile, (float*)lc_smem);
  }
  if (warp < 8) {
#pragma unroll
    for (int nt = 0; nt < 2 * NK; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = k0 + nt * 8 + 2 * t4 + (i & 1), col = half + g8 + (i >> 1) * 8;
        if (k < dk) st[k * VT + col] = sT[nt][i];
      }
  }
  if (KIND == SCAN_GATED_MAX) {
    __syncthreads();                                 // n is whole
    for (int i = tid; i < dk; i += LC_THREADS) st[dk * VT + i] = ns[i] + ns[DKP + i];
    if (tid == 0) st[dk * VT + dk] = gates[(nchunks - 1) & 1].m_end;
  }
}

template <int KIND, int VT, int NK>
static int launch_scan_chunk(const ScanArgs& a, dim3 grid, cudaStream_t st) {
  auto kernel = linear_scan_chunk_kernel<KIND, VT, NK>;
  static PerDevice allowed;
  const int rc = qv_allow_smem(kernel, LcShape<VT, NK>::BYTES, allowed);
  if (rc) return rc;
  return qv_launch(kernel, grid, dim3(LC_THREADS), (size_t)LcShape<VT, NK>::BYTES, st, a);
}

// ---------------------------------------------------------------- long portions: the chunks' outputs side by side
// Of a chunk only S_end = A S_0 + ... goes to the next one.  So for long portions the chunks' arithmetic (above) is dealt to three launches:
//   lp_gates_kernel     what a chunk's gates amount to (LpGates), a warp a chunk
//   lp_states_kernel    a CTA owns 64 keys x 64 value columns of a (segment, head) and walks the chunks; the state ahead of each goes to a
//                       workspace
//   lp_outputs_kernel   a CTA per (chunk, head, up to 256 value columns) forms q S_0 and W v, all chunks at once
// The states lie in the workspace as the products' accumulators lie in the lanes, and S^T's accumulators are S's operand for q S_0, so a
// state is written and read in whole 512-byte pieces and passes through no shared memory.  The update's arithmetic is that of
// linear_scan_chunk_kernel to the bit.  2,048 tokens of 4 heads of 256 x 512: 173 us in one kernel (32 chunks in a row, W formed again for each
// tile of 16 columns); gates 8, states 48, outputs 44 here.  Bound by the states' chain of chunks and, in the outputs, by the instructions that
// split float32 into three terms; the workspace (2 MB a chunk) is read from L2.
#define LP_KEYS 64                         // keys and value columns a CTA of lp_states_kernel holds
#define LP_COLS 256                        // value columns a CTA of lp_outputs_kernel forms
#define LP_THREADS 256
#define LP_NPARTS 4                        // sums that n is kept in
struct LpGates {                           // what a chunk's gates amount to; 16-byte pieces
  float2 G[LC_C], H[LC_C];                 // a number and what rounding it to float32 left over
  float A[LC_C], em[LC_C];                 // em: exp(-m_t)
  float R[3][LC_C], E[LC_C];               // blocks of 16 tokens, M_i the largest H in block i: exp(G_t + M_i) for t behind it, exp(H_j - M)
  float c[LC_C], A_end, m_end, pad[2];     // what the states' kernel reads
};

// One round of the three launches: some chunks of some segments, a slot of the workspace each.  What goes from a segment's round to its next
// one beside the state: the running maximum in its full width and n as the sums it is kept in, so that no bit depends on the rounds.
#define LP_ITEMS 32
struct LpWork {
  float* S;                                // [slots][H][col tiles of 16][key tiles of 8][32 lanes][4]
  float* n;                                // [slots][H][LP_NPARTS][dkp], n as sums
  LpGates* gates;                          // [slots][H]
  double* m;                               // [places][H]: the running maximum behind the round's last chunk
  float* n_end;                            // [places][H][LP_NPARTS][dkp]: n behind it
  int* odd;                                // [places][H][blocks of 64 columns]: some value of the round was infinite or NaN
  int dkp, ct, vt;                         // dkp: dk in whole runs of 32; ct: column tiles of 16; vt: columns a tile of the state
  PortionRound<LP_ITEMS> round;
};
static inline size_t lp_slot_bytes(int H, int dk, int dv) {
  const size_t dkp = (dk + 31) / 32 * 32, ct = (dv + 15) / 16;
  return (size_t)H * (ct * dkp * 64 + LP_NPARTS * dkp * 4 + sizeof(LpGates));
}
static inline size_t lp_place_bytes(int H, int dk, int dv) {
  return (size_t)H * (8 + LP_NPARTS * (size_t)((dk + 31) / 32 * 32) * 4 + (size_t)((dv + 63) / 64) * 4);
}

// grid (items, heads); a warp takes a chunk: two neighbouring tokens a lane, sums and maxima by scans over the warp.  Bound by the
// latency of its scans and functions.  In lp_states_kernel itself they cost more: a ninth warp there takes 2.5 us a chunk, which otherwise
// takes 1.4.
#define LP_GATE_WARPS 32
__global__ void __launch_bounds__(32 * LP_GATE_WARPS) lp_gates_kernel(const __grid_constant__ ScanArgs a, const __grid_constant__ LpWork w) {
  __shared__ double ends[LP_GATE_WARPS][2];          // F_63 and max H of the warps' chunks
  pdl_wait();
  pdl_launch_dependents();
  const PortionItem& it = w.round.item[blockIdx.x];
  const int s = it.seg, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  const int nchunks = (len + LC_C - 1) / LC_C, last = nchunks < it.first + it.count ? nchunks : it.first + it.count;
  const float b1 = a.p1 ? a.p1[h] : 0.f, b2 = a.p2 ? a.p2[h] : 0.f;
  const int tiles = (a.dv + w.vt - 1) / w.vt;
  double m_next = it.first ? w.m[(size_t)it.place * a.H + h]
                       : (double)a.state[(size_t)a.seg_slot[s] * a.slot_stride + (size_t)h * tiles * scan_tile_floats(SCAN_GATED_MAX, a.dk, w.vt) +
                                         (size_t)a.dk * w.vt + a.dk];
  for (int c1 = it.first; c1 < last; c1 += LP_GATE_WARPS) {
    const int c = c1 + warp;
    double lf[2], li[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = c * LC_C + 2 * lane + i;
      lf[i] = 0.0; li[i] = -1e30;                    // a token beyond the segment: keeps all, adds nothing
      if (c < last && t < len) {
        const size_t row = (size_t)(q0 + t);
        const float zf = a.cap * tanhf((a.g2[row * a.ld_g2 + h] + b2) / a.cap);
        lf[i] = (double)(fminf(zf, 0.f) - log1pf(expf(-fabsf(zf))));
        li[i] = (double)(a.cap * tanhf((a.g1[row * a.ld_g1 + h] + b1) / a.cap));
      }
    }
    double sum = lf[0] + lf[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    const double sum_ahead = __shfl_up_sync(0xffffffffu, sum, 1);
    double F[2], Hh[2], G[2], m[2], m_run = 0.0;
    F[1] = sum;
    F[0] = (lane ? sum_ahead : 0.0) + lf[0];         // (not sum - lf[1]: a token's gates say nothing about the token ahead of it)
    Hh[0] = li[0] - F[0]; Hh[1] = li[1] - F[1];
    double mx = fmax(Hh[0], Hh[1]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, mx, o);
      if (lane >= o) mx = fmax(mx, up);
    }
    if (lane == 31) { ends[warp][0] = F[1]; ends[warp][1] = mx; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < LP_GATE_WARPS; ++i) {
      if (i == warp) m_run = m_next;
      m_next = ends[i][0] + fmax(m_next, ends[i][1]);
    }
    const double ahead = __shfl_up_sync(0xffffffffu, mx, 1);
    const double before = lane ? fmax(m_run, ahead) : m_run;
    m[0] = F[0] + fmax(before, Hh[0]);
    m[1] = F[1] + fmax(m_run, mx);
    G[0] = F[0] - m[0]; G[1] = F[1] - m[1];
    const double G_end = __shfl_sync(0xffffffffu, G[1], 31), m_end = __shfl_sync(0xffffffffu, m[1], 31);
    double M = fmax(Hh[0], Hh[1]);                   // of the 16 tokens of eight lanes
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) M = fmax(M, __shfl_xor_sync(0xffffffffu, M, o));
    double Mi[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) Mi[i] = __shfl_sync(0xffffffffu, M, 8 * i);
    if (c < last) {
      LpGates& gt = w.gates[(size_t)(it.slot + c - it.first) * a.H + h];
      float2 pair[2];
      pair[0] = lc_pair(G[0]); pair[1] = lc_pair(G[1]);
      *(float4*)(gt.G + 2 * lane) = make_float4(pair[0].x, pair[0].y, pair[1].x, pair[1].y);
      pair[0] = lc_pair(Hh[0]); pair[1] = lc_pair(Hh[1]);
      *(float4*)(gt.H + 2 * lane) = make_float4(pair[0].x, pair[0].y, pair[1].x, pair[1].y);
      *(float2*)(gt.A + 2 * lane) = make_float2(expf((float)(G[0] + m_run)), expf((float)(G[1] + m_run)));
#pragma unroll
      for (int i = 0; i < 3; ++i)
        *(float2*)(gt.R[i] + 2 * lane) = lane >= 8 * i + 8 ? make_float2(expf((float)(G[0] + Mi[i])), expf((float)(G[1] + Mi[i]))) : make_float2(0.f, 0.f);
      *(float2*)(gt.E + 2 * lane) = make_float2(expf((float)(Hh[0] - M)), expf((float)(Hh[1] - M)));
      *(float2*)(gt.c + 2 * lane) = make_float2(expf((float)(G_end + Hh[0])), expf((float)(G_end + Hh[1])));
      *(float2*)(gt.em + 2 * lane) = make_float2(expf((float)-m[0]), expf((float)-m[1]));
      if (lane == 0) { gt.A_end = expf((float)(G_end + m_run)); gt.m_end = (float)m_end; }
    }
    __syncthreads();                                 // the ends have been read
  }
  if (threadIdx.x == 0) w.m[(size_t)it.place * a.H + h] = m_next;
}

// grid (items, heads, key blocks x column blocks, then the key blocks once more for n).  Eight warps hold the state as S^T, 16
// columns x 32 keys each.  The terms of c v are formed once a CTA, a chunk ahead of the products that read them, so a chunk is one stretch
// between barriers; k, v and the gates arrive ahead of that (cp.async).  Bound by the latency of a chunk's products and of the terms' way
// through shared memory: 1.4 us a chunk.  (With the terms formed in registers by both warps that share columns, and n by a ninth warp, three
// warps on one scheduler: 1.75.)
struct LpStatesSmem {
  bf16 k[3][LC_C][LP_KEYS + 8], v[2][LC_C][LP_KEYS + 8], terms[2][3][LC_C][LP_KEYS + 8];
  float c[3][LC_C + 4];                    // then A_end
};
__global__ void __launch_bounds__(LP_THREADS, 2) lp_states_kernel(const __grid_constant__ ScanArgs a, const __grid_constant__ LpWork w) {
  extern __shared__ __align__(16) unsigned char lp_smem[];
  LpStatesSmem& sm = *(LpStatesSmem*)lp_smem;
  pdl_wait();
  pdl_launch_dependents();
  const PortionItem& it = w.round.item[blockIdx.x];
  const int s = it.seg, h = blockIdx.y;
  const int nkb = (a.dk + LP_KEYS - 1) / LP_KEYS, ncb = (a.dv + LP_KEYS - 1) / LP_KEYS, kb = blockIdx.z % nkb, cb = blockIdx.z / nkb;
  const bool is_n = cb == ncb;                       // this CTA sums n
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  const int dk = a.dk, dv = a.dv, vt = w.vt, tiles = (dv + vt - 1) / vt, tf = scan_tile_floats(SCAN_GATED_MAX, dk, vt);
  const int nchunks = (len + LC_C - 1) / LC_C, count = (nchunks < it.first + it.count ? nchunks : it.first + it.count) - it.first;
  if (count <= 0) return;
  float* st = a.state + (size_t)a.seg_slot[s] * a.slot_stride + (size_t)h * tiles * tf;
  const int g8 = lane >> 2, t4 = lane & 3, mi = lane >> 3, r8 = lane & 7;
  const int kw = kb * LP_KEYS + (warp >> 2) * 32, cw = cb * LP_KEYS + (warp & 3) * 16;        // a warp's keys and columns
  const bool holds = !is_n && cw < dv && kw < w.dkp;
  const LpGates* gates = w.gates + (size_t)it.slot * a.H + h;

  // a thread copies, and splits, the same 16 bytes of every 32nd row
  const int row = tid >> 3, pc = tid & 7;
  const int token0 = q0 + it.first * LC_C, left0 = len - it.first * LC_C;
  const bf16* kp = (const bf16*)a.k + (size_t)(token0 + row) * a.ld_k + (size_t)(h / a.q_group) * dk + kb * LP_KEYS + pc * 8;
  const bf16* vp = (const bf16*)a.v + (size_t)(token0 + row) * a.ld_v + (size_t)h * dv + cb * LP_KEYS + pc * 8;
  const bool k_in = kb * LP_KEYS + pc * 8 < dk, v_in = !is_n && cb * LP_KEYS + pc * 8 < dv;
  auto issue = [&](int c) {
    if (c < count) {
      const int left = left0 - c * LC_C;
#pragma unroll
      for (int i = 0; i < LC_C; i += 32) {
        const bool lk = k_in && row + i < left, lv = v_in && row + i < left;
        lc_cp16(&sm.k[c % 3][row + i][pc * 8], lk ? kp + (size_t)(c * LC_C + i) * a.ld_k : (const bf16*)a.k, lk);
        if (!is_n) lc_cp16(&sm.v[c & 1][row + i][pc * 8], lv ? vp + (size_t)(c * LC_C + i) * a.ld_v : (const bf16*)a.v, lv);
      }
      if (tid < (LC_C + 4) / 4) lc_cp16(sm.c[c % 3] + tid * 4, gates[(size_t)c * a.H].c + tid * 4, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint32_t odd = 0;                                  // bits 15 and 31: a value had an exponent of all ones
  auto split = [&](int c) {                          // c_j v_j in three terms
#pragma unroll
    for (int i = 0; i < LC_C; i += 32) {
      const uint4 raw4 = *(const uint4*)&sm.v[c & 1][row + i][pc * 8];
      const uint32_t raw[4] = {raw4.x, raw4.y, raw4.z, raw4.w};
      const float cj = sm.c[c % 3][row + i];
      uint32_t t[4][3];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        odd |= (raw[e] & 0x7fff7fffu) + 0x00800080u;
        const __nv_bfloat162 vv = *(const __nv_bfloat162*)&raw[e];
        lc_split3(cj * __low2float(vv), cj * __high2float(vv), t[e]);
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) *(uint4*)&sm.terms[c & 1][x][row + i][pc * 8] = make_uint4(t[0][x], t[1][x], t[2][x], t[3][x]);
    }
  };
  issue(0);
  issue(1);
  float sT[4][4] = {};                               // S^T: value columns cw + g8 (+ 8), keys kw + 8 nt + 2 t4 (+ 1)
  if (holds) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = kw + nt * 8 + 2 * t4 + (i & 1), col = cw + g8 + (i >> 1) * 8;
        if (k < dk && col < tiles * vt) sT[nt][i] = st[(size_t)(col / vt) * tf + k * vt + col % vt];
      }
  }
  const int nk = kb * LP_KEYS + 2 * lane;            // n: two keys a lane, a quarter of the tokens a warp
  float n0 = 0.f, n1 = 0.f;
  auto n_end = [&]() { return (float2*)(w.n_end + (((size_t)it.place * a.H + h) * LP_NPARTS + warp) * w.dkp + nk); };
  if (is_n && warp < LP_NPARTS && nk < dk) {
    if (it.first) { n0 = n_end()->x; n1 = n_end()->y; }
    else if (warp == 0) { n0 = st[dk * vt + nk]; n1 = st[dk * vt + nk + 1]; }
  }
  if (!is_n) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    split(0);
  }
  for (int c = 0; c < count; ++c) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                 // chunk c + 1 is in place, and chunk c's terms; everyone is done with chunk c - 1
    issue(c + 2);
    const float* cs = sm.c[c % 3];
    const bf16(*ks)[LP_KEYS + 8] = sm.k[c % 3];
    const size_t slot = (size_t)(it.slot + c) * a.H + h;
    if (is_n) {
      if (warp < LP_NPARTS) {
        if (nk < w.dkp) *(float2*)(w.n + (slot * LP_NPARTS + warp) * w.dkp + nk) = make_float2(n0, n1);
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int j = 0; j < LC_C / LP_NPARTS; j += 4) {
          const float4 c4 = *(const float4*)(cs + warp * (LC_C / LP_NPARTS) + j);
          const float cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const __nv_bfloat162 kv = *(const __nv_bfloat162*)&ks[warp * (LC_C / LP_NPARTS) + j + u][2 * lane];
            a0 = fmaf(cc[u], __low2float(kv), a0);
            a1 = fmaf(cc[u], __high2float(kv), a1);
          }
        }
        n0 = fmaf(cs[LC_C], n0, a0);
        n1 = fmaf(cs[LC_C], n1, a1);
      }
      continue;
    }
    if ((warp & 4) && c + 1 < count) split(c + 1);   // (half of the warps ahead of their products, the others behind them)
    if (holds) {
      float* ws = w.S + ((slot * w.ct + (cw >> 4)) * (w.dkp >> 3) + (kw >> 3)) * 128 + lane * 4;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) *(float4*)(ws + nt * 128) = make_float4(sT[nt][0], sT[nt][1], sT[nt][2], sT[nt][3]);
      float up[4][4], lo[4][4];
#pragma unroll
      for (int kk = 0; kk < LC_C; kk += 16) {
        uint32_t af[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x) lc_ldsm4t(af[x], &sm.terms[c & 1][x][kk + (mi >> 1) * 8 + r8][(warp & 3) * 16 + (mi & 1) * 8]);
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          uint32_t bk[4];
          lc_ldsm4t(bk, &ks[kk + (mi & 1) * 8 + r8][(warp >> 2) * 32 + nb * 16 + (mi >> 1) * 8]);
#pragma unroll
          for (int x = 2; x >= 0; --x) {
            lc_mma(kk == 0 && x != 1, x ? lo[2 * nb] : up[2 * nb], af[x], bk[0], bk[1]);
            lc_mma(kk == 0 && x != 1, x ? lo[2 * nb + 1] : up[2 * nb + 1], af[x], bk[2], bk[3]);
          }
        }
      }
      const float ae = cs[LC_C];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int x = 0; x < 4; ++x) sT[nt][x] = fmaf(ae, sT[nt][x], up[nt][x] + lo[nt][x]);
    }
    if (!(warp & 4) && c + 1 < count) split(c + 1);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (is_n) {
    float2* sums = (float2*)sm.terms;                // [LP_NPARTS][32]: the terms' place, which these CTAs do not use
    if (warp < LP_NPARTS) {
      sums[warp * 32 + lane] = make_float2(n0, n1);
      if (nk < dk) *n_end() = make_float2(n0, n1);
    }
    __syncthreads();
    if (nk < dk) {
      const float2 x0 = sums[lane], x1 = sums[32 + lane], x2 = sums[64 + lane], x3 = sums[96 + lane];
      n0 = (x0.x + x1.x) + (x2.x + x3.x);
      n1 = (x0.y + x1.y) + (x2.y + x3.y);
      for (int tile = warp; tile < tiles; tile += LP_THREADS / 32) {
        float* np = st + (size_t)tile * tf + dk * vt;
        np[nk] = n0;
        np[nk + 1] = n1;
      }
    }
    return;
  }
  const int any_odd = __syncthreads_or(odd & 0x80008000u);
  if (kb == 0 && tid == 0) w.odd[((size_t)it.place * a.H + h) * ncb + cb] = any_odd != 0;
  if (any_odd) return;                               // the outputs' kernel goes token by token from the state as it is
  if (holds) {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = kw + nt * 8 + 2 * t4 + (i & 1), col = cw + g8 + (i >> 1) * 8;
        if (k < dk && col < tiles * vt) st[(size_t)(col / vt) * tf + k * vt + col % vt] = sT[nt][i];
      }
  }
  if (kb == 0) {
    const int tile = cb * LP_KEYS / vt + tid;
    if (tid < LP_KEYS / vt && tile < tiles) st[(size_t)tile * tf + dk * vt + dk] = gates[(size_t)(count - 1) * a.H].m_end;
  }
}

// grid (slots, heads, blocks of LP_COLS value columns).  The warps form W's blocks of 16 x 16 tokens (above the diagonal there is nothing):
// a warp the diagonal's block of 16 rows, with an exponential an entry, another those ahead of it, with two factors an entry (G_t + M and
// H_j - M are <= 0 for M the largest H of tokens all ahead of t); the one with nothing to do forms n . q.  W takes k's place in shared
// memory in three terms.  Then a warp takes 16 columns: q S_0 in runs of 32 keys, the next run's state in flight, then W v.
struct LpOutShape {
  int ldq, ldv, k_bytes, bytes;
  __host__ __device__ LpOutShape(int dkp, int cols) {
    ldq = dkp + 8;
    ldv = cols + 8;
    const int wterms = 3 * LC_C * (LC_C + 8) * 2, kb = LC_C * ldq * 2;
    k_bytes = kb > wterms ? kb : wterms;
    bytes = LC_C * ldq * 2 + k_bytes + LC_C * ldv * 2 + (int)sizeof(LpGates) + LC_C * 3 * 4 + dkp * 4;
  }
};
__global__ void __launch_bounds__(LP_THREADS, 2) lp_outputs_kernel(const __grid_constant__ ScanArgs a, const __grid_constant__ LpWork w) {
  extern __shared__ __align__(16) unsigned char lp_smem[];
  constexpr int LDW = LC_C + 8;
  pdl_wait();
  pdl_launch_dependents();
  int i_item = 0;
  while (i_item + 1 < w.round.items && w.round.item[i_item + 1].slot <= (int)blockIdx.x) ++i_item;
  const PortionItem& it = w.round.item[i_item];
  const int s = it.seg, cr = (int)blockIdx.x - it.slot, c = it.first + cr, h = blockIdx.y;
  const int q0 = a.seg_q_start[s], len = a.seg_q_start[s + 1] - q0;
  if (c * LC_C >= len) return;
  const int dk = a.dk, dv = a.dv, dkp = w.dkp;
  const int col0 = blockIdx.z * LP_COLS, cols = dv - col0 < LP_COLS ? (dv - col0 + 15) / 16 * 16 : LP_COLS;
  const LpOutShape sh(dkp, cols);
  bf16* qs = (bf16*)lp_smem;                                         // [64][ldq]
  bf16* ks = qs + LC_C * sh.ldq;                                     // [64][ldq], then
  bf16* wt = ks;                                                     // [3][64][LDW] the terms of W
  bf16* vs = (bf16*)(lp_smem + LC_C * sh.ldq * 2 + sh.k_bytes);      // [64][ldv]
  LpGates& gt = *(LpGates*)(vs + LC_C * sh.ldv);
  float* rowsum = (float*)(&gt + 1);                                 // [64][2]
  float* nq = rowsum + 2 * LC_C;                                     // [64] n_0 . q_t
  float* ns = nq + LC_C;                                             // [dkp]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g8 = lane >> 2, t4 = lane & 3, mi = lane >> 3, r8 = lane & 7;
  const size_t slot = (size_t)blockIdx.x * a.H + h;
  const size_t t0 = (size_t)q0 + (size_t)c * LC_C;
  const int left = len - c * LC_C;
  {
    const int pq = dkp >> 3, pv = cols >> 3;
    const bool q_in = lane * 8 < dk, v_in = col0 + lane * 8 < dv;
    const bf16* qp = (const bf16*)a.q + (t0 + warp) * a.ld_q + (size_t)(h / a.q_group) * dk + lane * 8;
    const bf16* kp = (const bf16*)a.k + (t0 + warp) * a.ld_k + (size_t)(h / a.q_group) * dk + lane * 8;
    const bf16* vp = (const bf16*)a.v + (t0 + warp) * a.ld_v + (size_t)h * dv + col0 + lane * 8;
    bf16 *qd = qs + warp * sh.ldq + lane * 8, *kd = ks + warp * sh.ldq + lane * 8, *vd = vs + warp * sh.ldv + lane * 8;
#pragma unroll
    for (int i = 0; i < LC_C; i += 8) {
      const bool live = warp + i < left, lq = live && q_in, lv = live && v_in;
      if (lane < pq) {
        lc_cp16(qd + i * sh.ldq, lq ? qp + (size_t)(i * a.ld_q) : (const bf16*)a.q, lq);
        lc_cp16(kd + i * sh.ldq, lq ? kp + (size_t)(i * a.ld_k) : (const bf16*)a.k, lq);
      }
      if (lane < pv) lc_cp16(vd + i * sh.ldv, lv ? vp + (size_t)(i * a.ld_v) : (const bf16*)a.v, lv);
    }
    for (int i = tid; i < (int)sizeof(LpGates) / 16; i += LP_THREADS) lc_cp16((char*)&gt + i * 16, (const char*)(w.gates + slot) + i * 16, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // a warp's first runs of 32 keys of the state, on their way meanwhile
  const int ncg = cols >> 4;
  int cg = warp;
  const float* Sp = w.S + (slot * w.ct + (col0 >> 4) + cg) * (size_t)(dkp >> 3) * 128 + lane * 4;
  float4 next[4];
  if (cg < ncg) {
#pragma unroll
    for (int i = 0; i < 4; ++i) next[i] = *(const float4*)(Sp + i * 128);
  }
  if (tid < dkp / 4) {
    const float4* np = (const float4*)(w.n + slot * LP_NPARTS * dkp) + tid;
    const float4 x0 = np[0], x1 = np[dkp / 4], x2 = np[dkp / 2], x3 = np[dkp / 4 * 3];
    *(float4*)(ns + tid * 4) = make_float4((x0.x + x1.x) + (x2.x + x3.x), (x0.y + x1.y) + (x2.y + x3.y), (x0.z + x1.z) + (x2.z + x3.z),
                                           (x0.w + x1.w) + (x2.w + x3.w));
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  {
    const int mt = warp >> 1;
    const bool diag = warp & 1;
    const int jb0 = diag ? mt : 0, nblk = diag ? 1 : mt;
    float f[3][2][4] = {};
    if (nblk) {
      for (int k4 = 0; k4 < dkp; k4 += 32) {         // runs of two products, added up in float32
        float part[3][2][4];
#pragma unroll
        for (int kk = k4; kk < k4 + 32; kk += 16) {
          uint32_t af[4], bq[4];
          lc_ldsm4(af, qs + (mt * 16 + (mi & 1) * 8 + r8) * sh.ldq + kk + (mi >> 1) * 8);
#pragma unroll
          for (int b = 0; b < 3; ++b)
            if (b < nblk) {
              lc_ldsm4(bq, ks + ((jb0 + b) * 16 + (mi >> 1) * 8 + r8) * sh.ldq + kk + (mi & 1) * 8);
              lc_mma(kk == k4, part[b][0], af, bq[0], bq[1]);
              lc_mma(kk == k4, part[b][1], af, bq[2], bq[3]);
            }
        }
#pragma unroll
        for (int b = 0; b < 3; ++b)
          if (b < nblk) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
              for (int x = 0; x < 4; ++x) f[b][nt][x] += part[b][nt][x];
          }
      }
    }
    float rs[2] = {0.f, 0.f};
    if (diag) {
      const float2 Gt[2] = {gt.G[mt * 16 + g8], gt.G[mt * 16 + g8 + 8]};
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          const int jr = nt * 8 + 2 * t4 + jj;
          const float2 Hj = gt.H[mt * 16 + jr];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const float x = jr <= g8 + r * 8 ? f[0][nt][2 * r + jj] * lc_exp_sum(Gt[r], Hj) : 0.f;
            f[0][nt][2 * r + jj] = x;
            rs[r] += x;
          }
        }
    } else {
#pragma unroll
      for (int b = 0; b < 3; ++b)
        if (b < nblk) {
          const float R[2] = {gt.R[b][mt * 16 + g8], gt.R[b][mt * 16 + g8 + 8]};
#pragma unroll
          for (int nt = 0; nt < 2; ++nt) {
            const float2 E = *(const float2*)(gt.E + b * 16 + nt * 8 + 2 * t4);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              f[b][nt][2 * r] *= R[r] * E.x;
              f[b][nt][2 * r + 1] *= R[r] * E.y;
              rs[r] += f[b][nt][2 * r] + f[b][nt][2 * r + 1];
            }
          }
        }
    }
    if (warp == 0) {                               // n . q, two tokens a lane
      float sum[2] = {0.f, 0.f};
      for (int k4 = 0; k4 < dkp; k4 += 32) {         // runs of 32 keys, two sums each
        float part[2][2] = {};
#pragma unroll
        for (int k = k4; k < k4 + 32; k += 8) {
          const float4 na = *(const float4*)(ns + k), nb = *(const float4*)(ns + k + 4);
          const float nn[8] = {na.x, na.y, na.z, na.w, nb.x, nb.y, nb.z, nb.w};
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const uint4 qv = *(const uint4*)(qs + (u * 32 + lane) * sh.ldq + k);
            const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162 q2 = *(const __nv_bfloat162*)&qw[i];
              part[u][0] = fmaf(nn[2 * i], __low2float(q2), part[u][0]);
              part[u][1] = fmaf(nn[2 * i + 1], __high2float(q2), part[u][1]);
            }
          }
        }
        sum[0] += part[0][0] + part[0][1];
        sum[1] += part[1][0] + part[1][1];
      }
      nq[lane] = sum[0];
      nq[32 + lane] = sum[1];
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      rs[x] += __shfl_xor_sync(0xffffffffu, rs[x], 1);
      rs[x] += __shfl_xor_sync(0xffffffffu, rs[x], 2);
      if (t4 == 0) rowsum[(mt * 16 + g8 + x * 8) * 2 + (warp & 1)] = rs[x];
    }
    __syncthreads();                                 // all are done with k
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (b < nblk) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            uint32_t t[3];
            lc_split3(f[b][nt][2 * r], f[b][nt][2 * r + 1], t);
#pragma unroll
            for (int x = 0; x < 3; ++x) *(uint32_t*)(wt + (x * LC_C + mt * 16 + g8 + r * 8) * LDW + (jb0 + b) * 16 + nt * 8 + 2 * t4) = t[x];
          }
      }
  }
  __syncthreads();                                   // W's terms, its rows' sums and n . q are in place
  const int* odd = w.odd + ((size_t)it.place * a.H + h) * ((dv + LP_KEYS - 1) / LP_KEYS);
  for (; cg < ncg; cg += LP_THREADS / 32) {
    float acc[4][2][4] = {};
    const float* Snext = Sp + (size_t)(LP_THREADS / 32) * (dkp >> 3) * 128;    // the warp's next 16 columns
    for (int run = 0; run < dkp >> 5; ++run) {
      uint32_t b0[2][2][3], b1[2][2][3];             // [key step][column tile][term]
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        lc_split3(next[2 * kk].x, next[2 * kk].y, b0[kk][0]);
        lc_split3(next[2 * kk].z, next[2 * kk].w, b0[kk][1]);
        lc_split3(next[2 * kk + 1].x, next[2 * kk + 1].y, b1[kk][0]);
        lc_split3(next[2 * kk + 1].z, next[2 * kk + 1].w, b1[kk][1]);
      }
      const bool more = run + 1 < dkp >> 5;
      const float* np = more ? Sp + (run + 1) * 512 : Snext;
      if (more || cg + LP_THREADS / 32 < ncg) {
#pragma unroll
        for (int i = 0; i < 4; ++i) next[i] = *(const float4*)(np + i * 128);
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float hi[2][4], lo[2][4];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          uint32_t af[4];
          lc_ldsm4(af, qs + (m * 16 + (mi & 1) * 8 + r8) * sh.ldq + run * 32 + kk * 16 + (mi >> 1) * 8);
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) {
            lc_mma(kk == 0, lo[nb], af, b0[kk][nb][2], b1[kk][nb][2]);
            lc_mma(kk == 0, hi[nb], af, b0[kk][nb][0], b1[kk][nb][0]);
            lc_mma(lo[nb], af, b0[kk][nb][1], b1[kk][nb][1]);
          }
        }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[m][nb][x] += hi[nb][x] + lo[nb][x];
      }
    }
    Sp = Snext;
    const bool skip = odd[(col0 + cg * 16) / LP_KEYS] != 0;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      float yw[2][4] = {};
#pragma unroll
      for (int run = 0; run < 2; ++run) {            // runs of 32 tokens
        if (2 * run > mt) break;
        float hi[2][4], lo[2][4];
#pragma unroll
        for (int kk = 2 * run; kk < 2 * run + 2; ++kk) {
          if (kk > mt) break;
          uint32_t bv[4];
          lc_ldsm4t(bv, vs + (kk * 16 + (mi & 1) * 8 + r8) * sh.ldv + cg * 16 + (mi >> 1) * 8);
#pragma unroll
          for (int x = 2; x >= 0; --x) {
            uint32_t af[4];
            lc_ldsm4(af, wt + (x * LC_C + mt * 16 + (mi & 1) * 8 + r8) * LDW + kk * 16 + (mi >> 1) * 8);
            lc_mma(kk == 2 * run && x != 1, x ? lo[0] : hi[0], af, bv[0], bv[1]);
            lc_mma(kk == 2 * run && x != 1, x ? lo[1] : hi[1], af, bv[2], bv[3]);
          }
        }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
          for (int x = 0; x < 4; ++x) yw[nb][x] += hi[nb][x] + lo[nb][x];
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int t = mt * 16 + g8 + r * 8;
        if (t >= left || skip) continue;
        const float At = gt.A[t];
        const float den = fmaxf(fabsf((rowsum[2 * t] + rowsum[2 * t + 1] + At * nq[t]) * a.q_scale), gt.em[t]) + 1e-6f;
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          const int col = cg * 16 + nb * 8 + 2 * t4;
          if (col0 + col >= dv) continue;
          const float y0 = fmaf(At, acc[mt][nb][2 * r], yw[nb][2 * r]) * a.q_scale, y1 = fmaf(At, acc[mt][nb][2 * r + 1], yw[nb][2 * r + 1]) * a.q_scale;
          *(float2*)(a.out + (t0 + t) * a.ld_out + (size_t)h * dv + col0 + col) = make_float2(y0 / den, y1 / den);
        }
      }
    }
  }
  if (cr == 0) {
    const int end = (c + it.count) * LC_C < len ? (c + it.count) * LC_C : len;
    const int tiles = (dv + w.vt - 1) / w.vt;
    for (int b = col0 / LP_KEYS; b * LP_KEYS < col0 + cols; ++b) {
      if (!odd[b]) continue;
      __syncthreads();                               // all are done with shared memory
      for (int tile = b * LP_KEYS / w.vt; tile < (b + 1) * LP_KEYS / w.vt && tile < tiles; ++tile) {
        if (w.vt == 16) lc_token_by_token<SCAN_GATED_MAX, 16, LP_THREADS>(a, w.n + slot * LP_NPARTS * dkp, LP_NPARTS, dkp, s, (int)t0, end - c * LC_C, h, tile, (float*)lp_smem);
        else lc_token_by_token<SCAN_GATED_MAX, 32, LP_THREADS>(a, w.n + slot * LP_NPARTS * dkp, LP_NPARTS, dkp, s, (int)t0, end - c * LC_C, h, tile, (float*)lp_smem);
      }
    }
  }
}

#define LP_MAX_OUT_BYTES (112 * 1024)      // two CTAs an SM

static int launch_scan_parallel(const ScanArgs& a, PortionRounds& rounds, void* ws, cudaStream_t st, int* launches) {
  static PerDevice allowed[2];
  LpWork w;
  w.dkp = (a.dk + 31) / 32 * 32;
  w.ct = (a.dv + 15) / 16;
  w.vt = scan_vt(a.dk);
  const size_t cells = rounds.slots() * a.H, places = (size_t)rounds.places() * a.H;
  w.m = (double*)ws;
  w.S = (float*)(w.m + (places + 1) / 2 * 2);
  w.gates = (LpGates*)(w.S + cells * w.ct * w.dkp * 16);
  w.n = (float*)(w.gates + cells);
  w.n_end = w.n + cells * LP_NPARTS * w.dkp;
  w.odd = (int*)(w.n_end + places * LP_NPARTS * w.dkp);
  const int cols = a.dv < LP_COLS ? (a.dv + 15) / 16 * 16 : LP_COLS;
  const int out_bytes = LpOutShape(w.dkp, cols).bytes, token_bytes = (a.dk * (w.vt + 3) + LP_THREADS + 4) * 4;
  const int smem = out_bytes > token_bytes ? out_bytes : token_bytes, states = (int)sizeof(LpStatesSmem);
  const int kblocks = (a.dk + LP_KEYS - 1) / LP_KEYS, cblocks = (a.dv + LP_KEYS - 1) / LP_KEYS;
  int rc = qv_allow_smem(lp_states_kernel, states, allowed[0]);
  if (!rc) rc = qv_allow_smem(lp_outputs_kernel, LP_MAX_OUT_BYTES, allowed[1]);
  while (!rc && rounds.next(w.round)) {
    rc = qv_launch(lp_gates_kernel, dim3(w.round.items, a.H), dim3(32 * LP_GATE_WARPS), 0, st, a, w);
    if (!rc) rc = qv_launch(lp_states_kernel, dim3(w.round.items, a.H, kblocks * (cblocks + 1)), dim3(LP_THREADS), (size_t)states, st, a, w);
    const dim3 grid(w.round.slots, a.H, (a.dv + LP_COLS - 1) / LP_COLS);
    if (!rc) rc = qv_launch(lp_outputs_kernel, grid, dim3(LP_THREADS), (size_t)smem, st, a, w);
    *launches += 3;
  }
  return rc;
}

// Segments from this many tokens on take the three launches, if their gates have a running maximum.  A layer with 4 heads of 256 x 512, us with the
// one kernel and with these: 768 tokens 121 and 127 (two launches more of a step that is not captured), 900 150 and 144, 1,024 159 and 148, 2,048
// 271 and 201; with 4 heads of 128 x 256 1,024 tokens 117 and 102, 2,048 203 and 140.
// Scalar decays stay with linear_scan_chunk_kernel: many heads of small states fill the GPU as they are (64 heads of 128 x 64, 1,943 tokens
// in three segments: a layer 292 us, and 299 with these launches; one segment of 2,048: 282 and 317).
// Which sizes: linear_scan_chunk_kernel forms W again for every tile of value columns, so many tiles a head speak for the three launches; where few
// tiles of all heads together fill the GPU once (128 CTAs) it is at its best.  A rule on a segment's own length and the sizes, so that its
// neighbours do not decide which sums it gets.  us with the one kernel and with the three launches, captured, one segment and four of 1,024
// tokens: 4 heads of 256 x 512 86 and 64, 333 and 171; 4 heads of 128 x 256 71 and 53, 73 and 64 (768 x 4: 56 and 57);
// 16 heads of 256 x 64 85 and 54, 170 and 139 (768 x 2: 66 and 72); 32 heads of 128 x 128 73 and 81, 286 and 207 (2,048: 141 and
// 144, 558 and 419); 16 heads of 64 x 64 61 and 46, 62 and 75; 64 heads of 128 x 64 74 and 98, 288 and 298; 4 heads of 64 x 64 61 and 43, 61
// and 46; 1 head 61 and 44.
static inline int scan_parallel_from(int kind, int H, int dk, int dv) {
  const int never = 0x7fffffff;
  if (kind != SCAN_GATED_MAX || dk > 256) return never;
  const int vt = scan_vt(dk), tiles = (dv + vt - 1) / vt;
  if (tiles >= 16) return 896;
  if (tiles >= 6 || (tiles >= 4 && vt == 16) || (long long)H * tiles <= 8) return 1024;
  return tiles >= 4 ? 2048 : never;
}
extern "C" int qv_linear_scan_parallel_from(int kind, int H, int dk, int dv) { return scan_parallel_from(kind, H, dk, dv); }
// What the three launches take beside qv_linear_scan's operands, for `rest` segments that take them, of rest_max tokens each (where they are not
// alike: of their mean number of chunks): the states of as many chunks as LP_ROOM bytes hold, the next ones follow in launches of their
// own (so few of a segment, LP_FEW, only where the step has many).
#define LP_ROOM ((size_t)160 << 20)
#define LP_FEW 8
static inline size_t lp_room_slots(int H, int dk, int dv) {
  const size_t fit = LP_ROOM / lp_slot_bytes(H, dk, dv);
  return fit ? fit : 1;
}
static inline long long lp_bytes(size_t slots, int places, int H, int dk, int dv) {
  return (long long)(slots * lp_slot_bytes(H, dk, dv) + places * lp_place_bytes(H, dk, dv) + 32);
}
extern "C" long long qv_linear_scan_workspace_bytes(int kind, int rest, int rest_max, int H, int dk, int dv) {
  if (rest <= 0 || H <= 0 || dk <= 0 || dv <= 0 || rest_max < scan_parallel_from(kind, H, dk, dv)) return 0;
  const size_t chunks = (size_t)((rest_max + LC_C - 1) / LC_C) * rest, fit = lp_room_slots(H, dk, dv);
  return lp_bytes(chunks < fit ? chunks : fit, rest, H, dk, dv);
}

extern "C" long long qv_linear_scan_state_floats(int kind, int H, int dk, int dv) {
  const int vt = scan_vt(dk);
  return (long long)H * ((dv + vt - 1) / vt) * scan_tile_floats(kind, dk, vt);
}

// Segments from the first of SCAN_CHUNK_FROM tokens on take the chunks' kernel (those among them that are shorter leave it at once), so
// that single tokens, which come first in a step, add no CTAs to it: lead, the segments ahead of it; rest_max, rest_min, the longest and the
// shortest of the others (rest_min 0: not known; that costs a launch).  lens: the segments' tokens (host); ws,
// ws_bytes: as qv_linear_scan_workspace_bytes says for those of parallel_from tokens and more.  Either null: these take the chunks' kernel
// like the others.  *launches: how many kernels were launched.
#define SCAN_CHUNK_FROM 16
extern "C" int qv_linear_scan_chunk_from(void) { return SCAN_CHUNK_FROM; }
extern "C" int qv_linear_scan(int kind, float* out, int ld_out, const void* q, int ld_q, int q_group, const void* k, int ld_k,
                              const void* v, int ld_v, const float* g1, int ld_g1, const float* g2, int ld_g2, const float* p1,
                              const float* p2, const float* p3, float cap, float q_scale, float* state, long long slot_stride,
                              const int* seg_q_start, const int* seg_slot, int S, int lead, int rest_max, int rest_min, int H, int dk, int dv, int dt,
                              const int* lens, void* ws, long long ws_bytes, int* launches, void* stream) {
  *launches = 0;
  if (S <= 0) return 0;
  if (kind != SCAN_GATED_MAX && kind != SCAN_DECAY) return QV_ERR_UNSUPPORTED;
  if (H <= 0 || dk <= 0 || dv <= 0 || q_group <= 0 || H > 65535) return QV_ERR_UNSUPPORTED;
  const int vt = scan_vt(dk);
  const int tiles = (dv + vt - 1) / vt;
  const size_t smem = ((size_t)dk * SCAN_VT + 3 * (size_t)dk + SCAN_WARPS * SCAN_VT + 2) * sizeof(float);
  if (smem > 200 * 1024 || tiles > 65535) return QV_ERR_TOO_LARGE;
  ScanArgs a;
  a.out = out; a.ld_out = ld_out; a.q = q; a.ld_q = ld_q; a.q_group = q_group; a.k = k; a.ld_k = ld_k; a.v = v; a.ld_v = ld_v;
  a.g1 = g1; a.ld_g1 = ld_g1; a.g2 = g2; a.ld_g2 = ld_g2; a.p1 = p1; a.p2 = p2; a.p3 = p3; a.cap = cap; a.q_scale = q_scale;
  a.state = state; a.slot_stride = slot_stride; a.seg_q_start = seg_q_start; a.seg_slot = seg_slot; a.H = H; a.dk = dk; a.dv = dv;
  a.chunk_from = a.parallel_from = 0x7fffffff;
  dim3 grid(S, H, tiles);
  cudaStream_t st = (cudaStream_t)stream;
  // Portions of SCAN_CHUNK_FROM tokens and more take the tensor cores, the step's other segments the token-by-token kernel: which kernel a
  // segment runs through depends on its own length alone.  bfloat16 only (the 32-bit path keeps one order of sums for every cut).
  if (dt == QV_DT_BF16 && lead >= 0 && lead < S && rest_max >= SCAN_CHUNK_FROM && dk <= 256 && dk % 8 == 0 && dv % 8 == 0 && ld_q % 8 == 0 && ld_k % 8 == 0 &&
      ld_v % 8 == 0 && ld_out % 4 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) == 0) {
    a.chunk_from = SCAN_CHUNK_FROM;
    ScanArgs rest = a;
    rest.seg_q_start += lead;
    rest.seg_slot += lead;
    const dim3 rest_grid(S - lead, H, tiles);
    int rc = 0;
    const int parallel_from = scan_parallel_from(kind, H, dk, dv);
    if (ws && lens && ((uintptr_t)ws & 15) == 0 && rest_max >= parallel_from) {
      try {
        PortionRounds rounds(lens + lead, S - lead, LC_C, parallel_from, lp_room_slots(H, dk, dv), LP_FEW);
        if (ws_bytes < lp_bytes(rounds.slots(), rounds.places(), H, dk, dv)) return QV_ERR_UNSUPPORTED;
        a.parallel_from = rest.parallel_from = parallel_from;
        rc = launch_scan_parallel(rest, rounds, ws, st, launches);
      } catch (...) {
        return QV_ERR_TOO_LARGE;
      }
      if (rc || (lead == 0 && rest_min >= parallel_from)) return rc;
    }
    if (rest.parallel_from > rest_min) ++*launches;
    if (rest.parallel_from <= rest_min) rc = 0;              // none of them is left for the chunks' kernel
    else if (kind == SCAN_GATED_MAX)
      rc = vt == 16 ? launch_scan_chunk<SCAN_GATED_MAX, 16, 2>(rest, rest_grid, st)
                    : dk <= 64 ? launch_scan_chunk<SCAN_GATED_MAX, 32, 1>(rest, rest_grid, st) : launch_scan_chunk<SCAN_GATED_MAX, 32, 2>(rest, rest_grid, st);
    else
      rc = vt == 16 ? launch_scan_chunk<SCAN_DECAY, 16, 2>(rest, rest_grid, st)
                    : dk <= 64 ? launch_scan_chunk<SCAN_DECAY, 32, 1>(rest, rest_grid, st) : launch_scan_chunk<SCAN_DECAY, 32, 2>(rest, rest_grid, st);
    if (rest_min >= SCAN_CHUNK_FROM) grid.x = lead;          // none of them is left for the kernel below
    if (rc || grid.x == 0) return rc;
  }
  ++*launches;
  if (dk <= 8 * 32) {                      // the state fits the registers
    const size_t esz = dt == QV_DT_F32 ? 4 : 2;
    const size_t rowpad = (size_t)((dk + 7) & ~7);
    const size_t smem_r = ((4 * SCAN_TB * rowpad * esz + 3) / 4 + dk + SCAN_TB * SCAN_WARPS * SCAN_VT + SCAN_TB + 4 * SCAN_CH) * sizeof(float);
    const bool async = (dk * esz) % 16 == 0 && ((size_t)ld_q * esz) % 16 == 0 && ((size_t)ld_k * esz) % 16 == 0 &&
                       (((uintptr_t)q | (uintptr_t)k) & 15) == 0;
    const int rpt = dk <= 32 ? 4 : dk <= 64 ? 8 : 16;          // 129..256 rows: 16 columns a tile, two row groups a warp
#define LAUNCH_REG(TT, KIND, RPT)                                                                                             \
  do {                                                                                                                        \
    if (vt == 16) {                                                                                                           \
      if (async) return qv_launch(linear_scan_reg_kernel<TT, KIND, 16, true, 16>, grid, dim3(SCAN_VT * SCAN_WARPS), smem_r, st, a); \
      return qv_launch(linear_scan_reg_kernel<TT, KIND, 16, false, 16>, grid, dim3(SCAN_VT * SCAN_WARPS), smem_r, st, a);     \
    }                                                                                                                         \
    if (async) return qv_launch(linear_scan_reg_kernel<TT, KIND, RPT, true, 32>, grid, dim3(SCAN_VT * SCAN_WARPS), smem_r, st, a); \
    return qv_launch(linear_scan_reg_kernel<TT, KIND, RPT, false, 32>, grid, dim3(SCAN_VT * SCAN_WARPS), smem_r, st, a);      \
  } while (0)
#define LAUNCH_REG_RPT(TT, KIND)                  \
  do {                                            \
    if (rpt == 4) LAUNCH_REG(TT, KIND, 4);        \
    if (rpt == 8) LAUNCH_REG(TT, KIND, 8);        \
    LAUNCH_REG(TT, KIND, 16);                     \
  } while (0)
    if (dt == QV_DT_F32 && kind == SCAN_GATED_MAX) LAUNCH_REG_RPT(float, SCAN_GATED_MAX);
    if (dt == QV_DT_F32 && kind == SCAN_DECAY) LAUNCH_REG_RPT(float, SCAN_DECAY);
    if (dt == QV_DT_BF16 && kind == SCAN_GATED_MAX) LAUNCH_REG_RPT(bf16, SCAN_GATED_MAX);
    if (dt == QV_DT_BF16 && kind == SCAN_DECAY) LAUNCH_REG_RPT(bf16, SCAN_DECAY);
#undef LAUNCH_REG_RPT
#undef LAUNCH_REG
    return QV_ERR_UNSUPPORTED;
  }
#define LAUNCH_SCAN(TT, KIND)                                                                                               \
  do {                                                                                                                      \
    if (smem > 48 * 1024) cudaFuncSetAttribute(linear_scan_kernel<TT, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    return qv_launch(linear_scan_kernel<TT, KIND>, grid, dim3(SCAN_VT * SCAN_WARPS), smem, st, a);                          \
  } while (0)
  if (dt == QV_DT_F32 && kind == SCAN_GATED_MAX) LAUNCH_SCAN(float, SCAN_GATED_MAX);
  if (dt == QV_DT_F32 && kind == SCAN_DECAY) LAUNCH_SCAN(float, SCAN_DECAY);
  if (dt == QV_DT_BF16 && kind == SCAN_GATED_MAX) LAUNCH_SCAN(bf16, SCAN_GATED_MAX);
  if (dt == QV_DT_BF16 && kind == SCAN_DECAY) LAUNCH_SCAN(bf16, SCAN_DECAY);
#undef LAUNCH_SCAN
  return QV_ERR_UNSUPPORTED;
}

// ---------------------------------------------------------------- unit norm in equal parts, weight, gate
// y [T, width] float32 in `groups` equal parts; gate [T, width] in the compute type (row stride ld_gate).
//   gate_first = 0:  out = y / rms_part(y) * w * sigmoid(gate)
//   gate_first = 1:  u = y * silu(gate);  out = u / rms_part(u) * w
// One block per (token, part).
template <typename T>
__global__ void __launch_bounds__(1024) gated_group_norm_kernel(T* __restrict__ out, int ld_out, const float* __restrict__ y, int ld_y,
                                                               const T* __restrict__ gate, int ld_gate, const float* __restrict__ w,
                                                               int part, float eps, int gate_first) {
  __shared__ float red[33];
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, g = blockIdx.y;
  const float* yr = y + (size_t)t * ld_y + (size_t)g * part;
  const T* gr = gate + (size_t)t * ld_gate + (size_t)g * part;
  T* o = out + (size_t)t * ld_out + (size_t)g * part;
  const float* wr = w + (size_t)g * part;
  float ss = 0.f;
  for (int i = threadIdx.x; i < part; i += blockDim.x) {
    float v = yr[i];
    if (gate_first) { const float z = to_f(gr[i]); v *= z / (1.0f + expf(-z)); }
    ss += v * v;
  }
  const float total = block_sum(ss, red);
  const float sc = 1.0f / sqrtf(total / (float)part + eps);
  for (int i = threadIdx.x; i < part; i += blockDim.x) {
    const float z = to_f(gr[i]);
    float v = yr[i];
    if (gate_first) v = v * (z / (1.0f + expf(-z))) * sc * wr[i];
    else v = v * sc * wr[i] * (1.0f / (1.0f + expf(-z)));
    o[i] = from_f<T>(v);
  }
}

// The same with 16-byte accesses and the part's values kept in registers between the sum and the output (they were read twice, one element
// a thread: 34 us for 2,048 x 2,048 in parts of 512, 42 us for 1,943 x 4,096 in one part; now 11 and 15).  A thread holds Q pieces of
// four, `blockDim` pieces apart; part a multiple of 4 of at most 4 Q blockDim.
template <typename T, int Q>
__global__ void __launch_bounds__(512) gated_group_norm_vec_kernel(T* __restrict__ out, int ld_out, const float* __restrict__ y, int ld_y,
                                                                   const T* __restrict__ gate, int ld_gate, const float* __restrict__ w, int part,
                                                                   float eps, int gate_first) {
  struct alignas(4 * sizeof(T)) Pack { T v[4]; };
  __shared__ float red[33];
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, g = blockIdx.y, pieces = part >> 2;
  const float4* yr = (const float4*)(y + (size_t)t * ld_y + (size_t)g * part);
  const Pack* gr = (const Pack*)(gate + (size_t)t * ld_gate + (size_t)g * part);
  const float4* wr = (const float4*)(w + (size_t)g * part);
  Pack* o = (Pack*)(out + (size_t)t * ld_out + (size_t)g * part);
  float v[Q][4], z[Q][4];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int p = threadIdx.x + i * blockDim.x;
    float4 yv = make_float4(0.f, 0.f, 0.f, 0.f);
    Pack gv = {};
    if (p < pieces) { yv = yr[p]; gv = gr[p]; }
    v[i][0] = yv.x; v[i][1] = yv.y; v[i][2] = yv.z; v[i][3] = yv.w;
#pragma unroll
    for (int k = 0; k < 4; ++k) z[i][k] = to_f(gv.v[k]);
  }
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float s = 1.0f / (1.0f + expf(-z[i][k]));
      if (gate_first) v[i][k] *= z[i][k] * s;
      z[i][k] = s;
      ss = fmaf(v[i][k], v[i][k], ss);
    }
  const float sc = 1.0f / sqrtf(block_sum(ss, red) / (float)part + eps);
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const int p = threadIdx.x + i * blockDim.x;
    if (p >= pieces) break;
    const float4 wv = wr[p];
    const float ww[4] = {wv.x, wv.y, wv.z, wv.w};
    Pack r;
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = from_f<T>(v[i][k] * sc * ww[k] * (gate_first ? 1.0f : z[i][k]));
    o[p] = r;
  }
}

extern "C" int qv_gated_group_norm(void* out, int ld_out, const float* y, int ld_y, const void* gate, int ld_gate, const float* w,
                                   int T, int width, int groups, float eps, int gate_first, int dt, void* stream) {
  if (T <= 0) return 0;
  if (groups <= 0 || width % groups || groups > 65535) return QV_ERR_UNSUPPORTED;
  // one element a thread up to 1024; the block's size, and so the order of the sums, follows from the part's width alone
  const int part_w = width / groups;
  const int threads = part_w >= 1024 ? 1024 : (part_w <= 128 ? 128 : ((part_w + 31) / 32) * 32);
  const size_t esz = dt == QV_DT_F32 ? 4 : 2;
  if (part_w % 4 == 0 && part_w <= 8192 && ld_out % 4 == 0 && ld_y % 4 == 0 && ld_gate % 4 == 0 && (((uintptr_t)y | (uintptr_t)w) & 15) == 0 &&
      (((uintptr_t)out | (uintptr_t)gate) & (4 * esz - 1)) == 0) {
    const int pieces = part_w / 4;
    const int q = pieces <= 512 ? 1 : pieces <= 1024 ? 2 : 4;
    const dim3 block((((pieces + q - 1) / q) + 31) / 32 * 32);
#define GGN(TT, QQ)                                                                                                                \
  return qv_launch(gated_group_norm_vec_kernel<TT, QQ>, dim3(T, groups), block, 0, (cudaStream_t)stream, (TT*)out, ld_out, y, ld_y, \
                   (const TT*)gate, ld_gate, w, part_w, eps, gate_first)
    QV_DISPATCH_DT(dt, TT, if (q == 1) GGN(TT, 1); if (q == 2) GGN(TT, 2); GGN(TT, 4));
#undef GGN
  }
  QV_DISPATCH_DT(dt, TT,
                 return qv_launch(gated_group_norm_kernel<TT>, dim3(T, groups), dim3(threads), 0, (cudaStream_t)stream, (TT*)out, ld_out, y,
                                  ld_y, (const TT*)gate, ld_gate, w, width / groups, eps, gate_first));
  return QV_ERR_UNSUPPORTED;
}
