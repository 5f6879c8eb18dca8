// Routed feed-forward (mixture of experts): router, grouping of tokens by expert, the experts' products
// over the grouped rows, and the weighted sum back into token order.
//
// qv_moe_route    logits = Wr h in float32 (fixed summation order), the `top` largest per token (ties: the lower
//                 index), weights = softmax over the chosen logits only; optionally one more row of the router
//                 matrix' companion (a scalar gate per token: sigmoid(ws . h)).  With `correction`: scores = softmax over all
//                 logits, the choice by score + correction, weights = scores * w_scale (not renormalised).  In sigmoid mode:
//                 scores = sigmoid(logits), the choice by score + correction among the experts of the `keep` best of `groups`
//                 equal groups of neighbours (a group counts the sum of its two largest choice scores), weights = the chosen
//                 scores over their sum (+ 1e-20), times w_scale.
// qv_moe_route_table  no router: row `token id` of an integer table [vocab, top] lists the token's experts, each weighted 1/top.
// qv_moe_group    counting sort of the (token, choice) pairs by expert, all on the device (a step never waits
//                 for the host): row_token[r] = token of sorted row r, slot_row[token * top + j] = its sorted row,
//                 and a table of row tiles (expert, first row, rows) for the products' grids.
// qv_moe_experts  CUDA-core products over the grouped rows, float32 multiply-adds with k ascending:
//                   UP (1):   act[r] = glu(Wg_e h[row_token[r]], Wu_e h[row_token[r]])    (GluAct: SiLU, GELU, clamped)
//                   UP (2):   act[r] = relu(Wu_e h[row_token[r]])^2            (ungated experts)
//                   DOWN (0): y[r]   = Wd_e act[r]   (float32)
// qv_moe_combine  delta[t] = (mixer output) * s_mix + (sum_j weight[t, j] * y[slot_row[t, j]] + gate[t] * shared[t]) * s_ff
//                 in float32, choices summed in the order the router ranked them; s_mix, s_ff: per-feature factors or none.
//
// Choices at or beyond the number of experts are identity experts: they take no row in the grouping (slot_row -1) and
// the sum takes the token's own input for them.
#include "tc_common.cuh"

#define ROUTE_WARPS 8
// One warp's dot product of a weight row with the token's inputs (float32 in shared memory), summed over the warp.
template <typename TW>
__device__ __forceinline__ float route_dot(const TW* __restrict__ w, const float* __restrict__ xs, int d, int lane) {
  // 16-byte loads, eight in flight per lane, where the rows allow; the order of the sum depends on d only
    float acc = 0.f;
    constexpr int VEC = 16 / (int)sizeof(TW);
    int i = 0;
    if ((d % VEC) == 0 && (((uintptr_t)w) & 15) == 0) {
      for (i = lane * VEC; i + 7 * 32 * VEC < d; i += 8 * 32 * VEC) {
        uint4 wv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) wv[u] = *(const uint4*)(w + i + u * 32 * VEC);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const TW* p = (const TW*)&wv[u];
#pragma unroll
          for (int k = 0; k < VEC; ++k) acc = fmaf(to_f(p[k]), xs[i + u * 32 * VEC + k], acc);
        }
      }
      for (; i < d; i += 32 * VEC) {
        const uint4 wv = *(const uint4*)(w + i);
        const TW* p = (const TW*)&wv;
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc = fmaf(to_f(p[k]), xs[i + k], acc);
      }
    } else {
      for (i = lane; i + 7 * 32 < d; i += 8 * 32) {
        float wv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) wv[u] = to_f(w[i + u * 32]);
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = fmaf(wv[u], xs[i + u * 32], acc);
      }
      for (; i < d; i += 32) acc = fmaf(to_f(w[i]), xs[i], acc);
    }
    return warp_sum(acc);
}

// logits[t][e] = wr[e] . h[t] for e < E, and logits[t][E] = wg . h[t] when wg is given: eight rows a CTA, so that a
// step of few tokens still spreads the router's matrix over many SMs.
template <typename T, typename TW>
__global__ void __launch_bounds__(ROUTE_WARPS * 32) moe_logits_kernel(float* __restrict__ logits, const T* __restrict__ h, int ld_h,
                                                                      const TW* __restrict__ wr, const TW* __restrict__ wg, int d, int E) {
  extern __shared__ float xs_only[];
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* x = h + (size_t)t * ld_h;
  for (int i = threadIdx.x; i < d; i += blockDim.x) xs_only[i] = to_f(x[i]);
  __syncthreads();
  const int e = blockIdx.y * ROUTE_WARPS + warp;
  if (e >= E + (wg ? 1 : 0)) return;
  const float acc = route_dot(e < E ? wr + (size_t)e * d : wg, xs_only, d, lane);
  if (lane == 0) logits[(size_t)t * (E + 1) + e] = acc;
}

// The same dot products for ROUTE_TOKENS tokens and ROUTE_ROWS rows of the router at once: a weight is converted once for all tokens, an
// input once for all rows, and every (token, row) sum has the order route_dot gives it (a lane's elements ascending, then the warp's
// tree), so the logits do not depend on which kernel formed them.  xs: [ROUTE_TOKENS][d] in shared memory, as stored.
#define ROUTE_TOKENS 8
#define ROUTE_ROWS 4
template <typename T, int N>
__device__ __forceinline__ void load_floats(const T* p, float (&f)[N]) {       // N elements, 16-byte pieces
  constexpr int PER = 16 / (int)sizeof(T);
#pragma unroll
  for (int i = 0; i < N / PER; ++i) {
    const uint4 v = *(const uint4*)(p + i * PER);
    const T* e = (const T*)&v;
#pragma unroll
    for (int k = 0; k < PER; ++k) f[i * PER + k] = to_f(e[k]);
  }
}
template <typename T, typename TW>
__device__ __forceinline__ void route_dot_tile(const TW* const (&w)[ROUTE_ROWS], const T* __restrict__ xs, int d, int lane,
                                               float (&acc)[ROUTE_ROWS][ROUTE_TOKENS]) {
  constexpr int VEC = 16 / (int)sizeof(TW);
#pragma unroll
  for (int r = 0; r < ROUTE_ROWS; ++r)
#pragma unroll
    for (int t = 0; t < ROUTE_TOKENS; ++t) acc[r][t] = 0.f;
  bool vec = (d % VEC) == 0 && (d % (16 / (int)sizeof(T))) == 0;
#pragma unroll
  for (int r = 0; r < ROUTE_ROWS; ++r) vec = vec && (((uintptr_t)w[r]) & 15) == 0;
  if (vec) {
    // (VEC is 8 or 4 elements and a lane's pieces lie 32 * VEC apart, as in route_dot)
#pragma unroll 2
    for (int i = lane * VEC; i < d; i += 32 * VEC) {
      float wf[ROUTE_ROWS][VEC];
#pragma unroll
      for (int r = 0; r < ROUTE_ROWS; ++r) load_floats<TW, VEC>(w[r] + i, wf[r]);
#pragma unroll
      for (int t = 0; t < ROUTE_TOKENS; ++t) {
        float xf[VEC];
        if (VEC * sizeof(T) >= 16) load_floats<T, VEC>(xs + (size_t)t * d + i, xf);
        else {
#pragma unroll
          for (int k = 0; k < VEC; ++k) xf[k] = to_f(xs[(size_t)t * d + i + k]);
        }
#pragma unroll
        for (int r = 0; r < ROUTE_ROWS; ++r)
#pragma unroll
          for (int k = 0; k < VEC; ++k) acc[r][t] = fmaf(wf[r][k], xf[k], acc[r][t]);
      }
    }
  } else if ((d % VEC) == 0) {
    // rows that route_dot would read in pieces but this kernel cannot: the same order, element by element
#pragma unroll
    for (int r = 0; r < ROUTE_ROWS; ++r) {
      const bool piece = (((uintptr_t)w[r]) & 15) == 0;
      for (int i = piece ? lane * VEC : lane; i < d; i += piece ? 32 * VEC : 32)
        for (int k = 0; k < (piece ? VEC : 1); ++k) {
          const float wv = to_f(w[r][i + k]);
#pragma unroll
          for (int t = 0; t < ROUTE_TOKENS; ++t) acc[r][t] = fmaf(wv, to_f(xs[(size_t)t * d + i + k]), acc[r][t]);
        }
    }
  } else {
    for (int i = lane; i < d; i += 32) {
#pragma unroll
      for (int r = 0; r < ROUTE_ROWS; ++r) {
        const float wv = to_f(w[r][i]);
#pragma unroll
        for (int t = 0; t < ROUTE_TOKENS; ++t) acc[r][t] = fmaf(wv, to_f(xs[(size_t)t * d + i]), acc[r][t]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROUTE_ROWS; ++r)
#pragma unroll
    for (int t = 0; t < ROUTE_TOKENS; ++t) acc[r][t] = warp_sum(acc[r][t]);
}

// Many tokens: a CTA takes ROUTE_TOKENS tokens and walks over all rows, four rows a warp at a time.  What bounds it is the
// multiply-adds with the conversions around them: a row alone (eight tokens in float32 in shared memory, so 16 bytes read there for
// four multiply-adds) took 170 us for 2,048 tokens x 65 rows x 2,048.
// Router as a whole (us, 2,048 wide, 65 / 256 rows), with a row alone over tokens x groups of rows and with this kernel: 257 tokens 35 / 87
// and 26 / 58, 512 tokens 59 / 147 and 26 / 58, 1,024 tokens 89 / 267 and 27 / 59, 2,048 tokens 164 / 493 and 39 / 99.
template <typename T, typename TW>
__global__ void __launch_bounds__(ROUTE_WARPS * 32) moe_logits_tokens_kernel(float* __restrict__ logits, const T* __restrict__ h, int ld_h,
                                                                             const TW* __restrict__ wr, const TW* __restrict__ wg, int d,
                                                                             int E, int T_all) {
  extern __shared__ __align__(16) unsigned char xs_raw[];
  T* xs = (T*)xs_raw;
  pdl_wait();
  pdl_launch_dependents();
  const int t0 = blockIdx.x * ROUTE_TOKENS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int PER = 16 / (int)sizeof(T);
  if (d % PER == 0 && ld_h % PER == 0 && (((uintptr_t)h) & 15) == 0) {
    const int pieces = d / PER;
    for (int i = threadIdx.x; i < ROUTE_TOKENS * pieces; i += blockDim.x) {
      const int t = i / pieces, c = (i - t * pieces) * PER;
      *(uint4*)(xs + (size_t)t * d + c) = t0 + t < T_all ? *(const uint4*)(h + (size_t)(t0 + t) * ld_h + c) : make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
    for (int i = threadIdx.x; i < ROUTE_TOKENS * d; i += blockDim.x) {
      const int t = i / d, c = i - t * d;
      xs[i] = t0 + t < T_all ? h[(size_t)(t0 + t) * ld_h + c] : from_f<T>(0.f);
    }
  }
  __syncthreads();
  const int rows = E + (wg ? 1 : 0);
  for (int e0 = warp * ROUTE_ROWS; e0 < rows; e0 += ROUTE_WARPS * ROUTE_ROWS) {
    const TW* w[ROUTE_ROWS];
#pragma unroll
    for (int r = 0; r < ROUTE_ROWS; ++r) {
      const int e = e0 + r < rows ? e0 + r : rows - 1;
      w[r] = e < E ? wr + (size_t)e * d : wg;
    }
    float acc[ROUTE_ROWS][ROUTE_TOKENS];
    route_dot_tile<T, TW>(w, xs, d, lane, acc);
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < ROUTE_ROWS; ++r)
#pragma unroll
        for (int t = 0; t < ROUTE_TOKENS; ++t)
          if (e0 + r < rows && t0 + t < T_all) logits[(size_t)(t0 + t) * (E + 1) + e0 + r] = acc[r][t];
    }
  }
}

// The same for bfloat16 inputs and weights in whole 16-byte pieces: ROWS rows a warp (so that 65 rows are one walk over the inputs for eight warps)
// and multiply-adds two tokens at a time (fma.rn.f32x2: each half is the multiply-add it stands for, so every sum is the same to the
// bit).  2,048 tokens x 65 rows x 2,048: 41 us with the kernel above, 29 here; bound by the multiply-adds and the conversions beside them.
__device__ __forceinline__ unsigned long long pair_f32(float lo, float hi) {
  unsigned long long p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
  return p;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float bf16_of(uint32_t w, int hi) { return __uint_as_float(hi ? w & 0xffff0000u : w << 16); }
template <int ROWS>
__global__ void __launch_bounds__(ROUTE_WARPS * 32) moe_logits_rows_kernel(float* __restrict__ logits, const bf16* __restrict__ h, int ld_h,
                                                                           const bf16* __restrict__ wr, const bf16* __restrict__ wg, int d, int E,
                                                                           int T_all) {
  extern __shared__ __align__(16) unsigned char xs_raw[];
  bf16* xs = (bf16*)xs_raw;                          // [ROUTE_TOKENS][d]
  pdl_wait();
  pdl_launch_dependents();
  const int t0 = blockIdx.x * ROUTE_TOKENS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pieces = d >> 3;
  for (int t = 0; t < ROUTE_TOKENS; ++t)
    for (int c = threadIdx.x; c < pieces; c += ROUTE_WARPS * 32)
      *(uint4*)(xs + (size_t)t * d + c * 8) = t0 + t < T_all ? *(const uint4*)(h + (size_t)(t0 + t) * ld_h + c * 8) : make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const int rows = E + (wg ? 1 : 0);
  for (int e0 = warp * ROWS; e0 < rows; e0 += ROUTE_WARPS * ROWS) {
    const bf16* w[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const int e = e0 + r < rows ? e0 + r : rows - 1;
      w[r] = e < E ? wr + (size_t)e * d : wg;
    }
    unsigned long long acc[ROWS][ROUTE_TOKENS / 2];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int t = 0; t < ROUTE_TOKENS / 2; ++t) acc[r][t] = 0ull;
    uint4 next[ROWS];                                // the weights of the next piece, on their way while this one's are multiplied
#pragma unroll
    for (int r = 0; r < ROWS; ++r) next[r] = lane * 8 < d ? *(const uint4*)(w[r] + lane * 8) : make_uint4(0u, 0u, 0u, 0u);
    for (int i = lane * 8; i < d; i += 256) {
      uint4 wv[ROWS], xv[ROUTE_TOKENS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        wv[r] = next[r];
        if (i + 256 < d) next[r] = *(const uint4*)(w[r] + i + 256);
      }
#pragma unroll
      for (int t = 0; t < ROUTE_TOKENS; ++t) xv[t] = *(const uint4*)(xs + (size_t)t * d + i);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        unsigned long long x2[ROUTE_TOKENS / 2];
#pragma unroll
        for (int t = 0; t < ROUTE_TOKENS / 2; ++t)
          x2[t] = pair_f32(bf16_of(((const uint32_t*)&xv[2 * t])[k >> 1], k & 1), bf16_of(((const uint32_t*)&xv[2 * t + 1])[k >> 1], k & 1));
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float f = bf16_of(((const uint32_t*)&wv[r])[k >> 1], k & 1);
          const unsigned long long w2 = pair_f32(f, f);
#pragma unroll
          for (int t = 0; t < ROUTE_TOKENS / 2; ++t) fma2(acc[r][t], w2, x2[t]);
        }
      }
    }
    // four rows x eight tokens at a time over the 32 lanes: the tree of warp_sum, each lane ending with one sum
#pragma unroll
    for (int r0 = 0; r0 < ROWS; r0 += 4) {
      float v[32];
#pragma unroll
      for (int x = 0; x < 32; ++x) {
        const int r = r0 + (x >> 3) < ROWS ? r0 + (x >> 3) : ROWS - 1;
        const unsigned long long a = acc[r][(x & 7) >> 1];
        v[x] = __uint_as_float((uint32_t)(x & 1 ? a >> 32 : a));
      }
#pragma unroll
      for (int half = 16; half > 0; half >>= 1)
#pragma unroll
        for (int x = 0; x < half; ++x) {
          const bool up = lane & half;
          const float send = up ? v[x] : v[x + half], keep = up ? v[x + half] : v[x];
          v[x] = keep + __shfl_xor_sync(0xffffffffu, send, half);
        }
      const int r = r0 + (lane >> 3), t = lane & 7;
      if (r < ROWS && e0 + r < rows && t0 + t < T_all) logits[(size_t)(t0 + t) * (E + 1) + e0 + r] = v[0];
    }
  }
}
// Rows a warp of the kernel above takes: as few walks over the inputs as sums of nine rows allow.
static int route_rows(int rows) {
  const int per = (rows + ROUTE_WARPS - 1) / ROUTE_WARPS, walks = (per + 8) / 9, each = (per + walks - 1) / walks;
  return each <= 4 ? 4 : each <= 5 ? 5 : each <= 8 ? 8 : 9;
}

// pre: logits worked out by moe_logits_kernel ([T][E + 1]), or null: then this kernel forms them itself.
template <typename T, typename TW>
__global__ void __launch_bounds__(ROUTE_WARPS * 32) moe_route_kernel(int* __restrict__ top_idx, float* __restrict__ top_w, float* __restrict__ gate_out,
                                                        const T* __restrict__ h, int ld_h, const TW* __restrict__ wr,
                                                        const TW* __restrict__ wg, int d, int E, int top, const float* __restrict__ pre,
                                                        const float* __restrict__ correction, float w_scale, int sigmoid, int groups,
                                                        int keep) {
  extern __shared__ float logit[];           // E floats, then the token's d inputs
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* xs = logit + E;
  if (pre) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) logit[e] = pre[(size_t)t * (E + 1) + e];
    if (wg && threadIdx.x == 0) gate_out[t] = 1.0f / (1.0f + expf(-pre[(size_t)t * (E + 1) + E]));
  } else {
    const T* x = h + (size_t)t * ld_h;
    for (int i = threadIdx.x; i < d; i += blockDim.x) xs[i] = to_f(x[i]);
    __syncthreads();
  }
  for (int e = warp; e < E + (wg ? 1 : 0) && !pre; e += ROUTE_WARPS) {
    float acc = route_dot(e < E ? wr + (size_t)e * d : wg, xs, d, lane);
    if (lane == 0) {
      if (e < E) logit[e] = acc;
      else gate_out[t] = 1.0f / (1.0f + expf(-acc));
    }
  }
  __syncthreads();
  if (warp != 0) return;
  float* score = xs + d;                     // E floats, with `correction`: the scores, while logit[] holds what the choice is by
  if (sigmoid) {
    for (int e = lane; e < E; e += 32) {
      score[e] = 1.0f / (1.0f + expf(-logit[e]));
      logit[e] = score[e] + (correction ? correction[e] : 0.f);
    }
    __syncwarp();
    if (keep < groups) {
      float* gscore = score + E;             // one number per group
      const int each = E / groups;
      for (int g = lane; g < groups; g += 32) {
        float a = -INFINITY, b = -INFINITY;  // the two largest of the group
        for (int i = 0; i < each; ++i) {
          const float v = logit[g * each + i];
          if (v > a) { b = a; a = v; }
          else if (v > b) b = v;
        }
        gscore[g] = each > 1 ? a + b : a;
      }
      __syncwarp();
      for (int g = lane; g < groups; g += 32) {
        int ahead = 0;                       // groups that come before this one (ties: the lower index)
        for (int o = 0; o < groups; ++o) ahead += gscore[o] > gscore[g] || (gscore[o] == gscore[g] && o < g);
        if (ahead >= keep)
          for (int i = 0; i < each; ++i) logit[g * each + i] = -INFINITY;
      }
      __syncwarp();
    }
  } else if (correction) {
    float mx = -INFINITY, sum = 0.f;
    for (int e = lane; e < E; e += 32) mx = fmaxf(mx, logit[e]);
    mx = warp_max(mx);
    for (int e = lane; e < E; e += 32) {
      const float p = expf(logit[e] - mx);
      score[e] = p;
      sum += p;
    }
    sum = warp_sum(sum);
    for (int e = lane; e < E; e += 32) {
      score[e] /= sum;
      logit[e] = score[e] + correction[e];
    }
    __syncwarp();
  }
  float first = 0.f, denom = 0.f, chosen = 0.f;
  for (int j = 0; j < top; ++j) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int e = lane; e < E; e += 32) {
      const float v = logit[e];
      if (v > best) { best = v; bi = e; }      // ascending e: the lowest index wins a tie within a lane
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (j == 0) first = best;
    const float p = expf(best - first);         // the first choice is the largest: exponents are <= 0
    denom += p;
    if (lane == 0 && (correction || sigmoid)) {
      const float sv = score[bi < E ? bi : 0];
      top_idx[(size_t)t * top + j] = bi < E ? bi : 0;
      top_w[(size_t)t * top + j] = sigmoid ? sv : sv * w_scale;
      chosen += sv;
      if (bi < E) logit[bi] = -INFINITY;
    } else if (lane == 0) {
      top_idx[(size_t)t * top + j] = bi < E ? bi : 0;          // (not-a-number logits: still an expert that exists)
      top_w[(size_t)t * top + j] = p;
      if (bi < E) logit[bi] = -INFINITY;
    }
    __syncwarp();
  }
  if (sigmoid) {
    chosen = __shfl_sync(0xffffffffu, chosen, 0);
    for (int j = lane; j < top; j += 32) top_w[(size_t)t * top + j] = top_w[(size_t)t * top + j] / (chosen + 1e-20f) * w_scale;
    return;
  }
  if (correction) return;
  for (int j = lane; j < top; j += 32) top_w[(size_t)t * top + j] /= denom;
}

// logits_ws: room for T * (E + 1) floats, or null.  With it, the logits are formed in a launch of their own: for steps of up to
// 256 tokens over (tokens x groups of eight rows) CTAs, for longer ones a CTA per eight tokens; the
// result is the same whichever kernel forms them (same sums, same order).
// Whether moe_logits_rows_kernel forms the logits (where types and alignment let it): not of few rows over many tokens of short rows, whose time
// is the inputs' way to shared memory (us with moe_logits_tokens_kernel and with rows: 2,048 tokens of 512, 33 rows 14.0 and 15.2, 65 rows 18.0
// and 17.2, 33 rows of 1,024 entries 17.3 and 18.1, of 2,048 faster; 1,024 tokens of 512, 33 rows 9.7 and 8.2; 300 tokens, 9 rows of 512
// 6.6 and 6.9, of 1,024 7.8 and 7.6).
extern "C" int qv_moe_route_rows(int T, int rows, int d) { return T <= 1024 ? rows > 16 || d >= 1024 : rows > 40 || d >= 2048; }

extern "C" int qv_moe_route(int* top_idx, float* top_w, float* gate_out, const void* h, int ld_h, const void* wr, const void* wg,
                            float* logits_ws, int T, int d, int E, int top, int dt, int w_dt, const float* correction, float w_scale,
                            int sigmoid, int groups, int keep, void* stream) {
  if (T <= 0) return 0;
  if (E <= 0 || top <= 0 || top > E || E > 8192) return QV_ERR_UNSUPPORTED;
  if (groups < 1 || keep < 1 || keep > groups || E % groups || top > keep * (E / groups) || (groups > 1 && !sigmoid)) return QV_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t smem = (size_t)(E + d + (correction || sigmoid ? E : 0) + (keep < groups ? groups : 0)) * sizeof(float);
  if (smem > 48 * 1024) return QV_ERR_TOO_LARGE;
  const bool split = logits_ws && T <= 256;
  // more tokens: the logits by groups of tokens, where the group's rows fit shared memory
  const size_t tsmem = (size_t)ROUTE_TOKENS * d * (dt == QV_DT_BF16 ? 2 : 4);
  const bool tokens = logits_ws && !split && d % 4 == 0 && (size_t)ROUTE_TOKENS * d * sizeof(float) <= 160 * 1024;
  const dim3 lgrid(T, (E + (wg ? 1 : 0) + ROUTE_WARPS - 1) / ROUTE_WARPS);
  const dim3 tgrid((T + ROUTE_TOKENS - 1) / ROUTE_TOKENS);
  const bool rows16 = tokens && qv_moe_route_rows(T, E + (wg ? 1 : 0), d) && dt == QV_DT_BF16 && w_dt == QV_DT_BF16 && d % 8 == 0 && ld_h % 8 == 0 &&
                      (((uintptr_t)h | (uintptr_t)wr | (uintptr_t)wg) & 15) == 0;
  if (rows16) {
    const int rows = route_rows(E + (wg ? 1 : 0));
    auto kernel = rows == 4 ? moe_logits_rows_kernel<4> : rows == 5 ? moe_logits_rows_kernel<5> : rows == 8 ? moe_logits_rows_kernel<8>
                                                                                                             : moe_logits_rows_kernel<9>;
    if (tsmem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem);
    const int rc = qv_launch(kernel, tgrid, dim3(ROUTE_WARPS * 32), tsmem, st, logits_ws, (const bf16*)h, ld_h, (const bf16*)wr, (const bf16*)wg, d, E, T);
    if (rc) return rc;
  }
#define ROUTE(TT, TW)                                                                                                        \
  do {                                                                                                                       \
    if (rows16) {                                                                                                            \
    } else if (split) {                                                                                                             \
      const int rc = qv_launch(moe_logits_kernel<TT, TW>, lgrid, dim3(ROUTE_WARPS * 32), (size_t)d * sizeof(float), st, logits_ws, \
                               (const TT*)h, ld_h, (const TW*)wr, (const TW*)wg, d, E);                                      \
      if (rc) return rc;                                                                                                     \
    } else if (tokens) {                                                                                                     \
      if (tsmem > 48 * 1024)                                                                                                 \
        cudaFuncSetAttribute(moe_logits_tokens_kernel<TT, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsmem);     \
      const int rc = qv_launch(moe_logits_tokens_kernel<TT, TW>, tgrid, dim3(ROUTE_WARPS * 32), tsmem, st, logits_ws,        \
                               (const TT*)h, ld_h, (const TW*)wr, (const TW*)wg, d, E, T);                                   \
      if (rc) return rc;                                                                                                     \
    }                                                                                                                        \
    return qv_launch(moe_route_kernel<TT, TW>, dim3(T), dim3(ROUTE_WARPS * 32), smem, st, top_idx, top_w, gate_out, (const TT*)h, \
                     ld_h, (const TW*)wr, (const TW*)wg, d, E, top,                                                          \
                     (split || tokens) ? (const float*)logits_ws : (const float*)nullptr, correction, w_scale, sigmoid, groups, keep); \
  } while (0)
  if (dt == QV_DT_F32 && w_dt == QV_DT_F32) ROUTE(float, float);
  if (dt == QV_DT_BF16 && w_dt == QV_DT_BF16) ROUTE(bf16, bf16);
  if (dt == QV_DT_BF16 && w_dt == QV_DT_F32) ROUTE(bf16, float);
  if (dt == QV_DT_F32 && w_dt == QV_DT_BF16) ROUTE(float, bf16);
#undef ROUTE
  return QV_ERR_UNSUPPORTED;
}

// top_idx[t][j] = table[ids[t]][j] (an entry outside 0..E-1, which a sound table has not, reads as expert 0), top_w = 1/top.
__global__ void moe_route_table_kernel(int* __restrict__ top_idx, float* __restrict__ top_w, const int* __restrict__ table,
                                       const int* __restrict__ ids, int n, int top, int vocab, int E) {
  pdl_wait();
  pdl_launch_dependents();
  const float w = 1.0f / (float)top;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int t = i / top, j = i - t * top;
    int id = ids[t];
    if (id < 0 || id >= vocab) id = 0;
    const int e = table[(size_t)id * top + j];
    top_idx[i] = (e >= 0 && e < E) ? e : 0;
    top_w[i] = w;
  }
}

extern "C" int qv_moe_route_table(int* top_idx, float* top_w, const int* table, const int* ids, int T, int top, int vocab, int E,
                                  void* stream) {
  if (T <= 0) return 0;
  if (top <= 0 || E <= 0 || top > E) return QV_ERR_UNSUPPORTED;
  const int n = T * top;
  const int blocks = (n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8;
  return qv_launch(moe_route_table_kernel, dim3(blocks), dim3(256), 0, (cudaStream_t)stream, top_idx, top_w, table, ids, n, top, vocab, E);
}

// One block.  tiles: [max_tiles][3] = (expert or -1, first sorted row, rows).  Its time is that of a few trips to memory and through
// shared memory: the first GROUP_KEEP choices of a thread and their ranks stay in registers, experts' offsets and tiles come from a scan
// by all threads (25 us for 12,288 choices when one thread walked over the experts and wrote the tiles).
#define GROUP_KEEP 12
__global__ void __launch_bounds__(1024) moe_group_kernel(int* __restrict__ row_token, int* __restrict__ slot_row, int* __restrict__ tiles,
                                                         int max_tiles, const int* __restrict__ top_idx, int* __restrict__ rank_tmp,
                                                         int R, int top, int E, int bm) {
  extern __shared__ int cnt[];               // E counts, then E offsets
  __shared__ int part_rows[32], part_tiles[32], total_tiles;
  pdl_wait();
  pdl_launch_dependents();
  int* off = cnt + E;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < E; e += 1024) cnt[e] = 0;
  __syncthreads();
  int mine[GROUP_KEEP], rank[GROUP_KEEP];
#pragma unroll
  for (int i = 0; i < GROUP_KEEP; ++i) {
    const int r = threadIdx.x + i * 1024;
    mine[i] = r < R ? top_idx[r] : E;
  }
#pragma unroll
  for (int i = 0; i < GROUP_KEEP; ++i) rank[i] = mine[i] < E ? atomicAdd(&cnt[mine[i]], 1) : 0;
  for (int r = threadIdx.x + GROUP_KEEP * 1024; r < R; r += 1024)
    if (top_idx[r] < E) rank_tmp[r] = atomicAdd(&cnt[top_idx[r]], 1);
  __syncthreads();
  int row_base = 0, tile_base = 0;           // of the experts ahead of this round of 1024
  for (int e0 = 0; e0 < E; e0 += 1024) {
    const int e = e0 + threadIdx.x;
    const int n = e < E ? cnt[e] : 0, nt = (n + bm - 1) / bm;
    int rows = n, nts = nt;                  // inclusive sums over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, rows, o), b = __shfl_up_sync(0xffffffffu, nts, o);
      if (lane >= o) { rows += a; nts += b; }
    }
    if (lane == 31) { part_rows[warp] = rows; part_tiles[warp] = nts; }
    __syncthreads();
    int rows_before = row_base, tiles_before = tile_base, rows_all = 0, tiles_all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) { rows_before += part_rows[w]; tiles_before += part_tiles[w]; }
      rows_all += part_rows[w];
      tiles_all += part_tiles[w];
    }
    if (e < E) {
      const int first = rows_before + rows - n;
      off[e] = first;
      int at = tiles_before + nts - nt;
      for (int r0 = 0; r0 < n && at < max_tiles; r0 += bm, ++at) {
        tiles[3 * at] = e;
        tiles[3 * at + 1] = first + r0;
        tiles[3 * at + 2] = n - r0 < bm ? n - r0 : bm;
      }
    }
    row_base += rows_all;
    tile_base += tiles_all;
    if (threadIdx.x == 0) total_tiles = tile_base;
    __syncthreads();
  }
  for (int n = total_tiles + threadIdx.x; n < max_tiles; n += 1024) { tiles[3 * n] = -1; tiles[3 * n + 1] = 0; tiles[3 * n + 2] = 0; }
#pragma unroll
  for (int i = 0; i < GROUP_KEEP; ++i) {
    const int r = threadIdx.x + i * 1024;
    if (r >= R) break;
    if (mine[i] >= E) { slot_row[r] = -1; continue; }          // an identity expert
    const int pos = off[mine[i]] + rank[i];
    slot_row[r] = pos;
    row_token[pos] = r / top;
  }
  for (int r = threadIdx.x + GROUP_KEEP * 1024; r < R; r += 1024) {
    if (top_idx[r] >= E) { slot_row[r] = -1; continue; }
    const int pos = off[top_idx[r]] + rank_tmp[r];
    slot_row[r] = pos;
    row_token[pos] = r / top;
  }
}

#define MOE_BM 32
#define MOE_BN 64
#define MOE_BK 16

// Rows of a tile of grouped rows.  Tensor cores: a tile is the narrow operand of one accumulator and every tile of an expert reads the
// expert's matrices once, so a tile should hold all rows of a usual expert; the shared memory that its room takes is taken from the
// stages in flight.  R rows over E experts (0: not known): for steps of up to MOE_DIRECT tokens the first of 32, 64 that holds them all
// (there the tokens themselves are the operand), else the first of 64, 128, 256 that holds 4/3 of the mean (counts scatter around it).
// us a layer with rows gathered and with the tokens themselves, 32 experts of 704 x 1,024: 33 tokens 98 and 94, 64 tokens 98 and 94; 64 of
// 1,408 x 2,048: 33 tokens 210 and 206, 64 tokens 219 and 218, but 100 tokens, inputs not in L2, 223 and 229: there the operand is as many
// bytes of a stage as the weights.
#define MOE_DIRECT 64
extern "C" int qv_moe_tile_rows(int tensor_cores, int tokens, int R, int E) {
  if (!tensor_cores) return MOE_BM;
  if (tokens <= 0 || E <= 0) return 64;
  if (tokens <= MOE_DIRECT) return tokens <= 32 ? 32 : 64;
  const long long want = (4LL * R + 3LL * E - 1) / (3LL * E);
  return want <= 64 ? 64 : want <= 128 ? 128 : 256;
}

extern "C" int qv_moe_max_tiles(int R, int E, int bm) {
  const int a = (R + bm - 1) / bm + E;
  return a < R ? a : R;
}

extern "C" int qv_moe_group(int* row_token, int* slot_row, int* tiles, const int* top_idx, int* rank_tmp, int T, int top, int E,
                            int bm, void* stream) {
  if (T <= 0) return 0;
  if (E > 8192 || bm <= 0) return QV_ERR_UNSUPPORTED;
  const int R = T * top;
  if (E > 4096) cudaFuncSetAttribute(moe_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * 2 * (int)sizeof(int));
  return qv_launch(moe_group_kernel, dim3(1), dim3(1024), (size_t)2 * E * sizeof(int), (cudaStream_t)stream, row_token, slot_row, tiles,
                   qv_moe_max_tiles(R, E, bm), top_idx, rank_tmp, R, top, E, bm);
}

// Tile of 32 rows x 64 columns, 256 threads, each 2 rows x 4 columns; k in steps of 16, ascending.
// MODE 1 (gated up): a = h (rows gathered by row_token), w1/w2 = gate/up matrices [E][N][K]; out act [R, N] in the compute type.
// MODE 2 (ungated up): as 1 with w1 the up matrices alone and the square of relu as activation.
// MODE 0 (down): a = act [R, K]; w1 = down matrices [E][N][K]; out y [R, N] float32.
template <typename T, typename TW, int MODE>
__global__ void __launch_bounds__(256) moe_experts_kernel(void* __restrict__ out_, int ld_out, const T* __restrict__ a, int ld_a,
                                                          const TW* __restrict__ w1, const TW* __restrict__ w2,
                                                          const int* __restrict__ row_token, const int* __restrict__ tiles, int N, int K,
                                                          GluAct glu) {
  constexpr bool GATHER = MODE != 0;         // rows of a are gathered, the output is in the compute type
  constexpr bool UP = MODE == 1;             // a second matrix (the gate's partner)
  __shared__ float As[MOE_BK][MOE_BM + 1];
  __shared__ float B1[MOE_BK][MOE_BN + 1];
  __shared__ float B2[UP ? MOE_BK : 1][MOE_BN + 1];
  pdl_wait();
  pdl_launch_dependents();
  const int e = tiles[3 * blockIdx.y];
  if (e < 0) return;
  const int row0 = tiles[3 * blockIdx.y + 1], rows = tiles[3 * blockIdx.y + 2];
  const int n0 = blockIdx.x * MOE_BN;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const TW* W1 = w1 + (size_t)e * N * K;
  const TW* W2 = UP ? w2 + (size_t)e * N * K : nullptr;
  float acc1[2][4] = {}, acc2[2][4] = {};
  // loaders: A tile 32 x 16 (2 elements a thread), B tiles 64 x 16 (4 elements a thread)
  const int ar = threadIdx.x >> 3, ak = (threadIdx.x & 7) * 2;
  size_t a_row = 0;
  const bool a_ok = ar < rows;
  if (a_ok) a_row = GATHER ? (size_t)row_token[row0 + ar] : (size_t)(row0 + ar);
  const int bn = threadIdx.x >> 2, bk = (threadIdx.x & 3) * 4;
  for (int k0 = 0; k0 < K; k0 += MOE_BK) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = k0 + ak + i;
      As[ak + i][ar] = (a_ok && k < K) ? to_f(a[a_row * ld_a + k]) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + bk + i, n = n0 + bn;
      const bool ok = n < N && k < K;
      B1[bk + i][bn] = ok ? to_f(W1[(size_t)n * K + k]) : 0.f;
      if (UP) B2[bk + i][bn] = ok ? to_f(W2[(size_t)n * K + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MOE_BK; ++k) {
      const float a0 = As[k][ty * 2], a1 = As[k][ty * 2 + 1];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float b = B1[k][tx * 4 + c];
        acc1[0][c] = fmaf(a0, b, acc1[0][c]);
        acc1[1][c] = fmaf(a1, b, acc1[1][c]);
        if (UP) {
          const float b2 = B2[k][tx * 4 + c];
          acc2[0][c] = fmaf(a0, b2, acc2[0][c]);
          acc2[1][c] = fmaf(a1, b2, acc2[1][c]);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = ty * 2 + r;
    if (row >= rows) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int n = n0 + tx * 4 + c;
      if (n >= N) continue;
      if (UP) {
        ((T*)out_)[(size_t)(row0 + row) * ld_out + n] = from_f<T>(glu_apply(acc1[r][c], acc2[r][c], glu));
      } else if (MODE == 2) {
        const float g = fmaxf(acc1[r][c], 0.f);
        ((T*)out_)[(size_t)(row0 + row) * ld_out + n] = from_f<T>(g * g);
      } else {
        ((float*)out_)[(size_t)(row0 + row) * ld_out + n] = acc1[r][c];
      }
    }
  }
}

extern "C" int qv_moe_experts(int up, void* out, int ld_out, const void* a, int ld_a, const void* w1, const void* w2,
                              const int* row_token, const int* tiles, int R, int E, int N, int K, int dt, int w_dt, int act, float limit,
                              float slope, void* stream) {
  if (R <= 0) return 0;
  if (act < 0 || act > 2) return QV_ERR_UNSUPPORTED;
  const GluAct glu = {act, limit, slope};
  const int max_tiles = qv_moe_max_tiles(R, E, MOE_BM);
  if (max_tiles > 65535) return QV_ERR_TOO_LARGE;
  dim3 grid((N + MOE_BN - 1) / MOE_BN, max_tiles);
  cudaStream_t st = (cudaStream_t)stream;
#define EXPERTS(TT, TW)                                                                                                        \
  do {                                                                                                                         \
    if (up == 1) return qv_launch(moe_experts_kernel<TT, TW, 1>, grid, dim3(256), 0, st, out, ld_out, (const TT*)a, ld_a, (const TW*)w1, \
                                  (const TW*)w2, row_token, tiles, N, K, glu);                                                 \
    if (up == 2) return qv_launch(moe_experts_kernel<TT, TW, 2>, grid, dim3(256), 0, st, out, ld_out, (const TT*)a, ld_a, (const TW*)w1, \
                                  (const TW*)w2, row_token, tiles, N, K, glu);                                                 \
    return qv_launch(moe_experts_kernel<TT, TW, 0>, grid, dim3(256), 0, st, out, ld_out, (const TT*)a, ld_a, (const TW*)w1,      \
                     (const TW*)w2, row_token, tiles, N, K, glu);                                                              \
  } while (0)
  if (dt == QV_DT_F32 && w_dt == QV_DT_F32) EXPERTS(float, float);
  if (dt == QV_DT_BF16 && w_dt == QV_DT_BF16) EXPERTS(bf16, bf16);
  if (dt == QV_DT_BF16 && w_dt == QV_DT_F32) EXPERTS(bf16, float);
  if (dt == QV_DT_F32 && w_dt == QV_DT_BF16) EXPERTS(float, bf16);
#undef EXPERTS
  return QV_ERR_UNSUPPORTED;
}

// ---------------------------------------------------------------- the experts' products on the tensor cores (bfloat16)
// Weights are the 128-row operand of tcgen05.mma, a tile's grouped rows (or, for steps of up to MOE_DIRECT tokens, all tokens) the narrow one,
// so an expert's matrices are read once per tile of rows whatever the number of rows, and rows are padded to 16 only.  One CTA per SM
// walks over (tile, block of features) items, features fastest: the CTAs at work share a tile's rows in L2 and stream different weights.
//   warp 0      weights by contiguous bulk copies (packed tiles), rows by TMA in boxes of 32 rows x 64 k, through a ring of STAGES
//   warp 1      tcgen05.mma, accumulators double-buffered in tensor memory
//   warps 2..5  epilogue of the item before: activation, stores (a thread holds a feature, columns are rows)
// Gated up product: the 128 rows are 16 gate rows and the 16 up rows of the same features in turn, so a warp holds both halves.
// What bounds it: the matrices' bytes (few rows an expert) or what an SM takes in from L2 (16 KB of weights and the rows' tile a k
// block).
struct ExpertsArgs {
  void* out;
  const uint8_t* w1;
  const uint8_t* w2;
  const int* row_token;
  const int* tiles;
  int* err;
  int max_tiles, N, K, ld_out;
  int tokens;                                // > 0: the rows of the narrow operand are the tokens, and row_token says which a row is
  GluAct glu;
};

__device__ __forceinline__ uint32_t tmem_ld1(uint32_t taddr) {
  uint32_t r;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr));
  return r;
}

template <int MODE, int RT, int STAGES>
__global__ void __launch_bounds__(192) moe_experts_tc_kernel(const __grid_constant__ CUtensorMap map_a, const ExpertsArgs p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int W_BYTES = BM * BK * 2;               // 128 weight rows x 64 k
  constexpr int STAGE_BYTES = W_BYTES + RT * BK * 2;
  constexpr int TMEM_COLS = 2 * RT;
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(ring + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;               // [2]
  uint64_t* acc_empty = acc_full + 2;                // [2]
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 128); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();                                        // the tile table, the rows and the output belong to the kernels ahead until here
  const int NT = (p.N + 63) / 64, KT = (p.K + BK - 1) / BK;
  const int blocks = MODE == 1 ? NT : (NT + 1) / 2;  // items of a tile: 64 features of two matrices, or 128 of one
  const int items = p.max_tiles * blocks;

  if (warp == 0) {
    const bool leader = elect_one();
    int it = 0;
    bool ok = true;
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      const int t = item / blocks, fb = item - t * blocks;
      const int e = p.tiles[3 * t];
      if (e < 0) break;
      const int row0 = p.tokens ? 0 : p.tiles[3 * t + 1], rows = p.tokens ? p.tokens : p.tiles[3 * t + 2];
      const int boxes = (rows + 31) / 32;
      const int halves = MODE == 1 ? 2 : (2 * fb + 1 < NT ? 2 : 1);        // 8 KB weight tiles a stage
      const uint8_t* w1 = p.w1 + ((size_t)e * NT + (MODE == 1 ? fb : 2 * fb)) * KT * 8192;
      const uint8_t* w2 = MODE == 1 ? p.w2 + ((size_t)e * NT + fb) * KT * 8192 : w1 + (size_t)KT * 8192;
      for (int kb = 0; kb < KT; ++kb, ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1, p.err, 31)) { ok = false; break; }
        if (leader) {
          uint8_t* dst = ring + s * STAGE_BYTES;
          mbar_expect_tx(&full[s], halves * 8192 + boxes * 4096);
          const uint8_t* s1 = w1 + (size_t)kb * 8192;
          const uint8_t* s2 = w2 + (size_t)kb * 8192;
          if (MODE == 1) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {            // 16 gate rows, then the 16 up rows of the same features
              bulk_load_1d(dst + q * 4096, s1 + q * 2048, &full[s], 2048);
              bulk_load_1d(dst + q * 4096 + 2048, s2 + q * 2048, &full[s], 2048);
            }
          } else {
            bulk_load_1d(dst, s1, &full[s], 8192);
            if (halves == 2) bulk_load_1d(dst + 8192, s2, &full[s], 8192);
          }
          for (int x = 0; x < boxes; ++x) tma_load_2d(dst + W_BYTES + x * 4096, &map_a, &full[s], kb * BK, row0 + 32 * x);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    int it = 0, local = 0;
    bool ok = true;
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x, ++local) {
      const int t = item / blocks;
      if (p.tiles[3 * t] < 0) break;
      const int rows = p.tokens ? p.tokens : p.tiles[3 * t + 2];
      const uint32_t idesc = umma_idesc(BM, (rows + 15) & ~15);
      const int b = local & 1;
      ok = mbar_wait(&acc_empty[b], ((local >> 1) & 1) ^ 1, p.err, 34);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + (uint32_t)(b * RT);
      for (int kb = 0; kb < KT; ++kb, ++it) {
        const int s = it % STAGES;
        ok = mbar_wait(&full[s], (it / STAGES) & 1, p.err, 32);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(ring + s * STAGE_BYTES);
        const uint64_t da = umma_desc(a_addr), db = umma_desc(a_addr + W_BYTES);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) umma_f16(d_tmem, da + 2 * kk, db + 2 * kk, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          umma_commit(&empty[s]);
        }
        __syncwarp();
      }
      if (leader) umma_commit(&acc_full[b]);
      __syncwarp();
    }
  } else {
    const int q = warp & 3;
    int local = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x, ++local) {
      const int t = item / blocks, fb = item - t * blocks;
      if (p.tiles[3 * t] < 0) break;
      const int row0 = p.tiles[3 * t + 1], rows = p.tiles[3 * t + 2];
      const int b = local & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[b], (local >> 1) & 1, p.err, 33))) break;     // (the MMA warp then gives up too)
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * RT);
      const int feat = MODE == 1 ? fb * 64 + q * 16 + (lane & 15) : fb * 128 + q * 32 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < rows; c0 += 16) {
        uint32_t r[16];
        if (p.tokens) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            int col = p.row_token[row0 + (c0 + j < rows ? c0 + j : 0)];
            if ((unsigned)col >= (unsigned)p.tokens) col = 0;
            r[j] = tmem_ld1(taddr + col);
          }
          tmem_wait_ld();
        } else {
          tmem_ld16(taddr + c0, r);
          tmem_wait_ld();
        }
        if (MODE == 1) {
          // a lane of the lower half gives its gate value of the odd row for the up value of the even row
          const int up = lane >> 4;
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float give = __uint_as_float(up ? r[j] : r[j + 1]);
            const float got = __shfl_xor_sync(0xffffffffu, give, 16);
            const float g = up ? got : __uint_as_float(r[j]), u = up ? __uint_as_float(r[j + 1]) : got;
            const int row = c0 + j + up;
            if (row < rows && feat < p.N)
              ((bf16*)p.out)[(size_t)(row0 + row) * p.ld_out + feat] = __float2bfloat16_rn(glu_apply(g, u, p.glu));
          }
        } else if (feat < p.N) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (c0 + j >= rows) break;
            const float v = __uint_as_float(r[j]);
            const size_t at = (size_t)(row0 + c0 + j) * p.ld_out + feat;
            if (MODE == 2) ((bf16*)p.out)[at] = __float2bfloat16_rn(fmaxf(v, 0.f) * fmaxf(v, 0.f));
            else ((float*)p.out)[at] = v;
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[b]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// out[r] = a[row_token[r]]: the rows in grouped order, for the boxes above (16-byte pieces; rows beyond the last choice copy any row).
__global__ void __launch_bounds__(256) moe_gather_kernel(uint4* __restrict__ out, const uint4* __restrict__ a, int ld16, int pieces,
                                                         const int* __restrict__ row_token, int R, int T) {
  pdl_wait();
  pdl_launch_dependents();
  for (int r = blockIdx.x; r < R; r += gridDim.x) {
    int t = row_token[r];
    if ((unsigned)t >= (unsigned)T) t = 0;
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) out[(size_t)r * pieces + i] = a[(size_t)t * ld16 + i];
  }
}

static int moe_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0, v = 0;
    n = (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0) ? v : 148;
  }
  return n;
}

template <int MODE, int RT, int STAGES>
static int moe_experts_launch(const CUtensorMap& map, const ExpertsArgs& p, cudaStream_t st) {
  constexpr int smem = STAGES * (BM * BK * 2 + RT * BK * 2) + 1024 + 256;
  auto kernel = moe_experts_tc_kernel<MODE, RT, STAGES>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int NT = (p.N + 63) / 64;
  const long long items = (long long)p.max_tiles * (MODE == 1 ? NT : (NT + 1) / 2);
  if (items > 0x40000000LL) return QV_ERR_TOO_LARGE;
  return qv_launch(kernel, dim3((unsigned)(items < moe_sms() ? items : moe_sms())), dim3(192), (size_t)smem, st, map, p);
}

// w [E][N][K] -> the packed tiles (see qv_moe_experts_tc), zero where a matrix ends.  K a multiple of 8, w on 16 bytes.
__global__ void __launch_bounds__(256) moe_pack_kernel(uint4* __restrict__ out, const bf16* __restrict__ w, int N, int K, int NT, int KT) {
  pdl_wait();
  pdl_launch_dependents();
  const size_t tile = ((size_t)blockIdx.z * NT + blockIdx.y) * KT + blockIdx.x;
  const bf16* src = w + (size_t)blockIdx.z * N * K;
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const int r = i >> 3, c = i & 7, n = blockIdx.y * 64 + r, k = blockIdx.x * 64 + c * 8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (n < N && k < K) v = *(const uint4*)(src + (size_t)n * K + k);
    out[tile * 512 + r * 8 + (c ^ (r & 7))] = v;
  }
}

extern "C" int qv_moe_pack_experts(void* out, const void* w, int E, int N, int K, void* stream) {
  if (E <= 0 || N <= 0 || K < 8 || (K & 7) || (((uintptr_t)out | (uintptr_t)w) & 15)) return QV_ERR_UNSUPPORTED;
  const int NT = (N + 63) / 64, KT = (K + 63) / 64;
  if (E > 65535 || NT > 65535) return QV_ERR_TOO_LARGE;
  return qv_launch(moe_pack_kernel, dim3(KT, NT, E), dim3(256), 0, (cudaStream_t)stream, (uint4*)out, (const bf16*)w, N, K, NT, KT);
}

// As qv_moe_experts for bfloat16 operands, on the tensor cores, with the experts' matrices packed in tiles of 64 x 64
// ([E][ceil(N/64)][ceil(K/64)][64][64], zero-padded, the eight 16-byte chunks of row r at chunk ^ (r % 8): the image the product
// reads from shared memory).  tile_rows: what the tile table was made for (32, 64, 128 or 256).  a_rows: the rows of `a`.
// gathered: room for R rows of K elements, for up products of more tokens than MOE_DIRECT or a tile's rows.  Refuses rows of `a` that do not start on 16 bytes.
extern "C" int qv_moe_experts_tc(int up, void* out, int ld_out, const void* a, int ld_a, int a_rows, const void* w1, const void* w2,
                                 const int* row_token, const int* tiles, int R, int E, int N, int K, int act, float limit, float slope,
                                 int tile_rows, void* gathered, int* err, void* stream) {
  if (R <= 0) return 0;
  if (act < 0 || act > 2 || up < 0 || up > 2 || N <= 0 || K < 8 || (K & 7)) return QV_ERR_UNSUPPORTED;
  if ((ld_a & 7) || (((uintptr_t)a | (uintptr_t)w1 | (uintptr_t)w2) & 15)) return QV_ERR_UNSUPPORTED;
  const bool direct = up && a_rows <= MOE_DIRECT && a_rows <= tile_rows;
  cudaStream_t st = (cudaStream_t)stream;
  ExpertsArgs p;
  p.out = out; p.w1 = (const uint8_t*)w1; p.w2 = (const uint8_t*)w2; p.row_token = row_token; p.tiles = tiles; p.err = err;
  p.max_tiles = qv_moe_max_tiles(R, E, tile_rows); p.N = N; p.K = K; p.ld_out = ld_out; p.tokens = direct ? a_rows : 0;
  p.glu = {act, limit, slope};
  CUtensorMap map;
  if (up && !direct) {
    if (!gathered || ((uintptr_t)gathered & 15)) return QV_ERR_UNSUPPORTED;
    const int pieces = K / 8;
    const int rc = qv_launch(moe_gather_kernel, dim3(R < 148 * 16 ? R : 148 * 16), dim3(pieces >= 256 ? 256 : pieces >= 128 ? 128 : 64), 0, st,
                             (uint4*)gathered, (const uint4*)a, ld_a / 8, pieces, row_token, R, a_rows);
    if (rc) return rc;
    if (!make_map(&map, gathered, R, K, K, 32)) return QV_ERR_UNSUPPORTED;
  } else if (!make_map(&map, a, direct ? a_rows : R, K, ld_a, 32)) {
    return QV_ERR_UNSUPPORTED;
  }
#define EXPERTS_TC(RT, ST)                                                                    \
  do {                                                                                        \
    if (up == 1) return moe_experts_launch<1, RT, ST>(map, p, st);                            \
    if (up == 2) return moe_experts_launch<2, RT, ST>(map, p, st);                            \
    return moe_experts_launch<0, RT, ST>(map, p, st);                                         \
  } while (0)
  if (tile_rows == 32) EXPERTS_TC(32, 10);
  if (tile_rows == 64) EXPERTS_TC(64, 8);
  if (tile_rows == 128) EXPERTS_TC(128, 6);
  if (tile_rows == 256) EXPERTS_TC(256, 4);
#undef EXPERTS_TC
  return QV_ERR_UNSUPPORTED;
}

// delta [T, d] float32.  mix, shared, h (the tokens' inputs, read for identity experts): [T, d] in the compute type or null; gate
// [T] float32 or null.  VEC elements a thread: 4 where all rows allow 16-byte (8-byte) accesses.  It moves the choices' float32 rows
// once; one element a thread kept too few bytes in flight (2,048 tokens x 6 choices x 2,048: 44 us).
template <typename T, int VEC>
__global__ void __launch_bounds__(256) moe_combine_kernel(float* __restrict__ delta, const T* __restrict__ mix, const float* __restrict__ y,
                                                          const int* __restrict__ slot_row, const float* __restrict__ top_w,
                                                          const T* __restrict__ shared, const float* __restrict__ gate, int d, int top,
                                                          const float* __restrict__ s_mix, const float* __restrict__ s_ff,
                                                          const T* __restrict__ h, int ld_h) {
  struct alignas(sizeof(T) * VEC) PackT { T v[VEC]; };
  struct alignas(4 * VEC) PackF { float v[VEC]; };
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const float g = gate ? gate[t] : 1.f;
  for (int i = (blockIdx.y * blockDim.x + threadIdx.x) * VEC; i < d; i += gridDim.y * blockDim.x * VEC) {
    float routed[VEC] = {};
#pragma unroll 4
    for (int j = 0; j < top; ++j) {
      const int r = slot_row[(size_t)t * top + j];
      const float w = top_w[(size_t)t * top + j];
      PackF yv = {};
      if (r >= 0) {
        yv = *(const PackF*)(y + (size_t)r * d + i);
      } else if (h) {
        const PackT hv = *(const PackT*)(h + (size_t)t * ld_h + i);
#pragma unroll
        for (int k = 0; k < VEC; ++k) yv.v[k] = to_f(hv.v[k]);
      }
#pragma unroll
      for (int k = 0; k < VEC; ++k) routed[k] = fmaf(w, yv.v[k], routed[k]);
    }
    PackT sv = {}, mv = {};
    if (shared) sv = *(const PackT*)(shared + (size_t)t * d + i);
    if (mix) mv = *(const PackT*)(mix + (size_t)t * d + i);
    PackF o;
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      float v = routed[k];
      if (shared) v = fmaf(g, to_f(sv.v[k]), v);
      if (s_ff) v *= s_ff[i + k];
      if (mix) v = fmaf(to_f(mv.v[k]), s_mix ? s_mix[i + k] : 1.f, v);
      o.v[k] = v;
    }
    *(PackF*)(delta + (size_t)t * d + i) = o;
  }
}

extern "C" int qv_moe_combine(float* delta, const void* mix, const float* y, const int* slot_row, const float* top_w,
                              const void* shared, const float* gate, int T, int d, int top, int dt, const float* s_mix,
                              const float* s_ff, const void* h, int ld_h, void* stream) {
  if (T <= 0) return 0;
  const bool vec = d % 4 == 0 && ld_h % 4 == 0 && ((((uintptr_t)delta | (uintptr_t)y | (uintptr_t)mix | (uintptr_t)shared | (uintptr_t)h) & 15) == 0);
  const int per = vec ? 1024 : 256;
  const dim3 grid(T, T < 256 ? (d + per - 1) / per : 1);
#define COMBINE(TT, V)                                                                                                                \
  return qv_launch(moe_combine_kernel<TT, V>, grid, dim3(256), 0, (cudaStream_t)stream, delta, (const TT*)mix, y, slot_row, top_w,    \
                   (const TT*)shared, gate, d, top, s_mix, s_ff, (const TT*)h, ld_h)
  QV_DISPATCH_DT(dt, TT, if (vec) COMBINE(TT, 4); COMBINE(TT, 1));
#undef COMBINE
  return QV_ERR_UNSUPPORTED;
}
