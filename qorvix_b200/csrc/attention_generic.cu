// Causal grouped-query attention over the paged cache, one warp per (token, query head).
// It serves every kind of step (a prompt portion, a single decoded token, any mix) with
// the same arithmetic, in float32 whatever the storage type, and takes any head size.
// It is the attention of the true 32-bit path and the reference for the tensor-core kernels.
//
// Formula (reference: runtime/src/text_model.cpp:83-114; its CUDA twin keeps all scores in
// shared memory and runs the softmax on one thread, cuda/src/cuda_backend.cu:347-395):
//   kv head = h / (H / Hkv);  s_t = (q . K_t) * scale for lo <= t <= pos;
//   p = softmax(s);  out = sum_t p_t V_t          lo = 0, or pos - window + 1 with a window.
//
// Keys are visited in blocks of 32 aligned to absolute positions (0-31, 32-63, ...), with a
// running maximum and sum, so the result for a position depends on that position and the
// cache contents only: not on how the prompt was cut, nor on the rest of the batch.
#include "common.cuh"

#define MAX_HD 512

// NREG: output entries a lane holds (head sizes up to 32 NREG).  VEC: the heads' rows start on 16 bytes and are whole 16-byte pieces.
// A warp's time is that of its loads, so those of a key's row go out 64 entries at a time, the values of several keys together, and a
// block's first ones ahead of its scores (3 rows of 30 keys of 32 entries: 5.9 us with values of 8 keys behind the scores, 3.4 with 32
// ahead of them); what is added in which order does not change by it.
template <typename T, int NREG, bool VEC>
__global__ void __launch_bounds__(128) attention_generic_kernel(
    T* __restrict__ out, int ld_out, const T* __restrict__ q, int ld_q, const T* __restrict__ cache,
    const int* __restrict__ tok_pos, const int* __restrict__ tok_seg,
    const int* __restrict__ block_table, int max_blocks, int H, int Hkv, int hd, int page, int window,
    float scale) {
  extern __shared__ float qs_all[];              // 4 warps x hd floats
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x * 4 + warp;
  const int t = blockIdx.y;
  pdl_wait();
  pdl_launch_dependents();
  if (h >= H) return;                            // whole warp leaves together
  float* qs = qs_all + (size_t)warp * hd;
  const T* qrow = q + (size_t)t * ld_q + (size_t)h * hd;
  for (int i = lane; i < hd; i += 32) qs[i] = to_f(qrow[i]);
  __syncwarp();

  const int pos = tok_pos[t];
  const int* bt = block_table + (size_t)tok_seg[t] * max_blocks;
  const int kvh = h / (H / Hkv);
  const int lo = window > 0 ? (pos - window + 1 > 0 ? pos - window + 1 : 0) : 0;
  const size_t page_elems = (size_t)2 * Hkv * page * hd;
  const size_t v_off = (size_t)Hkv * page * hd;
  const size_t head_off = (size_t)kvh * page * hd;

  // Of heads above 128 entries two keys' values are all that fits, which does not pay for holding them over the scores (256 entries, float32:
  // 5 % more): they are fetched behind the scores, for the keys whose weight is not zero.
  constexpr bool AHEAD = NREG <= 4;
  constexpr int KEYS = NREG <= 1 ? 32 : NREG <= 2 ? 16 : NREG <= 4 ? 8 : 2;      // keys whose values are fetched together
  float o[NREG];
#pragma unroll
  for (int j = 0; j < NREG; ++j) o[j] = 0.f;
  float m = -INFINITY, l = 0.f;

  for (int kb = (lo >> 5) << 5; kb <= pos; kb += 32) {
    const int tk = kb + lane;
    const bool valid = tk >= lo && tk <= pos;
    size_t base = 0;
    float s = -INFINITY;
    if (valid) base = (size_t)bt[tk / page] * page_elems + head_off + (size_t)(tk % page) * hd;
    const int nk = pos - kb + 1 < 32 ? pos - kb + 1 : 32;
    T v[KEYS][NREG];
    auto values = [&](int j0) {
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        const T* vp = cache + __shfl_sync(0xffffffffu, (unsigned long long)base, (j0 + j) & 31) + v_off;
        const bool live = j0 + j < nk && kb + j0 + j >= lo;
#pragma unroll
        for (int r = 0; r < NREG; ++r) {
          const int i = lane + 32 * r;
          v[j][r] = live && i < hd ? vp[i] : from_f<T>(0.f);
        }
      }
    };
    if constexpr (AHEAD) values(0);
    if (valid) {
      const T* kp = cache + base;
      float dot = 0.f;
      if (VEC) {
        constexpr int PER = 16 / (int)sizeof(T), GO = 64 / PER;     // pieces of 16 bytes
        for (int i0 = 0; i0 < hd; i0 += 64) {
          uint4 kv[GO];
#pragma unroll
          for (int u = 0; u < GO; ++u)
            if (i0 + u * PER < hd) kv[u] = *(const uint4*)(kp + i0 + u * PER);
#pragma unroll
          for (int u = 0; u < GO; ++u) {
            if (i0 + u * PER >= hd) break;
            const T* e = (const T*)&kv[u];
#pragma unroll
            for (int x = 0; x < PER; ++x) dot = fmaf(qs[i0 + u * PER + x], to_f(e[x]), dot);
          }
        }
      } else {
        for (int i = 0; i < hd; ++i) dot = fmaf(qs[i], to_f(kp[i]), dot);
      }
      s = dot * scale;
    }
    const float m_new = fmaxf(m, warp_max(s));   // finite: the block holds at least one valid key
    const float p = valid ? expf(s - m_new) : 0.f;
    const float corr = expf(m - m_new);          // exp(-inf) = 0 for the first block
    l = l * corr + warp_sum(p);
#pragma unroll
    for (int j = 0; j < NREG; ++j) o[j] *= corr;
    for (int j0 = 0; j0 < nk; j0 += KEYS) {
      float pj[KEYS];
      if constexpr (AHEAD) {
        if (j0) values(j0);
      }
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        pj[j] = __shfl_sync(0xffffffffu, p, (j0 + j) & 31);
        if (j0 + j >= nk) pj[j] = 0.f;
        if constexpr (!AHEAD) {
          const T* vp = cache + __shfl_sync(0xffffffffu, (unsigned long long)base, (j0 + j) & 31) + v_off;
#pragma unroll
          for (int r = 0; r < NREG; ++r) {
            const int i = lane + 32 * r;
            v[j][r] = pj[j] != 0.f && i < hd ? vp[i] : from_f<T>(0.f);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < KEYS; ++j) {
        if (pj[j] == 0.f) continue;                  // masked (before the window) or underflowed: adds nothing
#pragma unroll
        for (int r = 0; r < NREG; ++r) o[r] = fmaf(pj[j], to_f(v[j][r]), o[r]);
      }
    }
    m = m_new;
  }
  T* orow = out + (size_t)t * ld_out + (size_t)h * hd;
  const float inv = 1.0f / l;
#pragma unroll
  for (int r = 0; r < NREG; ++r) {
    const int i = lane + 32 * r;
    if (i < hd) orow[i] = from_f<T>(o[r] * inv);
  }
}

extern "C" int qv_attention_generic(void* out, int ld_out, const void* q, int ld_q, const void* cache,
                                    const int* tok_pos, const int* tok_seg, const int* block_table,
                                    int max_blocks, int T, int H, int Hkv, int hd, int page,
                                    int window, float scale, int dt, void* stream) {
  if (T <= 0) return 0;
  if (hd > MAX_HD || hd <= 0 || Hkv <= 0 || H % Hkv) return QV_ERR_UNSUPPORTED;
  if (T > 65535 * 32) return QV_ERR_TOO_LARGE;
  dim3 grid((H + 3) / 4, T);
  if (grid.y > 65535) {
    // split over several launches; rows are independent
    int done = 0;
    while (done < T) {
      const int n = T - done < 65535 ? T - done : 65535;
      const size_t esz = dt == QV_DT_F32 ? 4 : 2;
      int rc = qv_attention_generic((char*)out + (size_t)done * ld_out * esz, ld_out,
                                    (const char*)q + (size_t)done * ld_q * esz, ld_q, cache,
                                    tok_pos + done, tok_seg + done, block_table, max_blocks, n, H, Hkv,
                                    hd, page, window, scale, dt, stream);
      if (rc) return rc;
      done += n;
    }
    return 0;
  }
  const size_t smem = (size_t)4 * hd * sizeof(float);
  const bool vec = hd % (dt == QV_DT_F32 ? 4 : 8) == 0 && ((uintptr_t)cache & 15) == 0;
#define AG_LAUNCH(TT, NR, V)                                                                                                     \
  return qv_launch(attention_generic_kernel<TT, NR, V>, grid, dim3(128), smem, (cudaStream_t)stream, (TT*)out, ld_out, (const TT*)q, ld_q, \
                   (const TT*)cache, tok_pos, tok_seg, block_table, max_blocks, H, Hkv, hd, page, window, scale)
  QV_DISPATCH_DT(dt, TT, {
    if (!vec) AG_LAUNCH(TT, MAX_HD / 32, false);
    if (hd <= 32) AG_LAUNCH(TT, 1, true);
    if (hd <= 64) AG_LAUNCH(TT, 2, true);
    if (hd <= 128) AG_LAUNCH(TT, 4, true);
    AG_LAUNCH(TT, MAX_HD / 32, true);
  });
#undef AG_LAUNCH
  return QV_ERR_UNSUPPORTED;
}
