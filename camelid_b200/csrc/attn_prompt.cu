// Reference-order attention for long steps of one sequence (prompts): a CTA serves R neighbouring rows x the G query heads of
// one KV head, M = R * G queries, so that a key or value is read, widened to f32 and brought to shared memory once for all of
// them.  The same f32 operations in the same order as the other reference-order kernels (attention_context_for_head,
// src/inference.rs:30287-30466):
//   score_p = (sum over d, in order, of q_d * k_pd) * scale;  e_p = expf(score_p - max);  sum = e_0 + e_1 + ... in position
//   order;  w_p = e_p * (1 / sum);  out_d = ((0 + w_0 * v_0d) + w_1 * v_1d) + ...
// Both products are outer-product tiles, every output a chain of its own: scores 128 positions x M queries with the head
// dimension running, outputs HD dimensions x M queries with the positions running; a thread holds W x A of them (W = 8 or 4
// positions or dimensions) and multiplies and adds two at a time.  Bound by the FP32 units (a multiplication and an addition per term); keys and
// values travel through registers into two buffers of 16 terms, one barrier per 16.
// attn_rows_kernel, one CTA per row, reads a key from shared memory for every head and row and widens it each time.
// Per layer and step of 512 rows: 8B width, prompt of 1024 tokens 503 -> 249 us (the FP32 units' share is 119 us), 1B width,
// 1500 tokens 381 -> 254 us, 8B width from position 1500 on 2160 -> 1180 us, from 3500 on 5180 -> 3510 us.
#include "common.cuh"
#include "expf_exact.cuh"
#include "packed_f32.cuh"

namespace cmld {

namespace {

constexpr int kPromptTile = 128;  // positions per tile of scores
constexpr int kPromptK = 16;      // terms per buffer

__host__ __device__ constexpr int prompt_pitch(int a) { return 8 * a + (a & 1 ? 1 : 2); }  // floats between positions (or dimensions) of the queries' values

template <int A>
__device__ __forceinline__ void prompt_queries(const float *x, uint64_t (&xx)[A]) {
  if (A == 2) {
    const float2 v = *reinterpret_cast<const float2 *>(x);
    xx[0] = both(v.x);
    xx[A - 1] = both(v.y);
  } else {
#pragma unroll
    for (int c = 0; c < A; ++c) xx[c] = both(x[c]);
  }
}

template <int G, int HD, int A, int W>
__global__ void __launch_bounds__(1024 / W) attn_prompt_kernel(AttnArgs a, float neg_zero) {
  constexpr int M = 8 * A, R = M / G, PITCH = prompt_pitch(A), T = 1024 / W, PAIRS = W / 2;
  constexpr int OPAIRS = W == 8 ? HD / 32 : 2;  // pairs of dimensions of a thread's outputs
  extern __shared__ __align__(16) float prompt_smem[];
  float *buf = prompt_smem;                        // [2][kPromptK][128]
  float *q_s = buf + 2 * kPromptK * kPromptTile;   // [HD][PITCH]
  float *sc = q_s + HD * PITCH;                    // [positions][PITCH]
  __shared__ float s_max[8 / W][M], s_inv[M];
  __shared__ int s_rows[R];  // context length of each row
  const int kvh = blockIdx.x, tid = threadIdx.x, rg = (tid >> 1) & 15;
  // neighbouring lanes share positions and differ in their queries: a 16-byte load whose lanes pair up so takes half the time.
  // A thread's positions (dimensions): r0 .. r0 + 3 and, W = 8, 64 + the same; W = 4: warps 4..7 take the upper 64
  const int half = tid >> 7, ag = ((tid >> 4) & 6) | (tid & 1), r0 = 64 * half + 4 * rg;
  const int b0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * R;  // the longest contexts start first
  const int slot = a.slots[b0];
  const __half *kbase = a.k_cache + ((int64_t)slot * a.n_kv_heads + kvh) * a.max_pos * HD;
  const __half *vbase = a.v_cache + ((int64_t)slot * a.n_kv_heads + kvh) * a.max_pos * HD;
  if (tid < R) s_rows[tid] = a.positions[min(b0 + tid, a.batch - 1)] + 1;
  for (int i = tid; i < M * HD; i += T) {
    const int m = i / HD, d = i % HD, row = min(b0 + m / G, a.batch - 1);
    q_s[d * PITCH + m] = a.q[(int64_t)row * a.q_stride + ((int64_t)kvh * G + m % G) * HD + d];
  }
  __syncthreads();
  int n_min = s_rows[0], n_max = s_rows[0];
#pragma unroll
  for (int r = 1; r < R; ++r) n_min = min(n_min, s_rows[r]), n_max = max(n_max, s_rows[r]);
  int len[A];  // context lengths of this thread's queries
#pragma unroll
  for (int c = 0; c < A; ++c) len[c] = s_rows[(ag * A + c) / G];
  const uint64_t nz = both(neg_zero);

  // ---- scores
  constexpr int KCH = HD / kPromptK;
  const int steps = (n_max + kPromptTile - 1) / kPromptTile * KCH;
  constexpr int KW = kPromptK * kPromptTile / T / 8;  // 16-byte pieces of a key per thread
  uint4 raw[KW];
  const int kp = tid & 127, kd = (tid >> 7) * (8 * KW);
  auto load_k = [&](int s) {  // this thread's position and dimensions of a buffer
    const int p = min(s / KCH * kPromptTile + kp, n_max - 1);
    const uint4 *src = reinterpret_cast<const uint4 *>(kbase + (int64_t)p * HD + s % KCH * kPromptK + kd);
#pragma unroll
    for (int j = 0; j < KW; ++j) raw[j] = __ldg(src + j);
  };
  auto store_k = [&](int s) {
    float *dst = buf + (s & 1) * (kPromptK * kPromptTile) + kd * kPromptTile + kp;
#pragma unroll
    for (int j = 0; j < KW; ++j) {
      const uint32_t w[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        dst[(8 * j + 2 * i) * kPromptTile] = f.x;
        dst[(8 * j + 2 * i + 1) * kPromptTile] = f.y;
      }
    }
  };
  float mx[A];
#pragma unroll
  for (int c = 0; c < A; ++c) mx[c] = -INFINITY;
  uint64_t acc[A][PAIRS];
  load_k(0);
  store_k(0);
  __syncthreads();
  for (int s = 0; s < steps; ++s) {
    if (s + 1 < steps) load_k(s + 1);
    if (s % KCH == 0)
#pragma unroll
      for (int c = 0; c < A; ++c)
#pragma unroll
        for (int p = 0; p < PAIRS; ++p) acc[c][p] = 0;
    const float *w = buf + (s & 1) * (kPromptK * kPromptTile) + r0, *x = q_s + s % KCH * kPromptK * PITCH + ag * A;
#pragma unroll 8
    for (int k = 0; k < kPromptK; ++k) {
      uint64_t v[PAIRS], xx[A];
#pragma unroll
      for (int p = 0; p < PAIRS; p += 2) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(w + k * kPromptTile + 32 * p);
        v[p] = t.x;
        v[p + 1] = t.y;
      }
      prompt_queries<A>(x + k * PITCH, xx);
#pragma unroll
      for (int c = 0; c < A; ++c)
#pragma unroll
        for (int p = 0; p < PAIRS; ++p) acc[c][p] = add2(acc[c][p], mul2(xx[c], v[p], nz));
    }
    if (s % KCH == KCH - 1) {
      const int p0 = s / KCH * kPromptTile + r0;
#pragma unroll
      for (int i = 0; i < W; ++i) {
        const int p = p0 + 64 * (i >> 2) + (i & 3);
#pragma unroll
        for (int c = 0; c < A; ++c) {
          const float2 v = halves(acc[c][i >> 1]);
          const float f = __fmul_rn(i & 1 ? v.y : v.x, a.scale);
          if (p < n_max) sc[(int64_t)p * PITCH + ag * A + c] = f;
          if (p < len[c]) mx[c] = fmaxf(mx[c], f);
        }
      }
    }
    if (s + 1 < steps) store_k(s + 1);  // into the buffer that every thread left before the barrier below
    __syncthreads();
  }
  // ---- maxima, exponentials, sums in position order, weights
#pragma unroll
  for (int c = 0; c < A; ++c) {
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
    if (rg == 0) s_max[half][ag * A + c] = mx[c];
  }
  const int v_steps = (n_max + kPromptK - 1) / kPromptK;
  constexpr int VPIECES = kPromptK * HD / 8, VLOADS = (VPIECES + T - 1) / T;  // 16-byte pieces of a buffer's values
  uint4 vr[VLOADS];
  auto load_v = [&](int s) {
#pragma unroll
    for (int j = 0; j < VLOADS; ++j) {
      const int i = min(tid + j * T, VPIECES - 1), p = min(s * kPromptK + i / (HD / 8), n_max - 1);
      vr[j] = __ldg(reinterpret_cast<const uint4 *>(vbase + (int64_t)p * HD) + i % (HD / 8));
    }
  };
  auto store_v = [&](int s) {
    float *dst = buf + (s & 1) * (kPromptK * kPromptTile);
#pragma unroll
    for (int j = 0; j < VLOADS; ++j) {
      const int i = tid + j * T;
      if (i >= VPIECES) break;
      const uint32_t w[4] = {vr[j].x, vr[j].y, vr[j].z, vr[j].w};
      float2 f[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) f[t] = __half22float2(*reinterpret_cast<const __half2 *>(&w[t]));
      float4 *o = reinterpret_cast<float4 *>(dst + i * 8);  // [position][HD]
      o[0] = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
      o[1] = make_float4(f[2].x, f[2].y, f[3].x, f[3].y);
    }
  };
  load_v(0);
  __syncthreads();
  // thread: query m, every PS-th position, four at a time (the latencies of one hide behind the others)
  constexpr int PS = T / M;
  const int m = tid % M, own = tid < PS * M ? s_rows[m / G] : 0;
  if (W == 4 && tid < M) s_max[0][tid] = fmaxf(s_max[0][tid], s_max[8 / W - 1][tid]);
  if (W == 4) __syncthreads();
  const float top = s_max[0][m];
  for (int p = tid / M; p < own; p += 4 * PS) {
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = sc[(int64_t)min(p + j * PS, own - 1) * PITCH + m];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = expf_exact_flat(__fsub_rn(e[j], top));
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (p + j * PS < own) sc[(int64_t)(p + j * PS) * PITCH + m] = e[j];
  }
  store_v(0);
  __syncthreads();
  if (tid < M) {
    const int n = s_rows[tid / G];
    const float *e = sc + tid;
    float sum = 0.0f, v[8];
    if (n >= 8)
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = e[j * PITCH];
    int p = 0;
    for (; p + 8 <= n; p += 8) {
      float next[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) next[j] = e[(int64_t)min(p + 8 + j, n - 1) * PITCH];
#pragma unroll
      for (int j = 0; j < 8; ++j) sum = __fadd_rn(sum, v[j]);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = next[j];
    }
    for (; p < n; ++p) sum = __fadd_rn(sum, e[(int64_t)p * PITCH]);
    s_inv[tid] = __fdiv_rn(1.0f, sum);
  }
  __syncthreads();
  const float inv = s_inv[m];
  for (int p = tid / M; p < own; p += 4 * PS) {
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = sc[(int64_t)min(p + j * PS, own - 1) * PITCH + m];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (p + j * PS < own) sc[(int64_t)(p + j * PS) * PITCH + m] = __fmul_rn(e[j], inv);
  }
  __syncthreads();
  // ---- weighted values: dimensions r0 .. r0 + 3 (and 64 + the same) of A queries per thread
  const bool active = r0 < HD;
  uint64_t out[A][OPAIRS];
#pragma unroll
  for (int c = 0; c < A; ++c)
#pragma unroll
    for (int p = 0; p < OPAIRS; ++p) out[c][p] = 0;
  for (int s = 0; s < v_steps; ++s) {
    if (s + 1 < v_steps) load_v(s + 1);
    const float *w = buf + (s & 1) * (kPromptK * kPromptTile) + r0, *x = sc + (int64_t)s * kPromptK * PITCH + ag * A;
    if (!active) {
    } else if ((s + 1) * kPromptK <= n_min) {
#pragma unroll 8
      for (int k = 0; k < kPromptK; ++k) {
        uint64_t v[OPAIRS], xx[A];
#pragma unroll
        for (int p = 0; p < OPAIRS; p += 2) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(w + k * HD + 32 * p);
          v[p] = t.x;
          v[p + 1] = t.y;
        }
        prompt_queries<A>(x + k * PITCH, xx);
#pragma unroll
        for (int c = 0; c < A; ++c)
#pragma unroll
          for (int p = 0; p < OPAIRS; ++p) out[c][p] = add2(out[c][p], mul2(xx[c], v[p], nz));
      }
    } else {  // the last positions: a row adds only what lies in its context
      const int cnt = min(kPromptK, n_max - s * kPromptK);
      for (int k = 0; k < cnt; ++k) {
        uint64_t xx[A];
        prompt_queries<A>(x + k * PITCH, xx);
#pragma unroll
        for (int c = 0; c < A; ++c)
          if (s * kPromptK + k < len[c])
#pragma unroll
            for (int p = 0; p < OPAIRS; ++p)
              out[c][p] = add2(out[c][p], mul2(xx[c], *reinterpret_cast<const uint64_t *>(w + k * HD + 64 * (p >> 1) + 2 * (p & 1)), nz));
      }
    }
    if (s + 1 < v_steps) store_v(s + 1);
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < A; ++c) {
    const int q = ag * A + c, row = b0 + q / G;
    if (!active || row >= a.batch) continue;
    float *o = a.out + (int64_t)row * a.q_stride + ((int64_t)kvh * G + q % G) * HD + r0;
#pragma unroll
    for (int p = 0; p < OPAIRS; p += 2) {
      const float2 lo = halves(out[c][p]), hi = halves(out[c][p + 1]);
      *reinterpret_cast<float4 *>(o + 32 * p) = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
  }
}

size_t prompt_smem_bytes(int HD, int A, int64_t n_pos) { return 4 * (size_t)(2 * kPromptK * kPromptTile + (HD + n_pos) * prompt_pitch(A)); }
constexpr size_t kPromptTwo = 112 * 1024, kPromptOne = 220 * 1024;  // shared memory of which two CTAs, or one, fit an SM

template <int G, int HD, int A, int W>
int32_t launch_prompt(const AttnArgs &a, int64_t n_pos, cudaStream_t s) {
  constexpr int R = 8 * A / G;
  const size_t smem = prompt_smem_bytes(HD, A, n_pos);
  static SmemLimit limit;
  CMLD_TRY(allow_smem(limit, attn_prompt_kernel<G, HD, A, W>, smem));
  dim3 grid((unsigned)a.n_kv_heads, (unsigned)((a.batch + R - 1) / R));
  attn_prompt_kernel<G, HD, A, W><<<grid, 1024 / W, smem, s>>>(a, -0.0f);
  CMLD_CUDA(cudaGetLastError());
  return CMLD_OK;
}

// Eight threads side by side cover 8 * A queries, a multiple of G.  Contexts whose scores would leave room for one CTA per SM
// only take half the queries, or (G = 3) twice the threads and half the outputs per thread.
template <int G, int HD>
int32_t launch_prompt(const AttnArgs &a, int64_t n_pos, cudaStream_t s) {
  if constexpr (G == 3) {
    return prompt_smem_bytes(HD, 3, n_pos) > kPromptTwo ? launch_prompt<G, HD, 3, 4>(a, n_pos, s) : launch_prompt<G, HD, 3, 8>(a, n_pos, s);
  } else {
    return prompt_smem_bytes(HD, 2, n_pos) > kPromptTwo ? launch_prompt<G, HD, 1, 8>(a, n_pos, s) : launch_prompt<G, HD, 2, 8>(a, n_pos, s);
  }
}

}  // namespace

// n_pos: bound on positions[b] + 1 of every row; every row of the step belongs to one slot.
bool attention_prompt_fits(int n_heads, int n_kv_heads, int head_dim, int batch, int64_t n_pos, int sms) {
  if (n_kv_heads < 1 || n_heads % n_kv_heads) return false;
  const int G = n_heads / n_kv_heads;
  if (!(G == 1 || G == 2 || G == 3 || G == 4 || G == 8) || !(head_dim == 64 || head_dim == 128)) return false;
  // a CTA for every SM, or the row kernel's many small ones are faster (8B width: 36 rows at 700 positions 73 us against about
  // 50, 128 rows at 200 positions 47 us against 100)
  const int R = 8 * (G == 3 ? 3 : 2) / G;
  return (batch + R - 1) / R * n_kv_heads >= sms && n_pos > 0 && prompt_smem_bytes(head_dim, G == 3 ? 3 : 1, n_pos) <= kPromptOne;
}

int32_t launch_attention_prompt(const AttnArgs &a, int64_t n_pos, int sms, cudaStream_t s) {
  if (!attention_prompt_fits(a.n_heads, a.n_kv_heads, a.head_dim, a.batch, n_pos, sms)) return CMLD_ERR_UNSUPPORTED;
  if (a.tree_mask || a.fuse_rope) return fail(CMLD_ERR_INVALID, "attention (prompt): tree masks and fused RoPE are not supported here");
#define CMLD_PROMPT(GG) \
  case GG: return a.head_dim == 128 ? launch_prompt<GG, 128>(a, n_pos, s) : launch_prompt<GG, 64>(a, n_pos, s);
  switch (a.n_heads / a.n_kv_heads) {
    CMLD_PROMPT(1)
    CMLD_PROMPT(2)
    CMLD_PROMPT(3)
    CMLD_PROMPT(4)
    CMLD_PROMPT(8)
  }
#undef CMLD_PROMPT
  return CMLD_ERR_UNSUPPORTED;
}

}  // namespace cmld
