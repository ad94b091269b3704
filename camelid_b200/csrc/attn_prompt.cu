// Reference-order attention for long steps of one sequence (prompts).  The same f32 operations in the same order as the other
// reference-order kernels (attention_context_for_head, src/inference.rs:30287-30466):
//   score_p = (sum over d, in order, of q_d * k_pd) * scale;  e_p = expf(score_p - max);  sum = e_0 + e_1 + ... in position
//   order;  w_p = e_p * (1 / sum);  out_d = ((0 + w_0 * v_0d) + w_1 * v_1d) + ...
// A block of 64 queries is R neighbouring rows x the G query heads of a KV head.  Three kernels, the scores between them in memory
// (a scratch of the engine's, most of it still in L2 when it is read):
//   prompt_scores_kernel   64 queries x 128 positions per CTA, the head dimension running; a thread holds 8 x 8 scores
//   prompt_weights_kernel  a CTA per block: maxima, exponentials in place, each query's sum by one thread in position order
//   prompt_values_kernel   64 queries x 64 dimensions per CTA, the positions running; a thread holds 8 x 4 outputs
// Both products are outer-product tiles, every output a chain of its own, multiplied and added two at a time; they are bound by the
// FP32 units (a multiplication and an addition per term, and 64 or 32 of them per three or four loads from shared memory).
// One kernel that kept a block's scores in shared memory instead (16 queries, two CTAs of four warps per SM) left the FP32 units idle
// for half of the time.  Us of attention, that | this: 1024 tokens of the 8B width, 4 layers, 1992 | 1454 (scores 702, weights 163, values
// 589; the FP32 units' share of the products is 956); 1500 tokens of the 1B width 3040 | 2007; 333 tokens of the 3B width from
// position 700 on 1097 | 785.  What is left: the last CTAs of the scores (a CTA takes 26 us), the widening of keys and values.
#include "common.cuh"
#include "expf_exact.cuh"
#include "packed_f32.cuh"

namespace cmld {

namespace {

constexpr int kQ = 64;        // queries of a block
constexpr int kTileP = 128;   // positions of a tile of scores
constexpr int kStepP = 32;    // positions of a buffer of weights and values
constexpr int kStepD = 32;    // dimensions of a buffer of keys
constexpr int kThreads = 128;

struct PromptArgs {
  AttnArgs a;
  float *scores;     // [block][n_alloc][kQ]: scores, then exponentials
  float *tile_max;   // [block][n_alloc / 32][kQ]
  float *inv;        // [block][kQ]
  int64_t n_alloc;   // positions, a multiple of kTileP
  int32_t group, rows, first, blocks;  // query heads per KV head; rows of a block; this launch's blocks of rows
  float neg_zero;
};

// The rows of a block: the longest contexts start first.
struct Rows {
  int b0, kvh, block;
  __device__ __forceinline__ Rows(const PromptArgs &p, int y, int z) {
    const int rb = p.blocks - 1 - y;
    b0 = (p.first + rb) * p.rows;
    kvh = z;
    block = rb * p.a.n_kv_heads + z;
  }
  // context length of query m; 0: no such query
  __device__ __forceinline__ int length(const PromptArgs &p, int m) const {
    const int r = m / p.group, b = b0 + r;
    return r < p.rows && b < p.a.batch ? p.a.positions[b] + 1 : 0;
  }
  __device__ __forceinline__ int last_length(const PromptArgs &p) const { return p.a.positions[min(b0 + p.rows, p.a.batch) - 1] + 1; }
};

template <int HD>
__global__ void __launch_bounds__(kThreads) prompt_scores_kernel(const __grid_constant__ PromptArgs p) {
  extern __shared__ __align__(16) float scores_smem[];
  float *qs = scores_smem, *ks = qs + HD * kQ;  // [HD][kQ], [2][kStepD][kTileP]
  const Rows R(p, blockIdx.y, blockIdx.z);
  const int n_max = R.last_length(p), p0 = blockIdx.x * kTileP, tid = threadIdx.x, lane = tid & 31;
  if (p0 >= n_max) return;
  const AttnArgs &a = p.a;
  const uint4 *src = reinterpret_cast<const uint4 *>(a.k_cache + (((int64_t)a.slots[R.b0] * a.n_kv_heads + R.kvh) * a.max_pos + min(p0 + tid, n_max - 1)) * HD);
  uint4 raw[kStepD / 8];
  auto load = [&](int s) {  // this thread's position
#pragma unroll
    for (int j = 0; j < kStepD / 8; ++j) raw[j] = __ldg(src + s * (kStepD / 8) + j);
  };
  auto store = [&](int s) {
    float *dst = ks + (s & 1) * (kStepD * kTileP) + tid;
#pragma unroll
    for (int j = 0; j < kStepD / 8; ++j) {
      const uint32_t w[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        dst[(8 * j + 2 * i) * kTileP] = f.x;
        dst[(8 * j + 2 * i + 1) * kTileP] = f.y;
      }
    }
  };
  load(0);
  {
    const int m = tid & (kQ - 1), row = min(R.b0 + min(m / p.group, p.rows - 1), a.batch - 1);
    const float4 *q = reinterpret_cast<const float4 *>(a.q + (int64_t)row * a.q_stride + ((int64_t)R.kvh * p.group + m % p.group) * HD);
#pragma unroll 4
    for (int j = tid / kQ; j < HD / 4; j += kThreads / kQ) {
      const float4 v = q[j];
      qs[(4 * j) * kQ + m] = v.x, qs[(4 * j + 1) * kQ + m] = v.y, qs[(4 * j + 2) * kQ + m] = v.z, qs[(4 * j + 3) * kQ + m] = v.w;
    }
  }
  store(0);
  __syncthreads();
  // A warp has all queries and 32 positions (which, differs from CTA to CTA: the last tile's upper warps have nothing to do).
  // Neighbouring lanes share positions, next but one queries: a 16-byte load whose lanes pair up so takes half the time.
  const int pq = ((tid >> 5) + blockIdx.x + blockIdx.y) & 3, qg = (lane & 1) | ((lane >> 1) & 6), pg = ((lane >> 1) & 1) | ((lane >> 3) & 2);
  const int r0 = 32 * pq + 4 * pg;
  const bool any = p0 + 32 * pq < n_max;
  const uint64_t nz = both(p.neg_zero);
  uint64_t acc[8][4];  // [position r0 + i, r0 + 16 + i][pair of queries 4 qg, 4 qg + 2, 32 + the same]
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0;
#pragma unroll 1
  for (int s = 0; s < HD / kStepD; ++s) {
    if (s + 1 < HD / kStepD) load(s + 1);
    const float *qp = qs + s * (kStepD * kQ) + 4 * qg, *kp = ks + (s & 1) * (kStepD * kTileP) + r0;
    if (any) {
#pragma unroll 4
      for (int d = 0; d < kStepD; ++d) {
        const ulonglong2 q0 = *reinterpret_cast<const ulonglong2 *>(qp + d * kQ), q1 = *reinterpret_cast<const ulonglong2 *>(qp + d * kQ + 32);
        const float4 k0 = *reinterpret_cast<const float4 *>(kp + d * kTileP), k1 = *reinterpret_cast<const float4 *>(kp + d * kTileP + 16);
        const float kv[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
        const uint64_t q[4] = {q0.x, q0.y, q1.x, q1.y};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint64_t k = both(kv[i]);
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][c] = add2(acc[i][c], mul2(q[c], k, nz));
        }
      }
    }
    if (s + 1 < HD / kStepD) store(s + 1);  // into the buffer that every thread left before the barrier below
    __syncthreads();
  }
  if (!any) return;
  float mx[8];
  int len[8];
#pragma unroll
  for (int x = 0; x < 8; ++x) mx[x] = -INFINITY, len[x] = R.length(p, 4 * qg + 32 * (x >> 2) + (x & 3));
  float *out = p.scores + ((int64_t)R.block * p.n_alloc + p0) * kQ + 4 * qg;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + 16 * (i >> 2) + (i & 3);
    float f[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 v = halves(acc[i][c]);
      f[2 * c] = __fmul_rn(v.x, a.scale);
      f[2 * c + 1] = __fmul_rn(v.y, a.scale);
    }
#pragma unroll
    for (int x = 0; x < 8; ++x)
      if (p0 + r < len[x]) mx[x] = fmaxf(mx[x], f[x]);
    *reinterpret_cast<float4 *>(out + (int64_t)r * kQ) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4 *>(out + (int64_t)r * kQ + 32) = make_float4(f[4], f[5], f[6], f[7]);
  }
#pragma unroll
  for (int x = 0; x < 8; ++x) {
    mx[x] = fmaxf(mx[x], __shfl_xor_sync(0xffffffffu, mx[x], 2));
    mx[x] = fmaxf(mx[x], __shfl_xor_sync(0xffffffffu, mx[x], 16));
  }
  if (pg == 0) {
    float *t = p.tile_max + ((int64_t)R.block * (p.n_alloc / 32) + p0 / 32 + pq) * kQ + 4 * qg;
    *reinterpret_cast<float4 *>(t) = make_float4(mx[0], mx[1], mx[2], mx[3]);
    *reinterpret_cast<float4 *>(t + 32) = make_float4(mx[4], mx[5], mx[6], mx[7]);
  }
}

constexpr int kWeightThreads = 256, kWeightP = 64, kWeightN = kWeightP * kQ / kWeightThreads;

__global__ void __launch_bounds__(kWeightThreads) prompt_weights_kernel(const __grid_constant__ PromptArgs p) {
  __shared__ float e_s[2][kWeightP][kQ];
  __shared__ float s_max[kWeightThreads / kQ][kQ];
  constexpr int PARTS = kWeightThreads / kQ;
  const Rows R(p, blockIdx.y, blockIdx.x);
  const int n_max = R.last_length(p), tid = threadIdx.x, q = tid & (kQ - 1), part = tid / kQ, len = R.length(p, q);
  const float *t = p.tile_max + (int64_t)R.block * (p.n_alloc / 32) * kQ + q;
  float mx = -INFINITY;
  for (int i = part; i < (n_max + 31) / 32; i += PARTS) mx = fmaxf(mx, t[(int64_t)i * kQ]);
  s_max[part][q] = mx;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PARTS; ++i) mx = fmaxf(mx, s_max[i][q]);
  float *s = p.scores + (int64_t)R.block * p.n_alloc * kQ + q;
  float sum = 0.0f, v[kWeightN];
  // (positions beyond a query's context, up to n_alloc, hold some value; nothing of them is kept)
#pragma unroll
  for (int j = 0; j < kWeightN; ++j) v[j] = s[(int64_t)(part + PARTS * j) * kQ];
  for (int t0 = 0, buf = 0; t0 < n_max; t0 += kWeightP, buf ^= 1) {
#pragma unroll
    for (int j = 0; j < kWeightN; ++j) {
      const int r = part + PARTS * j;
      const float e = expf_exact_flat(__fsub_rn(v[j], mx));
      e_s[buf][r][q] = e;
      if (t0 + r < len) s[(int64_t)(t0 + r) * kQ] = e;
    }
    if (t0 + kWeightP < n_max)
#pragma unroll
      for (int j = 0; j < kWeightN; ++j) v[j] = s[(int64_t)(t0 + kWeightP + part + PARTS * j) * kQ];
    __syncthreads();
    if (part == 0) {
      const float *e = &e_s[buf][0][q];
      const int n = min(kWeightP, len - t0);
      if (n == kWeightP) {
#pragma unroll
        for (int i = 0; i < kWeightP; ++i) sum = __fadd_rn(sum, e[i * kQ]);
      } else {
        for (int i = 0; i < n; ++i) sum = __fadd_rn(sum, e[i * kQ]);
      }
    }
  }
  if (part == 0) p.inv[R.block * kQ + q] = __fdiv_rn(1.0f, sum);
}

template <int HD>
__global__ void __launch_bounds__(kThreads) prompt_values_kernel(const __grid_constant__ PromptArgs p) {
  __shared__ __align__(16) float ws[2][kStepP][kQ], vs[2][kStepP][64];
  const Rows R(p, blockIdx.y, blockIdx.x / (HD / 64));
  const int tid = threadIdx.x, lane = tid & 31, d0 = blockIdx.x % (HD / 64) * 64;
  const AttnArgs &a = p.a;
  const int n_max = R.last_length(p), n_min = a.positions[R.b0] + 1;
  const __half *vbase = a.v_cache + ((int64_t)a.slots[R.b0] * a.n_kv_heads + R.kvh) * a.max_pos * HD + d0;
  const float *wbase = p.scores + (int64_t)R.block * p.n_alloc * kQ + 4 * (tid & 15);
  const float4 inv = *reinterpret_cast<const float4 *>(p.inv + R.block * kQ + 4 * (tid & 15));
  uint4 vr[2];
  float4 wr[4];
  auto load = [&](int s) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
      vr[j] = __ldg(reinterpret_cast<const uint4 *>(vbase + (int64_t)min(s * kStepP + 16 * j + (tid >> 3), n_max - 1) * HD) + (tid & 7));
#pragma unroll
    for (int j = 0; j < 4; ++j) wr[j] = *reinterpret_cast<const float4 *>(wbase + (int64_t)(s * kStepP + 8 * j + (tid >> 4)) * kQ);
  };
  auto store = [&](int b) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t w[4] = {vr[j].x, vr[j].y, vr[j].z, vr[j].w};
      float2 f[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) f[i] = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
      float4 *o = reinterpret_cast<float4 *>(&vs[b][16 * j + (tid >> 3)][8 * (tid & 7)]);
      o[0] = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
      o[1] = make_float4(f[2].x, f[2].y, f[3].x, f[3].y);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4 *>(&ws[b][8 * j + (tid >> 4)][4 * (tid & 15)]) =
          make_float4(__fmul_rn(wr[j].x, inv.x), __fmul_rn(wr[j].y, inv.y), __fmul_rn(wr[j].z, inv.z), __fmul_rn(wr[j].w, inv.w));
  };
  // lanes paired as in the scores: neighbours share dimensions, next but one queries
  const int qg = (lane & 1) | ((lane >> 1) & 6), dg = 4 * (tid >> 5) + (((lane >> 1) & 1) | ((lane >> 3) & 2));
  const uint64_t nz = both(p.neg_zero);
  uint64_t acc[4][4];  // [dimension 4 dg + i][pair of queries 4 qg, 4 qg + 2, 32 + the same]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0;
  const int steps = (n_max + kStepP - 1) / kStepP;
  load(0);
  store(0);
  __syncthreads();
  for (int s = 0; s < steps; ++s) {
    if (s + 1 < steps) load(s + 1);
    const float *w = &ws[s & 1][0][4 * qg], *v = &vs[s & 1][0][4 * dg];
    if ((s + 1) * kStepP <= n_min) {
#pragma unroll 4
      for (int k = 0; k < kStepP; ++k) {
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2 *>(w + k * kQ), w1 = *reinterpret_cast<const ulonglong2 *>(w + k * kQ + 32);
        const float4 vv = *reinterpret_cast<const float4 *>(v + k * 64);
        const float vd[4] = {vv.x, vv.y, vv.z, vv.w};
        const uint64_t q[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t x = both(vd[i]);
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[i][c] = add2(acc[i][c], mul2(q[c], x, nz));
        }
      }
    } else {  // the last positions: a query adds only what lies in its context
      int len[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) len[x] = R.length(p, 4 * qg + 32 * (x >> 2) + (x & 3)) - s * kStepP;
      const int cnt = min(kStepP, n_max - s * kStepP);
      for (int k = 0; k < cnt; ++k) {
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2 *>(w + k * kQ), w1 = *reinterpret_cast<const ulonglong2 *>(w + k * kQ + 32);
        const float4 vv = *reinterpret_cast<const float4 *>(v + k * 64);
        const float vd[4] = {vv.x, vv.y, vv.z, vv.w};
        const uint64_t q[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t x = both(vd[i]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float2 o = halves(acc[i][c]), n = halves(add2(acc[i][c], mul2(q[c], x, nz)));
            acc[i][c] = pair(k < len[2 * c] ? n.x : o.x, k < len[2 * c + 1] ? n.y : o.y);
          }
        }
      }
    }
    if (s + 1 < steps) store((s + 1) & 1);  // into the buffer that every thread left before the barrier below
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float2 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = halves(acc[i][c]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int m = 4 * qg + 32 * (c >> 1) + 2 * (c & 1) + h;
      if (R.length(p, m) == 0) continue;
      float *o = a.out + (int64_t)(R.b0 + m / p.group) * a.q_stride + ((int64_t)R.kvh * p.group + m % p.group) * HD + d0 + 4 * dg;
      *reinterpret_cast<float4 *>(o) = h ? make_float4(v[0].y, v[1].y, v[2].y, v[3].y) : make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
    }
  }
}

int64_t padded(int64_t n_pos) { return (n_pos + kTileP - 1) / kTileP * kTileP; }
// floats of scratch for a block of rows: scores, maxima and inverse sums of every KV head's 64 queries
int64_t block_floats(int n_kv_heads, int64_t n_pos) { return n_kv_heads * (padded(n_pos) * kQ + padded(n_pos) / 32 * kQ + kQ); }

template <int HD>
int32_t launch_prompt(PromptArgs &p, int64_t n_pos, int64_t scratch_floats, cudaStream_t s, int64_t *launches) {
  const int kv = p.a.n_kv_heads, all = (p.a.batch + p.rows - 1) / p.rows;
  const int per = (int)std::min<int64_t>(all, scratch_floats / block_floats(kv, n_pos));
  const size_t smem = (size_t)(HD * kQ + 2 * kStepD * kTileP) * 4;
  static SmemLimit limit;
  CMLD_TRY(allow_smem(limit, prompt_scores_kernel<HD>, smem, true));
  float *scratch = p.scores;
  for (p.first = 0; p.first < all; p.first += per) {
    p.blocks = std::min(per, all - p.first);
    p.tile_max = scratch + (int64_t)p.blocks * kv * p.n_alloc * kQ;
    p.inv = p.tile_max + (int64_t)p.blocks * kv * (p.n_alloc / 32) * kQ;
    prompt_scores_kernel<HD><<<dim3((unsigned)(p.n_alloc / kTileP), (unsigned)p.blocks, (unsigned)kv), kThreads, smem, s>>>(p);
    prompt_weights_kernel<<<dim3((unsigned)kv, (unsigned)p.blocks), kWeightThreads, 0, s>>>(p);
    prompt_values_kernel<HD><<<dim3((unsigned)kv * (HD / 64), (unsigned)p.blocks), kThreads, 0, s>>>(p);
    CMLD_CUDA(cudaGetLastError());
    if (launches) *launches += 3;
  }
  return CMLD_OK;
}

}  // namespace

// Scratch of an engine whose prompt steps have up to `rows` rows and whose contexts up to `max_pos` positions: a whole step's, at most
// half a GB (longer contexts then go by groups of rows).
int64_t attention_prompt_scratch_floats(int n_heads, int n_kv_heads, int head_dim, int rows, int64_t max_pos) {
  if (n_kv_heads < 1 || n_heads % n_kv_heads || n_heads / n_kv_heads > kQ || !(head_dim == 64 || head_dim == 128)) return 0;
  const int R = kQ / (n_heads / n_kv_heads);
  return std::min<int64_t>((int64_t)1 << 27, (rows + R - 1) / R * block_floats(n_kv_heads, max_pos));
}

// n_pos: bound on positions[b] + 1 of every row; the rows of the step are neighbours in one slot.
bool attention_prompt_fits(int n_heads, int n_kv_heads, int head_dim, int batch, int64_t n_pos, int sms, int64_t scratch_floats) {
  if (n_kv_heads < 1 || n_heads % n_kv_heads || !(head_dim == 64 || head_dim == 128) || n_pos < 1) return false;
  const int G = n_heads / n_kv_heads;
  if (G > kQ) return false;
  const int R = kQ / G, all = (batch + R - 1) / R;
  const int per_block = n_kv_heads * (head_dim / 64), wanted = std::min(all, (sms + per_block - 1) / per_block);
  // Half a machine of CTAs: a CTA walks its positions alone, where the row kernel's many small CTAs share the machine.  Us per layer, row
  // kernel | here: 8B width, 128 rows at 200 positions 74 | 62, 64 at 200 38 | 46, 36 at 700 53 | 78, 64 at 2000 325 | 205; 1B width, 100 rows at
  // 200 35 | 47, 200 at 700 170 | 110; 3B width, 100 at 200 52 | 48, 40 at 200 26 | 42.
  if (scratch_floats < wanted * block_floats(n_kv_heads, n_pos)) return false;
  const int64_t ctas = (int64_t)all * per_block;
  if (ctas * 2 >= sms) return true;
  // Down to a quarter at long contexts, where the row kernel is not done in few rounds of the machine: per 1000 positions a round takes it 41, 35
  // and 25 us at the 8B, 3B and 1B widths (10 us and 0.06 per query head of a group and dimension), a CTA here 83 us, and 50 to 70 more
  // whatever the context.  Two layers, us, row kernel | here, rows from position p on: 8B 36 from 2000 937 | 1054, 33 from 6000 1586 | 1718, 40 from 1000
  // 888 | 899; 1B 72 from 2000 731 | 796, 80 from 1000 616 | 637, 96 from 1000 662 | 647; 3B 48 from 2000 799 | 839, 56 from 1000 686 | 676.
  const double rounds = (double)(((int64_t)batch * n_kv_heads + sms - 1) / sms);
  return ctas * 4 >= sms && n_pos >= 1024 && (double)n_pos * (rounds * (10.0 + 0.06 * G * head_dim) - 83.0) > 50000.0;
}

int32_t launch_attention_prompt(const AttnArgs &a, int64_t n_pos, int sms, float *scratch, int64_t scratch_floats, cudaStream_t s, int64_t *launches) {
  if (!attention_prompt_fits(a.n_heads, a.n_kv_heads, a.head_dim, a.batch, n_pos, sms, scratch_floats)) return CMLD_ERR_UNSUPPORTED;
  if (a.tree_mask || a.fuse_rope) return fail(CMLD_ERR_INVALID, "attention (prompt): tree masks and fused RoPE are not supported here");
  PromptArgs p{};
  p.a = a;
  p.scores = scratch;
  p.n_alloc = padded(n_pos);
  p.group = a.n_heads / a.n_kv_heads;
  p.rows = kQ / p.group;
  p.neg_zero = -0.0f;
  return a.head_dim == 128 ? launch_prompt<128>(p, n_pos, scratch_floats, s, launches) : launch_prompt<64>(p, n_pos, scratch_floats, s, launches);
}

}  // namespace cmld
