// Matrix-vector products with bfloat16 weights and 32-bit activations for one or two rows: one pass over the weights.
//
// Bound by HBM.  Persistent grid, one CTA of 16 warps per SM, each with its share of the output rows.  Rows two at a time (they share the
// operand's loads), 256 columns a step; a CTA's steps go to its warps in sixteen equal runs, whatever the number of rows: a row whose steps
// lie in several warps is added up at the end.  (With whole rows per warp 14336 rows were 3.03 rounds, so four.)  A lane copies the weights
// that it uses itself, 16 bytes at a time, into a private ring in shared memory, 64 KB of them in flight all the time; the first are asked
// for before the kernel waits for its predecessor (weights never depend on earlier kernels), then every CTA prepares the operand itself:
// the boundary between sublayers, an RMS norm (with a sigmoid gate, or over groups of columns with a SiLU gate), or a plain copy, with all
// its loads in flight at once.  Two products that do not depend on each other can share a launch: the first `n_first` CTAs work on one.
// One row, one after the other in a graph, before (whole rows per warp, weights in registers, fetched when the last were used up) and now:
// 14336 x 4096 25.4 -> 19.7 us, 4096 x 14336 24.3 -> 20.6, 32000 x 4096 47.1 -> 41.7 (6.3 TB/s), 6144 x 1536 6.7 -> 5.4; two rows 29.4 -> 20.8,
// 29.9 -> 21.7 and, of the last, 8.3 -> 6.3.  The operand of two rows is asked for together (14336 x 4096 23.0 -> 20.8), and so are a group's values,
// gate and weights (two rows of a pair of products with groups of 128, 25.0 us before, cold; a model's step of two rows 395 -> 337).
// Narrow matrices have too few steps to pay for rows that lie in several warps: up to kMvWholeCols columns and as many rows as there are
// warps, a row goes whole to a warp (1024 x 1024 2.8 -> 2.4 us, two rows 3.7 -> 2.5; at 2048 columns, 768 rows, 3.1 -> 3.3: not there).
// What is left is 4 to 5 us a launch: the wait, the operand, the last CTA.  Rings of 48, 96 and 160 KB
// measured 21.1, 20.1 and 19.7 us for 14336 x 4096 and 16.6, 16.4 and 16.9 ms for a request that 64 KB serve in 16.1 (4 layers, 32 tokens).
// Registers keep it at one CTA per SM: where two fit, the CTAs of the next launch pile up on some SMs (42 us in place of 23).
#include "layered.cuh"

namespace cmld {

namespace {

constexpr int kMvThreads = 512, kMvWarps = kMvThreads / 32;
constexpr int kMvRing = 64 * 1024;  // bytes
constexpr int kMvWholeCols = 1024;  // rows of up to so many columns go whole to a warp where every warp has at most one
constexpr size_t kMvMaxCols = 220 * 1024, kMvMaxSmem = 224 * 1024;  // (kMvRing + two thirds of kMvMaxCols is less)

__host__ __device__ constexpr int mv_kpad(int cols) { return (cols + 255) & ~255; }

// 16 bytes, zeros where `there` is false
__device__ __forceinline__ void mv_copy16(uint32_t dst, const void *src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// The prepared rows sit in shared memory as f32, the two 16-byte units of a lane's eight values changing places in every other four lanes:
// no two of a quarter warp meet in a bank.
__device__ __forceinline__ int mv_unit(int i) { return i ^ (i >> 3 & 1); }

// The operand of row r, value by value: any width, alignment and prologue.  (Apart, for the registers.)
__device__ __noinline__ void mv_prologue(const LinMvArgs &a, int r, float *xr, float *red, bool store) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, K = a.w.cols;
  const float *x = a.x + r * a.x_ld;
  if (a.prologue == kProStreams) {
    stream_mix_row(a.mix, r, xr, red, store);
  } else if (a.prologue == kProRmsGroups) {
    // a warp per group of columns
    const float *gate = a.gate + r * a.gate_ld;
    for (int c0 = warp * a.group; c0 < K; c0 += kMvWarps * a.group) {
      float s = 0.0f;
      if (a.group <= 128) {  // everything asked for at once
        float xv[4], gv[4], nw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int i = lane + 32 * j;
          const bool in = i < a.group;
          xv[j] = in ? x[c0 + i] : 0.0f, gv[j] = in ? gate[c0 + i] : 0.0f, nw[j] = in ? a.norm_w[i] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) s = fmaf(xv[j], xv[j], s);
        const float inv = 1.0f / sqrtf(warp_sum(s) / (float)a.group + a.eps);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (lane + 32 * j < a.group) xr[c0 + lane + 32 * j] = xv[j] * inv * nw[j] * silu_f(gv[j]);
        continue;
      }
      for (int i = lane; i < a.group; i += 32) s = fmaf(x[c0 + i], x[c0 + i], s);
      const float inv = 1.0f / sqrtf(warp_sum(s) / (float)a.group + a.eps);
      for (int i = lane; i < a.group; i += 32) xr[c0 + i] = x[c0 + i] * inv * a.norm_w[i] * silu_f(gate[c0 + i]);
    }
  } else {
    float inv = 1.0f;
    if (a.prologue != kProPlain) {
      float s = 0.0f;
      for (int i = tid; i < K; i += kMvThreads) s = fmaf(x[i], x[i], s);
      inv = 1.0f / sqrtf(cta_total(s, red) / (float)K + a.eps);
    }
    for (int i = tid; i < K; i += kMvThreads) {
      float v = x[i];
      if (a.prologue != kProPlain) {
        v = v * inv * a.norm_w[i];
        if (a.prologue == kProRmsGate) v *= sigmoid_f(a.gate[r * a.gate_ld + i]);
      }
      xr[i] = v;
    }
  }
}

template <int R, int ROWS>
__device__ __forceinline__ void lin_mv_cta(const LinMvArgs &a, int cta, int ctas) {
  constexpr int kStages = kMvRing / (ROWS * kMvThreads * 16);
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(8) float red[2 * kMvWarps];
  __shared__ float coef[kMixCoefs];
  __shared__ float part[kMvWarps][2][ROWS][R];  // sums of a row that other warps share: of its end (0), of its beginning (1)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = a.w.cols, kp = mv_kpad(K), nit = kp / 256;
  uint4 *ring = reinterpret_cast<uint4 *>(smem) + tid;  // [stage][ROWS][thread]
  float *xs = smem + kMvRing / 4;                       // [R][kp]
  const int groups = (a.w.rows + ROWS - 1) / ROWS;
  // groups * c / ctas and steps * w / kMvWarps, rounded down, without 64-bit divisions
  const unsigned whole = (unsigned)groups / (unsigned)ctas, rest = (unsigned)groups - whole * ctas;
  auto group_of = [&](int c) { return (int)(whole * c + rest * c / (unsigned)ctas); };
  const int g0 = group_of(cta), mine = group_of(cta + 1) - g0, steps = mine * nit;
  auto run_of = [&](int w) { return steps / kMvWarps * w + steps % kMvWarps * w / kMvWarps; };
  const bool rows_whole = ROWS == 1 && mine <= kMvWarps && K <= kMvWholeCols;  // a row per warp, all of it asked for at once
  const int lo = rows_whole ? min(warp, mine) * nit : run_of(warp), hi = rows_whole ? min(warp + 1, mine) * nit : run_of(warp + 1);

  // Step s of the CTA: columns s % nit * 256 .. of the ROWS rows s / nit; a lane copies what it will use itself.
  const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring);
  const bf16 *src;
  int64_t below;  // from the first row to the second
  int left;       // steps of these rows still to be copied
  auto rows_at = [&](int s) {
    const int grp = g0 + s / nit, it = s % nit;
    src = a.w.w + (int64_t)grp * ROWS * a.w.ld + it * 256 + lane * 8;
    below = grp * ROWS + 1 < a.w.rows ? a.w.ld : 0;
    left = nit - it;
  };
  auto copy = [&](int slot) {
    const bool there = left > 1 || (nit - 1) * 256 + lane * 8 < a.w.ld;  // the row's padding is zero
#pragma unroll
    for (int i = 0; i < ROWS; ++i) mv_copy16(ring_at + (slot * ROWS + i) * (kMvThreads * 16), there ? src + i * below : a.w.w, there);
    src += 256;
  };
  pdl_launch();
  if (rows_whole) {
    src = a.w.w + (int64_t)(g0 + warp) * a.w.ld + lane * 8, below = 0, left = nit;
  } else if (lo < hi) {
    rows_at(lo);
  }
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) {
    if (lo + i < hi) {
      copy(i);
      if (--left == 0 && lo + i + 1 < hi) rows_at(lo + i + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const bool mixed = a.prologue == kProStreams && mix_row_fits(a.mix, 2, kMvThreads);
  if (mixed && tid < kMixCoefs) coef[tid] = mix_coef(a.mix, tid);
  pdl_wait();

  const auto aligned = [](const float *p, int64_t ld) { return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)(4 * ld)) & 15) == 0; };
  const bool quads = K % 4 == 0 && aligned(a.x, a.x_ld) && aligned(a.gate, a.gate_ld) && aligned(a.norm_w, 0);
  const int n4 = K / 4;
  if (K < kp) {  // zeros behind the rows, in place before anything of them is
    for (int i = tid; i < 64 * R; i += kMvThreads) reinterpret_cast<float4 *>(xs + (i / 64 + 1) * kp)[i % 64 - 64] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
  }
  if (quads && a.prologue == kProPlain) {
    constexpr int N = 8 / R;
    for (int i0 = tid; i0 < n4; i0 += N * kMvThreads) {
      float4 v[R][N];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (i0 + j * kMvThreads < n4) v[r][j] = reinterpret_cast<const float4 *>(a.x + r * a.x_ld)[i0 + j * kMvThreads];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < N; ++j)
          if (i0 + j * kMvThreads < n4) reinterpret_cast<float4 *>(xs + r * kp)[mv_unit(i0 + j * kMvThreads)] = v[r][j];
    }
  } else
#pragma unroll 1
  for (int r = 0; r < R; ++r) {
    float *xr = xs + r * kp;
    float4 *x4 = reinterpret_cast<float4 *>(xr);
    if (mixed) {
      mix_row<2>(a.mix, a.mix.row_map ? a.mix.row_map[r] : r, coef, red, cta == 0, [&](int i, float4 v) { x4[mv_unit(i)] = v; });
    } else if (quads && (a.prologue == kProRms || a.prologue == kProRmsGate) && n4 <= 2 * kMvThreads) {
      const float4 *x = reinterpret_cast<const float4 *>(a.x + r * a.x_ld), *gate = reinterpret_cast<const float4 *>(a.gate + r * a.gate_ld);
      const float4 *nw = reinterpret_cast<const float4 *>(a.norm_w);
      const bool gated = a.prologue == kProRmsGate;
      float4 v[2], w[2], z[2];
      float s = 0.0f;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int i = tid + j * kMvThreads;
        v[j] = w[j] = z[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n4) {
          v[j] = x[i];
          w[j] = nw[i];
          if (gated) z[j] = gate[i];
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) s += dot4(v[j], v[j]);
      const float inv = 1.0f / sqrtf(cta_total(s, red) / (float)K + a.eps);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int i = tid + j * kMvThreads;
        float4 o = make_float4(v[j].x * inv * w[j].x, v[j].y * inv * w[j].y, v[j].z * inv * w[j].z, v[j].w * inv * w[j].w);
        if (gated) o = make_float4(o.x * sigmoid_f(z[j].x), o.y * sigmoid_f(z[j].y), o.z * sigmoid_f(z[j].z), o.w * sigmoid_f(z[j].w));
        if (i < n4) x4[mv_unit(i)] = o;
      }
    } else {
      mv_prologue(a, r, xr, red, cta == 0);
      __syncthreads();
      for (int i = tid; i < kp / 8; i += kMvThreads)
        if (mv_unit(2 * i) != 2 * i) {
          const float4 v = x4[2 * i];
          x4[2 * i] = x4[2 * i + 1];
          x4[2 * i + 1] = v;
        }
    }
  }
  __syncthreads();

  auto finish = [&](int g, const float (&sum)[ROWS][R]) {  // by one lane
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float v[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int row = g * ROWS + i;
        v[i] = fmaf(sum[i][r], a.scale, a.bias && row < a.w.rows ? a.bias[row] : 0.0f);
        if (row < a.w.rows && a.act != kActSwiGlu) a.y[r * a.y_ld + row] = lin_activate(v[i], a.act, row < a.act_rows);
      }
      if (ROWS == 2 && a.act == kActSwiGlu) a.y[r * a.y_ld + g] = silu_f(v[0]) * v[ROWS - 1];
    }
  };
  int g = rows_whole ? g0 + warp : g0 + lo / nit, it = rows_whole ? 0 : lo - (g - g0) * nit;
  const bool joins = it != 0 && lo < hi;  // the warp's first row began in another warp
  bool head = joins;
  const float *x = xs + it * 256 + lane * 8;
  const int odd = lane & 4;
  float acc[ROWS][R];
#pragma unroll
  for (int i = 0; i < ROWS; ++i)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[i][r] = 0.0f;
  if (!rows_whole && lo + kStages - 1 < hi) rows_at(lo + kStages - 1);
  for (int s0 = lo; s0 < hi; s0 += kStages) {
#pragma unroll
    for (int j = 0; j < kStages; ++j) {
      const int s = s0 + j;
      if (s >= hi) break;
      if (s + kStages - 1 < hi) {  // into the stage of step s - 1, whose bytes this thread has used
        copy((j + kStages - 1) % kStages);
        if (--left == 0 && s + kStages < hi) rows_at(s + kStages);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
      uint4 w[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) w[i] = ring[(j * ROWS + i) * kMvThreads];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 lo4 = *reinterpret_cast<const float4 *>(x + r * kp + odd), hi4 = *reinterpret_cast<const float4 *>(x + r * kp + (odd ^ 4));
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
          float t = acc[i][r];
          t = fmaf(bf16_lo(w[i].x), lo4.x, t);
          t = fmaf(bf16_hi(w[i].x), lo4.y, t);
          t = fmaf(bf16_lo(w[i].y), lo4.z, t);
          t = fmaf(bf16_hi(w[i].y), lo4.w, t);
          t = fmaf(bf16_lo(w[i].z), hi4.x, t);
          t = fmaf(bf16_hi(w[i].z), hi4.y, t);
          t = fmaf(bf16_lo(w[i].w), hi4.z, t);
          t = fmaf(bf16_hi(w[i].w), hi4.w, t);
          acc[i][r] = t;
        }
      }
      x += 256;
      const bool ends = ++it == nit;
      if (ends || s + 1 == hi) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int r = 0; r < R; ++r) acc[i][r] = warp_sum(acc[i][r]);
        if (lane == 0) {
          if (ends && !head) {
            finish(g, acc);
          } else {
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
#pragma unroll
              for (int r = 0; r < R; ++r) part[warp][head ? 0 : 1][i][r] = acc[i][r];
          }
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int r = 0; r < R; ++r) acc[i][r] = 0.0f;
        head = false;
        if (ends) it = 0, ++g, x = xs + lane * 8;
      }
    }
  }
  if (rows_whole) return;
  __syncthreads();
  // a row that begins in this warp and ends in another: `it` of its steps were done here
  if (lane == 0 && lo < hi && it != 0 && (!joins || g > g0 + lo / nit)) {
    float sum[ROWS][R];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int r = 0; r < R; ++r) sum[i][r] = part[warp][1][i][r];
    const int end = (g - g0 + 1) * nit;
    for (int w = warp + 1, at = hi; at < end; ++w) {
      const int upto = run_of(w + 1);
      if (upto > at) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
#pragma unroll
          for (int r = 0; r < R; ++r) sum[i][r] += part[w][0][i][r];
      }
      at = upto;
    }
    finish(g, sum);
  }
}

template <int R, int ROWS>
__global__ void __launch_bounds__(kMvThreads, 1) lin_mv_kernel(const __grid_constant__ LinMvArgs a) {
  lin_mv_cta<R, ROWS>(a, blockIdx.x, gridDim.x);
}

template <int R, int ROWS>
__global__ void __launch_bounds__(kMvThreads, 1) lin_mv_pair_kernel(const __grid_constant__ LinMvArgs a, const __grid_constant__ LinMvArgs b, int n_first) {
  const bool first = (int)blockIdx.x < n_first;
  lin_mv_cta<R, ROWS>(first ? a : b, first ? blockIdx.x : blockIdx.x - n_first, first ? n_first : gridDim.x - n_first);
}

size_t mv_smem(int cols, int batch) { return kMvRing + (size_t)batch * mv_kpad(cols) * 4; }

int mv_sms() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int R, int ROWS>
int32_t mv_launch(const LinMvArgs &a, bool pdl, cudaStream_t s) {
  static SmemLimit limit;
  CMLD_TRY(allow_smem(limit, lin_mv_kernel<R, ROWS>, kMvMaxSmem, true));
  const int groups = (a.w.rows + ROWS - 1) / ROWS;
  return launch_kernel(lin_mv_kernel<R, ROWS>, dim3(std::min(groups, mv_sms())), dim3(kMvThreads), mv_smem(a.w.cols, R), pdl, s, a);
}

template <int R, int ROWS>
int32_t mv_launch_pair(const LinMvArgs &a, const LinMvArgs &b, bool pdl, cudaStream_t s) {
  static SmemLimit limit;
  CMLD_TRY(allow_smem(limit, lin_mv_pair_kernel<R, ROWS>, kMvMaxSmem, true));
  const int sms = mv_sms();
  const double wa = (double)a.w.rows * a.w.ld, wb = (double)b.w.rows * b.w.ld;
  const int first = std::min(sms - 1, std::max(1, (int)(sms * wa / (wa + wb) + 0.5)));
  return launch_kernel(lin_mv_pair_kernel<R, ROWS>, dim3(sms), dim3(kMvThreads), mv_smem(std::max(a.w.cols, b.w.cols), R), pdl, s, a, b, first);
}

}  // namespace

bool lin_mv_fits(int32_t cols, int32_t batch) { return batch >= 1 && batch <= 2 && (size_t)(batch + 1) * mv_kpad(cols) * 4 <= kMvMaxCols; }

int32_t launch_lin_mv(const LinMvArgs &a, bool pdl, cudaStream_t s) {
  if (!lin_mv_fits(a.w.cols, a.batch)) return fail(CMLD_ERR_SHAPE, "matrix-vector product of %d columns and %d rows does not fit", a.w.cols, a.batch);
  if (a.act == kActSwiGlu) {
    if (a.w.rows % 2) return fail(CMLD_ERR_SHAPE, "linear: gated pairs need an even number of rows");
    return a.batch == 1 ? mv_launch<1, 2>(a, pdl, s) : mv_launch<2, 2>(a, pdl, s);
  }
  // single rows only where pairs would leave SMs without work or with one more than others (576 x 4096: 3.2 us, in pairs 3.4; 1536 x 4096: 4.8
  // and 4.5, 4096 x 4096: 8.0 and 7.6), and where rows go whole to warps
  const bool single = a.w.rows <= 4 * mv_sms() || (a.w.rows <= kMvWarps * mv_sms() && a.w.cols <= kMvWholeCols);
  if (a.batch == 1) return single ? mv_launch<1, 1>(a, pdl, s) : mv_launch<1, 2>(a, pdl, s);
  return single ? mv_launch<2, 1>(a, pdl, s) : mv_launch<2, 2>(a, pdl, s);
}

int32_t launch_lin_mv_pair(const LinMvArgs &a, const LinMvArgs &b, bool pdl, cudaStream_t s) {
  if (a.batch != b.batch || a.act == kActSwiGlu || b.act == kActSwiGlu || !lin_mv_fits(a.w.cols, a.batch) || !lin_mv_fits(b.w.cols, b.batch))
    return fail(CMLD_ERR_SHAPE, "a pair of matrix-vector products does not fit one launch");
  return a.batch == 1 ? mv_launch_pair<1, 2>(a, b, pdl, s) : mv_launch_pair<2, 2>(a, b, pdl, s);
}

}  // namespace cmld
