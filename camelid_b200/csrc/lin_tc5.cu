// Linear layers on the 5th-generation tensor cores: out[r][o] = act(scale * sum_k w[o][k] x[r][k] + bias[o]), bfloat16
// operands, f32 accumulators in tensor memory.
//
// The weights are operand A (tiles of 128 output rows), the activation rows operand B (tiles of n_tile rows, 16 to 256), both K-major
// and brought by TMA in 128-byte-swizzled boxes of 64 columns.  Persistent CTAs, one per SM; warp roles:
//   warps 0, 1  TMA: every other operand stage each (one elected lane)
//   warp 2      MMA issue (one elected lane), tensor-memory allocation
//   warps 3-10  epilogue: tcgen05.ld, activation, stores, two warps for each quarter of the accumulator lanes (every
//               other 16 columns); two accumulator slots, so that a tile's epilogue overlaps the next tile's products
// Many rows: bound by what an SM takes from L2, about 64 bytes a cycle for the 128 + n_tile rows of a step.  The tiles that read the same weights
// are neighbours, on different SMs at the same time, so that the weights come from HBM once and are in L2 for the others (all
// weights for each tile of rows: 22544 x 4096 with 2048 rows 369 us, now 275; 32000 x 4096 511 -> 389), and the rows are cut into tiles that fill the SMs,
// of equal size (300 rows as 2 x 160 in place of 2 x 256 or 4 x 80 in place of 5 x 64: 22544 x 4096 92 -> 63 us, 4096 x 14336 79 -> 66).
// Few rows: bound by HBM, as far as every SM has as much to do.  Few tiles: `split` CTAs of a thread-block cluster share a tile's inner
// dimension, leave their partial accumulators in shared memory, and each of them adds the partials of its share of the columns in rank order.
// (All CTAs with equal runs of the steps of all tiles took 22544 x 4096 with 8 rows from 45.6 to 35.3 us, but adds in another order.)
// The first weight boxes are asked for before the kernel waits for its predecessor.
// Every wait is bounded: one that runs out sets the status word and an abort flag, all roles leave their loops, tensor
// memory is freed and the kernel returns.
#include <cuda.h>

#include "layered.cuh"

namespace cmld {

namespace {

constexpr int kEpiWarps = 8, kThreads = (3 + kEpiWarps) * 32, kBM = 128, kBK = 64, kMaxStages = 8;
constexpr uint32_t kSpin = 1u << 22;
constexpr int kABytes = kBM * kBK * 2;
constexpr int kBarBytes = 256, kSmem = 226 * 1024;

__host__ __device__ constexpr int stage_bytes(int n_tile) { return kABytes + n_tile * kBK * 2; }
constexpr int stages(int n_tile) { return std::min(kMaxStages, (kSmem - kBarBytes - 1024) / stage_bytes(n_tile)); }
constexpr int smem_bytes(int n_tile) { return stages(n_tile) * stage_bytes(n_tile) + kBarBytes + 1024; }  // + slack to align the base to 1024

struct TcLinArgs {
  int32_t m_rows, n_rows, n_k, tiles_n, tiles, n_tile, split, stages, slot_cols;
  void *out;
  int64_t out_ld;
  int32_t act, act_rows;
  const float *bias;
  float scale;
  int32_t *status;
};

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int32_t *status) {
  for (uint32_t i = 0; i < kSpin; ++i) {
    if (bar_try(bar, parity)) return true;
    if ((i & 255u) == 255u && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicExch(status, (int32_t)CMLD_ERR_TIMEOUT);
  return false;
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x),
               "r"(y), "r"(bar)
               : "memory");
}
// K-major operand in 128-byte-swizzled rows: groups of eight rows are 1024 bytes apart (descriptor version 1, layout
// type 2 = 128-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t t, float (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&f"(r[0]), "=&f"(r[1]), "=&f"(r[2]), "=&f"(r[3]), "=&f"(r[4]), "=&f"(r[5]), "=&f"(r[6]), "=&f"(r[7]), "=&f"(r[8]), "=&f"(r[9]),
        "=&f"(r[10]), "=&f"(r[11]), "=&f"(r[12]), "=&f"(r[13]), "=&f"(r[14]), "=&f"(r[15])
      : "r"(t)
      : "memory");
}
__device__ __forceinline__ void put(float *p, float v) { *p = v; }
__device__ __forceinline__ void put(bf16 *p, float v) { *p = __float2bfloat16_rn(v); }

// The tile of a cluster, whose partial accumulators [n_tile][128] lie at `base` of each CTA: the elements are shared out over all threads and
// their partials, all of them asked for first, added in rank order.  Few rows: an element per thread, neighbours side by side (four to a
// thread in 16-byte loads leave whole warps without any and store quarters of a line).  Many rows, from four rounds of all threads on: four
// to a thread.  Us, four | one: 2048 x 2048 with 16 rows 10.3 | 9.1, 768 x 2048 with 16 4.7 | 4.0, 1536 x 4096 with 8 7.0 | 6.6, 4096 x 4096 with 100
// 14.7 | 16.1.  One loop per number of CTAs, four elements of a thread at once, did as well with every launch alike (9.3, 4.2, 6.5, 14.5) and was
// slower among other kernels, where its code is fetched anew: a step of the 2k Tokovik at 12 rows 410 us, here 406, 421 with four to a thread.
template <typename OutT>
__device__ __forceinline__ void add_parts(const TcLinArgs &a, uint32_t base, int rank) {
  OutT *out = static_cast<OutT *>(a.out);
  const int t = (int)blockIdx.x / a.split, m0 = (t / a.tiles_n) * kBM, n0 = (t % a.tiles_n) * a.n_tile;
  const int n_el = min(a.n_tile, a.n_rows - n0) * kBM, step = a.split * kThreads;
  const int per = (a.n_k + a.split - 1) / a.split, parts = (a.n_k + per - 1) / per;  // (the last CTAs may have none)
  if (n_el > 4 * step) {
    for (int e = 4 * (rank * kThreads + (int)threadIdx.x); e < n_el; e += 4 * step) {
      const int o = m0 + e % kBM;
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f), u[8];
#pragma unroll
      for (int p = 0; p < 8; ++p)
        if (p < parts) u[p] = ld_peer4(base + 4u * e, p);
#pragma unroll
      for (int p = 0; p < 8; ++p)
        if (p < parts) v = make_float4(v.x + u[p].x, v.y + u[p].y, v.z + u[p].z, v.w + u[p].w);
      float r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) r[j] = fmaf(r[j], a.scale, a.bias && o + j < a.m_rows ? a.bias[o + j] : 0.0f);
      OutT *p = out + (int64_t)(n0 + e / kBM) * a.out_ld;
      if (a.act == kActSwiGlu) {
#pragma unroll
        for (int j = 0; j < 4; j += 2)
          if (o + j < a.m_rows) put(p + ((o + j) >> 1), silu_f(r[j]) * r[j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (o + j < a.m_rows) put(p + o + j, lin_activate(r[j], a.act, o + j < a.act_rows));
      }
    }
    return;
  }
#pragma unroll 1
  for (int e = rank * kThreads + (int)threadIdx.x; e < n_el; e += step) {  // (all counts are multiples of 32: a warp's lanes agree on what is there)
    float u[8], v = 0.0f;
#pragma unroll
    for (int p = 0; p < 8; ++p)
      if (p < parts) u[p] = ld_peer(base + 4u * e, p);
#pragma unroll
    for (int p = 0; p < 8; ++p)
      if (p < parts) v += u[p];
    const int o = m0 + e % kBM;
    v = fmaf(v, a.scale, a.bias && o < a.m_rows ? a.bias[o] : 0.0f);
    OutT *q = out + (int64_t)(n0 + e / kBM) * a.out_ld;
    if (a.act == kActSwiGlu) {
      const float next = __shfl_down_sync(0xffffffffu, v, 1);
      if (!(e & 1) && o < a.m_rows) put(q + (o >> 1), silu_f(v) * next);
    } else if (o < a.m_rows) {
      put(q + o, lin_activate(v, a.act, o < a.act_rows));
    }
  }
}

template <typename OutT>
__global__ void __launch_bounds__(kThreads, 1)
    lin_tc5_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap, const TcLinArgs a) {
  const int NS = a.stages, stage = stage_bytes(a.n_tile);
  extern __shared__ uint8_t raw[];
  uint8_t *smem = raw + ((1024u - (s32(raw) & 1023u)) & 1023u);
  const uint32_t base = s32(smem), bars = base + NS * stage;
  auto full = [&](int i) { return bars + 8u * i; };
  auto empty = [&](int i) { return bars + 8u * (kMaxStages + i); };
  auto acc_full = [&](int i) { return bars + 8u * (2 * kMaxStages + i); };
  auto acc_empty = [&](int i) { return bars + 8u * (2 * kMaxStages + 2 + i); };
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + NS * stage + 8 * (2 * kMaxStages + 4));
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // A cluster of `split` CTAs works on one tile, each on its share of the inner columns.  Tiles that read the same weights are neighbours.
  const int rank = (int)blockIdx.x % a.split, per = (a.n_k + a.split - 1) / a.split, k_lo = min(rank * per, a.n_k), nk = min(k_lo + per, a.n_k) - k_lo;
  const int t_lo = (int)blockIdx.x / a.split, t_step = (int)gridDim.x / a.split;
  const int total = t_lo < a.tiles ? ((a.tiles - 1 - t_lo) / t_step + 1) * nk : 0;  // steps of this CTA
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.n_tile >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);

  if (tid == 0) {
    for (int i = 0; i < NS; ++i) {
      bar_init(full(i), 1);
      bar_init(empty(i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      bar_init(acc_full(i), 1);
      bar_init(acc_empty(i), kEpiWarps);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(2 * a.slot_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tbase = *tmem_slot;
  pdl_launch();

  if (warp < 2) {
    // every other step each: waiting for a stage and issuing its two copies takes one thread longer than the products of a step
    if (lane == 0 && total > 0) {
      const int early = min(total, NS);
      int q, kb, t;
      auto begin = [&] {
        q = warp, kb = k_lo + warp, t = t_lo;
        while (kb >= k_lo + nk) kb -= nk, t += t_step;
      };
      auto advance = [&] {
        q += 2, kb += 2;
        while (kb >= k_lo + nk) kb -= nk, t += t_step;
      };
      auto load_w = [&](int st) {
        bar_expect(full(st), stage);
        tma_2d(base + st * stage, &wmap, kb * kBK, t / a.tiles_n * kBM, full(st));
      };
      auto load_x = [&](int st) { tma_2d(base + st * stage + kABytes, &xmap, kb * kBK, t % a.tiles_n * a.n_tile, full(st)); };
      for (begin(); q < early; advance()) load_w(q);
      pdl_wait();
      for (begin(); q < early; advance()) load_x(q);
      int st = q - NS;
      for (uint32_t parity = 0; q < total; advance()) {
        if (!bar_wait(empty(st), parity, abort_flag, a.status)) break;
        load_w(st);
        load_x(st);
        st += 2;
        if (st >= NS) st -= NS, parity ^= 1;
      }
      if (*abort_flag) __nanosleep(1000000);  // copies in flight land before the shared memory is given back
    }
  } else if (warp == 2) {
    if (lane == 0) {
      int i = 0, st = 0;
      uint32_t parity = 0;
      bool ok = true;
      for (int q = 0; q < total && ok; ++i) {
        const int slot = i & 1, end = q + nk;
        if (i >= 2) ok = bar_wait(acc_empty(slot), (uint32_t)((i / 2 - 1) & 1), abort_flag, a.status);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (bool more = false; q < end && ok; ++q) {
          ok = bar_wait(full(st), parity, abort_flag, a.status);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = smem_desc(base + st * stage), db = smem_desc(base + st * stage + kABytes);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            mma_bf16(tbase + slot * a.slot_cols, da + 2 * k, db + 2 * k, idesc, more);
            more = true;
          }
          mma_commit(empty(st));
          if (++st == NS) st = 0, parity ^= 1;
        }
        if (ok) mma_commit(acc_full(slot));
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, half = (warp - 3) >> 2;  // the 32 accumulator lanes this warp may read; its column groups
    pdl_wait();                    // the output buffer may still be read by the predecessor
    int i = 0;
    OutT *out = static_cast<OutT *>(a.out);
    for (int q = 0, t = t_lo; q < total; ++i, q += nk, t += t_step) {
      const int slot = i & 1, o = (t / a.tiles_n) * kBM + quarter * 32 + lane, n0 = (t % a.tiles_n) * a.n_tile;
      if (!bar_wait(acc_full(slot), (uint32_t)((i / 2) & 1), abort_flag, a.status)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int n_live = min(a.n_tile, a.n_rows - n0);
      const bool silu = a.act == kActSilu && o < a.act_rows, relu2 = a.act == kActRelu2, swiglu = a.act == kActSwiGlu;
      const float bias = a.bias && o < a.m_rows ? a.bias[o] : 0.0f;
      const bool odd = lane & 1;
      // columns c .. c + 15 of the tile
      auto finish = [&](int c, float (&r)[16]) {
        OutT *p = out + (int64_t)(n0 + c) * a.out_ld + (swiglu ? o >> 1 : o);
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = fmaf(r[j], a.scale, bias);
        if (swiglu) {
          // a lane holds the gate (even rows) or the other factor (odd rows); of two columns the even lane finishes one,
          // the odd lane the other
          OutT *w = p + (odd ? a.out_ld : 0);
#pragma unroll
          for (int j = 0; j < 16; j += 2, w += 2 * a.out_ld) {
            const float t = __shfl_xor_sync(0xffffffffu, odd ? r[j] : r[j + 1], 1);
            const float v = odd ? silu_f(t) * r[j + 1] : silu_f(r[j]) * t;
            if (o < a.m_rows && c + j + (odd ? 1 : 0) < n_live) put(w, v);
          }
          return;
        }
        if (silu) {
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = silu_f(r[j]);
        } else if (relu2) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float v = fmaxf(r[j], 0.0f);
            r[j] = v * v;
          }
        }
        if (o < a.m_rows) {
          OutT *w = p;
          if (c + 16 <= n_live) {
#pragma unroll
            for (int j = 0; j < 16; ++j, w += a.out_ld) put(w, r[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j, w += a.out_ld)
              if (c + j < n_live) put(w, r[j]);
          }
        }
      };
#pragma unroll 1
      for (int c = 16 * half; c < n_live; c += 32) {
        float r[16];
        tmem_ld16(tbase + slot * a.slot_cols + c + ((uint32_t)(quarter * 32) << 16), r);
        if (a.split == 1) {
          finish(c, r);
        } else {
          float *part = reinterpret_cast<float *>(smem);  // [n_tile][128]: the operand stages are free by now
#pragma unroll
          for (int j = 0; j < 16; ++j) part[(c + j) * kBM + quarter * 32 + lane] = r[j];
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(acc_empty(slot));
    }
  }
  __syncwarp();
  if (a.split > 1) {
    // one tile per cluster: add the partial accumulators in rank order
    cluster_sync();
    if (!*abort_flag) add_parts<OutT>(a, base, rank);
    cluster_sync();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(2 * a.slot_cols) : "memory");
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int32_t make_map(CUtensorMap *map, const void *p, int64_t cols, int64_t rows, int64_t ld, int box_rows) {
  static EncodeFn encode = nullptr;
  if (!encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    CMLD_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    if (!fn || q != cudaDriverEntryPointSuccess) return fail(CMLD_ERR_CUDA, "the driver does not offer cuTensorMapEncodeTiled");
    encode = reinterpret_cast<EncodeFn>(fn);
  }
  if ((reinterpret_cast<uintptr_t>(p) & 15) || (ld & 7)) return fail(CMLD_ERR_SHAPE, "tensor-core operand is not 16-byte aligned");
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {kBK, (cuuint32_t)box_rows}, es[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(p), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(CMLD_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return CMLD_OK;
}

template <typename OutT>
int32_t launch_out(const LinArgs &L, int32_t sms, int32_t *status, bool pdl, cudaStream_t s) {
  static SmemLimit limit;
  CMLD_TRY(allow_smem(limit, lin_tc5_kernel<OutT>, kSmem, true));
  // Row tiles of equal size, as many as make (rounds over the SMs) x (rows of both operands that an SM takes in a step) least.
  const int n_k = (L.w.cols + kBK - 1) / kBK, tiles_m = (L.w.rows + kBM - 1) / kBM;
  int n_tile = 0;
  int64_t least = 0;
  for (int parts = (L.rows + 255) / 256; parts <= (L.rows + 63) / 64; ++parts) {
    const int n = ((L.rows + parts - 1) / parts + 15) & ~15;
    const int64_t rounds = ((int64_t)tiles_m * ((L.rows + n - 1) / n) + sms - 1) / sms, cost = rounds * (kBM + n);
    if (!n_tile || cost < least) n_tile = n, least = cost;
  }
  // Few tiles of few rows: spread a tile's inner dimension until the machine is full.
  const int few = L.rows <= 16 ? 16 : L.rows <= 32 ? 32 : 64;
  int split = 1;
  if (L.rows <= 64 || tiles_m * ((L.rows + 127) / 128) * 2 <= sms)
    while (split < 8 && tiles_m * ((L.rows + few - 1) / few) * split * 2 <= sms && n_k >= 4 * split) split *= 2;
  if (split > 1) n_tile = std::min(few, (L.rows + 15) & ~15);
  CUtensorMap wmap, xmap;
  CMLD_TRY(make_map(&wmap, L.w.w, L.w.cols, L.w.rows, L.w.ld, kBM));
  CMLD_TRY(make_map(&xmap, L.x, L.w.cols, L.rows, L.x_ld, n_tile));
  TcLinArgs a{};
  a.m_rows = L.w.rows;
  a.n_rows = L.rows;
  a.n_k = n_k;
  a.n_tile = n_tile;
  a.stages = stages(n_tile);
  a.slot_cols = 32;
  while (a.slot_cols < n_tile) a.slot_cols *= 2;
  a.tiles_n = (L.rows + n_tile - 1) / n_tile;
  a.tiles = tiles_m * a.tiles_n;
  a.split = split;
  a.out = L.out;
  a.out_ld = L.out_ld;
  a.act = L.act;
  a.act_rows = L.act_rows;
  a.bias = L.bias;
  a.scale = L.scale;
  a.status = status;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(a.split > 1 ? a.tiles * a.split : std::min(a.tiles, sms)));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_bytes(n_tile);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (a.split > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)a.split;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  CMLD_CUDA(cudaLaunchKernelEx(&cfg, lin_tc5_kernel<OutT>, wmap, xmap, a));
  return CMLD_OK;
}

}  // namespace

int32_t launch_lin_tc5(const LinArgs &a, int32_t sms, int32_t *status, bool pdl, cudaStream_t s) {
  if (a.rows < 1) return CMLD_OK;
  if (a.act == kActSwiGlu && a.w.rows % 2) return fail(CMLD_ERR_SHAPE, "linear: gated pairs need an even number of rows");
  return a.out_half ? launch_out<bf16>(a, sms, status, pdl, s) : launch_out<float>(a, sms, status, pdl, s);
}

}  // namespace cmld
