// Batched quantised matrix products on the 5th-generation tensor cores (tcgen05.mma, accumulators in tensor memory), with
// the CPU path's order of f32 operations in the epilogue, so that a row's result is bit-identical to the one-row kernels'.
//
// What the tensor cores compute is the INTEGER part of the reference's dot products, which is exact in any order; the f32
// steps that follow are done per (activation row, weight row) in block order:
//   Q8_0 (src/inference.rs:26191-26199): per 32-value block, isum = sum q*y is one K=32 MMA into its own accumulator
//     columns; then acc += ((float)isum * ws) * xs, block after block.
//   Q4_K (src/diffusion_gemma/refmath.rs:504-562): per superblock S = sum_g sc_g * (q.y)_g and P = sum_g min_g * bsum_g;
//     then acc = fma(-(xd*dmin), P, acc); acc = fma(xd*d, S, acc).  The 6-bit scale is split sc = 8*s1 + s0 and the weight
//     operand holds s1*q and s0*q (<= 105), so S = 8*S1 + S0 comes from two accumulators that run over the whole superblock.
//     P is one kind::f16 MMA: the mins (each twice) times the sums of 16 codes (|.| <= 2048: exact in f16, and every
//     partial sum stays below 2^24, so the f32 accumulator holds P itself).
//   Q6_K (src/inference.rs:25545-25581): eight f32 lanes by (index mod 8): per superblock aux[l] = sum_g sc_g * sum_{k in g,
//     k = l mod 8} (q_k - 32) * y_k, then sums[l] += (d*xd) * aux[l], and at the end 0 + sums[0] + ... + sums[7].  The K
//     dimension is permuted so that MMA l covers the 32 values with index = l mod 8; the weight operand holds
//     sc*(q-32) = 128*vh + vl (vh signed, vl in 0..127), and aux[l] = 128*D_hi + D_lo.
//
// The activation rows are operand A (M = 128), the weight rows operand B: a tile is 128 activation rows x NW weight rows, so
// that unpacking a weight is shared by 128 rows.  Steps of up to 32 rows have a kernel of their own (gemv_rows.cu).
//
// One CTA per SM, K step = 256 columns.  Warp roles (16 or 24 warps):
//   epilogue    8 or 16 warps that share the weight rows: tcgen05.ld, integer fix-up, f32 chains
//   weights     4 warps: cp.async of the raw wire bytes into a ring, unpack into the K-major operand layout; Q8_0 codes are
//               copied straight into that layout
//   MMA         one lane issues the MMAs and commits them to the mbarriers
//   activations one lane brings a step's packed record by bulk copies
// Accumulators: Q4_K two slots of a whole step; Q6_K and Q8_0 four slots that each hold a quarter of a step (two classes,
// two blocks), so that the tensor cores fill one while the epilogue reads another.
// Why this split: with the weights as operand A (128 rows) and at most 32 activation rows per pass, unpacking (about 300
// instructions of one thread per 64 Q6_K values) was repeated for every 8 to 32 activation rows and bound the launch: 45 ms of a
// 1024-token prompt's 55.8 ms (4 layers of the 8B width).  With the activations as A those launches take 7.1 ms.
// What bounds it now, at 512 rows: the epilogue, then unpacking (Q6_K 4096 x 14336: 461 us, 301 without the f32 steps, 361 without
// unpacking, 401 with half of the MMAs; Q4_K 28672 x 4096: 276, 229, 227, 266).
// Every wait is bounded: a wait that runs out sets the status word and an abort flag, all roles leave their loops, tensor
// memory is freed and the kernel returns.
#include "tc5_record.cuh"

namespace cmld {

namespace {

constexpr int kTcMaxStages = 8;
constexpr int kTcPrefetchAhead = 8;  // K steps by which a row's wire bytes are asked into L2 before they are copied
constexpr uint32_t kTcSpin = 1u << 22;
constexpr int kMR = kTc5Rows;  // activation rows of a tile

__host__ __device__ constexpr int kq_bytes(int qt) { return qt == CMLD_Q4_K ? 144 : qt == CMLD_Q6_K ? 208 : 256; }  // of a row per K step

// shared memory of one stage of weights
__host__ __device__ constexpr int b_planes(int qt) { return qt == CMLD_Q8_0 ? 1 : 2; }
__host__ __device__ constexpr int b_p(int qt, int nw) { return qt == CMLD_Q4_K ? nw * 32 : 0; }
__host__ __device__ constexpr int b_scales(int qt, int nw) { return (qt == CMLD_Q8_0 ? 8 : qt == CMLD_Q4_K ? 2 : 1) * nw * 4; }
__host__ __device__ constexpr int b_bytes(int qt, int nw) { return b_planes(qt) * nw * 256 + b_p(qt, nw) + b_scales(qt, nw); }
// ring of the weight warps: wire bytes (Q6_K: and the words that hold the f16 scales), or the f16 scales of Q8_0
__host__ __device__ constexpr int raw_bytes(int qt, int nw) { return qt == CMLD_Q8_0 ? nw * 16 : nw * (kq_bytes(qt) + (qt == CMLD_Q6_K ? 4 : 0)); }
// Groups of four warps.  Q8_0's epilogue (16 waits for tensor memory a step, few registers) hides them behind one another with
// twice the warps: 1B gate and up, 512 rows, 104 -> 93 us per launch on average; Q4_K does not gain (131 -> 147 us: its weight
// path loses registers), Q6_K has none to spare.
__host__ __device__ constexpr int epi_groups(int qt, int nw) { return qt == CMLD_Q8_0 && nw == 64 ? 4 : 2; }
__host__ __device__ constexpr int tc_threads(int qt, int nw) { return 128 * (epi_groups(qt, nw) + 2); }
constexpr int kLoadAhead = 2;  // steps by which the loads of weights run ahead of their use; their ring holds one more
__host__ __device__ constexpr int ring_bytes(int qt, int nw) { return (kLoadAhead + 1) * raw_bytes(qt, nw); }

__host__ __device__ constexpr int acc_groups(int qt) { return qt == CMLD_Q4_K ? 1 : 4; }  // accumulator slots filled per step
__host__ __device__ constexpr int acc_slots(int qt) { return qt == CMLD_Q4_K ? 2 : 4; }
__host__ __device__ constexpr int slot_cols(int qt, int nw) { return qt == CMLD_Q4_K ? 3 * nw : qt == CMLD_Q6_K ? 4 * nw : 2 * nw; }
__host__ __device__ constexpr uint32_t tmem_cols(int qt, int nw) {
  uint32_t c = 32;
  while ((int)c < acc_slots(qt) * slot_cols(qt, nw)) c *= 2;
  return c;
}

struct TcJob {
  const uint8_t *w;
  int32_t rows, first_tile;
  int64_t stride;
  float *y;
  const float *residual;
  int64_t y_stride;
};

struct TcArgs {
  TcJob job[3];
  int32_t n_jobs, w_tiles, m_tiles, nks, batch;
  int32_t a_stages, b_stages;
  int32_t off_b, off_raw, off_bar;
  const uint8_t *pack;
  int32_t *status;
};

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(s32(bar)), "r"(parity)
               : "memory");
  return ok != 0;
}
// Bounded wait.  Gives up when the limit is reached or another role has already given up.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int32_t *status) {
  for (uint32_t i = 0; i < kTcSpin; ++i) {
    if (bar_try(bar, parity)) return true;
    if ((i & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  if (status) atomicExch(status, (int32_t)CMLD_ERR_TIMEOUT);
  return false;
}

__device__ __forceinline__ void cp16(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst_smem, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const uint8_t *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(s32(bar))
               : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand without swizzle: 8 rows x 16 bytes are contiguous; LBO = bytes between the 16-byte chunks along K, SBO =
// bytes between groups of eight rows (descriptor version 1 in bits 46-47).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// kind::i8: D = S32, A and B signed; kind::f16: D = F32, A and B f16; both K-major, M = 128
__device__ __forceinline__ constexpr uint32_t idesc_i8(int n) { return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }
__device__ __forceinline__ constexpr uint32_t idesc_f16(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | (8u << 24); }
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
      "l"(da), "l"(db), "r"(idesc), "r"(0u), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
// tcgen05.ld is asynchronous: its registers are valid only after tcgen05.wait::ld.  Load(s) and wait sit in ONE asm
// statement, so the compiler cannot move a use of the registers between them, and every output is an early clobber: an
// address operand sharing a register with an output of an earlier load in the same statement would be overwritten
// whenever that load's write-back lands first.
__device__ __forceinline__ void tmem_ld8x3(uint32_t t0, int (&a)[8], uint32_t t1, int (&b)[8], uint32_t t2, int (&c)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]), "=&r"(b[0]), "=&r"(b[1]),
        "=&r"(b[2]), "=&r"(b[3]), "=&r"(b[4]), "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7]), "=&r"(c[0]), "=&r"(c[1]), "=&r"(c[2]), "=&r"(c[3]),
        "=&r"(c[4]), "=&r"(c[5]), "=&r"(c[6]), "=&r"(c[7])
      : "r"(t0), "r"(t1), "r"(t2)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8x2(uint32_t t0, int (&a)[8], uint32_t t1, int (&b)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]), "=&r"(b[0]), "=&r"(b[1]),
        "=&r"(b[2]), "=&r"(b[3]), "=&r"(b[4]), "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7])
      : "r"(t0), "r"(t1)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16x2(uint32_t t0, int (&a)[16], uint32_t t1, int (&b)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(a[0]), "=&r"(a[1]), "=&r"(a[2]), "=&r"(a[3]), "=&r"(a[4]), "=&r"(a[5]), "=&r"(a[6]), "=&r"(a[7]),
        "=&r"(a[8]), "=&r"(a[9]), "=&r"(a[10]), "=&r"(a[11]), "=&r"(a[12]), "=&r"(a[13]), "=&r"(a[14]), "=&r"(a[15]),
        "=&r"(b[0]), "=&r"(b[1]), "=&r"(b[2]), "=&r"(b[3]), "=&r"(b[4]), "=&r"(b[5]), "=&r"(b[6]), "=&r"(b[7]),
        "=&r"(b[8]), "=&r"(b[9]), "=&r"(b[10]), "=&r"(b[11]), "=&r"(b[12]), "=&r"(b[13]), "=&r"(b[14]), "=&r"(b[15])
      : "r"(t0), "r"(t1)
      : "memory");
}

__device__ __forceinline__ int tc_tile_job(const TcArgs &a, int t) {
  int j = 0;
  if (a.n_jobs > 1 && t >= a.job[1].first_tile) j = 1;
  if (a.n_jobs > 2 && t >= a.job[2].first_tile) j = 2;
  return j;
}

// ---------------------------------------------------------------- activation packing

// Quantised rows in the global layout (codes | f32 scales | i16 sums of 16) rearranged into records: a warp per row and K step.
__global__ void __launch_bounds__(256) tc5_pack_kernel(const uint8_t *act, int64_t cols, int tiles, uint8_t *rec4, uint8_t *rec6, uint8_t *rec0) {
  const int lane = threadIdx.x & 31, b = blockIdx.y;
  const int64_t ch = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (ch >= cols / 256) return;
  const uint8_t *row = act + b * act_row_stride(cols);
  const uint2 pk = *reinterpret_cast<const uint2 *>(row + ch * 256 + lane * 8);
  const float *scales = reinterpret_cast<const float *>(row + act_scale_off(cols));
  if (rec0) tc5_store_0(pk, scales[ch * 8 + (lane >> 2)], lane, b, ch, tiles, rec0);
  else tc5_store_k(pk, scales[ch], lane, b, ch, tiles, rec4, rec6);
}

// ---------------------------------------------------------------- weight path

// 16-byte chunk c of row r in a weight operand of R rows
template <int R>
__device__ __forceinline__ uint8_t *chunk_of(uint8_t *b, int c, int r) { return b + c * (R * 16) + r * 16; }

__device__ __forceinline__ uint4 mul4(uint4 v, uint32_t s) { return make_uint4(v.x * s, v.y * s, v.z * s, v.w * s); }

// A raw stage is the plain image of the tile's superblocks of one K step: row r at r * 144 (208) bytes, an odd multiple of
// 16, so that lanes reading the same field of consecutive rows hit distinct banks.
// Rows 0..NW-1 of the operand hold s1*q, rows NW..2NW-1 s0*q.  Thread: row r, group pairs jl0 .. jl0 + NJ - 1 (of four).
template <int NW, int NJ>
__device__ __forceinline__ void unpack_q4k(const uint8_t *raw_stage, uint8_t *b, int r, int jl0) {
  const uint8_t *blk = raw_stage + r * 144;
  const uint4 meta = *reinterpret_cast<const uint4 *>(blk);
  // 6-bit scales and mins as bytes (q4_k_scale_min, src/tensor/mod.rs:5997-6006)
  const uint32_t sc03 = meta.y & 0x3f3f3f3fu, sc47 = (meta.w & 0x0f0f0f0fu) | ((meta.y >> 2) & 0x30303030u);
#pragma unroll
  for (int n = 0; n < NJ; ++n) {
    const int j = jl0 + n;  // 64 values: low nibbles are group 2j, high nibbles group 2j + 1
    const uint32_t scw = (j & 2) ? sc47 : sc03;
    const uint32_t sc_lo = (scw >> (16 * (j & 1))) & 0xffu, sc_hi = (scw >> (16 * (j & 1) + 8)) & 0xffu;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint4 w = *reinterpret_cast<const uint4 *>(blk + 16 + 32 * j + 16 * e);
      const uint4 ql = make_uint4(w.x & 0x0f0f0f0fu, w.y & 0x0f0f0f0fu, w.z & 0x0f0f0f0fu, w.w & 0x0f0f0f0fu);
      const uint4 qh = make_uint4((w.x >> 4) & 0x0f0f0f0fu, (w.y >> 4) & 0x0f0f0f0fu, (w.z >> 4) & 0x0f0f0f0fu, (w.w >> 4) & 0x0f0f0f0fu);
      // sc = 8*s1 + s0: bytes s1*q and s0*q stay below 106, so the four bytes of a word multiply at once
      *reinterpret_cast<uint4 *>(chunk_of<2 * NW>(b, 4 * j + e, r)) = mul4(ql, sc_lo >> 3);
      *reinterpret_cast<uint4 *>(chunk_of<2 * NW>(b, 4 * j + e, NW + r)) = mul4(ql, sc_lo & 7u);
      *reinterpret_cast<uint4 *>(chunk_of<2 * NW>(b, 4 * j + 2 + e, r)) = mul4(qh, sc_hi >> 3);
      *reinterpret_cast<uint4 *>(chunk_of<2 * NW>(b, 4 * j + 2 + e, NW + r)) = mul4(qh, sc_hi & 7u);
    }
  }
  if (jl0 == 0) {
    // the mins operand: f16, every min twice (its group of 32 is two sums of 16), and the row's f32 scales
    const uint32_t m[2] = {meta.z & 0x3f3f3f3fu, ((meta.w >> 4) & 0x0f0f0f0fu) | ((meta.z >> 2) & 0x30303030u)};
    uint8_t *p = b + 2 * NW * 256;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t h[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {  // 0x6400 + v is the f16 number 1024 + v
        const uint32_t v = (m[c] >> (8 * x)) & 0x3fu;
        const __half2 hv = __hsub2(__halves2half2(__ushort_as_half((uint16_t)(0x6400u + v)), __ushort_as_half((uint16_t)(0x6400u + v))),
                                   __halves2half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400)));
        h[x] = *reinterpret_cast<const uint32_t *>(&hv);
      }
      *reinterpret_cast<uint4 *>(chunk_of<NW>(p, c, r)) = make_uint4(h[0], h[1], h[2], h[3]);
    }
    float *s = reinterpret_cast<float *>(p + NW * 32);
    s[r] = f16_bits_to_f32((uint16_t)(meta.x & 0xffff));
    s[NW + r] = f16_bits_to_f32((uint16_t)(meta.x >> 16));
  }
}

// prmt in its default mode: a selector nibble with bit 3 set yields the sign of the selected byte replicated (0x00 for the
// codes here, which are below 128).  __byte_perm documents only the three low bits of a nibble.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// Rows 0..NW-1 of the operand hold vh, rows NW..2NW-1 vl.  Thread: row r, half h (128 values), classes 4e .. 4e + 3.
// The 128 values of a half are four quarters of 32; value l' of quarter qd has the 6-bit code (ql[32*(qd&1) + l'] >>
// 4*(qd>>1)) & 15 | ((qh[l'] >> 2*qd) & 3) << 4 and the scale 2*qd + l'/16.  Class l takes from each quarter the values
// l' = l, 8+l, 16+l, 24+l: byte l%4 of the words l/4, 2+l/4 (scale 2qd) and 4+l/4, 6+l/4 (scale 2qd+1), so a thread needs
// the words of one parity only.  Two 16-bit lanes per multiply-add form v + 32768 = sc*q + (32768 - 32*sc), in 28672..36864;
// its low seven bits are vl and bits 7..14 are vh as a signed byte.
template <int NW>
__device__ __forceinline__ void unpack_q6k(const uint8_t *raw_stage, uint8_t *b, int r, int h, int e) {
  const uint8_t *blk = raw_stage + r * 208;
  uint32_t QL[8], QH[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const uint4 v = *reinterpret_cast<const uint4 *>(blk + 64 * h + 16 * s);
    QL[2 * s] = e ? v.y : v.x, QL[2 * s + 1] = e ? v.w : v.z;
  }
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint4 v = *reinterpret_cast<const uint4 *>(blk + 128 + 32 * h + 16 * s);
    QH[2 * s] = e ? v.y : v.x, QH[2 * s + 1] = e ? v.w : v.z;
  }
  const uint2 scw = *reinterpret_cast<const uint2 *>(blk + 192 + 8 * h);
  uint32_t oh[4][4], ol[4][4];  // [class][quarter]
#pragma unroll
  for (int qd = 0; qd < 4; ++qd) {
    uint32_t Q[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const uint32_t lo4 = (QL[4 * (qd & 1) + m] >> (4 * (qd >> 1))) & 0x0f0f0f0fu;
      const uint32_t hi2 = qd < 2 ? (QH[m] << (4 - 2 * qd)) : (QH[m] >> (2 * qd - 4));
      Q[m] = lo4 | (hi2 & 0x30303030u);
    }
    const uint32_t sw = qd < 2 ? scw.x : scw.y;
    const int sa = (int8_t)(sw >> (16 * (qd & 1))), sb = (int8_t)(sw >> (16 * (qd & 1) + 8));
    const uint32_t ba = (uint32_t)(32768 - 32 * sa) * 0x10001u, bb = (uint32_t)(32768 - 32 * sb) * 0x10001u;
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const uint32_t sel = (uint32_t)l | 0x80u | ((uint32_t)(4 + l) << 8) | 0x8000u;  // [x.b, 0, y.b, 0]
      const uint32_t u01 = prmt(Q[0], Q[1], sel) * (uint32_t)sa + ba;
      const uint32_t u23 = prmt(Q[2], Q[3], sel) * (uint32_t)sb + bb;
      ol[l][qd] = __byte_perm(u01, u23, 0x6420) & 0x7f7f7f7fu;
      oh[l][qd] = __byte_perm(u01 >> 7, u23 >> 7, 0x6420);
    }
  }
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const int c = 2 * (4 * e + l) + h;
    *reinterpret_cast<uint4 *>(chunk_of<2 * NW>(b, c, r)) = make_uint4(oh[l][0], oh[l][1], oh[l][2], oh[l][3]);
    *reinterpret_cast<uint4 *>(chunk_of<2 * NW>(b, c, NW + r)) = make_uint4(ol[l][0], ol[l][1], ol[l][2], ol[l][3]);
  }
}

// ---------------------------------------------------------------- the kernel

template <int QT, int NW>
__global__ void __launch_bounds__(tc_threads(QT, NW), 1) gemv_tc5_kernel(const TcArgs a) {
  constexpr int EG = epi_groups(QT, NW), EW = 4 * EG;   // epilogue warps
  constexpr int CW = NW / EG;                           // weight rows of one epilogue thread
  constexpr int MMA_WARP = EW + 4, ACT_WARP = MMA_WARP + 1;
  constexpr int REC = tc5_rec(QT), BB = b_bytes(QT, NW), RB = raw_bytes(QT, NW);
  constexpr int G = acc_groups(QT), NS = acc_slots(QT), SC = slot_cols(QT, NW);
  constexpr uint32_t TCOLS = tmem_cols(QT, NW);
  constexpr int PL = b_planes(QT) * NW * 256;  // bytes of the operand planes
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + a.off_bar);
  uint64_t *a_full = bars, *a_empty = bars + kTcMaxStages, *b_full = bars + 2 * kTcMaxStages, *b_empty = bars + 3 * kTcMaxStages;
  uint64_t *acc_full = bars + 4 * kTcMaxStages, *acc_empty = acc_full + 4;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 4);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  uint8_t *a_ring = smem, *b_ring = smem + a.off_b;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int NA = a.a_stages, NB = a.b_stages, nks = a.nks;
  const int total_tiles = a.w_tiles * a.m_tiles, cta = (int)blockIdx.x, n_ctas = (int)gridDim.x;
  const int n_mine = cta < total_tiles ? (total_tiles - cta + n_ctas - 1) / n_ctas : 0;
  const int total_steps = n_mine * nks;

  if (tid == 0) {
    for (int i = 0; i < kTcMaxStages; ++i) {
      bar_init(&a_full[i], 1);
      bar_init(&a_empty[i], EW);
      bar_init(&b_full[i], 4);
      bar_init(&b_empty[i], EW);
    }
    for (int i = 0; i < 4; ++i) {
      bar_init(&acc_full[i], 1);
      bar_init(&acc_empty[i], EW);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(TCOLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tmem_slot;

  // The epilogue threads hold up to 128 sums each and take registers from the other warpgroups
  // (2 x 128 x 184 + 2 x 128 x 72 = the 512 x 128 of the launch).
  if (tc_threads(QT, NW) == 512) {
    if (warp < EW) asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  }

  if (warp < EW) {
    // ------------------------------------------------ epilogue
    const int wg = warp >> 2, quarter = warp & 3;
    const int m = quarter * 32 + lane;                      // row within the activation tile
    const int col0 = wg * CW;                               // first weight row of this thread
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    int sa = 0, sb = 0, pa = 0, pb = 0, slot = 0, pc = 0;
    bool ok = true;
    for (int it = 0; it < n_mine && ok; ++it) {
      const int t = cta + it * n_ctas, wt = t / a.m_tiles, mt = t % a.m_tiles;
      float acc[CW][QT == CMLD_Q6_K ? 8 : 1];
#pragma unroll
      for (int i = 0; i < CW; ++i)
#pragma unroll
        for (int l = 0; l < (QT == CMLD_Q6_K ? 8 : 1); ++l) acc[i][l] = 0.0f;
      for (int ks = 0; ks < nks; ++ks) {
        const uint8_t *as = a_ring + sa * REC;
        const uint8_t *bs = b_ring + sb * BB;
        const float *xs = reinterpret_cast<const float *>(as + kMR * 256 + tc5_rec_p(QT)) + m;
        const float *ws = reinterpret_cast<const float *>(bs + PL + b_p(QT, NW)) + col0;
        // the record's bytes arrive through the async proxy and the scales of the weights through other warps: each reader
        // observes their barriers itself (both phases completed before the step's MMAs were issued, and neither is re-armed
        // before this warp gives the stages back)
        ok = bar_wait(&a_full[sa], (uint32_t)pa, abort_flag, a.status) && bar_wait(&b_full[sb], (uint32_t)pb, abort_flag, a.status);
        float dd[CW];  // Q6_K: the products of the scales
        const float xd = QT == CMLD_Q8_0 ? 0.0f : *xs;
        if (QT == CMLD_Q6_K) {
#pragma unroll
          for (int i = 0; i < CW; i += 4) {
            const float4 w4 = *reinterpret_cast<const float4 *>(ws + i);
            dd[i] = __fmul_rn(w4.x, xd), dd[i + 1] = __fmul_rn(w4.y, xd);  // src/inference.rs:25545
            dd[i + 2] = __fmul_rn(w4.z, xd), dd[i + 3] = __fmul_rn(w4.w, xd);
          }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
          ok = ok && bar_wait(&acc_full[slot], (uint32_t)pc, abort_flag, a.status);
          // The lanes leave the polling loops at different iterations; tcgen05.ld is a .sync.aligned instruction and must
          // be executed by the whole warp together, so the warp is brought back together here (a diverged warp returned
          // wrong values in the last registers of a load now and then).
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d0 = tbase + lane_base + (uint32_t)(slot * SC + col0);
          if constexpr (QT == CMLD_Q4_K) {
#pragma unroll
            for (int u = 0; u < CW; u += 8) {
              int s1[8], s0[8], pf[8];
              tmem_ld8x3(d0 + u, s1, d0 + NW + u, s0, d0 + 2 * NW + u, pf);
#pragma unroll
              for (int i = 0; i < 8; i += 4) {
                const float4 dw = *reinterpret_cast<const float4 *>(ws + u + i), dm = *reinterpret_cast<const float4 *>(ws + NW + u + i);
                const float dwv[4] = {dw.x, dw.y, dw.z, dw.w}, dmv[4] = {dm.x, dm.y, dm.z, dm.w};
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                  // sumf = fma(-dmin, P, sumf); sumf = fma(d, S, sumf) with d = xd*dw, dmin = xd*dminw (refmath.rs:529, :560)
                  float &o = acc[u + i + x][0];
                  o = __fmaf_rn(-__fmul_rn(xd, dmv[x]), __int_as_float(pf[i + x]), o);
                  o = __fmaf_rn(__fmul_rn(xd, dwv[x]), (float)(8 * s1[i + x] + s0[i + x]), o);
                }
              }
            }
          } else if constexpr (QT == CMLD_Q6_K) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              // as many columns per wait as there are: tensor memory's latency, not its rate, is what a wait costs
              int vh[CW], vl[CW];
              if constexpr (CW == 16) tmem_ld16x2(d0 + 2 * c * NW, vh, d0 + (2 * c + 1) * NW, vl);
              else tmem_ld8x2(d0 + 2 * c * NW, vh, d0 + (2 * c + 1) * NW, vl);
#pragma unroll
              for (int i = 0; i < CW; ++i) {
                // sums[l] += (d*xd) * (float)aux[l], each of the eight lanes on its own (independent chains)
                float &o = acc[i][2 * g + c];
                o = __fadd_rn(o, __fmul_rn(dd[i], (float)(128 * vh[i] + vl[i])));
              }
            }
          } else {
            const float x0 = xs[(2 * g) * kMR], x1 = xs[(2 * g + 1) * kMR];
#pragma unroll
            for (int u = 0; u < CW; u += 8) {
              int i0[8], i1[8];
              tmem_ld8x2(d0 + u, i0, d0 + NW + u, i1);
#pragma unroll
              for (int i = 0; i < 8; i += 4) {
                const float4 w0 = *reinterpret_cast<const float4 *>(ws + (2 * g) * NW + u + i), w1 = *reinterpret_cast<const float4 *>(ws + (2 * g + 1) * NW + u + i);
                const float w0v[4] = {w0.x, w0.y, w0.z, w0.w}, w1v[4] = {w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int x = 0; x < 4; ++x) {  // src/inference.rs:26198
                  float &o = acc[u + i + x][0];
                  o = __fadd_rn(o, __fmul_rn(__fmul_rn((float)i0[i + x], w0v[x]), x0));
                  o = __fadd_rn(o, __fmul_rn(__fmul_rn((float)i1[i + x], w1v[x]), x1));
                }
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) bar_arrive(&acc_empty[slot]);
          if (++slot == NS) slot = 0, pc ^= 1;
        }
        if (!ok) break;
        // The stages go back AFTER the step's f32 work, so that every value read from them has been consumed by an
        // instruction: a shared-memory load that is merely issued is not ordered before the arrival, and the next bulk copy
        // into the stage (async proxy) overtook such loads now and then.  The proxy fence orders this thread's generic
        // reads before async-proxy writes that follow the arrival.  (The step's MMAs have read both stages: the last
        // accumulator barrier of the step was committed behind them.)
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          bar_arrive(&a_empty[sa]);
          bar_arrive(&b_empty[sb]);
        }
        if (++sa == NA) sa = 0, pa ^= 1;
        if (++sb == NB) sb = 0, pb ^= 1;
      }
      if (!ok) break;
      const TcJob &J = a.job[tc_tile_job(a, wt)];
      const int b = mt * kMR + m, row0 = (wt - J.first_tile) * NW + col0;
      if (b < a.batch) {
        float *y = J.y + (int64_t)b * J.y_stride + row0;
        const float *res = J.residual ? J.residual + (int64_t)b * J.y_stride + row0 : nullptr;
        const bool vec = row0 + CW <= J.rows && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(res)) & 15) == 0;
#pragma unroll
        for (int i = 0; i < CW; i += 4) {
          float v[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            v[x] = acc[i + x][0];
            if (QT == CMLD_Q6_K) {
              v[x] = 0.0f;  // 0 + sums[0] + ... + sums[7] (src/inference.rs:25578-25580)
#pragma unroll
              for (int l = 0; l < 8; ++l) v[x] = __fadd_rn(v[x], acc[i + x][l]);
            }
          }
          if (vec) {
            if (res) {
              const float4 r4 = __ldcg(reinterpret_cast<const float4 *>(res + i));
              v[0] = __fadd_rn(r4.x, v[0]), v[1] = __fadd_rn(r4.y, v[1]), v[2] = __fadd_rn(r4.z, v[2]), v[3] = __fadd_rn(r4.w, v[3]);
            }
            *reinterpret_cast<float4 *>(y + i) = make_float4(v[0], v[1], v[2], v[3]);
          } else {
#pragma unroll
            for (int x = 0; x < 4; ++x)
              if (row0 + i + x < J.rows) y[i + x] = res ? __fadd_rn(__ldcg(res + i + x), v[x]) : v[x];
          }
        }
      }
    }
  } else if (warp < MMA_WARP) {
    // ------------------------------------------------ weight path
    const int tu = tid - EW * 32, wu = tu >> 5;
    constexpr int SEG = QT == CMLD_Q8_0 ? 1 : kq_bytes(QT) / 16;  // 16-byte pieces of a row (Q8_0: its scales of the step)
    constexpr int NP = (NW * SEG + 127) / 128;
    constexpr int RS = kLoadAhead + 1;
    uint8_t *raw = smem + a.off_raw;
    // state of the loads: the step they have reached, its tile, K step and raw stage
    int lq = 0, l_it = 0, l_ks = 0, l_stage = 0;
    const uint8_t *l_base = nullptr;
    int l_left = 0;
    int64_t l_stride = 0;
    auto open_tile = [&]() {
      if (l_it >= n_mine) return;
      const int wt = (cta + l_it * n_ctas) / a.m_tiles;
      const TcJob &J = a.job[tc_tile_job(a, wt)];
      const int r0 = (wt - J.first_tile) * NW;
      l_base = J.w + (int64_t)r0 * J.stride;
      l_left = J.rows - r0 - 1;  // last row that exists
      l_stride = J.stride;
    };
    open_tile();
    bool ok = true;
    auto load_step = [&]() {
      if (lq < total_steps && ok) {
        if (QT == CMLD_Q8_0) {
          // codes are int8 in K order already: straight into the operand layout (its stage must have been given back).  A
          // warp instruction covers 8 rows x 4 chunks: 64 contiguous bytes per row from memory, four contiguous 128-byte
          // pieces in shared memory.
          const int st = lq % NB;
          if (lq >= NB) ok = bar_wait(&b_empty[st], (uint32_t)((lq / NB - 1) & 1), abort_flag, a.status);
          if (ok) {
            const uint32_t dst = s32(b_ring + st * BB);
            const int r8 = lane & 7, cc = lane >> 3;
#pragma unroll
            for (int j = 0; j < NW / 8; ++j) {
              const int rr = 8 * ((NW / 32) * wu + (j >> 2)) + r8, c = 4 * (j & 3) + cc;
              cp16(dst + c * (NW * 16) + rr * 16, l_base + (int64_t)min(rr, l_left) * l_stride + (int64_t)l_ks * 256 + 16 * c);
            }
            if (tu < NW) cp16(s32(raw + l_stage * RB) + tu * 16, l_base + (int64_t)min(tu, l_left) * l_stride + (int64_t)nks * 256 + 16 * l_ks);
          }
        } else {
          const uint32_t dst = s32(raw + l_stage * RB);
#pragma unroll
          for (int j = 0; j < NP; ++j) {
            const int ci = tu + 128 * j;
            if (ci < NW * SEG) {
              const int rr = ci / SEG, sg = ci - rr * SEG;
              cp16(dst + ci * 16, l_base + (int64_t)min(rr, l_left) * l_stride + (int64_t)l_ks * kq_bytes(QT) + 16 * sg);
            }
          }
          if (QT == CMLD_Q6_K && tu < NW)  // the word that holds this step's f16 scale
            cp4(dst + NW * 208 + 4 * tu, l_base + (int64_t)min(tu, l_left) * l_stride + (int64_t)nks * 208 + 4 * (l_ks >> 1));
        }
        if (tu < NW && l_ks + kTcPrefetchAhead < nks) {  // a later step's bytes into L2, one request per line
          const uint8_t *pf = l_base + (int64_t)min(tu, l_left) * l_stride + (int64_t)(l_ks + kTcPrefetchAhead) * kq_bytes(QT);
          asm volatile("prefetch.global.L2 [%0];" ::"l"(pf));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(pf + kq_bytes(QT) - 16));
        }
      }
      cp_commit();
      ++lq;
      if (++l_ks == nks) {
        l_ks = 0;
        ++l_it;
        open_tile();
      }
      if (++l_stage == RS) l_stage = 0;
    };
    for (int q = 0; q < kLoadAhead; ++q) load_step();
    int u_ks = 0, stage = 0;
    for (int q = 0; q < total_steps; ++q) {
      const int st = q % NB;
      uint8_t *b = b_ring + st * BB;
      cp_wait<kLoadAhead - 1>();  // this thread's pieces of step q have landed
      if (QT != CMLD_Q8_0 && q >= NB && ok) ok = bar_wait(&b_empty[st], (uint32_t)((q / NB - 1) & 1), abort_flag, a.status);
      // One barrier per step over the 128 threads: everybody's pieces of step q are visible, everybody is done
      // reading the stage that the next load overwrites, and the verdict of the bounded waits is shared.
      uint32_t all_ok;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.and.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(all_ok)
                   : "r"(ok ? 1u : 0u), "r"(1)
                   : "memory");
      ok = all_ok != 0;
      if (!ok) break;
      load_step();
      const uint8_t *raw_stage = raw + stage * RB;
      if (QT == CMLD_Q4_K) {
        if (NW == 64) unpack_q4k<NW, 2>(raw_stage, b, tu & 63, 2 * (tu >> 6));
        else unpack_q4k<NW, 1>(raw_stage, b, lane, wu);
      } else if (QT == CMLD_Q6_K) {
        unpack_q6k<NW>(raw_stage, b, lane, wu & 1, wu >> 1);
        if (tu < NW) reinterpret_cast<float *>(b + PL)[tu] = f16_bits_to_f32(reinterpret_cast<const uint16_t *>(raw_stage + NW * 208)[2 * tu + (u_ks & 1)]);
      } else {
        float *s = reinterpret_cast<float *>(b + PL);
        for (int i = tu; i < NW * 8; i += 128) s[i] = f16_bits_to_f32(reinterpret_cast<const uint16_t *>(raw_stage)[(i % NW) * 8 + i / NW]);
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) bar_arrive(&b_full[st]);
      if (++stage == RS) stage = 0;
      if (++u_ks == nks) u_ks = 0;
    }
    cp_wait<0>();
  } else if (warp == ACT_WARP) {
    // ------------------------------------------------ activation records
    if (lane == 0) {
      for (int q = 0; q < total_steps; ++q) {
        const int st = q % NA;
        if (q >= NA && !bar_wait(&a_empty[st], (uint32_t)((q / NA - 1) & 1), abort_flag, a.status)) break;
        const int mt = (cta + (q / nks) * n_ctas) % a.m_tiles;
        const uint8_t *src = a.pack + ((int64_t)(q % nks) * a.m_tiles + mt) * REC;
        bar_expect_tx(&a_full[st], (uint32_t)REC);
        bulk_load(s32(a_ring + st * REC), src, REC, &a_full[st]);
      }
    }
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------ MMA issue
    if (lane == 0) {
      int sa = 0, sb = 0, pa = 0, pb = 0, slot = 0, pc = 0;
      bool ok = true;
      for (int q = 0; q < total_steps && ok; ++q) {
        if (!bar_wait(&a_full[sa], (uint32_t)pa, abort_flag, a.status)) break;
        if (!bar_wait(&b_full[sb], (uint32_t)pb, abort_flag, a.status)) break;
        const uint32_t a_addr = s32(a_ring + sa * REC), b_addr = s32(b_ring + sb * BB);
        constexpr int BR = b_planes(QT) * NW;  // rows of the weight operand
#pragma unroll
        for (int g = 0; g < G; ++g) {
          // a slot is free when the epilogue has given back its previous contents (the first round needs no wait)
          if (q * G + g >= NS && !bar_wait(&acc_empty[slot], (uint32_t)(pc ^ 1), abort_flag, a.status)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d0 = tbase + (uint32_t)(slot * SC);
          if (QT == CMLD_Q4_K) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              mma_i8(d0, smem_desc(a_addr + j * 256, 128, 2048), smem_desc(b_addr + j * 2 * (BR * 16), BR * 16, 128), idesc_i8(BR), j > 0);
            mma_f16(d0 + 2 * NW, smem_desc(a_addr + kMR * 256, 128, 256), smem_desc(b_addr + PL, NW * 16, 128), idesc_f16(NW));
          } else {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int j = 2 * g + c;
              mma_i8(d0 + c * BR, smem_desc(a_addr + j * 256, 128, 2048), smem_desc(b_addr + j * 2 * (BR * 16), BR * 16, 128), idesc_i8(BR), false);
            }
          }
          mma_commit(&acc_full[slot]);
          if (++slot == NS) slot = 0, pc ^= 1;
        }
        if (++sa == NA) sa = 0, pa ^= 1;
        if (++sb == NB) sb = 0, pb ^= 1;
      }
    }
  }
  cp_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(TCOLS) : "memory");
  }
}

int g_tc_sms = 0;

}  // namespace

static bool tc5_qt_ok(int qt) { return qt == CMLD_Q4_K || qt == CMLD_Q6_K || qt == CMLD_Q8_0; }
// Bytes of packed activation records a step of `batch` rows needs for `cols` columns of any type.
int64_t gemv_tc5_pack_bytes(int64_t cols, int32_t batch) {
  return cols / 256 * ((batch + kMR - 1) / kMR) * (int64_t)tc5_rec(CMLD_Q4_K);
}

bool gemv_tc5_fits(const GemvJob *jobs, int n_jobs, int32_t batch) {
  if (n_jobs < 1 || n_jobs > 3 || batch < 1) return false;
  for (int i = 0; i < n_jobs; ++i) {
    if (!tc5_qt_ok(jobs[i].qt) || jobs[i].cols != jobs[0].cols || jobs[i].cols % 256 != 0 || jobs[i].cols < 256 || jobs[i].rows < 1) return false;
  }
  return true;
}

template <int QT, int NW>
static int32_t launch_tc(TcArgs &a, const GemvJob *jobs, cudaStream_t s) {
  static SmemLimit limit;
  CMLD_TRY(allow_smem(limit, gemv_tc5_kernel<QT, NW>, 227 * 1024));
  int tiles = 0;
  for (int i = 0; i < a.n_jobs; ++i) {
    TcJob &J = a.job[i];
    J.w = jobs[i].w;
    J.rows = (int32_t)jobs[i].rows;
    J.stride = jobs[i].stride;
    J.y = jobs[i].y;
    J.residual = jobs[i].residual;
    J.y_stride = jobs[i].y_stride;
    J.first_tile = tiles;
    tiles += (int32_t)((jobs[i].rows + NW - 1) / NW);
  }
  a.w_tiles = tiles;
  constexpr int bar_bytes = 8 * (4 * kTcMaxStages + 8) + 16, a_stages = 3;
  constexpr int left = 227 * 1024 - bar_bytes - a_stages * tc5_rec(QT) - ring_bytes(QT, NW);
  constexpr int b_stages = std::min(kTcMaxStages, left / b_bytes(QT, NW));
  // Q8_0 loads go straight into the operand ring: it must hold more than the steps that are loaded ahead, or a load would
  // wait for a step that is not yet complete.
  static_assert(b_stages >= 2 && (QT != CMLD_Q8_0 || b_stages > kLoadAhead), "shared memory");
  a.a_stages = a_stages;
  a.b_stages = b_stages;
  a.off_b = a_stages * tc5_rec(QT);
  a.off_raw = a.off_b + b_stages * b_bytes(QT, NW);
  a.off_bar = (a.off_raw + ring_bytes(QT, NW) + 15) & ~15;
  const int grid = std::min(tiles * a.m_tiles, g_tc_sms);
  gemv_tc5_kernel<QT, NW><<<grid, tc_threads(QT, NW), a.off_bar + bar_bytes, s>>>(a);
  CMLD_CUDA(cudaGetLastError());
  return CMLD_OK;
}

// Matrices of ONE type; `pack`: their records.
static int32_t launch_tc5_qt(const GemvJob *jobs, int n_jobs, int32_t batch, const uint8_t *pack, int32_t *status, cudaStream_t s) {
  const int qt = jobs[0].qt;
  TcArgs a{};
  a.n_jobs = n_jobs;
  a.nks = (int32_t)(jobs[0].cols / 256);
  a.batch = batch;
  a.m_tiles = (batch + kMR - 1) / kMR;
  a.pack = pack;
  a.status = status;
  // Tiles of 64 weight rows, or of 32 where those leave the last wave of CTAs emptier.  A tile of 32 takes about 0.6 of the time of
  // one of 64 (it repeats the step's hand-offs for half of the rows), hence 3 rounds against 5.  Us with 32 | 64: Q4_K 28672 x 4096, 512
  // rows, 383 | 276; Q4_K 4096 x 4096 67 | 48, and at 128 rows, one round either way, 21.8 | 26.9; Q8_0 2048 x 8192 at 512 rows 110 | 85,
  // at 128 rows 58 | 84; Q8_0 3072 x 2048 at 512 rows 46.2 | 48.6.  The rule takes the faster one in each.
  auto rounds = [&](int nw) {
    int64_t t = 0;
    for (int i = 0; i < n_jobs; ++i) t += (jobs[i].rows + nw - 1) / nw;
    return (t * a.m_tiles + g_tc_sms - 1) / g_tc_sms;
  };
  const bool wide = rounds(64) * 5 <= rounds(32) * 3;
  int32_t rc;
  if (qt == CMLD_Q4_K) rc = wide ? launch_tc<CMLD_Q4_K, 64>(a, jobs, s) : launch_tc<CMLD_Q4_K, 32>(a, jobs, s);
  else if (qt == CMLD_Q6_K) rc = launch_tc<CMLD_Q6_K, 32>(a, jobs, s);
  else rc = wide ? launch_tc<CMLD_Q8_0, 64>(a, jobs, s) : launch_tc<CMLD_Q8_0, 32>(a, jobs, s);
  return rc;
}

int32_t launch_tc5_pack(const uint8_t *act, int64_t cols, int32_t batch, uint8_t *rec4, uint8_t *rec6, uint8_t *rec0, cudaStream_t s) {
  // (grid.y, the rows, is at most 65535: the callers' passes are of 2048)
  tc5_pack_kernel<<<dim3((unsigned)((cols / 256 + 7) / 8), (unsigned)batch), 256, 0, s>>>(act, cols, (batch + kMR - 1) / kMR, rec4, rec6, rec0);
  CMLD_CUDA(cudaGetLastError());
  return CMLD_OK;
}

// The records: rec4 for Q4_K matrices, rec6 for Q6_K, rec0 for Q8_0 (those of the types that occur), gemv_tc5_pack_bytes(cols, batch)
// each.  Matrices of different types are served by one launch per type.  CMLD_ERR_UNSUPPORTED (no message) when the shapes do not fit.
int32_t launch_gemv_tc5(const GemvJob *jobs, int n_jobs, int32_t batch, const uint8_t *rec4, const uint8_t *rec6, const uint8_t *rec0,
                        int32_t *status, cudaStream_t s, int64_t *launches) {
  if (!gemv_tc5_fits(jobs, n_jobs, batch)) return CMLD_ERR_UNSUPPORTED;
  if (g_tc_sms == 0) {
    int dev = 0;
    CMLD_CUDA(cudaGetDevice(&dev));
    CMLD_CUDA(cudaDeviceGetAttribute(&g_tc_sms, cudaDevAttrMultiProcessorCount, dev));
  }
  bool done[3] = {false, false, false};
  for (int i = 0; i < n_jobs; ++i) {
    if (done[i]) continue;
    const int qt = jobs[i].qt;
    GemvJob same[3];
    int n = 0;
    for (int k = i; k < n_jobs; ++k)
      if (!done[k] && jobs[k].qt == qt) {
        same[n++] = jobs[k];
        done[k] = true;
      }
    const uint8_t *rec = qt == CMLD_Q4_K ? rec4 : qt == CMLD_Q6_K ? rec6 : rec0;
    if (!rec) return fail(CMLD_ERR_INVALID, "gemv: activation records missing");
    CMLD_TRY(launch_tc5_qt(same, n, batch, rec, status, s));
    if (launches) *launches += 1;
  }
  return CMLD_OK;
}

}  // namespace cmld
