// Quantised matrix products of a few activation rows (decode steps of several sequences, short prompt steps), with every f32
// operation in the order of the CPU path, so that a row's result is bit-identical to the one-row kernels'.
//
// Weights go from memory into the operand registers of mma.m16n8k32 without a stop: a warp copies the wire bytes of 16 weight
// rows x one unit of columns (a superblock; 128 columns of Q8_0) into a private ring by cp.async, unpacks them in the layout of
// operand A, multiplies them by the activation records (rows_record.cuh; operand B, eight rows at a time) and has the integer parts
// of the reference's dots in its own registers, where the f32 steps follow:
//   Q4_K (src/diffusion_gemma/refmath.rs:504-562): S = sum_g sc_g * (q.y)_g, one MMA and one multiply-add per group of 32 (the
//     high nibbles stay in place, as 16 q, and the low groups' scales take a factor of 16; 16 S < 2^29); P = sum_g min_g * bsum_g is
//     one f16 MMA (every partial sum below 2^24: exact in f32); acc = fma(-(xd*dmin), P, acc); acc = fma(xd*d, S, acc).
//   Q6_K (src/inference.rs:25545-25581): eight accumulators by index mod 8; MMA l takes the columns of class l.  The scaled codes
//     sc*(q-32) = 256*vh + vl enter as a signed and an unsigned 8-bit operand.
//   Q8_0 (src/inference.rs:26191-26199): acc += ((float)isum * ws) * xs, an MMA per block.
// An accumulator that starts at the bits of 1.5*2^23 is, read as f32, that number plus the sum, exactly (|sum| < 2^22): one
// subtraction instead of a conversion.
//
// Two forms share this:
//   rows_whole_kernel  a warp walks a tile of 16 weight rows, its sums stay in its registers; the step's records lie in shared
//                      memory.  For matrices of one type with five tiles per SM or more whose records leave room for two ring stages
//                      of every warp; of Q6_K, whose sums take the registers, at most eight activation rows.  (At the 128 registers of
//                      512 threads Q6_K and 25 to 32 rows of Q4_K spill 88 and 48 bytes.)
//   rows_split_kernel  sixteen warps share a tile, a warp per unit, and hand the f32 terms of a pass (sixteen units) through shared
//                      memory to four warps that add them in block order, a thread per output.  For matrices whose tiles are too few
//                      to give every warp one (4096 rows: 1.7 tiles per SM).  Their operand B comes from L2, asked for one exchange
//                      ahead.  A launch may hold Q4_K and Q6_K matrices, on CTAs of their own.  All that the other form does not take.
//
// Measured, us per launch (records from quantised rows included, 2.3; weights beyond L2): the staged kernel at 3 and 6 rows and the tcgen05
// one (the rows four times over as its 128-row operand A) at 16 and 32 | here:
//   rows                       3              6             16             32
//   Q4_K 28672 x 4096     27.9 | 19.7    64.6 | 19.7    67.1 | 23.4    68.3 | 35.3
//   Q4_K  4096 x 4096      8.4 |  7.9    16.3 |  7.9    20.4 |  9.4    20.5 | 11.7
//   Q6_K  4096 x 14336    33.6 | 24.6    65.9 | 24.6    81.2 | 33.0    81.4 | 47.7
//   Q8_0 16384 x 2048     26.0 | 11.3    48.3 | 11.3    35.2 | 13.4    35.3 | 19.6
// What bounds it: neither memory (a launch whose weights lie in L2 is 1.3 us shorter) nor one unit of the SM: at eight rows a warp
// spends 270 instructions on a Q4_K unit and 850 on a Q6_K one (340 of them unpacking, at two cycles each), three or four warps a
// scheduler, half of the issue slots used; at 32 rows the MMAs (8 cycles each) and the multiply-adds behind them come to the same.
// Tried and slower: warps that pass the running sums on from unit to unit instead of the terms (600 cycles a hand-over: Q6_K 27 -> 39
// us), the multiplying warps adding the terms themselves between two barriers (31 us) or fetching a weight row each (29.5 us), one bulk
// copy per weight row and unit in the whole form (the sixteen copies are issued one after another: 20 -> 28 us).
#include "rows_record.cuh"

namespace cmld {

namespace {

constexpr int kWarps = 16;               // that multiply
constexpr int kSplitWarps = kWarps + 4;  // split form: and four that add up the terms
constexpr int kSplitThreads = kSplitWarps * 32;
constexpr int kSlice = 2048;  // a warp's f32 terms of one exchange: 128 outputs x 16 bytes
constexpr int kMagicBits = 0x4B400000;
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23, the number with these bits
constexpr int kSmemMax = 226 * 1024;
constexpr int kMaxStages = 4;
constexpr uint32_t kRowsSpin = 1u << 22;  // polls after which a wait gives up

// a weight row of one unit in the ring: the wire bytes, padded to an odd multiple of 32 (Q6_K: with the word that holds the f16
// scale), so that the eight rows x four lanes of a load meet distinct banks
__host__ __device__ constexpr int unit_bytes(int qt) { return qt == CMLD_Q4_K ? 144 : qt == CMLD_Q6_K ? 208 : 128; }  // of a row, without Q6_K's and Q8_0's scales
__host__ __device__ constexpr int raw_pitch(int qt) { return qt == CMLD_Q6_K ? 224 : 160; }
__host__ __device__ constexpr int raw_bytes(int qt) { return 16 * raw_pitch(qt); }

struct RowsJob {
  const uint8_t *w;
  int32_t qt, rows, units, first_tile;
  int64_t stride;
  float *y;
  const float *residual;
  int64_t y_stride;
  const uint8_t *rec;  // the records of this type
};

struct RowsArgs {
  RowsJob job[3];
  int32_t n_jobs, tiles, batch;
  int32_t tiles0, ctas0;  // split form: the tiles of the first type (Q4_K before Q6_K) and the CTAs that take them
  int32_t stages, stage_bytes;  // of the CTA's ring (split form), of a warp's (whole form)
  int32_t bufs;                 // split form: exchange buffers
  int32_t off_ring, off_sums;
  int32_t lose_one;             // split form, a self-test: the terms' barriers expect an arrival that never comes
  int32_t *status;
};

__device__ __forceinline__ uint32_t s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp8(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all groups but the last `stages` - 2 have landed
__device__ __forceinline__ void cp_wait_stages(int stages) {
  if (stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
  else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else asm volatile("cp.async.wait_group 2;" ::: "memory");
}

__device__ __forceinline__ void mma_s8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void mma_u8(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, int c) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%4,%5}, {%6,%7}, {%8,%8,%8,%8};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {  // a selector nibble with bit 3 set: the byte's sign
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// ---------------------------------------------------------------- weights

// A lane's part of copying 16 rows of one unit into a ring stage: chunk i lies `from[i]` behind the tile's first row and goes to
// `to[i]`; of the last Q6_K chunk the upper lanes have none.
template <int QT>
struct RawCopy {
  static constexpr int SEG = unit_bytes(QT) / 16, N = (16 * SEG + 31) / 32;
  int from[N], to[N], scale;
  // last: the tile's last row that exists
  __device__ __forceinline__ void place(int last, int64_t stride, int units, int lane) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int ci = min(lane + 32 * i, 16 * SEG - 1), r = ci / SEG, sg = ci - r * SEG;
      from[i] = min(r, last) * (int)stride + sg * 16;
      to[i] = r * raw_pitch(QT) + sg * 16;
    }
    scale = min(lane & 15, last) * (int)stride + units * unit_bytes(QT);
  }
  __device__ __forceinline__ void copy(uint32_t dst, const uint8_t *base, int unit, int lane) const {
    const uint8_t *src = base + (int64_t)unit * unit_bytes(QT);
#pragma unroll
    for (int i = 0; i < N; ++i) cp16(dst + to[i], src + from[i]);  // (a chunk that does not exist: the last one once more)
    if (QT != CMLD_Q4_K && lane < 16) {
      const uint32_t d = dst + lane * raw_pitch(QT) + unit_bytes(QT);
      if (QT == CMLD_Q6_K) cp4(d, base + scale + 4 * (unit >> 1));  // the word with this unit's f16
      else cp8(d, base + scale + 8 * unit);
    }
  }
};

// Lane (g, t) holds of rows g and g + 8 the operand bytes its place in the MMA wants.
struct Q4Unit {
  uint32_t c[4][4];   // [pair of groups of 32]: the even group in the low nibbles, the odd one in the high ones
  int sc[2][8];       // [row][group], the even groups' times 16
  uint32_t m[2];      // mins of groups 2t, 2t + 1 as f16
  float d[2], dm[2];
};
template <int P>
__device__ __forceinline__ void unpack_head(Q4Unit &u, const uint8_t *raw, const uint8_t *, int g, int t) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint8_t *blk = raw + (g + 8 * r) * P;
    const uint4 meta = *reinterpret_cast<const uint4 *>(blk);
    u.d[r] = f16_bits_to_f32((uint16_t)(meta.x & 0xffff));
    u.dm[r] = f16_bits_to_f32((uint16_t)(meta.x >> 16));
    // 6-bit scales and mins as bytes (q4_k_scale_min, src/tensor/mod.rs:5997-6006)
    const uint32_t sc[2] = {meta.y & 0x3f3f3f3fu, (meta.w & 0x0f0f0f0fu) | ((meta.y >> 2) & 0x30303030u)};
    const uint32_t mn = t < 2 ? meta.z & 0x3f3f3f3fu : ((meta.w >> 4) & 0x0f0f0f0fu) | ((meta.z >> 2) & 0x30303030u);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t even = (sc[h] << 4) & 0x0ff00ff0u, odd = (sc[h] >> 8) & 0x00ff00ffu;
      u.sc[r][4 * h] = (int)(even & 0xffffu), u.sc[r][4 * h + 2] = (int)(even >> 16);
      u.sc[r][4 * h + 1] = (int)(odd & 0xffffu), u.sc[r][4 * h + 3] = (int)(odd >> 16);
    }
    // 0x6400 + v is the f16 number 1024 + v
    const uint32_t hv = prmt(mn, 0x64646464u, t & 1 ? 0x4342u : 0x4140u);
    const __half2 k = __halves2half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400));
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&hv), k);
    u.m[r] = *reinterpret_cast<const uint32_t *>(&v);
  }
}
template <int P>
__device__ __forceinline__ void unpack_codes(Q4Unit &u, const uint8_t *raw, int g, int t, int) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint8_t *blk = raw + (g + 8 * r) * P;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint2 w = *reinterpret_cast<const uint2 *>(blk + 16 + 32 * j + 8 * t);
      u.c[j][r] = w.x, u.c[j][2 + r] = w.y;
    }
  }
}

struct Q6Unit {
  uint32_t hi[4][4], lo[4][4];  // of four classes: [class][operand register]
  int sc[2][4];
  float d[2];
};
template <int P>
__device__ __forceinline__ void unpack_head(Q6Unit &s, const uint8_t *raw, const uint8_t *scales, int g, int t) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint8_t *blk = raw + (g + 8 * r) * P;
    s.d[r] = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(scales + (g + 8 * r) * P));
    const uint2 w = *reinterpret_cast<const uint2 *>(blk + 192 + 8 * (t >> 1));  // groups 2q + c of the half
    const int sh = 8 * (t & 1);
    s.sc[r][0] = (int8_t)(w.x >> sh), s.sc[r][1] = (int8_t)(w.x >> (16 + sh));
    s.sc[r][2] = (int8_t)(w.y >> sh), s.sc[r][3] = (int8_t)(w.y >> (16 + sh));
  }
}
// Classes 4e .. 4e + 3.  The 128 values of a half are four quarters of 32: value l' of quarter q has the code (ql[32*(q&1) + l'] >>
// 4*(q>>1)) & 15 | ((qh[l'] >> 2q) & 3) << 4.  Of the lane's 16 values of a quarter, class l takes l and l + 8: byte l % 4 of
// the words e and e + 2.  Two 16-bit lanes per multiply-add form v + 32768 = sc*q + (32768 - 32*sc), in 28672..36864.
template <int P>
__device__ __forceinline__ void unpack_codes(Q6Unit &u, const uint8_t *raw, int g, int t, int e) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint8_t *blk = raw + (g + 8 * r) * P + 16 * (t & 1);
    const uint4 v0 = *reinterpret_cast<const uint4 *>(blk + 64 * (t >> 1)), v1 = *reinterpret_cast<const uint4 *>(blk + 64 * (t >> 1) + 32);
    const uint4 vh = *reinterpret_cast<const uint4 *>(blk + 128 + 32 * (t >> 1));
    const uint32_t ql[2][2] = {{e ? v0.y : v0.x, e ? v0.w : v0.z}, {e ? v1.y : v1.x, e ? v1.w : v1.z}};
    const uint32_t qh[2] = {e ? vh.y : vh.x, e ? vh.w : vh.z};
    uint32_t c[4][4];  // [quarter][class]: 16-bit lanes of the values l and l + 8
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t w[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const uint32_t low = ql[q & 1][x] >> (4 * (q >> 1)), high = q < 2 ? qh[x] << (4 - 2 * q) : qh[x] >> (2 * q - 4);
        w[x] = (low & 0x0f0f0f0fu) | (high & 0x30303030u);
      }
      const uint32_t bias = 0x80008000u - 32u * 0x10001u * (uint32_t)u.sc[r][q];
#pragma unroll
      for (int l = 0; l < 4; ++l) c[q][l] = prmt(w[0], w[1], (uint32_t)l | 0x80u | ((uint32_t)(4 + l) << 8) | 0x8000u) * (uint32_t)u.sc[r][q] + bias;
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      u.lo[l][r] = __byte_perm(c[0][l], c[1][l], 0x6420), u.lo[l][2 + r] = __byte_perm(c[2][l], c[3][l], 0x6420);
      u.hi[l][r] = __byte_perm(c[0][l], c[1][l], 0x7531) ^ 0x80808080u, u.hi[l][2 + r] = __byte_perm(c[2][l], c[3][l], 0x7531) ^ 0x80808080u;
    }
  }
}

struct Q8Unit {
  uint32_t a[4][4];
  float ws[2][4];
};
template <int P>
__device__ __forceinline__ void unpack_head(Q8Unit &u, const uint8_t *, const uint8_t *scales, int g, int) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint2 s = *reinterpret_cast<const uint2 *>(scales + (g + 8 * r) * P);
    u.ws[r][0] = f16_bits_to_f32((uint16_t)(s.x & 0xffff)), u.ws[r][1] = f16_bits_to_f32((uint16_t)(s.x >> 16));
    u.ws[r][2] = f16_bits_to_f32((uint16_t)(s.y & 0xffff)), u.ws[r][3] = f16_bits_to_f32((uint16_t)(s.y >> 16));
  }
}
template <int P>
__device__ __forceinline__ void unpack_codes(Q8Unit &u, const uint8_t *raw, int g, int t, int) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint8_t *blk = raw + (g + 8 * r) * P;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint2 w = *reinterpret_cast<const uint2 *>(blk + 32 * k + 8 * t);
      u.a[k][r] = w.x, u.a[k][2 + r] = w.y;
    }
  }
}

template <int QT>
struct Sums {  // of one output, between passes of the split form
  typedef float type;
};
template <>
struct Sums<CMLD_Q6_K> {
  typedef float4 type;
};
template <int QT>
struct UnitOf {
  typedef Q8Unit type;
};
template <>
struct UnitOf<CMLD_Q4_K> {
  typedef Q4Unit type;
};
template <>
struct UnitOf<CMLD_Q6_K> {
  typedef Q6Unit type;
};

// ---------------------------------------------------------------- products of one unit and eight activation rows

// A lane's part of a record.  From shared memory it is read where it is used; from global memory (L2) it is asked for one exchange ahead.
struct Operand {
  uint4 c[4];
  uint2 p;
  float2 x[4];
};
template <bool GLOBAL, typename T>
__device__ __forceinline__ T fetch(const uint8_t *p) {
  if (GLOBAL) return __ldcg(reinterpret_cast<const T *>(p));
  return *reinterpret_cast<const T *>(p);
}
template <int QT, bool GLOBAL>
__device__ __forceinline__ void fetch_operand(Operand &o, const uint8_t *rec, int half, int lane) {
#pragma unroll
  for (int j = 0; j < (QT == CMLD_Q4_K ? 4 : 2); ++j) o.c[j] = fetch<GLOBAL, uint4>(rec + (2 * half + j) * 512 + lane * 16);
  const int t = lane & 3;
  if (QT == CMLD_Q4_K) {
    o.p = fetch<GLOBAL, uint2>(rec + 2048 + lane * 8);
    o.x[0] = fetch<GLOBAL, float2>(rec + 2304 + 8 * t);
  } else if (QT == CMLD_Q6_K) {
    o.x[0] = fetch<GLOBAL, float2>(rec + 2048 + 8 * t);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) o.x[k] = fetch<GLOBAL, float2>(rec + 1024 + 32 * k + 8 * t);
  }
}

// Outputs of a lane: i = 0: (row g, column 2t), 1: (g, 2t + 1), 2: (g + 8, 2t), 3: (g + 8, 2t + 1)

// put(i, {xd*d, S, -(xd*dmin), P})
template <typename Put>
__device__ __forceinline__ void product(Q4Unit &u, const Operand &o, Put &&put) {
  int s[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    int c[4];
    uint32_t a[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      asm volatile("" : "+r"(u.c[j][i]));  // (masked anew for every row group: the masked words of all groups would not fit the registers)
      a[i] = u.c[j][i] & 0x0f0f0f0fu;
    }
    mma_u8(c, a, o.c[j].x, o.c[j].y, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] += c[i] * u.sc[i >> 1][2 * j];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = u.c[j][i] & 0xf0f0f0f0u;
    mma_u8(c, a, o.c[j].z, o.c[j].w, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] += c[i] * u.sc[i >> 1][2 * j + 1];
  }
  float p[4];
  mma_f16(p, u.m[0], u.m[1], o.p.x, o.p.y);
  const float xd[2] = {o.x[0].x, o.x[0].y};
#pragma unroll
  for (int i = 0; i < 4; ++i)  // (the conversion rounds 16 S as it would S)
    put(i, make_float4(__fmul_rn(xd[i & 1], u.d[i >> 1]), __fmul_rn((float)s[i], 0.0625f), -__fmul_rn(xd[i & 1], u.dm[i >> 1]), p[i]));
}
// put(i, (d*xd) * aux[l] of the half's four classes)
template <typename Put>
__device__ __forceinline__ void product(Q6Unit &u, const Operand &o, Put &&put) {
  const float xd[2] = {o.x[0].x, o.x[0].y};
  float dd[4], f[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) dd[i] = __fmul_rn(u.d[i >> 1], xd[i & 1]);  // src/inference.rs:25545
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    int h[4], w[4];
    const uint4 b = o.c[l >> 1];
    mma_s8(h, u.hi[l], l & 1 ? b.z : b.x, l & 1 ? b.w : b.y, kMagicBits);
    mma_u8(w, u.lo[l], l & 1 ? b.z : b.x, l & 1 ? b.w : b.y, kMagicBits);
#pragma unroll
    for (int i = 0; i < 4; ++i)  // |aux| <= 32 * 127 * 4096 < 2^24: exact
      f[i][l] = __fmul_rn(dd[i], __fmaf_rn(256.0f, __fsub_rn(__int_as_float(h[i]), kMagic), __fsub_rn(__int_as_float(w[i]), kMagic)));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) put(i, make_float4(f[i][0], f[i][1], f[i][2], f[i][3]));
}
// put(i, (isum * ws) * xs of the four blocks)
template <typename Put>
__device__ __forceinline__ void product(Q8Unit &u, const Operand &o, Put &&put) {
  float f[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    int c[4];
    const uint4 b = o.c[k >> 1];
    mma_s8(c, u.a[k], k & 1 ? b.z : b.x, k & 1 ? b.w : b.y, kMagicBits);
#pragma unroll
    for (int i = 0; i < 4; ++i)  // src/inference.rs:26198
      f[i][k] = __fmul_rn(__fmul_rn(__fsub_rn(__int_as_float(c[i]), kMagic), u.ws[i >> 1][k]), i & 1 ? o.x[k].y : o.x[k].x);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) put(i, make_float4(f[i][0], f[i][1], f[i][2], f[i][3]));
}

// The same for all row groups at once, onto the sums: a group's codes are masked once and the products of the row groups are
// independent of one another.  rec: the unit's records, in shared memory.
template <int NT>
__device__ __forceinline__ void products(const Q4Unit &u, const uint8_t *rec, int lane, float (&acc)[NT][4][1]) {
  int s[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int i = 0; i < 4; ++i) s[nt][i] = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) lo[i] = u.c[j][i] & 0x0f0f0f0fu, hi[i] = u.c[j][i] & 0xf0f0f0f0u;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const uint4 b = *reinterpret_cast<const uint4 *>(rec + nt * rows_rec(CMLD_Q4_K) + j * 512 + lane * 16);
      int c[4], d[4];
      mma_u8(c, lo, b.x, b.y, 0);
      mma_u8(d, hi, b.z, b.w, 0);
#pragma unroll
      for (int i = 0; i < 4; ++i) s[nt][i] += c[i] * u.sc[i >> 1][2 * j] + d[i] * u.sc[i >> 1][2 * j + 1];
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const uint8_t *r = rec + nt * rows_rec(CMLD_Q4_K);
    const uint2 b = *reinterpret_cast<const uint2 *>(r + 2048 + lane * 8);
    const float2 x = *reinterpret_cast<const float2 *>(r + 2304 + 8 * (lane & 3));
    const float xd[2] = {x.x, x.y};
    float p[4];
    mma_f16(p, u.m[0], u.m[1], b.x, b.y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float &o = acc[nt][i][0];
      o = __fmaf_rn(-__fmul_rn(xd[i & 1], u.dm[i >> 1]), p[i], o);
      o = __fmaf_rn(__fmul_rn(xd[i & 1], u.d[i >> 1]), __fmul_rn((float)s[nt][i], 0.0625f), o);
    }
  }
}

__device__ __forceinline__ int tile_job(const RowsArgs &a, int tile) {
  int j = 0;
  if (a.n_jobs > 1 && tile >= a.job[1].first_tile) j = 1;
  if (a.n_jobs > 2 && tile >= a.job[2].first_tile) j = 2;
  return j;
}

// ---------------------------------------------------------------- tiles shared by a team

// A row of a pass (up to kWarps units) in a stage: the codes, then the scales behind them (Q6_K, Q8_0), padded so that neighbouring
// rows lie 32 bytes apart modulo 128.
__host__ __device__ constexpr int pass_pitch(int qt) { return qt == CMLD_Q4_K ? 2304 + 32 : qt == CMLD_Q6_K ? 3328 + 32 : 2048 + 128 + 32; }

__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(bar)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(s32(bar)), "r"(parity)
               : "memory");
  return ok;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const uint8_t *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(s32(bar))
               : "memory");
}

// Where a thread of the split form stands.
struct Split {
  int first, step, n_mine;   // tiles of this CTA: first + k * step
  int stage, stage_phase;    // ring stage of the next pass
  int buf, buf_phase;        // buffer of the next exchange
  int lk, lu, ls;            // the next load: tile of this CTA's list, first unit, ring stage
  uint8_t *smem;
  uint64_t *landed, *full, *empty;  // mbarriers of the stages; of the exchange buffers
  volatile int *gave_up;            // a wait of this CTA ran out
};
__device__ __forceinline__ void give_up(const RowsArgs &a, const Split &s) {
  *s.gave_up = 1;
  if (a.status) atomicExch(a.status, (int32_t)CMLD_ERR_TIMEOUT);
}
// Bounded.  Once a wait of the CTA has run out, the others give up after a few polls and no more weights are fetched: the roles run through
// their loops without a result, and the host reports the error.  (Roles that leave their loops instead need the verdict of all lanes of a
// warp: 1 % of a launch.)
__device__ __forceinline__ void bar_wait(const RowsArgs &a, const Split &s, uint64_t *bar, uint32_t parity) {
  for (uint32_t i = 0; i < kRowsSpin; ++i) {
    if (bar_try(bar, parity)) return;
    if ((i & 7u) == 7u && *s.gave_up) return;
  }
  give_up(a, s);
}
__device__ __forceinline__ void next_stage(const RowsArgs &a, Split &s) {
  if (++s.stage == a.stages) s.stage = 0, s.stage_phase ^= 1;
}
__device__ __forceinline__ void next_buf(const RowsArgs &a, Split &s) {
  if (++s.buf == a.bufs) s.buf = 0, s.buf_phase ^= 1;
}

// The next pass of this CTA's tiles into its stage: each of the four adding warps four weight rows, a lane per row.  (A warp's copies are
// issued one after another, about 60 cycles each: all of a pass by one warp kept the sums waiting.  Us per launch so | here: Q6_K
// 4096 x 14336 27.1 | 24.6 at 8 rows, 55.8 | 47.7 at 32.)
template <int QT>
__device__ __forceinline__ void load_pass(const RowsArgs &a, Split &s, int warp, int lane) {
  if (s.lk >= s.n_mine) return;
  const int tile = s.first + s.lk * s.step;
  const RowsJob &J = a.job[tile_job(a, tile)];
  const int row0 = (tile - J.first_tile) * 16, cnt = min(kWarps, J.units - s.lu);
  constexpr int UB = unit_bytes(QT);
  const int codes = cnt * UB, scales = QT == CMLD_Q4_K ? 0 : QT == CMLD_Q6_K ? (2 * cnt + 15) & ~15 : 8 * cnt;
  const bool stop = __shfl_sync(0xffffffffu, *s.gave_up, 0);
  if (lane == 0) {
    if (stop) bar_arrive(&s.landed[s.ls]);
    else bar_expect(&s.landed[s.ls], (uint32_t)(4 * (codes + scales)));
  }
  __syncwarp();
  if (lane < 4 && !stop) {
    const int r = 4 * warp + lane;
    const uint8_t *row = J.w + (int64_t)min(row0 + r, J.rows - 1) * J.stride;
    const uint32_t dst = s32(s.smem + a.off_ring + s.ls * a.stage_bytes) + r * pass_pitch(QT);
    bulk_load(dst, row + (int64_t)s.lu * UB, (uint32_t)codes, &s.landed[s.ls]);
    if (scales) bulk_load(dst + kWarps * UB, row + (int64_t)J.units * UB + s.lu * (QT == CMLD_Q6_K ? 2 : 8), (uint32_t)scales, &s.landed[s.ls]);
  }
  if (++s.ls == a.stages) s.ls = 0;
  s.lu += kWarps;
  if (s.lu >= J.units) s.lu = 0, ++s.lk;
}

// A unit's terms of one output onto its sums: the next two multiply-adds of Q4_K, four classes of Q6_K, the next four blocks of Q8_0.
template <int QT>
__device__ __forceinline__ void add_terms(float *s, const float4 &v) {
  if constexpr (QT == CMLD_Q4_K) {
    s[0] = __fmaf_rn(v.x, v.y, __fmaf_rn(v.z, v.w, s[0]));
  } else if constexpr (QT == CMLD_Q6_K) {
    s[0] = __fadd_rn(s[0], v.x), s[1] = __fadd_rn(s[1], v.y), s[2] = __fadd_rn(s[2], v.z), s[3] = __fadd_rn(s[3], v.w);
  } else {
    s[0] = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s[0], v.x), v.y), v.z), v.w);
  }
}

// The products of one tile: warp `warp` takes one unit of each pass, `first` of the first.
template <int QT, int NT>
__device__ __forceinline__ void split_products(const RowsArgs &a, const RowsJob &J, int first, int lane, Split &s) {
  constexpr int HALVES = QT == CMLD_Q6_K ? 2 : 1, P = pass_pitch(QT), UB = unit_bytes(QT);
  const int g = lane >> 2, t = lane & 3, units = J.units;
  const uint8_t *rec = J.rec + (int64_t)first * NT * rows_rec(QT);
  Operand o;
  if (first < units) fetch_operand<QT, true>(o, rec, 0, lane);
  for (int u = first; u < units + kWarps - 1; u += kWarps, rec += kWarps * NT * rows_rec(QT)) {
    if (u - first >= units) break;  // no such pass
    const bool mine = u < units;
    bar_wait(a, s, &s.landed[s.stage], (uint32_t)s.stage_phase);
    __syncwarp();
    const uint8_t *raw = s.smem + a.off_ring + s.stage * a.stage_bytes + first * UB;
    const uint8_t *scales = raw + (kWarps - first) * UB + first * (QT == CMLD_Q6_K ? 2 : 8);
    next_stage(a, s);
    typename UnitOf<QT>::type w;
    if (mine) unpack_head<P>(w, raw, scales, g, t);
#pragma unroll
    for (int e = 0; e < HALVES; ++e) {
      if (mine) unpack_codes<P>(w, raw, g, t, e);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        bar_wait(a, s, &s.empty[s.buf], (uint32_t)(s.buf_phase ^ 1));
        if (mine) {
          float4 *dst = reinterpret_cast<float4 *>(s.smem + s.buf * (kWarps * kSlice) + first * kSlice) + lane;
          product(w, o, [&](int i, const float4 &f) { dst[i == 0 ? 0 : i == 1 ? 64 : i == 2 ? 32 : 96] = f; });
          // the operand of the next exchange, asked for before this one
          if (nt + 1 < NT) fetch_operand<QT, true>(o, rec + (nt + 1) * rows_rec(QT), e, lane);
          else if (e + 1 < HALVES) fetch_operand<QT, true>(o, rec, e + 1, lane);
          else if (u + kWarps < units) fetch_operand<QT, true>(o, rec + kWarps * NT * rows_rec(QT), 0, lane);
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&s.full[s.buf]);
        next_buf(a, s);
      }
    }
  }
}

// The sums of one tile: four warps, a thread per output of a row group (its place in a slice: idx).  Between passes the running sums
// lie in shared memory, a float (Q6_K: two float4, the halves' classes) per row group.
template <int QT, int NT>
__device__ __forceinline__ void split_sums(const RowsArgs &a, const RowsJob &J, int row0, int idx, Split &s) {
  constexpr int HALVES = QT == CMLD_Q6_K ? 2 : 1, NL = QT == CMLD_Q6_K ? 4 : 1;
  typedef typename Sums<QT>::type sum_t;
  const int lane = idx & 31;
  sum_t *sums = reinterpret_cast<sum_t *>(s.smem + a.off_sums) + idx;
  for (int u0 = 0; u0 < J.units; u0 += kWarps) {
    const int cnt = min(kWarps, J.units - u0);
#pragma unroll 1
    for (int x = 0; x < HALVES * NT; ++x) {
      float acc[NL];
      if (u0 > 0) {
        const sum_t v = sums[x * 128];
#pragma unroll
        for (int l = 0; l < NL; ++l) acc[l] = reinterpret_cast<const float *>(&v)[l];
      } else {
#pragma unroll
        for (int l = 0; l < NL; ++l) acc[l] = 0.0f;
      }
      bar_wait(a, s, &s.full[s.buf], (uint32_t)s.buf_phase);
      __syncwarp();
      const float4 *p = reinterpret_cast<const float4 *>(s.smem + s.buf * (kWarps * kSlice)) + idx;
      if (cnt == kWarps) {
        float4 v[kWarps];
#pragma unroll
        for (int i = 0; i < kWarps; ++i) v[i] = p[i * (kSlice / 16)];
#pragma unroll
        for (int i = 0; i < kWarps; ++i) add_terms<QT>(acc, v[i]);
      } else {
        for (int i = 0; i < cnt; ++i) add_terms<QT>(acc, p[i * (kSlice / 16)]);
      }
      __syncwarp();
      if (lane == 0) bar_arrive(&s.empty[s.buf]);
      next_buf(a, s);
      // the pass's last terms were there: nobody reads its stage any more
      if (x + 1 == HALVES * NT) load_pass<QT>(a, s, idx >> 5, lane);
      sum_t v;
#pragma unroll
      for (int l = 0; l < NL; ++l) reinterpret_cast<float *>(&v)[l] = acc[l];
      sums[x * 128] = v;
    }
  }
  const int r = row0 + ((idx >> 2) & 15);
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int b = nt * 8 + 2 * (idx & 3) + (idx >> 6);
    if (b < a.batch && r < J.rows) {
      float v;
      if constexpr (QT == CMLD_Q6_K) {
        const float4 lo = sums[nt * 128], hi = sums[(NT + nt) * 128];
        v = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(0.0f, lo.x), lo.y), lo.z), lo.w);  // 0 + sums[0] + ... + sums[7] (src/inference.rs:25578-25580)
        v = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(v, hi.x), hi.y), hi.z), hi.w);
      } else {
        v = sums[nt * 128];
      }
      const int64_t at = (int64_t)b * J.y_stride + r;
      J.y[at] = J.residual ? __fadd_rn(__ldcg(J.residual + at), v) : v;
    }
  }
}

// After a wait that ran out, what was fetched may still be on its way into this CTA's shared memory: the adding warps stay until it is there.
// (All of them have arrived for every pass by the time the last of them is here.)
__device__ __forceinline__ void drain(const RowsArgs &a, const Split &s, int lane) {
  if (!*s.gave_up || lane != 0) return;
  int loads = 0;
  for (int k = 0; k < s.n_mine; ++k) loads += (a.job[tile_job(a, s.first + k * s.step)].units + kWarps - 1) / kWarps;
  for (int i = max(0, loads - a.stages); i < loads; ++i)
    for (uint32_t n = 0; n < kRowsSpin && !bar_try(&s.landed[i % a.stages], (uint32_t)(i / a.stages & 1)); ++n) {
    }
}

// The two roles over all tiles of this CTA.
template <int QT, int NT>
__device__ __forceinline__ void split_multiply(const RowsArgs &a, int warp, int lane, Split &s) {
  for (int k = 0; k < s.n_mine; ++k) {
    const RowsJob &J = a.job[tile_job(a, s.first + k * s.step)];
    split_products<QT, NT>(a, J, (warp - k * J.units) & (kWarps - 1), lane, s);  // (who has no unit in a short pass differs from tile to tile)
  }
}
template <int QT, int NT>
__device__ __forceinline__ void split_add(const RowsArgs &a, int warp, int lane, Split &s) {
  for (int i = 0; i < a.stages; ++i) load_pass<QT>(a, s, warp, lane);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int k = 0; k < s.n_mine; ++k) {
    const int tile = s.first + k * s.step;
    const RowsJob &J = a.job[tile_job(a, tile)];
    split_sums<QT, NT>(a, J, (tile - J.first_tile) * 16, warp * 32 + lane, s);
  }
}

template <int NT>
__global__ void __launch_bounds__(kSplitThreads, 1) rows_split_kernel(const __grid_constant__ RowsArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];  // exchange buffers [buffer][unit of the pass][kSlice], then the stages
  __shared__ __align__(8) uint64_t bars[3 * kMaxStages];
  __shared__ int gave_up;
  asm volatile("griddepcontrol.launch_dependents;");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxStages; ++i) {
      bar_init(&bars[i], kSplitWarps - kWarps);
      bar_init(&bars[kMaxStages + i], kWarps + a.lose_one);
      bar_init(&bars[2 * kMaxStages + i], kSplitWarps - kWarps);
    }
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  Split s{};
  const int cta = (int)blockIdx.x, n_ctas = (int)gridDim.x;
  const bool second = cta >= a.ctas0;
  s.first = second ? a.tiles0 + cta - a.ctas0 : cta;
  s.step = second ? n_ctas - a.ctas0 : a.ctas0;
  s.n_mine = ((second ? a.tiles : a.tiles0) - s.first + s.step - 1) / s.step;
  s.smem = smem;
  s.landed = bars, s.full = bars + kMaxStages, s.empty = bars + 2 * kMaxStages;
  s.gave_up = &gave_up;
  // the adding warps hold few values: they leave registers to the others
  const int qt = a.job[tile_job(a, s.first)].qt;
  if (warp < kWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");  // 512 x 104 + 128 x 64 = the 640 x 96 of the launch
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (a.lose_one && threadIdx.x == 0) give_up(a, s);
    if (qt == CMLD_Q4_K) split_multiply<CMLD_Q4_K, NT>(a, warp, lane, s);
    else if (qt == CMLD_Q6_K) split_multiply<CMLD_Q6_K, NT>(a, warp, lane, s);
    else split_multiply<CMLD_Q8_0, NT>(a, warp, lane, s);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (qt == CMLD_Q4_K) split_add<CMLD_Q4_K, NT>(a, warp - kWarps, lane, s);
    else if (qt == CMLD_Q6_K) split_add<CMLD_Q6_K, NT>(a, warp - kWarps, lane, s);
    else split_add<CMLD_Q8_0, NT>(a, warp - kWarps, lane, s);
    drain(a, s, lane);
  }
}

// ---------------------------------------------------------------- a tile per warp

template <int QT, int NT>
__global__ void __launch_bounds__(kWarps * 32, 1) rows_whole_kernel(const __grid_constant__ RowsArgs a) {
  constexpr int NL = QT == CMLD_Q6_K ? 8 : 1, HALVES = QT == CMLD_Q6_K ? 2 : 1;
  extern __shared__ __align__(128) uint8_t smem[];  // the records of all units, then the rings
  asm volatile("griddepcontrol.launch_dependents;");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, n_warps = (int)blockDim.x >> 5;
  const int grid = (int)gridDim.x, cta = (int)blockIdx.x, S = a.stages;
  const int n_mine = (a.tiles - cta + grid - 1) / grid, units = a.job[0].units;
  const uint8_t *ring_p = smem + a.off_ring + warp * S * raw_bytes(QT);
  const uint32_t ring = s32(ring_p);

  RawCopy<QT> rc;
  const uint8_t *lbase = nullptr;
  int lk = warp, lu = 0, ls = 0;
  auto issue = [&]() {
    if (lk < n_mine) {
      if (lu == 0) {
        const int tile = cta + lk * grid;
        const RowsJob &J = a.job[tile_job(a, tile)];
        const int row0 = (tile - J.first_tile) * 16;
        lbase = J.w + (int64_t)row0 * J.stride;
        rc.place(J.rows - row0 - 1, J.stride, units, lane);
      }
      rc.copy(ring + ls * raw_bytes(QT), lbase, lu, lane);
      if (++lu == units) lu = 0, lk += n_warps;
    }
    cp_commit();
    if (++ls == S) ls = 0;
  };
  for (int i = 0; i < S - 1; ++i) issue();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int n16 = units * NT * rows_rec(QT) / 16;
  for (int i = threadIdx.x; i < n16; i += (int)blockDim.x) cp16(s32(smem) + i * 16, a.job[0].rec + (int64_t)i * 16);
  cp_commit();
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  int stage = 0;
  for (int k = warp; k < n_mine; k += n_warps) {
    const int tile = cta + k * grid;
    const RowsJob &J = a.job[tile_job(a, tile)];
    const int row0 = (tile - J.first_tile) * 16;
    float acc[NT][4][NL];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int l = 0; l < NL; ++l) acc[n][i][l] = 0.0f;
    for (int u = 0; u < units; ++u) {
      cp_wait_stages(S);
      __syncwarp();
      issue();
      const uint8_t *raw = ring_p + stage * raw_bytes(QT);
      if (++stage == S) stage = 0;
      const uint8_t *rec = smem + u * NT * rows_rec(QT);
      typename UnitOf<QT>::type w;
      unpack_head<raw_pitch(QT)>(w, raw, raw + (QT == CMLD_Q6_K ? 208 + 2 * (u & 1) : 128), g, t);
#pragma unroll
      for (int e = 0; e < HALVES; ++e) {
        unpack_codes<raw_pitch(QT)>(w, raw, g, t, e);
        if constexpr (QT == CMLD_Q4_K) {
          products<NT>(w, rec, lane, acc);
        } else {
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            Operand o;
            fetch_operand<QT, false>(o, rec + nt * rows_rec(QT), e, lane);
            product(w, o, [&](int i, const float4 &f) { add_terms<QT>(&acc[nt][i][4 * e], f); });
          }
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int b = nt * 8 + 2 * t + (i & 1), r = row0 + g + 8 * (i >> 1);
        float v = acc[nt][i][0];
        if constexpr (QT == CMLD_Q6_K) {
          v = 0.0f;
#pragma unroll
          for (int l = 0; l < NL; ++l) v = __fadd_rn(v, acc[nt][i][l]);
        }
        if (b < a.batch && r < J.rows) {
          const int64_t at = (int64_t)b * J.y_stride + r;
          J.y[at] = J.residual ? __fadd_rn(__ldcg(J.residual + at), v) : v;
        }
      }
  }
}

// ---------------------------------------------------------------- records from quantised rows in the global layout

__global__ void __launch_bounds__(256) rows_pack_kernel(const uint8_t *act, int64_t cols, int nt, uint8_t *rec4, uint8_t *rec6, uint8_t *rec0) {
  const int lane = threadIdx.x & 31, b = blockIdx.y;
  const int64_t ch = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (ch >= cols / 256) return;
  const uint8_t *row = act + b * act_row_stride(cols);
  const uint2 pk = *reinterpret_cast<const uint2 *>(row + ch * 256 + lane * 8);
  const float *scales = reinterpret_cast<const float *>(row + act_scale_off(cols));
  if (rec0) rows_store_0(pk, scales[ch * 8 + (lane >> 2)], lane, b, ch, nt, rec0);
  else rows_store_k(pk, scales[ch], lane, b, ch, nt, rec4, rec6);
}

int sm_count() {
  static const int n = [] {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) v = 0;
    return v;
  }();
  return n;
}

template <typename K>
int32_t launch(SmemLimit &limit, K kernel, const RowsArgs &a, int grid, int threads, int smem, cudaStream_t s, bool pdl) {
  CMLD_TRY(allow_smem(limit, kernel, (size_t)kSmemMax, true));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  CMLD_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
  return CMLD_OK;
}

template <int NT>
int32_t launch_split(const RowsArgs &a, int grid, int smem, cudaStream_t s, bool pdl) {
  static SmemLimit limit;
  return launch(limit, rows_split_kernel<NT>, a, grid, kSplitThreads, smem, s, pdl);
}
template <int QT, int NT>
int32_t launch_whole(const RowsArgs &a, int grid, int warps, int smem, cudaStream_t s, bool pdl) {
  static SmemLimit limit;
  return launch(limit, rows_whole_kernel<QT, NT>, a, grid, warps * 32, smem, s, pdl);
}
template <int QT>
int32_t launch_whole_nt(int nt, const RowsArgs &a, int grid, int warps, int smem, cudaStream_t s, bool pdl) {
  if constexpr (QT != CMLD_Q6_K) {
    switch (nt) {
      case 2: return launch_whole<QT, 2>(a, grid, warps, smem, s, pdl);
      case 3: return launch_whole<QT, 3>(a, grid, warps, smem, s, pdl);
      case 4: return launch_whole<QT, 4>(a, grid, warps, smem, s, pdl);
      default: break;
    }
  }
  return launch_whole<QT, 1>(a, grid, warps, smem, s, pdl);
}

}  // namespace

// Room for the records of one type (the widest: Q4_K) of a step of `batch` rows of `cols` columns.
int64_t gemv_rows_rec_bytes(int64_t cols, int32_t batch) { return (cols + 255) / 256 * ((batch + 7) / 8) * (int64_t)rows_rec(CMLD_Q4_K); }

bool gemv_rows_fits(const GemvJob *jobs, int n_jobs, int32_t batch) {
  if (n_jobs < 1 || n_jobs > 3 || batch < 1 || batch > kRowsMaxBatch) return false;
  for (int i = 0; i < n_jobs; ++i) {
    const int qt = jobs[i].qt;
    if (qt != CMLD_Q4_K && qt != CMLD_Q6_K && qt != CMLD_Q8_0) return false;
    if ((qt == CMLD_Q8_0) != (jobs[0].qt == CMLD_Q8_0) || jobs[i].cols != jobs[0].cols || jobs[i].cols % 256 != 0 || jobs[i].cols < 256 || jobs[i].rows < 1) return false;
    if (jobs[i].stride % 16 || (reinterpret_cast<uintptr_t>(jobs[i].w) & 15)) return false;
  }
  return true;
}

int32_t launch_rows_pack(const uint8_t *act, int64_t cols, int32_t batch, uint8_t *rec4, uint8_t *rec6, uint8_t *rec0, cudaStream_t s) {
  const dim3 grid((unsigned)((cols / 256 + 7) / 8), (unsigned)batch);
  rows_pack_kernel<<<grid, 256, 0, s>>>(act, cols, (batch + 7) / 8, rec4, rec6, rec0);
  CMLD_CUDA(cudaGetLastError());
  return CMLD_OK;
}

// The records: rec4 for Q4_K matrices, rec6 for Q6_K, rec0 for Q8_0 (those of the types that occur).  lose_one (a self-test): an arrival of
// the split form never comes and a wait counts as run out; shapes that take the other form, which has no such waits, are refused.
int32_t launch_gemv_rows(const GemvJob *jobs, int n_jobs, int32_t batch, const uint8_t *rec4, const uint8_t *rec6, const uint8_t *rec0,
                         int32_t *status, cudaStream_t s, bool pdl, bool lose_one) {
  if (!gemv_rows_fits(jobs, n_jobs, batch)) return CMLD_ERR_UNSUPPORTED;
  const int sms = sm_count(), nt = (batch + 7) / 8;
  if (sms < 1) return fail(CMLD_ERR_CUDA, "gemv: no device");
  RowsArgs a{};
  a.n_jobs = n_jobs;
  a.batch = batch;
  a.status = status;
  a.lose_one = lose_one;
  for (int pass = 0, k = 0; pass < 2; ++pass)  // Q6_K last
    for (int i = 0; i < n_jobs; ++i) {
      const int qt = jobs[i].qt;
      if ((qt == CMLD_Q6_K) != (pass == 1)) continue;
      RowsJob &J = a.job[k++];
      J = RowsJob{jobs[i].w, qt, (int32_t)jobs[i].rows, (int32_t)(jobs[i].cols / rows_unit(qt)), a.tiles, jobs[i].stride, jobs[i].y, jobs[i].residual,
                  jobs[i].y_stride, qt == CMLD_Q4_K ? rec4 : qt == CMLD_Q6_K ? rec6 : rec0};
      if (!J.rec) return fail(CMLD_ERR_INVALID, "gemv: activation records missing");
      a.tiles += (int32_t)((jobs[i].rows + 15) / 16);
      if (qt == a.job[0].qt) a.tiles0 = a.tiles;
    }
  const bool same = a.tiles0 == a.tiles;
  int grid = std::min(a.tiles, sms);
  const int per_cta = (a.tiles + grid - 1) / grid, qt = a.job[0].qt;
  const int warps = std::min(kWarps, per_cta), rec = a.job[0].units * nt * rows_rec(qt);
  const int fit = warps > 0 ? (kSmemMax - rec) / (warps * raw_bytes(qt)) : 0;
  if (same && per_cta >= 5 && fit >= 2 && (qt != CMLD_Q6_K || nt == 1)) {
    if (lose_one) return CMLD_ERR_UNSUPPORTED;
    a.stages = std::min(kMaxStages, fit);
    a.off_ring = rec;
    const int smem = rec + warps * a.stages * raw_bytes(qt);
    if (qt == CMLD_Q4_K) return launch_whole_nt<CMLD_Q4_K>(nt, a, grid, warps, smem, s, pdl);
    if (qt == CMLD_Q6_K) return launch_whole_nt<CMLD_Q6_K>(nt, a, grid, warps, smem, s, pdl);
    return launch_whole_nt<CMLD_Q8_0>(nt, a, grid, warps, smem, s, pdl);
  }
  a.ctas0 = grid;
  if (!same) {
    // two types: the CTAs in proportion to the work, a Q6_K tile counted as two of Q4_K
    const int work0 = a.tiles0, work1 = 2 * (a.tiles - a.tiles0);
    a.ctas0 = std::min(a.tiles0, std::max(1, std::min(grid - 1, (int)((int64_t)grid * work0 / (work0 + work1)))));
    grid = a.ctas0 + std::min(grid - a.ctas0, a.tiles - a.tiles0);
  }
  for (int i = 0; i < n_jobs; ++i) a.stage_bytes = std::max(a.stage_bytes, 16 * pass_pitch(jobs[i].qt));
  a.bufs = nt >= 3 ? 3 : 2;
  a.off_sums = a.bufs * kWarps * kSlice;
  a.off_ring = a.off_sums + nt * (a.tiles0 < a.tiles || qt == CMLD_Q6_K ? 2 * kSlice : kSlice / 4);
  a.stages = std::min(kMaxStages, (kSmemMax - a.off_ring) / a.stage_bytes);
  const int smem = a.off_ring + a.stages * a.stage_bytes;
  switch (nt) {
    case 1: return launch_split<1>(a, grid, smem, s, pdl);
    case 2: return launch_split<2>(a, grid, smem, s, pdl);
    case 3: return launch_split<3>(a, grid, smem, s, pdl);
    default: return launch_split<4>(a, grid, smem, s, pdl);
  }
}

}  // namespace cmld
