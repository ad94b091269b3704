// Activation records of the row-batched matvec (gemv_rows.cu): what one warp's tensor-core operand registers take of eight
// activation rows and one unit of columns (K-quants 256, Q8_0 128), in the order in which its lanes load it.
//
// mma.m16n8k32 wants of lane (g = lane / 4, t = lane % 4) eight bytes of activation row g; which eight of the 32 columns is free
// as long as the weight operand takes the same ones.
//   Q4_K, Q8_0: columns 8t .. 8t+7 of each 32.  Codes: [pair of 32-blocks][lane][block of the pair][8 bytes].
//   Q6_K: product l of a superblock covers the columns with index = l mod 8 (the CPU's eight accumulators); lane t = 2h + c holds
//     the half h (128 values) and the 16-value groups of parity c in it: bytes 2q, 2q+1 are the columns 128h + 32q + 16c + {l, l + 8},
//     q = 0..3.  Codes: [pair of classes l][lane][class of the pair][8 bytes].
// Behind the codes: Q4_K the sums of 16 codes as f16 (exact, |sum| <= 2032), [lane][{4t, 4t+2, 4t+1, 4t+3}], then a scale per row;
// Q6_K a scale per row; Q8_0 [4 blocks][8 rows] scales.
// A step's records lie [unit][group of eight rows].  Rows past the batch are not written: a row's results depend on no other.
#pragma once

#include "common.cuh"

namespace cmld {

__host__ __device__ constexpr int rows_unit(int qt) { return qt == CMLD_Q8_0 ? 128 : 256; }
__host__ __device__ constexpr int rows_rec(int qt) { return qt == CMLD_Q4_K ? 2048 + 256 + 32 : qt == CMLD_Q6_K ? 2048 + 32 : 1024 + 128; }

// One 256-value chunk of row b: pk = this lane's eight Q8_K codes, d the chunk's scale.  All lanes must call.
__device__ __forceinline__ void rows_store_k(uint2 pk, float d, int lane, int b, int64_t ch, int nt, uint8_t *rec4, uint8_t *rec6) {
  const int g = b & 7;
  if (rec4) {
    uint8_t *r = rec4 + (ch * nt + (b >> 3)) * rows_rec(CMLD_Q4_K);
    *reinterpret_cast<uint2 *>(r + (lane >> 3) * 512 + (g * 4 + (lane & 3)) * 16 + ((lane >> 2) & 1) * 8) = pk;
    int s = __dp4a((int)pk.y, 0x01010101, __dp4a((int)pk.x, 0x01010101, 0));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    const int m = lane >> 1;  // which sum of 16
    if ((lane & 1) == 0) *reinterpret_cast<__half *>(r + 2048 + (g * 4 + (m >> 2)) * 8 + (m & 1) * 4 + ((m >> 1) & 1) * 2) = __int2half_rn(s);
    if (lane == 0) *reinterpret_cast<float *>(r + 2304 + g * 4) = d;
  }
  if (rec6) {
    // lane = 16h + 4q + 2c + half holds classes 0..7 of its (half, q, c): three exchanges leave it with all eight bytes of one class
    const bool odd = lane & 1, q0 = lane & 4, q1 = lane & 8;
    const uint32_t r1 = __shfl_xor_sync(0xffffffffu, odd ? pk.x : pk.y, 1);
    const uint32_t a1 = odd ? r1 : pk.x, b1 = odd ? pk.y : r1;
    const uint32_t w01 = __byte_perm(a1, b1, 0x5140), w23 = __byte_perm(a1, b1, 0x7362);
    const uint32_t r2 = __shfl_xor_sync(0xffffffffu, q0 ? w01 : w23, 4);
    const uint32_t a2 = q0 ? r2 : w01, b2 = q0 ? w23 : r2;
    const uint32_t x = __byte_perm(a2, b2, 0x5410), y = __byte_perm(a2, b2, 0x7632);
    const uint32_t r3 = __shfl_xor_sync(0xffffffffu, q1 ? x : y, 8);
    const int l = 4 * (lane & 1) + 2 * ((lane >> 2) & 1) + ((lane >> 3) & 1), t = 2 * (lane >> 4) + ((lane >> 1) & 1);
    uint8_t *r = rec6 + (ch * nt + (b >> 3)) * rows_rec(CMLD_Q6_K);
    *reinterpret_cast<uint2 *>(r + (l >> 1) * 512 + (g * 4 + t) * 16 + (l & 1) * 8) = q1 ? make_uint2(r3, y) : make_uint2(x, r3);
    if (lane == 0) *reinterpret_cast<float *>(r + 2048 + g * 4) = d;
  }
}

// The same for Q8_0 codes; scale: that of this lane's 32-value block.
__device__ __forceinline__ void rows_store_0(uint2 pk, float scale, int lane, int b, int64_t ch, int nt, uint8_t *rec0) {
  const int g = b & 7, blk = (lane >> 2) & 3;
  uint8_t *r = rec0 + ((ch * 2 + (lane >> 4)) * nt + (b >> 3)) * rows_rec(CMLD_Q8_0);
  *reinterpret_cast<uint2 *>(r + (blk >> 1) * 512 + (g * 4 + (lane & 3)) * 16 + (blk & 1) * 8) = pk;
  if ((lane & 3) == 0) *reinterpret_cast<float *>(r + 1024 + blk * 32 + g * 4) = scale;
}

}  // namespace cmld
