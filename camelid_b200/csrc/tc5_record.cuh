// Activation records of the tcgen05 batched matvec (gemv_tc5.cu): operand A of one K step (256 columns) and one tile of 128 rows, as one
// bulk copy brings it into shared memory.
//   codes [row/8][k/16][row%8][16]  (Q6_K: K permuted, chunk 2l + h holds the sixteen values of half h with index = l mod 8, in the order
//                                   32q + {l, l + 8, l + 16, l + 24}, q = 0..3)
//   Q4_K: the sums of 16 codes as f16 [row/8][2][row%8][8]
//   scales f32 [128] (Q8_0: [8 blocks][128])
// A step's records lie [K step][tile].  Rows past the batch are not written: a row's results depend on no other.
#pragma once

#include "common.cuh"

namespace cmld {

constexpr int kTc5Rows = 128;
__host__ __device__ constexpr int tc5_rec_p(int qt) { return qt == CMLD_Q4_K ? kTc5Rows * 32 : 0; }
__host__ __device__ constexpr int tc5_rec_scales(int qt) { return (qt == CMLD_Q8_0 ? 8 : 1) * kTc5Rows * 4; }
__host__ __device__ constexpr int tc5_rec(int qt) { return kTc5Rows * 256 + tc5_rec_p(qt) + tc5_rec_scales(qt); }

// One 256-value chunk of row b: pk = this lane's eight Q8_K codes, d the chunk's scale.  All lanes must call.
__device__ __forceinline__ void tc5_store_k(uint2 pk, float d, int lane, int b, int64_t ch, int tiles, uint8_t *rec4, uint8_t *rec6) {
  const int row = b % kTc5Rows, g = row >> 3, i = row & 7;
  const int64_t at = ch * tiles + b / kTc5Rows;
  if (rec4) {
    uint8_t *r = rec4 + at * tc5_rec(CMLD_Q4_K);
    *reinterpret_cast<uint2 *>(r + g * 2048 + (lane >> 1) * 128 + i * 16 + (lane & 1) * 8) = pk;
    int s = __dp4a((int)pk.y, 0x01010101, __dp4a((int)pk.x, 0x01010101, 0));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    const int m = lane >> 1;  // which sum of 16
    uint8_t *p = r + kTc5Rows * 256;
    if ((lane & 1) == 0) *reinterpret_cast<__half *>(p + g * 256 + (m >> 3) * 128 + i * 16 + (m & 7) * 2) = __int2half_rn(s);
    if (lane == 0) reinterpret_cast<float *>(p + tc5_rec_p(CMLD_Q4_K))[row] = d;
  }
  if (rec6) {
    // lane = 16h + 4q + 2c + half holds the classes 0..7 of its eight values 128h + 32q + 16c + 8 half ..: exchanges over half and c
    // leave it with the four bytes {l, l + 8, l + 16, l + 24} of two classes, those over q with two such words of one class
    const bool odd = lane & 1, up = lane & 2, q0 = lane & 4;
    const uint32_t r1 = __shfl_xor_sync(0xffffffffu, odd ? pk.x : pk.y, 1);
    const uint32_t a1 = odd ? r1 : pk.x, b1 = odd ? pk.y : r1;
    const uint32_t w01 = __byte_perm(a1, b1, 0x5140), w23 = __byte_perm(a1, b1, 0x7362);  // classes 4 odd + {0, 1}, {2, 3}: (l, l + 8)
    const uint32_t r2 = __shfl_xor_sync(0xffffffffu, up ? w01 : w23, 2);
    const uint32_t a2 = up ? r2 : w01, b2 = up ? w23 : r2;
    const uint32_t x = __byte_perm(a2, b2, 0x5410), y = __byte_perm(a2, b2, 0x7632);      // classes 4 odd + 2 up + {0, 1}
    const uint32_t r3 = __shfl_xor_sync(0xffffffffu, q0 ? x : y, 4);
    const int l = 4 * (lane & 1) + 2 * ((lane >> 1) & 1) + ((lane >> 2) & 1), h = lane >> 4, pair = (lane >> 3) & 1;  // quarters 2 pair, 2 pair + 1
    uint8_t *r = rec6 + at * tc5_rec(CMLD_Q6_K);
    *reinterpret_cast<uint2 *>(r + g * 2048 + (2 * l + h) * 128 + i * 16 + 8 * pair) = q0 ? make_uint2(r3, y) : make_uint2(x, r3);
    if (lane == 0) reinterpret_cast<float *>(r + kTc5Rows * 256)[row] = d;
  }
}

// The same for Q8_0 codes; scale: that of this lane's 32-value block.
__device__ __forceinline__ void tc5_store_0(uint2 pk, float scale, int lane, int b, int64_t ch, int tiles, uint8_t *rec0) {
  const int row = b % kTc5Rows;
  uint8_t *r = rec0 + (ch * tiles + b / kTc5Rows) * tc5_rec(CMLD_Q8_0);
  *reinterpret_cast<uint2 *>(r + (row >> 3) * 2048 + (lane >> 1) * 128 + (row & 7) * 16 + (lane & 1) * 8) = pk;
  if ((lane & 3) == 0) reinterpret_cast<float *>(r + kTc5Rows * 256)[(lane >> 2) * kTc5Rows + row] = scale;
}

}  // namespace cmld
