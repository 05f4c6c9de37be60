// Operand-tile layout of the tensor-core Hankel transform (hankel_tc.cu), shared with the kernels
// that write its A operand directly (k_hankel_tc_prep, and the spectral update k_spec_point, which
// forms the next inverse transform's operand from the stage estimate it has just computed).
//
// A tile of 64 frequencies becomes 128 MMA rows (row 2j = Re A(w0 + j, .), row 2j + 1 = Im A(w0 + j,
// .)) by 64 reduction elements, bf16, in the K-major no-swizzle core-matrix layout: 8x8 core matrices
// of 128 contiguous bytes (8 rows of 16 bytes), core matrices adjacent in K 128 bytes apart, adjacent
// in M 1024 bytes apart.  Each FP32 value x is stored as x_hi = bf16(x) in the first 16 KB of the
// 32 KB tile pair and x_lo = bf16(x - x_hi) in the second.  Tiles of azimuthal mode m are ordered
// [m][w / 64][k / 64].
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "common.cuh"
#include "uppe_internal.h"

#define TC_ROWS 128  // MMA rows per tile (64 frequencies x re/im)
#define TC_W 64      // frequencies per tile
#define TC_N 128     // output columns per tile
#define TC_K 64      // reduction elements per shared tile (four K=16 MMAs)
#define TC_TILE_BYTES (TC_ROWS * TC_K * 2)  // 16 KB per bf16 operand tile

// Byte offset of element (row, k) of a 128 x 64 bf16 tile.
__device__ __forceinline__ uint32_t core_off(int row, int k) {
    return (uint32_t)((row >> 3) * 1024 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
    hi = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

// Element (w, k) of azimuthal mode m of the A operand: v split into its four bf16 parts.
__device__ __forceinline__ void tc_store_split(uint8_t* __restrict__ Atc, int nwt, int nkt, int m, int w, int k,
                                               float2 v) {
    __nv_bfloat16 rh, rl, ih, il;
    split_bf16(v.x, rh, rl);
    split_bf16(v.y, ih, il);
    const unsigned uw = (unsigned)w, uk = (unsigned)k;  // both >= 0: shifts and masks
    const int wl = (int)(uw % TC_W), kk = (int)(uk % TC_K);
    uint8_t* tile = Atc + (((size_t)m * nwt + uw / TC_W) * nkt + uk / TC_K) * (size_t)(2 * TC_TILE_BYTES);
    const uint32_t ore = core_off(2 * wl, kk), oim = core_off(2 * wl + 1, kk);
    *reinterpret_cast<__nv_bfloat16*>(tile + ore) = rh;
    *reinterpret_cast<__nv_bfloat16*>(tile + oim) = ih;
    *reinterpret_cast<__nv_bfloat16*>(tile + TC_TILE_BYTES + ore) = rl;
    *reinterpret_cast<__nv_bfloat16*>(tile + TC_TILE_BYTES + oim) = il;
}

// The bf16 halves of a pair of values as two 32-bit words, the first value in the low half.
__device__ __forceinline__ void split_bf16x2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a - __low2float(h), b - __high2float(h));
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// tc_store_split for neighbouring lanes k, k ^ 1 of one w (both active): the even lane stores the real row's two
// values, the odd lane the imaginary row's, 4 bytes a store instead of 2.  (In the spectral update and the operand pre-pass,
// whose eight neighbouring lanes already fill a 16-byte row, the exchange cost more than the stores saved.)
__device__ __forceinline__ void tc_store_pair(uint8_t* __restrict__ Atc, int nwt, int nkt, int m, int w, int k,
                                              float2 v) {
    const bool odd = k & 1;
    const float got = __shfl_xor_sync(3u << (threadIdx.x & 30), odd ? v.x : v.y, 1);
    uint32_t hi, lo;
    split_bf16x2(odd ? got : v.x, odd ? v.y : got, hi, lo);
    const unsigned uw = (unsigned)w, uk = (unsigned)k & ~1u;
    uint8_t* tile = Atc + (((size_t)m * nwt + uw / TC_W) * nkt + uk / TC_K) * (size_t)(2 * TC_TILE_BYTES);
    const uint32_t o = core_off(2 * (int)(uw % TC_W) + (odd ? 1 : 0), (int)(uk % TC_K));
    *reinterpret_cast<uint32_t*>(tile + o) = hi;
    *reinterpret_cast<uint32_t*>(tile + TC_TILE_BYTES + o) = lo;
}

// Eight columns k .. k + 7 (k a multiple of 8) of one row (part 0: re, 1: im of w) of azimuthal mode 0: x[0 .. 8)
// as one 16-byte store to each tile.
__device__ __forceinline__ void tc_store_row8(uint8_t* __restrict__ Atc, int nkt, int w, int part, int k,
                                              const float (&x)[8]) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) split_bf16x2(x[2 * i], x[2 * i + 1], h[i], l[i]);
    const unsigned uw = (unsigned)w, uk = (unsigned)k;
    uint8_t* tile = Atc + ((size_t)(uw / TC_W) * nkt + uk / TC_K) * (size_t)(2 * TC_TILE_BYTES);
    const uint32_t o = core_off(2 * (int)(uw % TC_W) + part, (int)(uk % TC_K));
    *reinterpret_cast<uint4*>(tile + o) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(tile + TC_TILE_BYTES + o) = make_uint4(l[0], l[1], l[2], l[3]);
}

// The next inverse transform's operand, written by the spectral update of the stage before it:
// Atc NULL when not asked.
struct TcNext {
    uint8_t* Atc;
    int logN2;         // azimuthal nodes (the fast axis of the field)
    int nwt, nkt, Nk;  // tile counts of the inverse transform (reduction over the Nk radial modes)
    StepArgs z;        // the next evaluation's z
};
