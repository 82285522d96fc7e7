// Pieces of the chunk-parallel recurrence kernels (gla_chunk.cu, delta_chunk.cu, gdn_chunk.cu): fp32 operands as a high and a low bf16 part,
// positions of the 64-token chunks, fragment loads, the triangular inverse.
#pragma once
#include "attn_device.cuh"
#include "ptx.cuh"

namespace tdb {
namespace chunk {

constexpr int kC = 64;            // tokens per chunk
constexpr int kFp = kC + 4;       // pitch of fp32 [64][64] matrices

// Lower 16 x 16 block (bi, bj) of a 64 x 64 matrix.
TDB_DEVICE constexpr int lower_block(int bi, int bj) { return bi * (bi + 1) / 2 + bj; }

struct HiLo {
  uint32_t hi, lo;
};
// Two fp32 values as packed bf16 high parts and packed bf16 remainders.
TDB_DEVICE HiLo split2(float a, float b) {
  HiLo r;
  r.hi = pack_bf16x2(a, b);
  const float2 h = unpack_bf16x2(r.hi);
  r.lo = pack_bf16x2(a - h.x, b - h.y);
  return r;
}
TDB_DEVICE float2 ld2(const __nv_bfloat16* p) { return unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p)); }

struct ChunkPos {
  int64_t t0;
  int n;       // tokens of the chunk
};
template <typename Args>
TDB_DEVICE ChunkPos chunk_pos(const Args& p, int chunk) {
  ChunkPos r;
  r.t0 = p.chunk_t0[chunk];
  const int64_t end = p.cu[p.chunk_seq[chunk] + 1];
  r.n = static_cast<int>(min(static_cast<int64_t>(kC), end - r.t0));
  return r;
}

TDB_DEVICE void ldmatrix_x4(uint32_t (&r)[4], const void* smem_row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_u32(smem_row)));
}

// Rows [0, 64) of `cols` bf16 columns starting at src (row stride ld) into smem with row pitch `pitch` elements, by `threads`
// threads; rows >= n are zero.  Asynchronous (cp.async).
TDB_DEVICE void load_tile(__nv_bfloat16* dst, int pitch, const __nv_bfloat16* src, int64_t ld, int cols, int n, int threads) {
  const int vec = cols >> 3;
  for (int i = threadIdx.x; i < kC * vec; i += threads) {
    const int r = i / vec, c = i - r * vec;
    attn::cp_async16(dst + r * pitch + c * 8, src + (r < n ? r * ld : 0) + c * 8, r < n);
  }
}

// A <- (I + A)^-1 for the strictly lower triangular A (blocks above the diagonal are scratch).
template <int THREADS>
TDB_DEVICE void invert_unit_lower(float* A) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp < 4) {                       // the 16 x 16 blocks on the diagonal by substitution, a column per lane
    float* D = A + (warp * 16) * kFp + warp * 16;
    float x[16];
    const int j = lane & 15;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float a = (i == j) ? 1.f : 0.f, b = 0.f;
#pragma unroll
      for (int m = 0; m < i; ++m) {
        if (m & 1) a = fmaf(-D[i * kFp + m], x[m], a);
        else b = fmaf(-D[i * kFp + m], x[m], b);
      }
      x[i] = a + b;
    }
    __syncwarp();
    if (lane < 16) {
#pragma unroll
      for (int i = 0; i < 16; ++i) D[i * kFp + j] = i >= j ? x[i] : 0.f;
    }
  }
  __syncthreads();
  // blocks below the diagonal, 16 then 32: A21 = -A22 (L21 A11); the product in brackets goes to the block above the diagonal.
  // A thread owns four neighbouring columns of a row.
#pragma unroll
  for (int n = 16; n <= 32; n *= 2) {
    const int per = n * n / 4, all = 32 / n * per;
    for (int i = tid; i < all; i += THREADS) {
      const int b = (i / per) * 2 * n, r = (i % per) / (n / 4), c = (i % (n / 4)) * 4;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int m = c & ~15; m < n; ++m) {
        const float l = A[(b + n + r) * kFp + b + m];
        const float4 v = *reinterpret_cast<const float4*>(A + (b + m) * kFp + b + c);
        a.x = fmaf(l, v.x, a.x); a.y = fmaf(l, v.y, a.y); a.z = fmaf(l, v.z, a.z); a.w = fmaf(l, v.w, a.w);
      }
      *reinterpret_cast<float4*>(A + (b + r) * kFp + b + n + c) = a;
    }
    __syncthreads();
    for (int i = tid; i < all; i += THREADS) {
      const int b = (i / per) * 2 * n, r = (i % per) / (n / 4), c = (i % (n / 4)) * 4;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int m = 0; m < (r & ~15) + 16; ++m) {
        const float l = -A[(b + n + r) * kFp + b + n + m];
        const float4 v = *reinterpret_cast<const float4*>(A + (b + m) * kFp + b + n + c);
        a.x = fmaf(l, v.x, a.x); a.y = fmaf(l, v.y, a.y); a.z = fmaf(l, v.z, a.z); a.w = fmaf(l, v.w, a.w);
      }
      *reinterpret_cast<float4*>(A + (b + n + r) * kFp + b + c) = a;
    }
    __syncthreads();
  }
}

}  // namespace chunk
}  // namespace tdb
