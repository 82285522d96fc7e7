// Gated delta rule forward in the chunk-parallel WY form on tensor cores (64-token chunks, K = 128).
//
// Per chunk (rows i, j of one chunk, gc = chunk-local cumulative log decay):
//     L[i][j] = beta_i (k_i . k_j) exp(gc_i - gc_j)        for i > j, else 0
//     A       = (I + L)^-1                                  (unit lower triangular)
//     w       = A (beta k exp(gc)),   u = A (beta v),       kd = k exp(gc_last - gc)
// then, sequentially over the chunks of a sequence with the state S [K x V] at the start of the chunk:
//     v_new   = u - w S
//     S      <- S exp(gc_last) + kd^T v_new
// and per chunk again:
//     o       = scale [ exp(gc) (q S) + tril(q k^T exp(gc_i - gc_j)) v_new ]
//
// The mathematics of the reference (python/triton_dist/kernels/nvidia/gdn.py:123 scaled-dot KK^T, :300 solve, :482 recompute
// w / u, :620 chunk state pass, :785 output; entry point :926).  Four launches, chained with programmatic dependent launch:
//   gdn_chunk_tables    one CTA: which chunk belongs to which sequence.  cu_seqlens is a device tensor; reading it on the host
//                       would make every call wait for the stream.
//   gdn_chunk_prepare   grid (chunks, H): KK^T, triangular inverse, w / u / kd
//   gdn_chunk_state     grid (V / 16 or V / 32, H, sequences): walks the chunks, S in fp32 registers
//   gdn_chunk_output    grid (chunks, H): q k^T, decay, two products
// Products use the warp-level bf16 MMA: 64 x 64 x 128 problems in a serial chain are too small for a tcgen05 / TMEM pipeline.
// What travels between the kernels (w, kd, u, v_new and S in bf16, as the tensor cores take them) is stored in the order in which
// the lanes of a warp hold the fragments of m16n8k16, so that every load is 16 coalesced bytes per lane and nothing is
// rearranged in the serial kernel.  Rows beyond the end of a sequence are zero.
//
// Bound by the state walk, a chain of dependent chunks.  One sequence of 8192 tokens, 16 heads, V = 128 (B200): with S in shared
// memory, 64 columns per CTA (32 CTAs) and row-major operands it took 6.5 us a chunk, now 0.95 us; the whole call 1606 -> 238 us
// (prepare 374 -> 65 us through the blocked inverse on all threads, output 292 -> 51 us, and no wait for the stream).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "tdb/chunk.cuh"
#include "tdb/gdn.h"
#include "tdb/launch.cuh"

namespace tdb {

namespace {

using attn::cp_async16;
using attn::cp_async_commit;
using attn::cp_async_wait;
using attn::ldmatrix_x4_trans;
using attn::mma_bf16;
using namespace chunk;

constexpr int kK = 128;            // head dim of q / k
constexpr int kKs = kK / 16;       // k-steps of a product over it
constexpr int kThreads = 256;      // prepare and output
constexpr int kLdK = kK + 8;       // bf16 row pitch of [64][128] tiles (272 bytes: ldmatrix without bank conflicts)
constexpr int kBlocks = 10;        // 16 x 16 blocks on and below the diagonal
constexpr int kWFrag = 4 * kKs * 32;       // uint4 of w and of kd per (chunk, head)
constexpr int kUFrag = 4 * 32;             // uint4 of u / v_new per 16 columns
constexpr int kSFrag = kKs * 32;           // uint4 of S per 16 columns

struct ChunkParams {
  const __nv_bfloat16* q;       // [T, H, K]
  const __nv_bfloat16* k;       // [T, H, K]
  const __nv_bfloat16* v;       // [T, H, V]
  const float* g;               // [T, H]
  const __nv_bfloat16* beta;    // [T, H]
  const int32_t* cu;            // [N + 1]
  int32_t* chunk_seq;           // [NC] sequence of every chunk
  int32_t* chunk_t0;            // [NC] first token of every chunk
  int32_t* seq_chunk0;          // [N + 1] first chunk of every sequence
  float* gcum;                  // [T, H] chunk-local cumulative log decay
  float* a_out;                 // [T, H, 64] or null
  float* decay;                 // [NC, H] exp(gc_last)
  uint4* w;                     // [NC, H, 4 row blocks, 8 k-steps, 32]     A fragments
  uint4* kd;                    // [NC, H, 8 row blocks of K, 4 k-steps, 32] A fragments of kd^T
  uint4* u;                     // [NC, H, V / 16, 4 row blocks, 32]        accumulator fragments of two 8-column tiles
  uint4* vnew;                  // [NC, H, V / 16, 4 k-steps, 32]           B fragments of two 8-column tiles
  uint4* hstate;                // [NC, H, V / 16, 8 k-steps, 32]           S at the start of the chunk, B fragments
  const float* h0;              // [N, H, K, V] or null
  float* ht;                    // [N, H, K, V] or null
  __nv_bfloat16* o;             // [T, H, V]
  int H, V, N, NC;              // NC: room in the tables, at least the number of chunks
  float scale;
};

// ------------------------------------------------------------------------------------------------------------------
// Kernel 0: chunk tables
// ------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) gdn_chunk_tables(const ChunkParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  pdl_launch_dependents();
  if (warp == 0) {
    int base = 0;
    for (int s0 = 0; s0 < p.N; s0 += 32) {
      const int s = s0 + lane;
      const int own = s < p.N ? (max(p.cu[s + 1] - p.cu[s], 0) + kC - 1) / kC : 0;
      int pre = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += x;
      }
      if (s < p.N) p.seq_chunk0[s] = min(base + pre - own, p.NC);
      base += __shfl_sync(0xffffffffu, pre, 31);
    }
    if (lane == 0) p.seq_chunk0[p.N] = min(base, p.NC);
  }
  __syncthreads();
  for (int s = warp; s < p.N; s += kThreads / 32) {
    const int c0 = p.seq_chunk0[s], c1 = p.seq_chunk0[s + 1], t0 = p.cu[s];
    for (int c = c0 + lane; c < c1; c += 32) {
      p.chunk_seq[c] = s;
      p.chunk_t0[c] = t0 + (c - c0) * kC;
    }
  }
}

// Two neighbouring accumulator tiles as one A fragment (also the form in which u travels).
TDB_DEVICE uint4 pack_tiles(const float (&a)[4], const float (&b)[4]) {
  return make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(b[0], b[1]), pack_bf16x2(b[2], b[3]));
}
TDB_DEVICE void zero(float (&a)[4]) { a[0] = a[1] = a[2] = a[3] = 0.f; }
TDB_DEVICE int block_row(int i) { return i < 1 ? 0 : i < 3 ? 1 : i < 6 ? 2 : 3; }

// 16 x 16 block (bi, bj) of X K^T, both [64][kLdK] in shared memory: two tiles of eight columns.
TDB_DEVICE void score_block(const __nv_bfloat16* x, const __nv_bfloat16* k, int bi, int bj, float (&acc)[2][4]) {
  const int lane = threadIdx.x & 31, mat = lane >> 3, mr = lane & 7;
  const __nv_bfloat16* a0 = x + (bi * 16 + (mat & 1) * 8 + mr) * kLdK + (mat >> 1) * 8;
  const __nv_bfloat16* b0 = k + (bj * 16 + (mat >> 1) * 8 + mr) * kLdK + (mat & 1) * 8;
  zero(acc[0]);
  zero(acc[1]);
#pragma unroll
  for (int ks = 0; ks < kKs; ++ks) {
    uint32_t a[4], b[4];
    ldmatrix_x4(a, a0 + ks * 16);
    ldmatrix_x4(b, b0 + ks * 16);
    mma_bf16(acc[0], a, b[0], b[1]);
    mma_bf16(acc[1], a, b[2], b[3]);
  }
}

// Four row blocks of (lower triangular X as fragments) x (64 tokens x 16 columns at b0 in shared memory).
TDB_DEVICE void lower_times(float (&acc)[4][2][4], const uint4* xf, const __nv_bfloat16* b0, int pitch) {
  const int lane = threadIdx.x & 31, mat = lane >> 3, mr = lane & 7;
#pragma unroll
  for (int rb = 0; rb < 4; ++rb) {
    zero(acc[rb][0]);
    zero(acc[rb][1]);
  }
#pragma unroll
  for (int kb = 0; kb < 4; ++kb) {
    uint32_t b[4];
    ldmatrix_x4_trans(b, b0 + (kb * 16 + (mat & 1) * 8 + mr) * pitch + (mat >> 1) * 8);
#pragma unroll
    for (int rb = kb; rb < 4; ++rb) {
      const uint4 x = xf[lower_block(rb, kb) * 32 + lane];
      const uint32_t a[4] = {x.x, x.y, x.z, x.w};
      mma_bf16(acc[rb][0], a, b[0], b[1]);
      mma_bf16(acc[rb][1], a, b[2], b[3]);
    }
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Kernel 1: per (chunk, head)
// ------------------------------------------------------------------------------------------------------------------
struct PrepSmem {
  __nv_bfloat16 k[kC][kLdK];
  union {
    float A[kC * kFp];                 // L, then (I + L)^-1
    struct {
      uint4 uf[kBlocks * 32];          // fragments of A beta
      uint4 wf[kBlocks * 32];          // fragments of A beta exp(gc)
    };
  };
  float gc[kC];
  float beta[kC];
  // followed by v [64][V + 8] bf16
};

__global__ void __launch_bounds__(kThreads, 3) gdn_chunk_prepare(const ChunkParams p) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  PrepSmem& s = *reinterpret_cast<PrepSmem*>(smem_raw);
  __nv_bfloat16* vs = reinterpret_cast<__nv_bfloat16*>(smem_raw + sizeof(PrepSmem));
  const int ldv = p.V + 8;
  const int c = blockIdx.x, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3, mat = lane >> 3, mr = lane & 7;
  pdl_wait();
  pdl_launch_dependents();
  if (c >= p.seq_chunk0[p.N]) return;
  const ChunkPos cp = chunk_pos(p, c);
  const int64_t Hk = static_cast<int64_t>(p.H) * kK, Hv = static_cast<int64_t>(p.H) * p.V;
  load_tile(&s.k[0][0], kLdK, p.k + cp.t0 * Hk + h * kK, Hk, kK, cp.n, kThreads);
  cp_async_commit();
  load_tile(vs, ldv, p.v + cp.t0 * Hv + static_cast<int64_t>(h) * p.V, Hv, p.V, cp.n, kThreads);
  cp_async_commit();
  const int64_t ch = static_cast<int64_t>(c) * p.H + h;
  if (warp == 0) {                      // inclusive scan of the log decays, two tokens per lane
    const int t = 2 * lane;
    const float a = t < cp.n ? p.g[(cp.t0 + t) * p.H + h] : 0.f;
    const float b = t + 1 < cp.n ? p.g[(cp.t0 + t + 1) * p.H + h] : 0.f;
    const float sum = a + b;
    float pre = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float x = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += x;
    }
    const float base = pre - sum;
    s.gc[t] = base + a;
    s.gc[t + 1] = base + a + b;
    if (t < cp.n) p.gcum[(cp.t0 + t) * p.H + h] = base + a;
    if (t + 1 < cp.n) p.gcum[(cp.t0 + t + 1) * p.H + h] = base + a + b;
    if (lane == 31) p.decay[ch] = __expf(base + a + b);
  } else if (warp == 1) {
    s.beta[lane] = lane < cp.n ? __bfloat162float(p.beta[(cp.t0 + lane) * p.H + h]) : 0.f;
    s.beta[lane + 32] = lane + 32 < cp.n ? __bfloat162float(p.beta[(cp.t0 + lane + 32) * p.H + h]) : 0.f;
  }
  cp_async_wait<1>();
  __syncthreads();
  for (int i = warp; i < kBlocks; i += kThreads / 32) {
    const int bi = block_row(i), bj = i - lower_block(bi, 0);
    float acc[2][4];
    score_block(&s.k[0][0], &s.k[0][0], bi, bj, acc);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = bi * 16 + g + 8 * (e >> 1), cc = bj * 16 + j * 8 + 2 * t4 + (e & 1);
        s.A[r * kFp + cc] = r > cc ? acc[j][e] * s.beta[r] * __expf(s.gc[r] - s.gc[cc]) : 0.f;
      }
  }
  // kd^T as A fragments, a warp per 16 rows of K
  {
    const float gl = s.gc[kC - 1];
    uint4* dst = p.kd + ch * kWFrag + warp * 4 * 32 + lane;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[4];
      ldmatrix_x4_trans(a, &s.k[ks * 16 + (mat >> 1) * 8 + mr][warp * 16 + (mat & 1) * 8]);
      const int t = ks * 16 + 2 * t4;
      const float f[4] = {__expf(gl - s.gc[t]), __expf(gl - s.gc[t + 1]), __expf(gl - s.gc[t + 8]), __expf(gl - s.gc[t + 9])};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 x = unpack_bf16x2(a[e]);
        a[e] = pack_bf16x2(x.x * f[2 * (e >> 1)], x.y * f[2 * (e >> 1) + 1]);
      }
      dst[ks * 32] = make_uint4(a[0], a[1], a[2], a[3]);
    }
  }
  __syncthreads();
  invert_unit_lower<kThreads>(s.A);
  if (p.a_out != nullptr) {
    for (int i = threadIdx.x; i < kC * kC; i += kThreads) {
      const int r = i / kC, cc = i - r * kC;
      if (r < cp.n) p.a_out[((cp.t0 + r) * p.H + h) * kC + cc] = r >= cc ? s.A[r * kFp + cc] : 0.f;
    }
  }
  // the fragments of A beta and A beta exp(gc) take the place of A
  {
    uint4 fu[2], fw[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = warp + 8 * r;
      if (i >= kBlocks) break;
      const int bi = block_row(i), c0 = (i - lower_block(bi, 0)) * 16 + 2 * t4;
      const float* a = s.A + (bi * 16 + g) * kFp + c0;
      const float* b = a + 8 * kFp;
      const float b0 = s.beta[c0], b1 = s.beta[c0 + 1], b2 = s.beta[c0 + 8], b3 = s.beta[c0 + 9];
      const float x[4] = {a[0] * b0, a[1] * b1, b[0] * b0, b[1] * b1}, y[4] = {a[8] * b2, a[9] * b3, b[8] * b2, b[9] * b3};
      const float e0 = __expf(s.gc[c0]), e1 = __expf(s.gc[c0 + 1]), e2 = __expf(s.gc[c0 + 8]), e3 = __expf(s.gc[c0 + 9]);
      const float xe[4] = {x[0] * e0, x[1] * e1, x[2] * e0, x[3] * e1}, ye[4] = {y[0] * e2, y[1] * e3, y[2] * e2, y[3] * e3};
      fu[r] = pack_tiles(x, y);
      fw[r] = pack_tiles(xe, ye);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = warp + 8 * r;
      if (i >= kBlocks) break;
      s.uf[i * 32 + lane] = fu[r];
      s.wf[i * 32 + lane] = fw[r];
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // w: a warp per 16 columns of K; u: a warp per 16 columns of V
  {
    float acc[4][2][4];
    lower_times(acc, s.wf, &s.k[0][warp * 16], kLdK);
    uint4* dst = p.w + ch * kWFrag + warp * 32 + lane;
#pragma unroll
    for (int rb = 0; rb < 4; ++rb) dst[rb * kKs * 32] = pack_tiles(acc[rb][0], acc[rb][1]);
  }
  const int vt = p.V / 16;
  for (int t = warp; t < vt; t += kThreads / 32) {
    float acc[4][2][4];
    lower_times(acc, s.uf, vs + t * 16, ldv);
    uint4* dst = p.u + (ch * vt + t) * kUFrag + lane;
#pragma unroll
    for (int rb = 0; rb < 4; ++rb) dst[rb * 32] = pack_tiles(acc[rb][0], acc[rb][1]);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Kernel 2: per (16 NP columns of V, head, sequence), sequential over the chunks.  Four warps: in the first product a warp owns 16
// tokens, in the second 32 rows of the state, which stays in its registers in fp32.  A chunk is two dependent products with an
// exchange through shared memory after each (S and v_new as B operands), about 500 cycles; its operands (34 KB) arrive STAGES - 1
// chunks ahead through cp.async.  The 16 columns keep the serial part short and spread 16 heads over 128 SMs; two such CTAs
// share an SM when there are more, and beyond two per SM a CTA takes 32 columns, which halves the operand traffic.
// ------------------------------------------------------------------------------------------------------------------
constexpr int kStateThreads = 128;
template <int NP>
struct StateLay {
  static constexpr int kStage = (2 * kWFrag + NP * kUFrag);      // uint4 of a stage: w | kd | u
  static constexpr int kPitch = NP * 16 + 8;                     // bf16 pitch of the exchange buffers
  static constexpr int smem(int stages) { return stages * kStage * 16 + (kK + kC) * kPitch * 2; }
};

template <int NP, int STAGES>
__global__ void __launch_bounds__(kStateThreads, 1) gdn_chunk_state(const ChunkParams p) {
  using L = StateLay<NP>;
  constexpr int kPitch = L::kPitch;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint4* ring = reinterpret_cast<uint4*>(smem_raw);
  __nv_bfloat16* sb = reinterpret_cast<__nv_bfloat16*>(ring + STAGES * L::kStage);     // [128][pitch] S
  __nv_bfloat16* vb = sb + kK * kPitch;                                                // [64][pitch] v_new
  const int tile0 = blockIdx.x * NP, h = blockIdx.y, seq = blockIdx.z, vt = p.V / 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3, mat = lane >> 3, mr = lane & 7;
  pdl_wait();
  pdl_launch_dependents();
  const int c0 = p.seq_chunk0[seq], nc = p.seq_chunk0[seq + 1] - c0;
  const int64_t st_off = ((static_cast<int64_t>(seq) * p.H + h) * kK + warp * 32 + g) * p.V + tile0 * 16 + 2 * t4;
  float S[2][2 * NP][4];
#pragma unroll
  for (int rb = 0; rb < 2; ++rb)
#pragma unroll
    for (int j = 0; j < 2 * NP; ++j) {
      zero(S[rb][j]);
      if (p.h0 != nullptr) {
        const float* src = p.h0 + st_off + static_cast<int64_t>(rb * 16) * p.V + j * 8;
        const float2 a = *reinterpret_cast<const float2*>(src), b = *reinterpret_cast<const float2*>(src + 8 * p.V);
        S[rb][j][0] = a.x; S[rb][j][1] = a.y; S[rb][j][2] = b.x; S[rb][j][3] = b.y;
      }
    }
  auto fetch = [&](int i) {            // chunk i of the sequence into stage i % STAGES
    if (i < nc) {
      const int64_t ch = static_cast<int64_t>(c0 + i) * p.H + h;
      uint4* st = ring + (i % STAGES) * L::kStage;
      const uint4 *w = p.w + ch * kWFrag, *kd = p.kd + ch * kWFrag, *u = p.u + (ch * vt + tile0) * kUFrag;
#pragma unroll
      for (int e = 0; e < kWFrag / kStateThreads; ++e) {
        const int at = e * kStateThreads + threadIdx.x;
        cp_async16(st + at, w + at, true);
        cp_async16(st + kWFrag + at, kd + at, true);
      }
#pragma unroll
      for (int e = 0; e < NP; ++e) {
        const int at = e * kStateThreads + threadIdx.x;
        cp_async16(st + 2 * kWFrag + at, u + at, true);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) fetch(i);
  float dec_next = nc > 0 ? p.decay[static_cast<int64_t>(c0) * p.H + h] : 0.f;
  cp_async_wait<STAGES - 2>();
  __syncthreads();
  uint4 wf[kKs];                       // this warp's 16 rows of w, loaded one chunk ahead
#pragma unroll
  for (int ks = 0; ks < kKs; ++ks) wf[ks] = ring[(warp * kKs + ks) * 32 + lane];
  for (int i = 0; i < nc; ++i) {
    const int64_t ch = static_cast<int64_t>(c0 + i) * p.H + h;
    const uint4* st = ring + (i % STAGES) * L::kStage;
    const float dec = dec_next;
    // S as bf16 for the tensor cores
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int j = 0; j < 2 * NP; ++j) {
        __nv_bfloat16* dst = sb + (warp * 32 + rb * 16 + g) * kPitch + j * 8 + 2 * t4;
        *reinterpret_cast<uint32_t*>(dst) = pack_bf16x2(S[rb][j][0], S[rb][j][1]);
        *reinterpret_cast<uint32_t*>(dst + 8 * kPitch) = pack_bf16x2(S[rb][j][2], S[rb][j][3]);
      }
    __syncthreads();                   // S complete; every warp has left the previous chunk, so its stage and v_new are free
    fetch(i + STAGES - 1);
    if (i + 1 < nc) dec_next = p.decay[ch + p.H];
    uint4 kf[2][4], uf[NP];
#pragma unroll
    for (int t = 0; t < NP; ++t) uf[t] = st[2 * kWFrag + t * kUFrag + warp * 32 + lane];
    // w S: even and odd k-steps in sums of their own, so that the chain of dependent products is half as long
    float acc[2][2 * NP][4];
#pragma unroll
    for (int j = 0; j < 2 * NP; ++j) {
      zero(acc[0][j]);
      zero(acc[1][j]);
    }
#pragma unroll
    for (int ks = 0; ks < kKs; ++ks) {
      const uint32_t a[4] = {wf[ks].x, wf[ks].y, wf[ks].z, wf[ks].w};
#pragma unroll
      for (int t = 0; t < NP; ++t) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, sb + (ks * 16 + (mat & 1) * 8 + mr) * kPitch + t * 16 + (mat >> 1) * 8);
        mma_bf16(acc[ks & 1][2 * t], a, b[0], b[1]);
        mma_bf16(acc[ks & 1][2 * t + 1], a, b[2], b[3]);
        if ((ks >> 1) == warp)         // the state before this chunk, for the output kernel
          p.hstate[((ch * vt + tile0 + t) * kKs + ks) * 32 + lane] = make_uint4(b[0], b[1], b[2], b[3]);
      }
    }
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) kf[rb][ks] = st[kWFrag + ((warp * 2 + rb) * 4 + ks) * 32 + lane];
    // v_new = u - w S
#pragma unroll
    for (int t = 0; t < NP; ++t) {
      const uint32_t uw[4] = {uf[t].x, uf[t].y, uf[t].z, uf[t].w};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 a = unpack_bf16x2(uw[2 * j]), b = unpack_bf16x2(uw[2 * j + 1]);
        __nv_bfloat16* dst = vb + (warp * 16 + g) * kPitch + t * 16 + j * 8 + 2 * t4;
        const float (&x)[4] = acc[0][2 * t + j], (&y)[4] = acc[1][2 * t + j];
        *reinterpret_cast<uint32_t*>(dst) = pack_bf16x2(a.x - (x[0] + y[0]), a.y - (x[1] + y[1]));
        *reinterpret_cast<uint32_t*>(dst + 8 * kPitch) = pack_bf16x2(b.x - (x[2] + y[2]), b.y - (x[3] + y[3]));
      }
    }
    cp_async_wait<STAGES - 2>();       // the next chunk's operands (this thread's part)
    __syncthreads();                   // v_new and the next stage complete
    {
      const uint4* nx = ring + ((i + 1) % STAGES) * L::kStage;
#pragma unroll
      for (int ks = 0; ks < kKs; ++ks) wf[ks] = nx[(warp * kKs + ks) * 32 + lane];
    }
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int j = 0; j < 2 * NP; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[rb][j][e] *= dec;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int t = 0; t < NP; ++t) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, vb + (ks * 16 + (mat & 1) * 8 + mr) * kPitch + t * 16 + (mat >> 1) * 8);
#pragma unroll
        for (int rb = 0; rb < 2; ++rb) {
          const uint32_t a[4] = {kf[rb][ks].x, kf[rb][ks].y, kf[rb][ks].z, kf[rb][ks].w};
          mma_bf16(S[rb][2 * t], a, b[0], b[1]);
          mma_bf16(S[rb][2 * t + 1], a, b[2], b[3]);
        }
        if (ks == warp) p.vnew[((ch * vt + tile0 + t) * 4 + ks) * 32 + lane] = make_uint4(b[0], b[1], b[2], b[3]);
      }
  }
  cp_async_wait<0>();
  if (p.ht != nullptr) {
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int j = 0; j < 2 * NP; ++j) {
        float* dst = p.ht + st_off + static_cast<int64_t>(rb * 16) * p.V + j * 8;
        *reinterpret_cast<float2*>(dst) = make_float2(S[rb][j][0], S[rb][j][1]);
        *reinterpret_cast<float2*>(dst + 8 * p.V) = make_float2(S[rb][j][2], S[rb][j][3]);
      }
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Kernel 3: per (chunk, head).  A warp owns 16 columns of V for RB of the four row blocks, so that S and v_new go from memory to
// its registers once; q and the masked scores are the shared operands.
// ------------------------------------------------------------------------------------------------------------------
struct OutSmem {
  __nv_bfloat16 q[kC][kLdK];
  __nv_bfloat16 k[kC][kLdK];
  uint4 pf[kBlocks * 32];          // masked, decayed scores as A fragments
  float gc[kC];
};

template <int RB>
__global__ void __launch_bounds__(kThreads, 2) gdn_chunk_output(const ChunkParams p) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  OutSmem& s = *reinterpret_cast<OutSmem*>(smem_raw);
  const int c = blockIdx.x, h = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3, mat = lane >> 3, mr = lane & 7;
  pdl_wait();
  pdl_launch_dependents();
  if (c >= p.seq_chunk0[p.N]) return;
  const ChunkPos cp = chunk_pos(p, c);
  const int64_t Hk = static_cast<int64_t>(p.H) * kK, ch = static_cast<int64_t>(c) * p.H + h;
  load_tile(&s.q[0][0], kLdK, p.q + cp.t0 * Hk + h * kK, Hk, kK, cp.n, kThreads);
  load_tile(&s.k[0][0], kLdK, p.k + cp.t0 * Hk + h * kK, Hk, kK, cp.n, kThreads);
  cp_async_commit();
  constexpr int kParts = 4 / RB, kTiles = kThreads / 32 / kParts;      // warps side by side
  const int part = warp / kTiles, vt = p.V / 16;
  uint4 sf[kKs], vf[4];
  auto fetch = [&](int t) {
#pragma unroll
    for (int ks = 0; ks < kKs; ++ks) sf[ks] = p.hstate[((ch * vt + t) * kKs + ks) * 32 + lane];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) vf[ks] = p.vnew[((ch * vt + t) * 4 + ks) * 32 + lane];
  };
  const int t_first = warp % kTiles;
  if (t_first < vt) fetch(t_first);
  if (threadIdx.x < kC) s.gc[threadIdx.x] = p.gcum[(cp.t0 + min(static_cast<int>(threadIdx.x), cp.n - 1)) * p.H + h];
  cp_async_wait<0>();
  __syncthreads();
  for (int i = warp; i < kBlocks; i += kThreads / 32) {
    const int bi = block_row(i), bj = i - lower_block(bi, 0);
    float acc[2][4];
    score_block(&s.q[0][0], &s.k[0][0], bi, bj, acc);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = bi * 16 + g + 8 * (e >> 1), cc = bj * 16 + j * 8 + 2 * t4 + (e & 1);
        acc[j][e] = r >= cc ? acc[j][e] * __expf(s.gc[r] - s.gc[cc]) : 0.f;
      }
    s.pf[i * 32 + lane] = pack_tiles(acc[0], acc[1]);
  }
  __syncthreads();
  for (int t = t_first; t < vt; t += kTiles) {
    if (t != t_first) fetch(t);
    float acc[RB][2][4];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const int rb = part * RB + r;
      zero(acc[r][0]);
      zero(acc[r][1]);
#pragma unroll
      for (int ks = 0; ks < kKs; ++ks) {
        uint32_t a[4];
        ldmatrix_x4(a, &s.q[rb * 16 + (mat & 1) * 8 + mr][ks * 16 + (mat >> 1) * 8]);
        mma_bf16(acc[r][0], a, sf[ks].x, sf[ks].y);
        mma_bf16(acc[r][1], a, sf[ks].z, sf[ks].w);
      }
      const float e0 = __expf(s.gc[rb * 16 + g]), e1 = __expf(s.gc[rb * 16 + g + 8]);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        acc[r][j][0] *= e0; acc[r][j][1] *= e0;
        acc[r][j][2] *= e1; acc[r][j][3] *= e1;
      }
#pragma unroll
      for (int kb = 0; kb < 4; ++kb) {
        if (kb > rb) break;
        const uint4 x = s.pf[lower_block(rb, kb) * 32 + lane];
        const uint32_t a[4] = {x.x, x.y, x.z, x.w};
        mma_bf16(acc[r][0], a, vf[kb].x, vf[kb].y);
        mma_bf16(acc[r][1], a, vf[kb].z, vf[kb].w);
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int row = rb * 16 + g + 8 * half;
        if (row >= cp.n) continue;
        __nv_bfloat16* dst = p.o + ((cp.t0 + row) * p.H + h) * p.V + t * 16 + 2 * t4;
#pragma unroll
        for (int j = 0; j < 2; ++j)
          *reinterpret_cast<uint32_t*>(dst + j * 8) = pack_bf16x2(acc[r][j][2 * half] * p.scale, acc[r][j][2 * half + 1] * p.scale);
      }
    }
  }
}

template <int NP, int STAGES>
cudaError_t launch_state(const ChunkParams& p, cudaStream_t stream) {
  static SmemOptIn opt;
  constexpr int smem = StateLay<NP>::smem(STAGES);
  const cudaError_t e = opt.ensure(gdn_chunk_state<NP, STAGES>, smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(gdn_chunk_state<NP, STAGES>, dim3(p.V / (16 * NP), p.H, p.N), dim3(kStateThreads), smem, stream, p);
}
template <int RB>
cudaError_t launch_output(const ChunkParams& p, cudaStream_t stream) {
  static SmemOptIn opt;
  constexpr int smem = static_cast<int>(sizeof(OutSmem));
  const cudaError_t e = opt.ensure(gdn_chunk_output<RB>, smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(gdn_chunk_output<RB>, dim3(p.NC, p.H), dim3(kThreads), smem, stream, p);
}

}  // namespace

cudaError_t launch_gdn_chunk_fwd(const GdnChunkArgs& a, cudaStream_t stream) {
  if (a.K != kK || a.V % 64 != 0 || a.V < 64 || a.V > 256 || a.num_seqs < 1 || a.num_chunks < 1) return cudaErrorInvalidValue;
  ChunkParams p;
  p.q = reinterpret_cast<const __nv_bfloat16*>(a.q);
  p.k = reinterpret_cast<const __nv_bfloat16*>(a.k);
  p.v = reinterpret_cast<const __nv_bfloat16*>(a.v);
  p.g = a.g;
  p.beta = reinterpret_cast<const __nv_bfloat16*>(a.beta);
  p.cu = a.cu_seqlens;
  p.chunk_seq = a.tables;
  p.chunk_t0 = a.tables + a.num_chunks;
  p.seq_chunk0 = a.tables + 2 * static_cast<int64_t>(a.num_chunks);
  p.gcum = a.g_cumsum;
  p.a_out = a.a_out;
  p.decay = a.decay;
  p.w = reinterpret_cast<uint4*>(a.w);
  p.kd = reinterpret_cast<uint4*>(a.kd);
  p.u = reinterpret_cast<uint4*>(a.u);
  p.vnew = reinterpret_cast<uint4*>(a.v_new);
  p.hstate = reinterpret_cast<uint4*>(a.h_chunks);
  p.h0 = a.initial_state;
  p.ht = a.final_state;
  p.o = reinterpret_cast<__nv_bfloat16*>(a.o);
  p.H = a.H; p.V = a.V; p.N = a.num_seqs; p.NC = a.num_chunks;
  p.scale = a.scale;
  cudaError_t e = launch_pdl(gdn_chunk_tables, dim3(1), dim3(kThreads), 0, stream, p);
  if (e != cudaSuccess) return e;
  static SmemOptIn opt;
  e = opt.ensure(gdn_chunk_prepare, 128 * 1024);
  if (e != cudaSuccess) return e;
  e = launch_pdl(gdn_chunk_prepare, dim3(a.num_chunks, a.H), dim3(kThreads), sizeof(PrepSmem) + kC * (a.V + 8) * 2, stream, p);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t ctas = static_cast<int64_t>(a.num_seqs) * a.H * (a.V / 16);
  e = ctas <= sms ? launch_state<1, 5>(p, stream) : ctas <= 2 * sms ? launch_state<1, 3>(p, stream) : launch_state<2, 3>(p, stream);
  if (e != cudaSuccess) return e;
  return a.V == 64 ? launch_output<2>(p, stream) : launch_output<4>(p, stream);
}

}  // namespace tdb
