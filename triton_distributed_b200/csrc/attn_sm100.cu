// Prefill / context attention on the 5th-generation tensor cores (head dim 128 or 64, bf16, GQA, var-len, causal).
//
// Two launches:
//   attn_pack_kv_kernel     gathers the visible KV of every sequence out of the paged cache into TMA-friendly dense
//                           tensors: K [B * Hkv][Lp][D] and V transposed, Vt [B * Hkv][D][Lp] (Lp = padded max length,
//                           zero beyond a sequence's length).  With V transposed both products of attention are plain
//                           K-major x K-major UMMAs, and paging no longer concerns the main kernel.  One read and one
//                           write of the KV, against O(S^2) work in the main kernel.
//   flash_fwd_sm100_kernel  one CTA = 128 query rows of one head.  Warp 0 loads Q once and streams K / Vt blocks of
//                           64 tokens by TMA (two stages); warp 1 issues tcgen05.mma: S = Q K^T (128 x 64, K = 128)
//                           into TMEM, and after the softmax warps have written P (bf16, 128B-swizzled shared
//                           memory) O += P V (128 x 128, K = 64), accumulated in a second TMEM buffer over all blocks;
//                           warps 2-5 (one thread per query row) read S with tcgen05.ld, apply scale / mask / softmax
//                           in the log2 domain and write P.  The output is NOT read back per block: the exponentials
//                           use a reference maximum that is only raised when the row maximum has grown by more than
//                           2^8 (P stays below 256, exact in the final division because O and the row sum share the
//                           reference); only then the warp rescales its O rows in TMEM (tcgen05.ld / st).  S of block
//                           j + 1 is issued as soon as S of block j has been read, so the tensor core works during the
//                           exponentials; the output row is read once, after the last block.
//   flash_fwd_sm100_duo_kernel  256 query rows per CTA, P in TMEM: longer sequences, and heads of 64.
// Every wait is bounded; a timeout is recorded, the CTA stops issuing work, frees its TMEM and returns.
//
// Reference behaviour being matched (not its code): mega_triton_kernel/kernels/flash_attn.py:33-372 (TMA +
// warp-specialised prefill attention), kernels/nvidia/sp_ag_attention_intra_node.py:256-425 (var-len cu_seqlens,
// causal offsets of context-parallel chunks).
#include <cuda.h>
#include <cuda_bf16.h>

#include "tdb/attn.h"
#include "tdb/attn_sm100.cuh"
#include "tdb/launch.cuh"
#include "tdb/ptx.cuh"
#include "tdb/status.h"

namespace tdb {

namespace {

constexpr int kD = 128;            // head dim
constexpr int kThreads = 192;      // warp 0 TMA, warp 1 MMA, warps 2-5 softmax
constexpr int kUmmaK = 16;
constexpr int kQBytes = kBM * kD * 2;        // 32 KB: two [128 x 64] swizzled halves
constexpr int kKBytes = kBN * kD * 2;        // 16 KB: two [64 x 64] halves
constexpr int kVBytes = kD * kBN * 2;        // 16 KB: Vt block [128 d x 64 tokens]
constexpr int kPBytes = kBM * kBN * 2;       // 16 KB
// Shared-memory layout for a ring of STAGES K / Vt blocks: Q | K ring | Vt ring | P | barriers
template <int STAGES>
struct Lay {
  static constexpr int kOffK = kQBytes;
  static constexpr int kOffV = kOffK + STAGES * kKBytes;
  static constexpr int kOffP = kOffV + STAGES * kVBytes;
  static constexpr int kOffBar = kOffP + kPBytes;
  static constexpr int kSmem = kOffBar + (2 * STAGES + 8) * 8 + 64;
};
static_assert(2 * (Lay<2>::kSmem + 1024) <= 227 * 1024, "two CTAs of the two-stage prefill kernel must fit one SM");
static_assert(Lay<5>::kSmem + 1024 <= 227 * 1024, "the five-stage prefill kernel must fit one SM");
constexpr int kTmemCols = 256;     // S: columns [0, 64), PV: columns [64, 192)

// ------------------------------------------------------------------------------------------------------------------
// KV packing: grid (Lp / 64, Hkv, B), 256 threads
// ------------------------------------------------------------------------------------------------------------------
struct PackParams {
  const __nv_bfloat16* k_cache;
  const __nv_bfloat16* v_cache;
  const int32_t* block_table;
  const int32_t* kv_lens;
  int max_pages, page_size, Hkv, Lp;
  __nv_bfloat16* k_out;        // [B * Hkv][Lp][D]
  __nv_bfloat16* vt_out;       // [B * Hkv][D][Lp]
  const float* k_scale;        // tied form (see AttnKV): V is the raw key, K the key times its factor
};

template <int D, bool TIED>
__global__ void __launch_bounds__(256) attn_pack_kv_kernel(const PackParams p) {
  __shared__ __align__(16) __nv_bfloat16 vs[kBN][D + 8];
  const int t0 = blockIdx.x * kBN, h = blockIdx.y, b = blockIdx.z;
  const int kv_len = p.kv_lens[b];
  // no block of 64 or 128 keys reaches that far (five prompts of 700 to 1600 keys, heads of 64: the call 88.7 us without this, 86.4 with)
  if (t0 >= (kv_len + 127) / 128 * 128) return;
  const int64_t bh = static_cast<int64_t>(b) * p.Hkv + h;
  for (int i = threadIdx.x; i < kBN * (D / 8); i += 256) {
    const int r = i / (D / 8), c = (i % (D / 8)) * 8;
    const int tok = t0 + r;
    uint4 kv = make_uint4(0u, 0u, 0u, 0u), vv = make_uint4(0u, 0u, 0u, 0u);
    if (tok < kv_len) {
      const int page = p.block_table[static_cast<int64_t>(b) * p.max_pages + tok / p.page_size];
      const int64_t off = ((static_cast<int64_t>(page) * p.page_size + tok % p.page_size) * p.Hkv + h) * D + c;
      kv = *reinterpret_cast<const uint4*>(p.k_cache + off);
      if constexpr (TIED) {
        vv = kv;
        const float f = p.k_scale[static_cast<int64_t>(page) * p.page_size + tok % p.page_size];
        uint32_t* w = reinterpret_cast<uint32_t*>(&kv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 x = unpack_bf16x2(w[i]);
          w[i] = pack_bf16x2(x.x * f, x.y * f);
        }
      } else {
        vv = *reinterpret_cast<const uint4*>(p.v_cache + off);
      }
    }
    *reinterpret_cast<uint4*>(p.k_out + (bh * p.Lp + tok) * D + c) = kv;
    *reinterpret_cast<uint4*>(&vs[r][c]) = vv;
  }
  __syncthreads();
  // Vt[d][t0 .. t0 + 63]: a thread writes D / 4 consecutive tokens of one d
  constexpr int kRun = kBN * D / 256;
  const int d = threadIdx.x % D, part = threadIdx.x / D;
  __nv_bfloat16* dst = p.vt_out + (bh * D + d) * p.Lp + t0 + part * kRun;
#pragma unroll
  for (int i = 0; i < kRun; i += 8) {
    __align__(16) __nv_bfloat16 tmp[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) tmp[j] = vs[part * kRun + i + j][d];
    *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(tmp);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Main kernel
// ------------------------------------------------------------------------------------------------------------------
template <int kStages, int kCtasPerSm, bool CAP>
__global__ void __launch_bounds__(kThreads, kCtasPerSm)
flash_fwd_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_vt, const FwdParams p) {
  // Two CTAs share an SM (one runs its exponentials while the other's products are on the tensor core), which leaves no
  // room for an alignment slack: the kernel has no static shared memory, so the dynamic window starts at offset 0 of the
  // CTA's allocation; the 1024-byte alignment the swizzled tiles need is checked, not assumed.
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && p.error_flag != nullptr) *p.error_flag = 2;
    return;
  }
  using L = Lay<kStages>;
  constexpr int kOffK = L::kOffK, kOffV = L::kOffV, kOffP = L::kOffP;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* q_full = bars;
  uint64_t* s_full = bars + 1;
  uint64_t* s_free = bars + 2;
  uint64_t* p_full = bars + 3;
  uint64_t* pv_full = bars + 4;
  uint64_t* kv_full = bars + 5;                 // [kStages]
  uint64_t* kv_empty = kv_full + kStages;       // [kStages]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(kv_empty + kStages);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int b = blockIdx.z, head = blockIdx.y;
  const int q_begin = p.cu_seqlens_q[b], q_len = p.cu_seqlens_q[b + 1] - q_begin;
  // causal tiles get longer towards the end of a sequence: the long ones are scheduled first (the block scheduler hands
  // out blockIdx.x in increasing order), so the tail of the launch consists of short tiles
  const int row0 = (p.causal ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x)) * kBM;
  if (row0 >= q_len) return;                      // whole CTA, before any barrier or TMEM use
  const int kv_len = p.kv_lens[b];
  const int pos0 = p.q_pos0 ? p.q_pos0[b] : (kv_len - q_len);
  const int hkv = head / p.group;
  const int rows_here = min(q_len - row0, kBM);
  int kv_end = p.causal ? min(kv_len, pos0 + row0 + rows_here) : kv_len;
  if (kv_end < 0) kv_end = 0;
  const int nblk = (kv_end + kBN - 1) / kBN;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, 128);
    mbar_init(p_full, 128);
    mbar_init(pv_full, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_s = tmem_base, tmem_pv = tmem_base + 64;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_vt);
      mbar_arrive_expect_tx(q_full, kQBytes);
      tma_load_2d(smem, &tmap_q, q_full, head * kD, q_begin + row0);
      tma_load_2d(smem + kQBytes / 2, &tmap_q, q_full, head * kD + 64, q_begin + row0);
      const int z = b * p.Hkv + hkv;
      for (int j = 0; j < nblk; ++j) {
        const int s = j % kStages;
        const uint32_t ph = (j / kStages) & 1;
        if (!mbar_wait(&kv_empty[s], ph ^ 1, abort_flag, kWaitNs)) {
          *abort_flag = 1;
          break;
        }
        mbar_arrive_expect_tx(&kv_full[s], kKBytes + kVBytes);
        uint8_t* sk = smem + kOffK + s * kKBytes;
        tma_load_3d(sk, &tmap_k, &kv_full[s], 0, j * kBN, z);
        tma_load_3d(sk + kKBytes / 2, &tmap_k, &kv_full[s], 64, j * kBN, z);
        tma_load_3d(smem + kOffV + s * kVBytes, &tmap_vt, &kv_full[s], j * kBN, 0, z);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc(1u, kBM, kBN);
      constexpr uint32_t idesc_pv = make_idesc(1u, kBM, kD);
      bool ok = mbar_wait(q_full, 0, abort_flag, kWaitNs);
      const uint32_t sq = smem_u32(smem);
      const uint32_t sp = smem_u32(smem + kOffP);
      auto issue_s = [&](int j) -> bool {
        const int s = j % kStages;
        if (!mbar_wait(&kv_full[s], (j / kStages) & 1, abort_flag, kWaitNs)) return false;
        if (j > 0 && !mbar_wait(s_free, (j - 1) & 1, abort_flag, kWaitNs)) return false;
        tc_fence_after_sync();
        const uint32_t sk = smem_u32(smem + kOffK + s * kKBytes);
#pragma unroll
        for (int k = 0; k < kD / kUmmaK; ++k) {
          const uint64_t adesc = make_smem_desc_sw128(sq + (k / 4) * (kQBytes / 2)) + 2 * (k % 4);
          const uint64_t bdesc = make_smem_desc_sw128(sk + (k / 4) * (kKBytes / 2)) + 2 * (k % 4);
          umma_f16(tmem_s, adesc, bdesc, idesc_s, k > 0 ? 1u : 0u);
        }
        umma_commit(s_full);
        return true;
      };
      if (ok && nblk > 0) ok = issue_s(0);
      for (int j = 0; j < nblk && ok; ++j) {
        // S of the next block goes out before this block's P is waited for: it only needs S of block j to have been read
        if (j + 1 < nblk) ok = issue_s(j + 1);
        if (!ok) break;
        if (!mbar_wait(p_full, j & 1, abort_flag, kWaitNs)) { ok = false; break; }
        tc_fence_after_sync();
        const int s = j % kStages;
        const uint32_t sv = smem_u32(smem + kOffV + s * kVBytes);
#pragma unroll
        for (int k = 0; k < kBN / kUmmaK; ++k)
          umma_f16(tmem_pv, make_smem_desc_sw128(sp) + 2 * k, make_smem_desc_sw128(sv) + 2 * k, idesc_pv,
                   (j > 0 || k > 0) ? 1u : 0u);   // O accumulates over all blocks
        umma_commit(pv_full);
        umma_commit(&kv_empty[s]);      // K (read by S of this block) and Vt of this stage are free again
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    // ------------------------------------------------------------ softmax + output (one thread per query row)
    TileCtx t;
    t.s_full = s_full; t.s_free = s_free; t.p_full = p_full; t.pv_full = pv_full;
    t.tmem_s = tmem_s; t.tmem_pv = tmem_pv;
    t.p_smem = smem + kOffP;
    t.row0 = row0; t.rows_here = rows_here; t.nblk = nblk;
    softmax_tile<kD, CAP>(p, t, warp, lane, q_begin, head, kv_len, pos0, abort_flag);
  }

  // ------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.error_flag != nullptr) *p.error_flag = 1;
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Two-tile form: one CTA per SM handles 256 query rows of a head as two 128-row tiles that share every block of 128 keys.  A tile's
// chain is serial (S, softmax, P V, next S), so the tiles take turns: while one is in its exponentials the other's products are on
// the tensor core.  P never leaves TMEM: a softmax thread reads its part of a row of S and writes P as bf16 over the first half of
// the row, where P V takes its A operand from.  With 128 keys a block and no P in shared memory an MMA reads no more than 64 bytes of
// shared memory a clock (with 64 keys, two buffers of S and products ahead of the softmax the kernel took 733 us for the 549 of
// this layout with four softmax warps a tile: an S of 64 keys reads more than it computes).
// Two threads share a row, 64 keys each: they exchange the maximum of a block and, at the end, the sums.  Eight warps a tile hide the
// latencies of TMEM, barriers and exponentials that four left open: 8192 tokens, 32 heads of 128: 549 us, now 508 for this kernel alone,
// which is 1080 TFLOP/s (with one tile per CTA and P in shared memory 790 us; the call with its packing launch takes 590, 931 TFLOP/s).
// 640 threads: warps 0-7 softmax of tile 0 (keys 0-63, then 64-127 of a block), 8-15 of tile 1, warp 16 TMA, warp 17 MMA; the
// fifth warpgroup gives registers to the others, which hold 64 scores a thread.  K and V
// blocks share one ring in the order K0 V0 K1 V1 ..., in which they are also released.  The tensor core executes one thread's MMAs in
// order, so S of the next block may be issued right behind the P V whose P it overwrites, and the commit behind it also says
// that this P V is done: one barrier per tile and direction.
// What bounds it: a pair of 128 x 128 blocks takes 3500 clocks, 1500 of a tile's exponentials and 1270 of its two products with 700 of
// hand-overs between them in turn.  The exponentials alone are 2048 (16 a clock and SM), the four products of D = 128 as long.
// A quarter of them by polynomial on the FMA pipe cost more instructions than it freed (537 us), and P V in two halves, the first
// issued while the second half's exponentials ran, gained nothing (521 us).
// ------------------------------------------------------------------------------------------------------------------
constexpr int kDuoThreads = 640;
constexpr int kDuoRegs = 96, kDuoSoftmaxRegs = 104, kDuoOtherRegs = 64;        // a thread: at launch, and after the split
static_assert(4 * kDuoSoftmaxRegs + kDuoOtherRegs <= 5 * kDuoRegs && kDuoThreads * kDuoRegs <= 65536, "the shares must add up to the launch's");
constexpr int kDuoBN = 128;
template <int D>
struct LayDuo {
  static constexpr int kHalf = kBM * 128;               // [128 rows x 64 elements], swizzled
  static constexpr int kQ = kBM * D * 2;
  static constexpr int kSlot = kDuoBN * D * 2;          // a block of K [128 keys x D] or of V^T [D x 128 keys]
  static constexpr int kSlots = D == 128 ? 5 : 8;
  static constexpr int kOffRing = 2 * kQ;
  static constexpr int kOffX = kOffRing + kSlots * kSlot;       // float [tile][half][128 rows]: what the two threads of a row exchange
  static constexpr int kOffBar = kOffX + 2 * 2 * kBM * 4;
  static constexpr int kSmem = kOffBar + (2 * kSlots + 5) * 8 + 16;
};
static_assert(LayDuo<128>::kSmem <= 227 * 1024 && LayDuo<64>::kSmem > 114 * 1024, "one CTA per SM: it takes all of TMEM");

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Half a query row of a tile over all its blocks.  s_full completes once per block and once more behind the last P V.  Every warp goes
// through all blocks even after a wait that gave up (the waits return at once then), because it meets its partner at each of them.
template <int D, bool CAP>
__device__ __forceinline__ void softmax_duo(const FwdParams& p, uint64_t* s_full, uint64_t* p_full, uint32_t tmem_s, uint32_t tmem_o, float* xch,
                                            int row0, int rows_here, int nblk, int warp, int lane, int q_begin, int head, int kv_len, int pos0,
                                            volatile int* abort_flag) {
  const int half = (warp >> 2) & 1;
  const int row = (warp & 3) * 32 + lane;
  const int bar = 1 + (warp >> 3) * 4 + (warp & 3);      // this warp and its partner
  float* mine = xch + half * kBM + row;
  const float* other = xch + (half ^ 1) * kBM + row;
  auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); };
  const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t ts = tmem_s + lane_off;
  const int lim = (p.causal ? min(kv_len, pos0 + row0 + row + 1) : kv_len) - half * 64;   // tokens [0, lim) from this half's first are visible
  // log2, see softmax_tile.  Heads of 64 follow every new maximum, so that the largest probability stays an exact one in bf16 as in
  // the mma.sync kernel that shorter prompts take
  constexpr float kRescaleStep = D == 64 ? 0.f : 8.f;
  const float scale = CAP ? 1.f : p.scale_log2;
  float m = -INFINITY, l = 0.f;
  bool ok = true;
  for (int j = 0; j < nblk; ++j) {
    ok = __all_sync(0xffffffffu, ok && mbar_wait(s_full, j & 1, abort_flag, kWaitNs));
    if (!ok) {
      *abort_flag = 1;
      meet();
      continue;
    }
    tc_fence_after_sync();
    uint32_t s[2][32];
    tmem_ld_32x32(ts + half * 64, s[0]);
    tmem_ld_32x32(ts + half * 64 + 32, s[1]);
    tmem_ld_wait();
    if constexpr (CAP) {
      attn::cap_scores(reinterpret_cast<float (&)[32]>(s[0]), p.to_cap, p.cap_log2);
      attn::cap_scores(reinterpret_cast<float (&)[32]>(s[1]), p.to_cap, p.cap_log2);
    }
    const int t0 = j * kDuoBN;
    if (!__all_sync(0xffffffffu, t0 + 64 <= lim)) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (t0 + c * 32 + i >= lim) s[c][i] = 0xff800000u;          // -inf
    }
    float mx4[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t* x = s[c >> 1] + (c & 1) * 16;
      mx4[c] = fmaxf(__uint_as_float(x[0]), __uint_as_float(x[1]));
#pragma unroll
      for (int i = 2; i < 16; i += 2) mx4[c] = max3(mx4[c], __uint_as_float(x[i]), __uint_as_float(x[i + 1]));
    }
    const float here = fmaxf(max3(mx4[0], mx4[1], mx4[2]), mx4[3]);
    // The partner's S is in its registers behind this as well: P may overwrite it.  The next block's exchange begins when both have
    // delivered this block's P.
    *mine = here;
    tc_fence_before_sync();
    meet();
    tc_fence_after_sync();
    const float mx = fmaxf(here, *other) * scale;         // scale > 0: the maximum commutes with it
    float alpha = 1.f;
    bool raise = false;
    if (mx > m) {
      if (m == -INFINITY) {
        m = mx;                                   // nothing accumulated for this row so far (its P were all zero)
      } else if (mx - m > kRescaleStep) {
        alpha = ex2(m - mx);
        m = mx;
        raise = true;
      }
    }
    if (__any_sync(0xffffffffu, raise)) {         // each half of the row's threads takes half of O
#pragma unroll 1
      for (int c = 0; c < D / 2; c += 16) {
        const uint32_t at = tmem_o + lane_off + half * (D / 2) + c;
        uint32_t r[16];
        tmem_ld_32x16(at, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
        tmem_st_32x16(at, r);
      }
    }
    const float m_use = (m == -INFINITY) ? 0.f : m;
    const float2 scale2 = make_float2(scale, scale), neg_m = make_float2(-m_use, -m_use);
    float2 sum[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t pk[16];
      sum[c] = make_float2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float2 x = fma2(make_float2(__uint_as_float(s[c][2 * i]), __uint_as_float(s[c][2 * i + 1])), scale2, neg_m);
        x = make_float2(ex2(x.x), ex2(x.y));
        sum[c] = add2(sum[c], x);
        pk[i] = pack_bf16x2(x.x, x.y);
      }
      tmem_st_32x16(ts + half * 32 + c * 16, pk);
    }
    tmem_st_wait();
    tc_fence_before_sync();
    mbar_arrive(p_full);
    const float2 all = add2(sum[0], sum[1]);
    l = l * alpha + (all.x + all.y);
  }
  if (nblk > 0) ok = __all_sync(0xffffffffu, ok && mbar_wait(s_full, nblk & 1, abort_flag, kWaitNs));
  if (!ok) *abort_flag = 1;
  *mine = l;
  meet();
  l += *other;
  write_row<D / 2>(p, tmem_o + lane_off + half * (D / 2), half * (D / 2), ok, nblk > 0, row < rows_here, m, l,
                   static_cast<int64_t>(q_begin) + row0 + row, head);
}

template <int D, bool CAP>
__global__ void __launch_bounds__(kDuoThreads, 1)
flash_fwd_sm100_duo_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                           const __grid_constant__ CUtensorMap tmap_vt, const FwdParams p) {
  // No room for an alignment slack: checked as in flash_fwd_sm100_kernel.
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && p.error_flag != nullptr) *p.error_flag = 2;
    return;
  }
  using L = LayDuo<D>;
  constexpr int kSlots = L::kSlots, kHalves = D / 64;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* s_full = q_full + 1;                // [2] per tile
  uint64_t* p_full = s_full + 2;                // [2]
  uint64_t* full = p_full + 2;                  // [kSlots]
  uint64_t* empty = full + kSlots;              // [kSlots]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + kSlots);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // The long causal tiles of all heads first (blocks are handed out in order of blockIdx.x, then y): no long tile in the last wave.
  const int b = blockIdx.z, head = blockIdx.x;
  const int q_begin = p.cu_seqlens_q[b], q_len = p.cu_seqlens_q[b + 1] - q_begin;
  const int row0 = (p.causal ? static_cast<int>(gridDim.y - 1 - blockIdx.y) : static_cast<int>(blockIdx.y)) * (2 * kBM);
  if (row0 >= q_len) return;                      // whole CTA, before any barrier or TMEM use
  const int kv_len = p.kv_lens[b];
  const int pos0 = p.q_pos0 ? p.q_pos0[b] : (kv_len - q_len);
  int rows_t[2], nblk_t[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    rows_t[t] = max(0, min(q_len - (row0 + t * kBM), kBM));
    const int kv_end = p.causal ? min(kv_len, pos0 + row0 + t * kBM + rows_t[t]) : kv_len;
    nblk_t[t] = rows_t[t] > 0 && kv_end > 0 ? (kv_end + kDuoBN - 1) / kDuoBN : 0;
  }
  const int nblk = max(nblk_t[0], nblk_t[1]);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp-uniform

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int t = 0; t < 2; ++t) {
      mbar_init(&s_full[t], 1);
      mbar_init(&p_full[t], 256);
    }
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 17) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;               // S / P of tile t at column 128 t, O at 256 + 128 t

  if (warp >= 16) {
    // in the role's branch: the compiler allocates each against its own limit
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kDuoOtherRegs));
    if (warp == 16 && lane == 0) {
      tma_prefetch_desc(&tmap_q);
      tma_prefetch_desc(&tmap_k);
      tma_prefetch_desc(&tmap_vt);
      // both Q tiles (rows beyond the sequence or the tensor read other rows or zeros; they are never written out)
      mbar_arrive_expect_tx(q_full, 2 * L::kQ);
#pragma unroll
      for (int i = 0; i < 2 * kHalves; ++i)
        tma_load_2d(smem + i * L::kHalf, &tmap_q, q_full, head * D + (i % kHalves) * 64, q_begin + row0 + i / kHalves * kBM);
      const int z = b * p.Hkv + head / p.group;
      for (int i = 0; i < 2 * nblk; ++i) {
        const int s = i % kSlots, j = i >> 1;
        if (!mbar_wait(&empty[s], ((i / kSlots) & 1) ^ 1, abort_flag, kWaitNs)) {
          *abort_flag = 1;
          break;
        }
        mbar_arrive_expect_tx(&full[s], L::kSlot);
        uint8_t* dst = smem + L::kOffRing + s * L::kSlot;
        if ((i & 1) == 0) {
#pragma unroll
          for (int h = 0; h < kHalves; ++h) tma_load_3d(dst + h * L::kHalf, &tmap_k, &full[s], h * 64, j * kDuoBN, z);
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) tma_load_3d(dst + h * (D * 128), &tmap_vt, &full[s], j * kDuoBN + h * 64, 0, z);
        }
      }
    } else if (warp == 17 && lane == 0) {
      constexpr uint32_t idesc_s = make_idesc(1u, kBM, kDuoBN), idesc_pv = make_idesc(1u, kBM, D);
      const uint32_t ring = smem_u32(smem + L::kOffRing);
      auto landed = [&](int i) { return mbar_wait(&full[i % kSlots], (i / kSlots) & 1, abort_flag, kWaitNs); };
      auto issue_s = [&](int t, int j) {
        const uint32_t sq = smem_u32(smem) + t * L::kQ, sk = ring + (2 * j) % kSlots * L::kSlot;
#pragma unroll
        for (int k = 0; k < D / kUmmaK; ++k)
          umma_f16(tmem + t * 128, make_smem_desc_sw128(sq + (k / 4) * L::kHalf) + 2 * (k % 4),
                   make_smem_desc_sw128(sk + (k / 4) * L::kHalf) + 2 * (k % 4), idesc_s, k > 0 ? 1u : 0u);
      };
      bool ok = mbar_wait(q_full, 0, abort_flag, kWaitNs);
      if (ok && nblk > 0) {
        ok = landed(0);
        tc_fence_after_sync();
        for (int t = 0; t < 2 && ok; ++t) {
          if (nblk_t[t] == 0) continue;
          issue_s(t, 0);
          umma_commit(&s_full[t]);
        }
        if (ok) umma_commit(&empty[0]);
      }
      for (int j = 0; j < nblk && ok; ++j) {
        ok = landed(2 * j + 1) && (j + 1 >= nblk || landed(2 * j + 2));
        const uint32_t sv = ring + (2 * j + 1) % kSlots * L::kSlot;
        for (int t = 0; t < 2 && ok; ++t) {
          if (j >= nblk_t[t]) continue;
          ok = mbar_wait(&p_full[t], j & 1, abort_flag, kWaitNs);
          if (!ok) break;
          tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < kDuoBN / kUmmaK; ++k)
            umma_f16_ts(tmem + 256 + t * 128, tmem + t * 128 + k * (kUmmaK / 2),
                        make_smem_desc_sw128(sv + (k / 4) * (D * 128)) + 2 * (k % 4), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
          if (j + 1 < nblk_t[t]) issue_s(t, j + 1);
          umma_commit(&s_full[t]);
        }
        if (!ok) break;
        umma_commit(&empty[(2 * j + 1) % kSlots]);
        if (j + 1 < nblk) umma_commit(&empty[(2 * j + 2) % kSlots]);
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kDuoSoftmaxRegs));
    const int t = warp >> 3;
    softmax_duo<D, CAP>(p, &s_full[t], &p_full[t], tmem + t * 128, tmem + 256 + t * 128, reinterpret_cast<float*>(smem + L::kOffX) + t * 2 * kBM,
                        row0 + t * kBM, rows_t[t], nblk_t[t], warp, lane, q_begin, head, kv_len, pos0, abort_flag);
  }

  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag != 0 && p.error_flag != nullptr) *p.error_flag = 1;
  if (warp == 17) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

constexpr int kDuoOverQ = 512;

}  // namespace

cudaError_t launch_flash_fwd_sm100(const FlashFwdSm100Args& a, cudaStream_t stream) {
  const int D = a.head_dim;
  if ((D != 128 && D != 64) || (D != 128 && a.kv.k_scale != nullptr) || a.num_q_heads % a.num_kv_heads != 0 || a.Lp % kBN != 0 || a.Lp <= 0) return cudaErrorInvalidValue;
  if (!(a.scale > 0.f)) return cudaErrorInvalidValue;   // the row maximum is taken before scaling
  if (a.batch == 0 || a.max_q_len == 0) return cudaSuccess;
  PackParams pk;
  pk.k_cache = reinterpret_cast<const __nv_bfloat16*>(a.kv.k_cache);
  pk.v_cache = reinterpret_cast<const __nv_bfloat16*>(a.kv.v_cache);
  pk.block_table = a.kv.block_table;
  pk.kv_lens = a.kv_lens;
  pk.max_pages = a.kv.max_pages;
  pk.page_size = a.kv.page_size;
  pk.Hkv = a.num_kv_heads;
  pk.Lp = a.Lp;
  pk.k_out = reinterpret_cast<__nv_bfloat16*>(a.k_dense);
  pk.vt_out = reinterpret_cast<__nv_bfloat16*>(a.vt_dense);
  pk.k_scale = a.kv.k_scale;
  const dim3 pack_grid(a.Lp / kBN, a.num_kv_heads, a.batch);
  if (pk.k_scale != nullptr)
    attn_pack_kv_kernel<128, true><<<pack_grid, 256, 0, stream>>>(pk);
  else if (D == 128)
    attn_pack_kv_kernel<128, false><<<pack_grid, 256, 0, stream>>>(pk);
  else
    attn_pack_kv_kernel<64, false><<<pack_grid, 256, 0, stream>>>(pk);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;

  // Three forms: (2) two CTAs of 128 rows per SM with a two-stage KV ring (one CTA's exponentials overlap the other's products),
  // (1) one such CTA per SM with a five-stage ring, (3) one CTA of 256 rows per SM, the only one for heads of 64.
  // TDB200_ATTN_FORM selects for heads of 128.  Short sequences fill 256 rows badly
  // (8 heads: 512 tokens 20.8 us with (2), 22.7 with (3); 1024 tokens 30.9 and 28.9; 32 heads, 7 x 292: 37.3 and 45.7, 6 x 1365: 206 and 180).
  static const int forced = [] {
    const char* e = std::getenv("TDB200_ATTN_FORM");
    return e != nullptr ? std::atoi(e) : 0;
  }();
  const int form = D == 64 ? 3 : forced != 0 ? forced : a.max_q_len > kDuoOverQ ? 3 : 2;
  const uint32_t block_n = form == 3 ? kDuoBN : kBN;
  TensorMap tq, tk, tv;
  const uint64_t bh = static_cast<uint64_t>(a.batch) * a.num_kv_heads;
  if (encode_tensor_map_2d(&tq, a.q, kBF16, static_cast<uint64_t>(a.total_q), static_cast<uint64_t>(a.num_q_heads) * D,
                           static_cast<uint64_t>(a.num_q_heads) * D * 2, kBM, 64, 128) != 0)
    return cudaErrorInvalidValue;
  if (encode_tensor_map_3d(&tk, a.k_dense, kBF16, bh, static_cast<uint64_t>(a.Lp), D, D * 2,
                           static_cast<uint64_t>(a.Lp) * D * 2, block_n, 64, 128) != 0)
    return cudaErrorInvalidValue;
  if (encode_tensor_map_3d(&tv, a.vt_dense, kBF16, bh, D, static_cast<uint64_t>(a.Lp), static_cast<uint64_t>(a.Lp) * 2,
                           static_cast<uint64_t>(a.Lp) * D * 2, D, 64, 128) != 0)
    return cudaErrorInvalidValue;
  FwdParams p;
  p.q = reinterpret_cast<const __nv_bfloat16*>(a.q);
  p.out = reinterpret_cast<__nv_bfloat16*>(a.out);
  p.lse = a.lse;
  p.cu_seqlens_q = a.cu_seqlens_q;
  p.q_pos0 = a.q_pos0;
  p.kv_lens = a.kv_lens;
  p.Hq = a.num_q_heads;
  p.Hkv = a.num_kv_heads;
  p.group = a.num_q_heads / a.num_kv_heads;
  p.causal = a.causal;
  p.dv = D;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  if (a.softcap < 0.f) return cudaErrorInvalidValue;
  p.cap_log2 = a.softcap * 1.4426950408889634f;
  p.to_cap = a.softcap > 0.f ? a.scale / a.softcap : 0.f;
  p.total_q = a.total_q;
  p.error_flag = a.error_flag;
  p.epi = a.epi;
  if (p.epi.gate != nullptr && (p.epi.ld_gate % 8 != 0 || (reinterpret_cast<uintptr_t>(p.epi.gate) & 15u) != 0))
    return cudaErrorInvalidValue;
  dim3 grid((a.max_q_len + kBM - 1) / kBM, a.num_q_heads, a.batch);
  CUtensorMap mq, mk, mv;
  memcpy(&mq, tq.bytes, sizeof(mq));
  memcpy(&mk, tk.bytes, sizeof(mk));
  memcpy(&mv, tv.bytes, sizeof(mv));
  auto launch = [&](auto kernel, SmemOptIn& opt, dim3 g, int threads, int smem) -> cudaError_t {
    const cudaError_t err = opt.ensure(kernel, smem);
    if (err != cudaSuccess) return err;
    kernel<<<g, threads, smem, stream>>>(mq, mk, mv, p);
    return cudaGetLastError();
  };
  static SmemOptIn opt1, opt2, opt3, opt64, cap1, cap2, cap3, cap64;
  const bool cap = a.softcap > 0.f;
  if (form == 3) {
    const dim3 duo(a.num_q_heads, (a.max_q_len + 2 * kBM - 1) / (2 * kBM), a.batch);
    if (D == 64)
      return cap ? launch(flash_fwd_sm100_duo_kernel<64, true>, cap64, duo, kDuoThreads, LayDuo<64>::kSmem)
                 : launch(flash_fwd_sm100_duo_kernel<64, false>, opt64, duo, kDuoThreads, LayDuo<64>::kSmem);
    return cap ? launch(flash_fwd_sm100_duo_kernel<128, true>, cap3, duo, kDuoThreads, LayDuo<128>::kSmem)
               : launch(flash_fwd_sm100_duo_kernel<128, false>, opt3, duo, kDuoThreads, LayDuo<128>::kSmem);
  }
  if (form == 1)
    return cap ? launch(flash_fwd_sm100_kernel<5, 1, true>, cap1, grid, kThreads, Lay<5>::kSmem)
               : launch(flash_fwd_sm100_kernel<5, 1, false>, opt1, grid, kThreads, Lay<5>::kSmem);
  return cap ? launch(flash_fwd_sm100_kernel<2, 2, true>, cap2, grid, kThreads, Lay<2>::kSmem)
             : launch(flash_fwd_sm100_kernel<2, 2, false>, opt2, grid, kThreads, Lay<2>::kSmem);
}

}  // namespace tdb
