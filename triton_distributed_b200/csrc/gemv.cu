// Decode GEMV for one to sixteen tokens:  out[M, N] = f(x)[M, K] * W[N, K]^T  (+ all-reduce) (+ residual).
//
// With so few tokens a linear layer is a pure weight stream: the tensor cores have nothing to amortise and the cost
// of a decode step is the HBM time of the weights plus whatever each launch adds around it.  This kernel therefore
// keeps the stream as plain as possible (every warp owns an equal span of the CTA's weight rows, fetched in 16-byte
// copies that stay many deep in flight, and sums on the tensor cores, so there are no atomics and no second pass) and
// folds the neighbouring small kernels of a transformer layer into its prologue and epilogue:
//   prologue   f = RMSNorm(x) * g      (the sum of squares is taken while the activations are staged)
//              f = SiLU(gate) * up     (x is the fused gate | up projection)
//   epilogue   SiLU(gate) * up on the fp32 sums, where the product is a gate | up projection
//              all-reduce of the result over the tensor-parallel ranks: every CTA publishes its columns in the
//              symmetric heap, exchanges one epoch flag per peer with the CTA of the same index there, and reads the
//              sum back with multimem.ld_reduce (or sums the peers' slots after a push when there is no multicast)
//              residual add, in place if wanted
// so a decoder layer is four GEMV launches plus attention.  SwiGLU belongs to the epilogue of the first product: as a prologue every
// CTA of the second one computed it for all K columns and all tokens (4096 x 12288, one token: 22.0 us
// with it, 20.0 without; a decode step of four layers of an 8B model with three tokens: 652 us, now 602).
//
// Reference behaviour being matched (not its code): the decode path of layers/nvidia/tp_attn.py:160-213 and
// tp_mlp.py:196-229 (rmsnorm -> linear -> ... -> linear -> all-reduce -> add) and the fused GEMM+AllReduce of
// kernels/nvidia/gemm_allreduce.py:124-315, specialised to M <= 8.
#include <cuda.h>

#include <cstdlib>

#include "tdb/attn_device.cuh"
#include "tdb/gemv.h"
#include "tdb/launch.cuh"
#include "tdb/symm_device.cuh"
#include "tdb/vec.cuh"

namespace tdb {

namespace {

constexpr int kGemvThreads = 512;
constexpr int kGemvWarps = kGemvThreads / 32;
constexpr int kRedBytes = 2 * kGemvWarps * 256;   // partial sums of eight tokens: two parts per warp, 8 x 8 floats each
constexpr int kMaxSmem = 200 * 1024;
constexpr int kMinRing = kGemvWarps * 2 * 512;
constexpr int kLaunchSmem = 225 * 1024;        // dynamic, beside at most 1.1 KB of static shared memory
static_assert(kMaxSmem + kRedBytes + kMinRing <= kLaunchSmem, "what fits without a ring must fit with the smallest");

struct GemvParams {
  int M, N, K;
  const __nv_bfloat16* x;
  int64_t ldx;
  const __nv_bfloat16* w;
  int64_t ldw;
  __nv_bfloat16* out;
  int64_t ld_out;
  const __nv_bfloat16* norm_w;
  float eps;
  int gated;
  int swiglu;                  // a group is four gate rows and the four up rows of the same output columns
  const __nv_bfloat16* residual;
  int64_t ld_res;
  int rows_per_cta;
  int all_reduce;
  int use_mc;
  __nv_bfloat16* partial;
  uint64_t partial_half;
  uint32_t* flags;
  int max_ctas;
  int m_cap;
  CtxDev* ctx;
  SymmInfo symm;
};

TDB_DEVICE void unpack8(const uint4& v, float (&f)[8]) {
  const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z), d = unpack_bf16x2(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
TDB_DEVICE uint4 pack8(const float (&f)[8]) {
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
  return o;
}

// One warp-wide tensor-core step: D[16 x 8] += A[16 x 16] * B[16 x 8], bf16 in, fp32 accumulate.
TDB_DEVICE void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Work layout.  A CTA owns `rows_per_cta` output columns = weight rows, in groups of 8 (the last one may be partly
// empty).  The steps of all its groups, laid end to end, are cut into sixteen equal spans, one per warp, so that every
// warp streams the same number of bytes whatever the shape: a span begins and ends anywhere inside a group, and a group
// that several warps share is summed through shared memory at the end (a warp has at most two such parts: one that begins
// inside its group, slot 2 warp, and one that begins with it, slot 2 warp + 1).  The kernel is bound by the weights'
// HBM time; with whole groups per warp, SMs waited for the warps that had one group more.
// Lane (g = lane / 4, t = lane % 4) streams row g of the group with 16-byte
// loads, 32 elements of K per step across the four t lanes.  The dot products run on the tensor cores: the eight
// loaded values of a lane are fed as the A fragments of two m16n8k16 steps (rows 8..15 of A are zero), the eight
// activations of the same K positions of token g as the B fragments.  A dot product does not care in which order K
// is walked, so the K positions are simply assigned to fragment slots in the order the 16-byte loads deliver them;
// the accumulator then holds [8 rows x 8 tokens] and no lane-wise reduction is needed.  What is left per lane and
// load is two shared-memory reads and two mma instructions.
// The weights land in shared memory (cp.async), in a ring of R batches of J steps per warp that only the lane that fetched
// a vector reads: no barrier.  Loads to registers need room in L1 while they are in flight, and next to attention kernels
// that have the SM configured for shared memory there is next to none: inside a decode step the register form ran at half
// the rate it had alone (lm_head of 151936 x 4096: 188 us alone and 240 to 410 us in the step; now 207 us in both.  gate | up of
// 24576 x 4096 with one token: 71 us in the step, now 33).
constexpr int kSpanSteps = 8;

// Steps of a warp when a CTA has `total`: whole batches, so that only a group's last batch is ever a partial one.
TDB_DEVICE int warp_span(int total) {
  const int per = (total + kGemvWarps - 1) / kGemvWarps;
  return (per + kSpanSteps - 1) / kSpanSteps * kSpanSteps;
}

template <int MP, int J, int R>   // tokens rounded up to 1, 2, 4, 8 or 16 (two 8-token MMA tiles); ring
__global__ void __launch_bounds__(kGemvThreads, 1) gemv_kernel(const GemvParams p) {
  extern __shared__ uint4 smem4[];
  __shared__ float s_part[kGemvWarps][MP];
  __shared__ float s_rstd[16];
  constexpr int NT = (MP + 7) / 8;          // 8-token tiles of the MMA's N dimension
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int kv = p.K >> 3;                       // 16-byte vectors per row
  const int xs_stride = kv + 4;                  // in vectors: rows 64 bytes apart modulo 128 (bank-conflict free)
  uint4* xs = smem4;                             // staged activations f(x): [MP][xs_stride]
  uint4* ring = smem4 + MP * xs_stride + warp * (R * J * 32) + lane;                           // [R][J][32 lanes] of this warp
  float* red = reinterpret_cast<float*>(smem4 + MP * xs_stride + kGemvWarps * R * J * 32);    // [2 per warp][8 rows][8 NT tokens]
  const int cols = p.swiglu ? p.N >> 1 : p.N;    // of the output
  const int r0 = blockIdx.x * p.rows_per_cta;
  const int r1 = min(cols, r0 + p.rows_per_cta);
  const int gshift = p.swiglu ? 2 : 3;           // log2 of the output columns of a group
  const int groups = (r1 - r0 + (1 << gshift) - 1) >> gshift;
  const int gcol = g & ((1 << gshift) - 1);      // this lane's column of a group, its weight row lies up_off further
  const int up_off = g >> gshift ? cols : 0;
  const int steps = (kv + 3) >> 2;               // steps of 4 vectors (32 elements of K) of a group
  const int span = warp_span(groups * steps);
  struct Seg {                                   // what is left of this warp's part of a group, and of its span behind st
    int grp, st, end, left;
  };
  Seg cur;
  cur.left = min(span, groups * steps - warp * span);
  cur.grp = warp * span / steps;
  cur.st = warp * span - cur.grp * steps;
  cur.end = min(steps, cur.st + cur.left);

  // The weights do not depend on the previous kernel: the first loads are issued before anything else, so that
  // their latency overlaps the predecessor's tail (programmatic dependent launch) and the staging of x.
  const int part0 = cur.st;      // where this warp's first part begins
  const int grp0 = cur.grp;
  auto fetch = [&](int slot, const Seg& s) {
    if (s.left > 0) {
      const int row = r0 + (s.grp << gshift) + gcol;
      const bool row_ok = row < r1;
      const __nv_bfloat16* wr = p.w + static_cast<int64_t>(row_ok ? row + up_off : r0) * p.ldw;
#pragma unroll
      for (int j = 0; j < J; ++j) {
        const int c = (s.st + j) * 4 + t;
        const bool ok = row_ok && s.st + j < s.end && c < kv;
        attn::cp_async16(ring + (slot * J + j) * 32, wr + (ok ? c * 8 : 0), ok);
      }
    }
    attn::cp_async_commit();
  };
  // The batch behind `s`: of the same segment, or the first of the next group.
  auto next = [&](const Seg& s) {
    const int done = min(J, s.end - s.st);
    Seg n{s.grp, s.st + done, s.end, s.left - done};
    if (n.st == steps) n = Seg{s.grp + 1, 0, min(steps, n.left), n.left};
    return n;
  };
  Seg ahead = cur;
#pragma unroll
  for (int i = 0; i < R - 1; ++i) {
    fetch(i, ahead);
    if (ahead.left > 0) ahead = next(ahead);
  }
  pdl_wait();
  pdl_launch_dependents();
  // the call epoch is advanced by the last CTA of the previous call: read it only after the dependency wait
  const uint32_t epoch = (p.ctx != nullptr) ? ld_volatile(&p.ctx->epoch) : 1u;
  const int par = epoch & 1;

  // ---- prologue: stage f(x) in shared memory; a thread takes one 16-byte column slice of every token, so the loads
  // of all tokens are in flight together and the staging time does not grow with the token count
  float ss[MP];
#pragma unroll
  for (int m = 0; m < MP; ++m) ss[m] = 0.f;
  constexpr int MB = MP < 4 ? MP : 4;      // tokens whose loads are in flight together (register budget)
  for (int c = tid; c < kv; c += kGemvThreads) {
    float gn[8];
    if (p.norm_w != nullptr) unpack8(ld_nc_v4(p.norm_w + c * 8), gn);
#pragma unroll
    for (int m0 = 0; m0 < MP; m0 += MB) {
      uint4 v[MB], u[MB];
#pragma unroll
      for (int i = 0; i < MB; ++i) {
        const int m = m0 + i;
        v[i] = (m < p.M) ? ld_v4(p.x + static_cast<int64_t>(m) * p.ldx + c * 8) : make_uint4(0u, 0u, 0u, 0u);
        if (p.gated)
          u[i] = (m < p.M) ? ld_v4(p.x + static_cast<int64_t>(m) * p.ldx + p.K + c * 8) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int i = 0; i < MB; ++i) {
        const int m = m0 + i;
        if (p.gated) {
          float gg[8], h[8];
          unpack8(v[i], gg);
          unpack8(u[i], h);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            gg[j] = (p.gated == 1 ? gg[j] / (1.f + __expf(-gg[j])) : gelu_tanh_f32(gg[j])) * h[j];
          v[i] = pack8(gg);
        } else if (p.norm_w != nullptr) {
          float a[8];
          unpack8(v[i], a);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            ss[m] += a[j] * a[j];
            a[j] *= gn[j];
          }
          v[i] = pack8(a);
        }
        xs[m * xs_stride + c] = v[i];
      }
    }
  }
  if (p.norm_w != nullptr) {
#pragma unroll
    for (int m = 0; m < MP; ++m) {
      const float tt = warp_sum(ss[m]);
      if (lane == 0) s_part[warp][m] = tt;
    }
    __syncthreads();
    if (tid < MP) {
      float tt = 0.f;
      for (int wi = 0; wi < kGemvWarps; ++wi) tt += s_part[wi][tid];
      s_rstd[tid] = rsqrtf(tt / static_cast<float>(p.K) + p.eps);
    }
  } else if (tid < 16) {
    s_rstd[tid] = 1.f;
  }
  __syncthreads();

  // ---- main loop
  __nv_bfloat16* pdst = nullptr;   // all-reduce: where this rank's partial result goes
  if (p.all_reduce)
    pdst = p.partial + par * p.partial_half + (p.use_mc ? 0ull : static_cast<uint64_t>(p.symm.rank) * p.m_cap * p.N);
  auto store = [&](int m, int row, float v, float up) {
    v *= s_rstd[m];
    if (p.swiglu) v = silu_f32(v) * (up * s_rstd[m]);
    if (p.all_reduce) {
      pdst[static_cast<int64_t>(m) * p.N + row] = __float2bfloat16(v);
    } else {
      if (p.residual != nullptr) v += __bfloat162float(p.residual[static_cast<int64_t>(m) * p.ld_res + row]);
      p.out[static_cast<int64_t>(m) * p.ld_out + row] = __float2bfloat16(v);
    }
  };
  float acc[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  for (int i = 0; cur.left > 0; ++i) {
    fetch((i + R - 1) % R, ahead);
    if (ahead.left > 0) ahead = next(ahead);
    attn::cp_async_wait<R - 1>();
    const uint4* src = ring + (i % R) * J * 32;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int cv = (cur.st + j) * 4 + t;
      const bool in_range = cur.st + j < cur.end && cv < kv;
      const uint4 wv = src[j * 32];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int tok = nt * 8 + g;               // token whose activations this lane feeds as the B fragment
        uint4 xv = make_uint4(0u, 0u, 0u, 0u);
        if (tok < MP && in_range) xv = xs[tok * xs_stride + cv];
        mma_bf16_16816(acc[nt], wv.x, 0u, wv.y, 0u, xv.x, xv.y);
        mma_bf16_16816(acc[nt], wv.z, 0u, wv.w, 0u, xv.z, xv.w);
      }
    }
    if (cur.st + J >= cur.end) {   // the part is complete: acc[0], acc[1] = (row g, tokens 2t, 2t + 1), rows 8..15 of the tile are zero
      const bool from_start = cur.grp != grp0 || part0 == 0;
      float* slot = red + ((2 * warp + (from_start ? 1 : 0)) * 8 + g) * (8 * NT) + 2 * t;
      const int row = r0 + (cur.grp << gshift) + gcol;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int m = nt * 8 + 2 * t + e;
          if (from_start && cur.end == steps) {        // the whole group; an up row is 16 lanes from its gate row
            const float up = p.swiglu ? __shfl_down_sync(0xffffffffu, acc[nt][e], 16) : 0.f;
            if (m < p.M && row < r1 && up_off == 0) store(m, row, acc[nt][e], up);
          } else {
            slot[nt * 8 + e] = acc[nt][e];
          }
        }
        acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
      }
    }
    cur = next(cur);
  }
  attn::cp_async_wait<0>();
  __syncthreads();

  // ---- groups that several warps share: sum their parts
  const int shown = groups << gshift;
  for (int i = tid; i < shown * p.M; i += kGemvThreads) {
    const int m = i / shown, rr = i - m * shown;                   // consecutive threads -> consecutive columns
    const int gi = rr >> gshift, gr = rr & ((1 << gshift) - 1);
    const int w0 = gi * steps / span, w1 = ((gi + 1) * steps - 1) / span;
    if (r0 + rr >= r1 || w0 == w1) continue;
    float v = 0.f, up = 0.f;
    for (int w = w0; w <= w1; ++w) {
      const float* part = red + ((2 * w + (w * span <= gi * steps ? 1 : 0)) * 8 + gr) * (8 * NT) + m;
      v += part[0];
      if (p.swiglu) up += part[4 * 8 * NT];
    }
    store(m, r0 + rr, v, up);
  }

  // ---- epilogue: all-reduce of this CTA's columns [r0, r1) (multiples of 8) with the same CTA of every rank
  if (p.all_reduce && r0 < p.N) {
    const int W = p.symm.world, rank = p.symm.rank;
    const int nvec = (r1 - r0) >> 3;
    __syncthreads();
    if (!p.use_mc) {
      // push this rank's slot of the columns to every peer
      for (int v = tid; v < p.M * nvec; v += kGemvThreads) {
        const int m = v / nvec, col = r0 + (v - m * nvec) * 8;
        __nv_bfloat16* src = pdst + static_cast<int64_t>(m) * p.N + col;
        const uint4 u = ld_v4(src);
        for (int j = 1; j < W; ++j) st_v4(symm_at(p.symm, src, (rank + j) % W), u);
      }
      __syncthreads();
    }
    bool ok = true;
    if (tid < W) {
      fence_acq_rel_sys();
      st_release_sys(symm_at(p.symm, p.flags + static_cast<int64_t>(rank) * p.max_ctas + blockIdx.x, (rank + tid) % W), epoch);
      ok = wait_until(p.symm, p.flags + static_cast<int64_t>(tid) * p.max_ctas + blockIdx.x, epoch, kCmpGe, kKernelGemv, 1,
                      tid, blockIdx.x);
    }
    ok = __syncthreads_and(ok);
    if (ok) {
      for (int v = tid; v < p.M * nvec; v += kGemvThreads) {
        const int m = v / nvec, col = r0 + (v - m * nvec) * 8;
        float s[8];
        if (p.use_mc) {
          const __nv_bfloat16* src = p.partial + par * p.partial_half + static_cast<int64_t>(m) * p.N + col;
          unpack8(multimem_ld_reduce_bf16x8(mc_ptr(p.symm, src)), s);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] = 0.f;
          for (int r = 0; r < W; ++r) {
            const __nv_bfloat16* src =
                p.partial + par * p.partial_half + (static_cast<uint64_t>(r) * p.m_cap + m) * p.N + col;
            float tt[8];
            unpack8(ld_relaxed_sys_v4(src), tt);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += tt[j];
          }
        }
        if (p.residual != nullptr) {
          float e[8];
          unpack8(ld_v4(p.residual + static_cast<int64_t>(m) * p.ld_res + col), e);
#pragma unroll
          for (int j = 0; j < 8; ++j) s[j] += e[j];
        }
        st_v4(p.out + static_cast<int64_t>(m) * p.ld_out + col, pack8(s));
      }
    }
  }

  // last CTA out advances the call epoch
  if (p.ctx != nullptr) {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      const uint32_t prev = atomicAdd(&p.ctx->done, 1u);
      if (prev == gridDim.x - 1) {
        p.ctx->done = 0;
        __threadfence();
        *reinterpret_cast<volatile uint32_t*>(&p.ctx->epoch) = epoch + 1;
      }
    }
  }
}

template <int M, int J, int R>
cudaError_t launch_ring(const GemvParams& p, int grid, size_t smem, cudaStream_t stream) {
  static SmemOptIn opt;
  cudaError_t e = opt.ensure(gemv_kernel<M, J, R>, kLaunchSmem);
  if (e != cudaSuccess) return e;
  // everything the kernel reads from its predecessor comes after pdl_wait()
  return launch_pdl(gemv_kernel<M, J, R>, dim3(grid), dim3(kGemvThreads), smem + kGemvWarps * J * R * 512, stream, p);
}

// The deepest ring that fits beside the activations and the partial sums (`smem` bytes).  40 KB per SM must be in flight to
// cover HBM's latency: the 128 KB ring has 96 KB, the 16 KB one is what the largest activations leave.  Four steps a batch ask for
// 256 bytes of a row at once: 4096 x 12288 takes 19.9 us, with two steps and eight batches 22.5, with eight and two 20.6.
template <int M>
cudaError_t launch_t(const GemvParams& p, int grid, size_t smem, cudaStream_t stream) {
  const int left = kLaunchSmem - static_cast<int>(smem);
  if (left >= kGemvWarps * 16 * 512) return launch_ring<M, 4, 4>(p, grid, smem, stream);
  if (left >= kGemvWarps * 8 * 512) return launch_ring<M, 2, 4>(p, grid, smem, stream);
  if (left >= kGemvWarps * 4 * 512) return launch_ring<M, 2, 2>(p, grid, smem, stream);
  return launch_ring<M, 1, 2>(p, grid, smem, stream);
}

}  // namespace

int gemv_max_k(int M) {
  const int mp = M <= 1 ? 1 : M <= 2 ? 2 : M <= 4 ? 4 : M <= 8 ? 8 : 16;
  // mp rows of (2 K + 64) bytes next to the partial-sum slots
  return (((kMaxSmem - kRedBytes) / mp - 64) / 2) & ~7;
}

cudaError_t launch_gemv(const GemvArgs& a, cudaStream_t stream) {
  if (a.M < 1 || a.M > 16 || a.K % 8 != 0 || a.K > gemv_max_k(a.M)) return cudaErrorInvalidValue;
  if (a.ldw % 8 != 0 || a.ldx % 8 != 0) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.x)) & 15u) return cudaErrorInvalidValue;
  if (a.norm_w != nullptr && a.gated) return cudaErrorInvalidValue;
  GemvParams p;
  p.M = a.M; p.N = a.N; p.K = a.K;
  p.x = reinterpret_cast<const __nv_bfloat16*>(a.x);
  p.ldx = a.ldx;
  p.w = reinterpret_cast<const __nv_bfloat16*>(a.w);
  p.ldw = a.ldw;
  p.out = reinterpret_cast<__nv_bfloat16*>(a.out);
  p.ld_out = a.ld_out;
  p.norm_w = reinterpret_cast<const __nv_bfloat16*>(a.norm_w);
  p.eps = a.eps;
  p.gated = a.gated;
  p.swiglu = a.swiglu;
  p.residual = reinterpret_cast<const __nv_bfloat16*>(a.residual);
  p.ld_res = a.ld_res;
  p.all_reduce = a.all_reduce;
  p.use_mc = (a.use_multimem && a.symm.mc_base != 0) ? 1 : 0;
  p.partial = reinterpret_cast<__nv_bfloat16*>(a.partial);
  p.m_cap = a.m_cap;
  p.partial_half = p.use_mc ? static_cast<uint64_t>(a.m_cap) * a.N : static_cast<uint64_t>(a.symm.world) * a.m_cap * a.N;
  p.flags = a.flags;
  p.max_ctas = a.max_ctas;
  p.ctx = a.ctx;
  static_assert(sizeof(SymmInfo) == sizeof(SymmInfoHost), "SymmInfo mirrors must match");
  memcpy(&p.symm, &a.symm, sizeof(SymmInfo));
  const int num_ctas = a.num_ctas < 1 ? 1 : a.num_ctas;
  // As even as it goes: 4096 columns are 28 for each of 147 CTAs, not 32 for 128.  In all-reduce mode every CTA gets
  // whole 16-byte vectors.
  if (a.swiglu && (a.N % 2 != 0 || a.all_reduce || a.residual != nullptr)) return cudaErrorInvalidValue;
  const int cols = a.swiglu ? a.N / 2 : a.N;
  if (cols == 0) return cudaSuccess;
  if (a.K == 0) {      // nothing to sum on any rank, no step to divide among the warps: the residual, or zeros
    const size_t width = static_cast<size_t>(cols) * 2, pitch = static_cast<size_t>(a.ld_out) * 2;
    if (a.residual == nullptr) return cudaMemset2DAsync(a.out, pitch, 0, width, a.M, stream);
    if (a.residual == a.out) return cudaSuccess;
    return cudaMemcpy2DAsync(a.out, pitch, a.residual, static_cast<size_t>(a.ld_res) * 2, width, a.M, cudaMemcpyDeviceToDevice, stream);
  }
  const int even = (cols + num_ctas - 1) / num_ctas;
  const int rows = a.all_reduce ? (even + 7) & ~7 : even;
  if (a.all_reduce) {
    // the residual / output rows must allow vector access
    if (a.N % 8 != 0 || a.ld_out % 8 != 0 || (a.residual != nullptr && a.ld_res % 8 != 0)) return cudaErrorInvalidValue;
    if (a.ctx == nullptr || a.partial == nullptr || a.flags == nullptr || a.M > a.m_cap) return cudaErrorInvalidValue;
  }
  p.rows_per_cta = rows;
  const int grid = (cols + rows - 1) / rows;
  if (a.all_reduce && grid > a.max_ctas) return cudaErrorInvalidValue;
  const int mp = a.M <= 1 ? 1 : a.M <= 2 ? 2 : a.M <= 4 ? 4 : a.M <= 8 ? 8 : 16;
  const size_t smem = static_cast<size_t>(mp) * (a.K * 2 + 64) + static_cast<size_t>(kRedBytes) * ((mp + 7) / 8);
  switch (mp) {
    case 1: return launch_t<1>(p, grid, smem, stream);
    case 2: return launch_t<2>(p, grid, smem, stream);
    case 4: return launch_t<4>(p, grid, smem, stream);
    case 8: return launch_t<8>(p, grid, smem, stream);
    default: return launch_t<16>(p, grid, smem, stream);
  }
}

}  // namespace tdb
