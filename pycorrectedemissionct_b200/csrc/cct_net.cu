// Warm-start network kernels (no reference counterpart): 3x3 convolutions as implicit GEMMs on
// the 5th-generation tensor cores (tcgen05.mma, BF16 x BF16 -> FP32 accumulators in TMEM), and
// the elementwise pieces of a small encoder-decoder (bias/ReLU, 2x2 average pooling, nearest
// upsampling, skip additions, MSE, Adam).
//
// Activations are NHWC bfloat16 with channel counts that are multiples of 16.  Weights are
// [Cout][3][3][Cin] bfloat16 ("K-major": k = tap * Cin + ci).
//
// Both GEMMs have M = 128 (one TMEM lane per row) and FP32 accumulators in TMEM, and read their
// operands as TMA boxes of pixels x channels in the 32-, 64- or 128-byte swizzled layout that the
// tensor core reads (blocks of 16, 32 or 64 channels).  Every wait is bounded; on timeout the kernel raises
// g_net_timeout, waits once more for its own copies and leaves.

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "cct_common.cuh"
#include "cct_internal.cuh"

namespace cct {

__device__ int g_net_timeout = 0;

constexpr int NET_TW = 8;                       // tile columns: 8 pixel rows of an operand are one swizzle atom
constexpr int NET_TH = 16;                      // tile rows of one M = 128 block
constexpr uint32_t NET_WAIT_LIMIT = 1u << 24;
constexpr int NET_SMEM_MAX = 223 * 1024;  // dynamic; 4 KB of the 227 are left to the static arrays

// n / d for n < 2^31 by one multiplication: (n * mul) >> (32 + shift), mul = floor(2^(32 + shift) / d) + 1
// with 2^shift >= d / 2 (d = 1: mul = 0 stands for n itself).
struct FastDiv {
  uint32_t d, mul, shift;
  FastDiv() = default;
  explicit FastDiv(int v) : d((uint32_t)v), mul(0), shift(0) {
    if (v == 1) return;
    while ((2u << shift) < d) ++shift;
    mul = (uint32_t)(((1ull << (32 + shift)) / d) + 1);
  }
  __device__ __forceinline__ void divmod(int n, int* q, int* r) const {
    const uint32_t x = mul == 0 ? (uint32_t)n : __umulhi((uint32_t)n, mul) >> shift;
    *q = (int)x;
    *r = n - (int)(x * d);
  }
};

struct ConvArgs {
  int batch, h, w, cin, cout;
  FastDiv by_n, by_x, by_y;  // n_tiles, tiles_x, tiles_y
  int ck;              // channels per operand block of x (64, 32 or 16: one 128-, 64- or 32-byte swizzled row)
  int tiles_x, tiles_y, tiles, n_tiles;
  const float* bias;   // [cout] or nullptr
  __nv_bfloat16* y;    // NHWC output
  int relu, wide;      // wide: y is 32-byte aligned
  int stages, resident;
  int whole;           // a stage holds the three boxes of a tile (one channel block, weights resident)
};

struct WgradArgs {
  int batch, h, w, cin, cout;
  int ckx, cky;        // channels per operand block of x and dy
  int bx, by;          // operand blocks of x (M) and dy (N) per CTA
  int n;               // N = by * cky
  int tiles_x, tiles_y, tiles;
  int sets;            // MMAs per K step: taps (or groups of taps) of one dx
  int stages;
  float* dw;           // [cout][9][cin] FP32, accumulated
};

__device__ __forceinline__ uint32_t net_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory operand of rows of `ck` BF16 elements (128, 64 or 32 bytes) as TMA writes them with the
// matching swizzle; 8 rows are an atom.  K-major: rows are M / N, lbo unused, sbo = atom.
// MN-major: rows are K, lbo = distance of the next ck elements along M / N, sbo = atom.
// The two words of the descriptor: a further operand in the same buffer adds its byte offset / 16 to
// the low one (one thread issues all MMAs, so what it computes per MMA is what an MMA costs).
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t addr, uint32_t lbo_bytes) {
  return ((addr >> 4) & 0x3FFF) | (((lbo_bytes >> 4) & 0x3FFF) << 16);
}
__device__ __forceinline__ uint32_t umma_desc_hi(int ck) {
  const uint32_t layout = ck == 64 ? 2 : ck == 32 ? 4 : 6;  // SWIZZLE_128B, _64B, _32B
  return ((16u * (uint32_t)ck) >> 4)                        // stride-byte offset: 8 rows
         | (1u << 14)                                       // descriptor version for sm_100
         | (layout << 29);
}
__device__ __forceinline__ uint64_t umma_desc(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }

// M = 128, BF16 x BF16 -> FP32; `mn_major`: both operands MN-major
__device__ __forceinline__ uint32_t umma_idesc(int n, bool mn_major) {
  return (1u << 4)                            // D format FP32
         | (1u << 7)                          // A format BF16
         | (1u << 10)                         // B format BF16
         | (mn_major ? (3u << 15) : 0u)       // A and B transposed
         | ((uint32_t)(n >> 3) << 17)         // N / 8
         | ((uint32_t)(128 >> 4) << 24);      // M / 16
}

__device__ __forceinline__ void umma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(net_smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void net_mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(net_smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void net_mbar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(net_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void net_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(net_smem_u32(bar)) : "memory");
}

// Bounded wait; when it runs out (or another warp's did) the CTA gives up: abort is set, the flag that
// the host reads is raised, and every role leaves its loop.
__device__ __forceinline__ bool net_mbar_wait(uint64_t* bar, uint32_t phase, volatile int* abort) {
  for (uint32_t it = 0; it < NET_WAIT_LIMIT; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(net_smem_u32(bar)), "r"(phase)
        : "memory");
    if (ok) return true;
    if (*abort) return false;
  }
  *abort = 1;
  atomicExch(&g_net_timeout, 1);
  return false;
}

// After a CTA gave up: waits (bounded each) until the last use of every barrier of a ring is complete, `uses`
// being the uses of the ring so far, so that no copy or MMA in flight outlives its shared memory or TMEM.
__device__ __noinline__ void net_drain(uint64_t* bars, int ring, int uses) {
  int none = 0;
  for (int k = 0; k < ring && k < uses; ++k) {
    const int idx = uses - 1 - k;
    net_mbar_wait(&bars[idx % ring], (uint32_t)((idx / ring) & 1), &none);
  }
}

__device__ __forceinline__ void tma_4d(void* dst, const CUtensorMap* map, int c, int x, int y, int b, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(net_smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(x), "r"(y), "r"(b), "r"(net_smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* map, int c, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(net_smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(x), "r"(y), "r"(net_smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(net_smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
// (.aligned: the whole warp takes part, joined here after its lanes' own branches)
__device__ __forceinline__ void tmem_dealloc(uint32_t base, uint32_t cols) {
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t addr, uint32_t (&r)[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__host__ __device__ inline uint32_t net_tmem_cols(int cols) {
  uint32_t c = 32;
  while ((int)c < cols) c *= 2;
  return c;
}

// ----------------------------------------------------------------------------------------------
// Forward (and data-gradient) convolution
//
// Persistent CTAs of ten warps: one thread loads operands by TMA, one issues the MMAs, eight warps
// write the results of the tile before from the other TMEM accumulator (a pair of warps per quarter
// of its lanes, each with half of the columns: with one warp per quarter and integer divisions
// for the tile's place, that chain of ~500 dependent instructions was what a tile took).  A tile is 8 columns x 16
// (or, in pairs that share the weights, 32) rows of output pixels, one TMEM lane each.  The sum runs
// over taps in row order, then channels: TMEM rounds by truncation, so another order moves the
// results, and 15 layers of BF16 rounding make 0.5 % of such a difference (dx outermost: 1.19 ms for the
// network instead of 1.21 ms).  Up to 64 x 64 channels the weights stay in shared memory and a
// stage is a tile's three boxes of 8 x 18 pixels, one per horizontal tap, zero outside the image:
// 8 pixels of a row are one swizzle atom, so a vertical tap is a box from dy rows on.  With more
// channels a stage is one tap: its box of pixels and, unless they stay, its weights.
// ----------------------------------------------------------------------------------------------
constexpr int CONV_THREADS = 320;

struct ConvItem {
  int nt, tx, ty, b;
};
__device__ __forceinline__ ConvItem conv_item(const ConvArgs& a, int it) {
  ConvItem i;
  int t, u;
  a.by_n.divmod(it, &t, &i.nt);
  a.by_x.divmod(t, &u, &i.tx);
  a.by_y.divmod(u, &i.b, &i.ty);
  return i;
}

template <int MT, int CK>
__global__ void __launch_bounds__(CONV_THREADS)
    conv_fwd_kernel(ConvArgs a, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w) {
  extern __shared__ __align__(1024) unsigned char net_smem[];
  __shared__ __align__(8) uint64_t full[8], empty[8], acc_full[2], acc_empty[2], w_full;
  __shared__ __align__(16) float bias_sh[512];
  __shared__ uint32_t tmem_sh;
  __shared__ int abort_sh;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort = &abort_sh;
  constexpr int ck = CK;
  const int chunks = a.cin / ck;
  const int bn = a.cout < 128 ? a.cout : 128;
  const uint32_t cols = net_tmem_cols(2 * MT * bn);
  const bool whole = a.whole != 0;
  const uint32_t x_bytes = (uint32_t)(NET_TW * (MT * NET_TH + (whole ? 2 : 0)) * ck * 2);
  const uint32_t w_bytes = (uint32_t)(bn * ck * 2);  // one tap
  const uint32_t x_pitch = (x_bytes + 1023) & ~1023u;
  const uint32_t stage_bytes = whole ? 3u * x_pitch : x_pitch + (a.resident ? 0u : w_bytes);
  const int steps = whole ? 1 : 9 * chunks;  // stages of a tile
  const uint32_t w_base = 0, ring = a.resident ? 9u * chunks * w_bytes : 0u;
  const int items = a.tiles * a.n_tiles;

  if (warp == 1) tmem_alloc(&tmem_sh, cols);
  for (int c = tid; c < a.cout; c += CONV_THREADS) bias_sh[c] = a.bias != nullptr ? a.bias[c] : 0.f;
  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      net_mbar_init(&full[s], 1);
      net_mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      net_mbar_init(&acc_full[s], 1);
      net_mbar_init(&acc_empty[s], 8);
    }
    net_mbar_init(&w_full, 1);
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_sh;
  int sent = 0, issued = 0;  // boxes' stages of the loading thread, stages consumed by the MMA thread

  if (warp == 0 && lane == 0) {
    // ---- loads
    if (a.resident && blockIdx.x < items) {
      net_mbar_expect(&w_full, 9u * chunks * w_bytes);
      for (int c = 0; c < chunks; ++c)
        for (int t = 0; t < 9; ++t)
          tma_3d(net_smem + w_base + (uint32_t)(c * 9 + t) * w_bytes, &tm_w, c * ck, t, 0, &w_full);
    }
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
      const ConvItem i = conv_item(a, it);
      for (int q = 0, t = 0, c = 0; q < steps; ++q, c + 1 == chunks ? (c = 0, ++t) : ++c) {
        if (sent >= a.stages && !net_mbar_wait(&empty[s], phase ^ 1u, abort)) {
          ok = false;
          break;
        }
        unsigned char* st = net_smem + ring + (uint32_t)s * stage_bytes;
        if (whole) {
          net_mbar_expect(&full[s], 3u * x_bytes);
          for (int dx = 0; dx < 3; ++dx)
            tma_4d(st + (uint32_t)dx * x_pitch, &tm_x, 0, i.tx * NET_TW + dx - 1, i.ty * MT * NET_TH - 1, i.b, &full[s]);
        } else {
          const int dy = t / 3;
          net_mbar_expect(&full[s], x_bytes + (a.resident ? 0u : w_bytes));
          tma_4d(st, &tm_x, c * ck, i.tx * NET_TW + t - 3 * dy - 1, i.ty * MT * NET_TH + dy - 1, i.b, &full[s]);
          if (!a.resident) tma_3d(st + x_pitch, &tm_w, c * ck, t, i.nt * bn, &full[s]);
        }
        ++sent;
        if (++s == a.stages) {
          s = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMAs
    const uint32_t idesc = umma_idesc(bn, false), hi = umma_desc_hi(CK), base = net_smem_u32(net_smem);
    int s = 0, done = 0;
    uint32_t phase = 0;
    bool ok = true;
    if (a.resident && blockIdx.x < items) ok = net_mbar_wait(&w_full, 0, abort);
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x, ++done) {
      const int buf = done & 1;
      if (done >= 2 && !net_mbar_wait(&acc_empty[buf], (uint32_t)(((done >> 1) & 1) ^ 1), abort)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int q = 0, t = 0, c = 0; q < steps; ++q) {
        if (!net_mbar_wait(&full[s], phase, abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t st = base + ring + (uint32_t)s * stage_bytes;
        const uint32_t xa = umma_desc_lo(st, 16);
        const uint32_t acc = tmem + (uint32_t)(buf * MT * bn);
        if (whole) {
          const uint32_t wb = umma_desc_lo(base + w_base, 16), w_step = w_bytes >> 4, x_step = x_pitch >> 4;
#pragma unroll
          for (int tap = 0; tap < 9; ++tap) {
#pragma unroll
            for (int k = 0; k < CK / 16; ++k) {
              const uint64_t bd = umma_desc(wb + tap * w_step + 2u * k, hi);
#pragma unroll
              for (int m = 0; m < MT; ++m)
                umma_bf16(acc + (uint32_t)(m * bn),
                          umma_desc(xa + (tap % 3) * x_step + (uint32_t)((m * NET_TH + tap / 3) * NET_TW * CK / 8) + 2u * k, hi),
                          bd, idesc, tap > 0 || k > 0);
            }
          }
        } else {
          const uint32_t wb = umma_desc_lo(a.resident ? base + w_base + (uint32_t)(c * 9 + t) * w_bytes : st + x_pitch, 16);
#pragma unroll
          for (int k = 0; k < CK / 16; ++k) {
            const uint64_t bd = umma_desc(wb + 2u * k, hi);
#pragma unroll
            for (int m = 0; m < MT; ++m)
              umma_bf16(acc + (uint32_t)(m * bn), umma_desc(xa + (uint32_t)(m * NET_TH * NET_TW * CK / 8) + 2u * k, hi), bd, idesc,
                        q > 0 || k > 0);
          }
        }
        umma_commit(&empty[s]);
        ++issued;
        if (++c == chunks) {
          c = 0;
          ++t;
        }
        if (++s == a.stages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (ok) umma_commit(&acc_full[buf]);
    }
  } else if (warp >= 2) {
    // ---- results: TMEM lane = pixel, warp % 4 selects its 32 lanes
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const int c_begin = half * ((bn / 16 + 1) / 2) * 16, c_end = half == 0 ? ((bn / 16 + 1) / 2) * 16 : bn;
    int done = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++done) {
      const int buf = done & 1;
      const ConvItem i = conv_item(a, it);
      const int x = i.tx * NET_TW + (row & 7), n0 = i.nt * bn;
      const bool ok = net_mbar_wait(&acc_full[buf], (uint32_t)((done >> 1) & 1), abort);
      if (!__all_sync(0xffffffffu, ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int m = 0; m < MT; ++m) {
        const int y = (i.ty * MT + m) * NET_TH + (row >> 3);
        const bool in = x < a.w && y < a.h;
        __nv_bfloat16* out = a.y + (((int64_t)i.b * a.h + y) * a.w + x) * a.cout + n0;
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_end; c0 += 16) {
          if (n0 + c0 >= a.cout) break;  // the whole warp
          uint32_t r[16];
          tmem_load16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((buf * MT + m) * bn + c0), r);
          uint32_t o[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float2 bias = *reinterpret_cast<const float2*>(&bias_sh[n0 + c0 + 2 * k]);
            float v0 = __uint_as_float(r[2 * k]) + bias.x, v1 = __uint_as_float(r[2 * k + 1]) + bias.y;
            if (a.relu) {
              v0 = fmaxf(v0, 0.f);
              v1 = fmaxf(v1, 0.f);
            }
            const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
            o[k] = *reinterpret_cast<const uint32_t*>(&h);
          }
          if (in && a.wide) {
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + c0), "r"(o[0]), "r"(o[1]),
                         "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7])
                         : "memory");
          } else if (in) {
            reinterpret_cast<uint4*>(out + c0)[0] = make_uint4(o[0], o[1], o[2], o[3]);
            reinterpret_cast<uint4*>(out + c0)[1] = make_uint4(o[4], o[5], o[6], o[7]);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) net_mbar_arrive(&acc_empty[buf]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_sh != 0) {  // whichever role gave up (all have ended, so abort no longer changes)
    if (tid == 0 && a.resident && blockIdx.x < items) net_drain(&w_full, 1, 1);
    if (tid == 0) net_drain(full, a.stages, sent);
    if (tid == 32) net_drain(empty, a.stages, issued);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, cols);
}

// ----------------------------------------------------------------------------------------------
// Weight gradient: dW[co][tap][ci] = sum over pixels p of dy[p][co] x[p + tap][ci]
//
// A GEMM with M = input channels (of several vertical taps), N = output channels and K = pixels.
// Both operands are used as TMA brings them (pixels x channels, channels contiguous: MN-major),
// 128 pixels per stage.  A CTA holds one horizontal tap dx and a range of pixel tiles; its box of
// x has two more rows, and the next vertical tap is the next atom, so that the descriptor's
// leading offset of one atom stacks taps along M: four of 32 channels (eight of 16), two of 64,
// and one of 128 channels (two boxes).  The sums of a tap past the third are not used.
//
// 64 x 64 channels over 16 x 128^2 pixels (19 GFLOP, 67 MB): 1465 us with operands gathered element by
// element, 60 us so.
//
// The tensor core's FP32 accumulation truncates, an error that grows with the number of steps (3e-5
// over 5,000 pixels): every WGRAD_GROUP tiles, 16 steps, the sums go to FP32 registers of eight warps,
// which add with rounding, while the next group fills the other TMEM buffer.
// ----------------------------------------------------------------------------------------------
constexpr int WGRAD_GROUP = 2;
constexpr int WGRAD_REGS = 8;  // blocks of 16 sums per thread

__global__ void __launch_bounds__(CONV_THREADS)
    conv_wgrad_kernel(WgradArgs a, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_dy) {
  extern __shared__ __align__(1024) unsigned char net_smem[];
  __shared__ __align__(8) uint64_t full[8], empty[8], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_sh;
  __shared__ int abort_sh;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort = &abort_sh;
  const uint32_t cols = net_tmem_cols(2 * a.sets * a.n);
  const uint32_t x_box = (uint32_t)(NET_TW * (NET_TH + 2) * a.ckx * 2), x_pitch = (x_box + 1023) & ~1023u;
  const uint32_t dy_box = (uint32_t)(NET_TW * NET_TH * a.cky * 2);
  const uint32_t stage_bytes = a.bx * x_pitch + a.by * ((dy_box + 1023) & ~1023u);
  const int dx = blockIdx.y % 3;
  const int cblock = blockIdx.y / 3;                    // (input block, output block)
  const int n_blocks = (a.cout + a.n - 1) / a.n;
  const int ci0 = cblock / n_blocks * a.bx * a.ckx, co0 = cblock % n_blocks * a.n;
  const int t0 = (int)((int64_t)blockIdx.x * a.tiles / gridDim.x), t1 = (int)((int64_t)(blockIdx.x + 1) * a.tiles / gridDim.x);

  if (warp == 1) tmem_alloc(&tmem_sh, cols);
  if (tid == 0) {
    for (int s = 0; s < a.stages; ++s) {
      net_mbar_init(&full[s], 1);
      net_mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      net_mbar_init(&acc_full[s], 1);
      net_mbar_init(&acc_empty[s], 8);
    }
    abort_sh = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_sh;
  int sent = 0, issued = 0;  // as in the forward

  if (warp == 0 && lane == 0) {
    int s = 0;
    uint32_t phase = 0;
    for (int tile = t0; tile < t1; ++tile) {
      const int tx = tile % a.tiles_x, ty = (tile / a.tiles_x) % a.tiles_y, b = tile / (a.tiles_x * a.tiles_y);
      if (sent >= a.stages && !net_mbar_wait(&empty[s], phase ^ 1u, abort)) break;
      unsigned char* st = net_smem + (uint32_t)s * stage_bytes;
      net_mbar_expect(&full[s], a.bx * x_box + a.by * dy_box);
      for (int k = 0; k < a.bx; ++k)
        tma_4d(st + k * x_pitch, &tm_x, ci0 + k * a.ckx, tx * NET_TW + dx - 1, ty * NET_TH - 1, b, &full[s]);
      for (int k = 0; k < a.by; ++k)
        tma_4d(st + a.bx * x_pitch + k * dy_box, &tm_dy, co0 + k * a.cky, tx * NET_TW, ty * NET_TH, b, &full[s]);
      ++sent;
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 1 && lane == 0) {
    const uint32_t idesc = umma_idesc(a.n, true);
    // along M the next ckx rows are the next vertical tap (one atom on), or the next box
    const uint32_t atom_x = 16u * a.ckx, atom_y = 16u * a.cky;
    const uint32_t lbo_x = a.bx > 1 ? x_pitch : atom_x, lbo_y = a.by > 1 ? dy_box : atom_y;
    const uint32_t set_step = ((a.ckx == 64 && a.bx == 1 ? 2u : 1u) * atom_x) >> 4;
    const uint32_t hi_x = umma_desc_hi(a.ckx), hi_y = umma_desc_hi(a.cky);
    int s = 0;
    uint32_t phase = 0;
    for (int tile = t0; tile < t1; ++tile) {
      const int group = (tile - t0) / WGRAD_GROUP, in_group = (tile - t0) % WGRAD_GROUP, buf = group & 1;
      if ((in_group == 0 && group >= 2 && !net_mbar_wait(&acc_empty[buf], (uint32_t)(((group >> 1) & 1) ^ 1), abort)) ||
          !net_mbar_wait(&full[s], phase, abort))
        break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem + (uint32_t)(buf * a.sets * a.n);
      const uint32_t xs = net_smem_u32(net_smem) + (uint32_t)s * stage_bytes;
      uint32_t xl = umma_desc_lo(xs, lbo_x), yl = umma_desc_lo(xs + a.bx * x_pitch, lbo_y);
#pragma unroll
      for (int k = 0; k < NET_TW * NET_TH / 16; ++k) {  // 16 pixels: two atoms
        const uint64_t bd = umma_desc(yl, hi_y);
        const bool acc = in_group > 0 || k > 0;
        umma_bf16(d, umma_desc(xl, hi_x), bd, idesc, acc);
        if (a.sets > 1) umma_bf16(d + (uint32_t)a.n, umma_desc(xl + set_step, hi_x), bd, idesc, acc);
        if (a.sets > 2) umma_bf16(d + (uint32_t)(2 * a.n), umma_desc(xl + 2 * set_step, hi_x), bd, idesc, acc);
        xl += atom_x >> 3;
        yl += atom_y >> 3;
      }
      umma_commit(&empty[s]);
      ++issued;
      if (in_group == WGRAD_GROUP - 1 || tile == t1 - 1) umma_commit(&acc_full[buf]);
      if (++s == a.stages) {
        s = 0;
        phase ^= 1u;
      }
    }
  } else if (warp >= 2) {
    // a pair of warps per quarter of the lanes, each with every other block of 16 columns
    const int quarter = warp & 3, half = (warp - 2) >> 2, row = quarter * 32 + lane;
    const int blocks = a.sets * a.n / 16;
    float sum[WGRAD_REGS][16];
#pragma unroll
    for (int j = 0; j < WGRAD_REGS; ++j)
#pragma unroll
      for (int k = 0; k < 16; ++k) sum[j][k] = 0.f;
    const int groups = (t1 - t0 + WGRAD_GROUP - 1) / WGRAD_GROUP;
    bool ok = true;
    for (int g = 0; g < groups; ++g) {
      const int buf = g & 1;
      ok = __all_sync(0xffffffffu, net_mbar_wait(&acc_full[buf], (uint32_t)((g >> 1) & 1), abort)) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int j = 0; j < WGRAD_REGS; ++j) {
        if (2 * j + half < blocks) {
          uint32_t r[16];
          tmem_load16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * a.sets * a.n + (2 * j + half) * 16), r);
#pragma unroll
          for (int k = 0; k < 16; ++k) sum[j][k] += __uint_as_float(r[k]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) net_mbar_arrive(&acc_empty[buf]);
    }
    if (ok) {
#pragma unroll
      for (int j = 0; j < WGRAD_REGS; ++j) {
        const int col = (2 * j + half) * 16, m = col / a.n, c0 = col - m * a.n;
        const int in_set = a.bx > 1 ? 0 : row / a.ckx;
        const int dy = m * (a.ckx == 64 && a.bx == 1 ? 2 : 1) + in_set;
        const int ci = ci0 + (a.bx > 1 ? row : row - in_set * a.ckx);
        if (2 * j + half >= blocks || dy >= 3 || ci >= a.cin) continue;
        float* out = a.dw + (3 * dy + dx) * a.cin + ci;
#pragma unroll
        for (int k = 0; k < 16; ++k)
          if (co0 + c0 + k < a.cout) atomicAdd(out + (int64_t)(co0 + c0 + k) * 9 * a.cin, sum[j][k]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_sh != 0) {
    if (tid == 0) net_drain(full, a.stages, sent);
    if (tid == 32) net_drain(empty, a.stages, issued);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, cols);
}

// ----------------------------------------------------------------------------------------------
// Launchers
// ----------------------------------------------------------------------------------------------
static int net_sms() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

static CUtensorMapSwizzle net_swizzle(int ck) {
  return ck == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : ck == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

// NHWC activations as (channel, x, y, image) with a box of ck channels x 8 columns x `rows` rows.
static bool net_map_nhwc(CUtensorMap* map, const void* p, int b, int h, int w, int c, int ck, int rows) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (enc == nullptr) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)b};
  const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)c * 2 * w, (cuuint64_t)c * 2 * w * h};
  const cuuint32_t box[4] = {(cuuint32_t)ck, (cuuint32_t)NET_TW, (cuuint32_t)rows, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, net_swizzle(ck), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Weights [cout][9][cin] as (channel, tap, output channel) with a box of one tap of bn outputs.
static bool net_map_weights(CUtensorMap* map, const void* p, int cin, int cout, int ck, int bn) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (enc == nullptr) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)cin, 9, (cuuint64_t)cout};
  const cuuint64_t strides[2] = {(cuuint64_t)cin * 2, (cuuint64_t)cin * 18};
  const cuuint32_t box[3] = {(cuuint32_t)ck, 1, (cuuint32_t)bn};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, net_swizzle(ck), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int net_fail(const char* msg) {
  cct_set_last_error(msg);
  return CCT_ERR_CUDA;
}

template <int MT, int CK>
static int launch_conv_fwd(ConvArgs a, const void* x, const void* wt, cudaStream_t st) {
  const int bn = a.cout < 128 ? a.cout : 128, chunks = a.cin / a.ck;
  a.tiles_x = (a.w + NET_TW - 1) / NET_TW;
  a.tiles_y = (a.h + MT * NET_TH - 1) / (MT * NET_TH);
  a.n_tiles = (a.cout + bn - 1) / bn;
  const int64_t tiles = (int64_t)a.batch * a.tiles_x * a.tiles_y;
  if (tiles * a.n_tiles > 0x7fffffffLL) return net_fail("the convolution has too many tiles");
  a.tiles = (int)tiles;
  a.by_n = FastDiv(a.n_tiles);
  a.by_x = FastDiv(a.tiles_x);
  a.by_y = FastDiv(a.tiles_y);
  a.whole = a.resident && chunks == 1;
  const int box_rows = MT * NET_TH + (a.whole ? 2 : 0);
  const int x_pitch = (NET_TW * box_rows * a.ck * 2 + 1023) / 1024 * 1024, w_tap = bn * a.ck * 2;
  const int weights = 9 * chunks * w_tap;
  const int stage = a.whole ? 3 * x_pitch : x_pitch + (a.resident ? 0 : w_tap);
  const int fixed = a.resident ? weights : 0;
  // two CTAs per SM where each still gets three stages, else as many stages as one CTA can hold
  const int half = 110 * 1024;
  const int per_sm = fixed + (a.whole ? 2 : 3) * stage <= half && 2 * net_tmem_cols(2 * MT * bn) <= 512 ? 2 : 1;
  const int room = (per_sm == 2 ? half : NET_SMEM_MAX - 1024) - fixed;
  a.stages = std::min(8, room / stage);
  if (a.stages < 2) return net_fail("the convolution's operands do not fit in shared memory");
  const int smem = fixed + a.stages * stage + 1024;
  CUtensorMap tm_x, tm_w;
  if (!net_map_nhwc(&tm_x, x, a.batch, a.h, a.w, a.cin, a.ck, box_rows) ||
      !net_map_weights(&tm_w, wt, a.cin, a.cout, a.ck, bn))
    return net_fail("cuTensorMapEncodeTiled refused the convolution's operands");
  if (!ensure_dynamic_smem<conv_fwd_kernel<MT, CK>>(NET_SMEM_MAX))
    return net_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed for the convolution kernel");
  const int64_t grid = std::min<int64_t>(tiles * a.n_tiles, (int64_t)net_sms() * per_sm);
  conv_fwd_kernel<MT, CK><<<(unsigned)grid, CONV_THREADS, smem, st>>>(a, tm_x, tm_w);
  return CCT_OK;
}

static int net_block(int c) { return c % 64 == 0 ? 64 : c % 32 == 0 ? 32 : 16; }

static int launch_conv_wgrad(WgradArgs a, const void* x, const void* dy, cudaStream_t st) {
  a.ckx = net_block(a.cin);
  a.cky = net_block(a.cout);
  a.bx = a.cin >= 128 ? 2 : 1;                               // cin is a power of two
  a.sets = a.bx > 1 ? 3 : a.ckx == 64 ? 2 : 1;
  // two buffers of sets x N sums fit the 512 TMEM columns and the registers of the eight warps
  a.by = std::max(1, std::min(a.cout, a.sets == 3 ? 64 : 128) / a.cky);
  a.n = a.by * a.cky;
  a.tiles_x = (a.w + NET_TW - 1) / NET_TW;
  a.tiles_y = (a.h + NET_TH - 1) / NET_TH;
  const int64_t tiles = (int64_t)a.batch * a.tiles_x * a.tiles_y;
  if (tiles > 0x7fffffffLL) return net_fail("the convolution has too many tiles");
  a.tiles = (int)tiles;
  const int x_pitch = (NET_TW * (NET_TH + 2) * a.ckx * 2 + 1023) / 1024 * 1024;
  const int dy_pitch = (NET_TW * NET_TH * a.cky * 2 + 1023) / 1024 * 1024;
  const int stage = a.bx * x_pitch + a.by * dy_pitch;
  a.stages = std::min(8, (NET_SMEM_MAX - 2048) / stage);
  // the taps past the third read up to five rows past the last box: 2048 spare bytes behind it
  const int smem = a.stages * stage + 2048;
  CUtensorMap tm_x, tm_dy;
  if (!net_map_nhwc(&tm_x, x, a.batch, a.h, a.w, a.cin, a.ckx, NET_TH + 2) ||
      !net_map_nhwc(&tm_dy, dy, a.batch, a.h, a.w, a.cout, a.cky, NET_TH))
    return net_fail("cuTensorMapEncodeTiled refused the convolution's operands");
  if (!ensure_dynamic_smem<conv_wgrad_kernel>(NET_SMEM_MAX))
    return net_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed for the weight-gradient kernel");
  const int groups = 3 * (a.cin / (a.bx * a.ckx)) * ((a.cout + a.n - 1) / a.n);
  // one CTA per SM over all groups, at least four tiles each (every CTA adds its sums atomically)
  const int split = (int)std::max<int64_t>(1, std::min<int64_t>(net_sms() / groups, (tiles + 3) / 4));
  conv_wgrad_kernel<<<dim3(split, groups), CONV_THREADS, smem, st>>>(a, tm_x, tm_dy);
  return CCT_OK;
}

// ----------------------------------------------------------------------------------------------
// Elementwise kernels (NHWC bf16 activations, FP32 parameters / gradients)
// ----------------------------------------------------------------------------------------------
__global__ void relu_bwd_kernel(const __nv_bfloat16* y, const __nv_bfloat16* dy, __nv_bfloat16* dx, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float g = __bfloat162float(y[i]) > 0.f ? __bfloat162float(dy[i]) : 0.f;
    dx[i] = __float2bfloat16_rn(g);
  }
}

// Eight BF16 channels (16 bytes) at a time: the tensors' channel counts are multiples of 16.
struct Bf16x8 {
  uint4 v;
  __device__ __forceinline__ void get(float (&f)[8]) const {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      f[2 * k] = __uint_as_float(w[k] << 16);
      f[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
    }
  }
  __device__ __forceinline__ void set(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
      w[k] = *reinterpret_cast<const uint32_t*>(&h);
    }
    v = make_uint4(w[0], w[1], w[2], w[3]);
  }
};

// 2x2 average pooling (stride 2) and its adjoint, V channels per thread (8, or 1 for channel counts or
// addresses that do not allow 16-byte accesses); grid y: rows of the small images.
// (Element by element with four divisions each, the network's three pools took 177 us on 8 x 512^2,
// the upsamplings 288 us and the additions 277 us, 4-5 times their memory time.)
template <int V>
__device__ __forceinline__ void ew_load(const __nv_bfloat16* p, float (&f)[V]) {
  if constexpr (V == 8) {
    Bf16x8 t;
    t.v = __ldg(reinterpret_cast<const uint4*>(p));
    t.get(f);
  } else {
    f[0] = __bfloat162float(*p);
  }
}
template <int V>
__device__ __forceinline__ void ew_store(__nv_bfloat16* p, const float (&f)[V]) {
  if constexpr (V == 8) {
    Bf16x8 t;
    t.set(f);
    *reinterpret_cast<uint4*>(p) = t.v;
  } else {
    *p = __float2bfloat16_rn(f[0]);
  }
}

// One row pair of the large image (row pitch `row` elements) and one row of the small one; `half`: the
// small image is their 2x2 mean (else their sum).  TO_SMALL reduces, else the small value (times 1/4
// for `half`) goes to the four large pixels.
template <int V, bool TO_SMALL>
__global__ void __launch_bounds__(256) resize2_kernel(const __nv_bfloat16* src, __nv_bfloat16* dst, int64_t rows, int w,
                                                      int c, int half) {
  // rows (of all images) and w: the small images
  const int cv = c / V, per_row = w * cv;
  for (int64_t y = blockIdx.y; y < rows; y += gridDim.y) {
    const __nv_bfloat16* s = src + y * (TO_SMALL ? 4 : 1) * (int64_t)w * c;
    __nv_bfloat16* d = dst + y * (TO_SMALL ? 1 : 4) * (int64_t)w * c;
    const int64_t row = 2 * (int64_t)w * c;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < per_row; i += gridDim.x * blockDim.x) {
      const int x = i / cv, ch = (i - x * cv) * V;
      const int64_t big = 2 * (int64_t)x * c + ch, small = (int64_t)x * c + ch;
      float v[V];
      if constexpr (TO_SMALL) {
        float a[V], b[V], e[V], f[V];
        ew_load<V>(s + big, a);
        ew_load<V>(s + big + c, b);
        ew_load<V>(s + big + row, e);
        ew_load<V>(s + big + row + c, f);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const float t = a[k] + b[k] + e[k] + f[k];
          v[k] = half ? 0.25f * t : t;
        }
        ew_store<V>(d + small, v);
      } else {
        ew_load<V>(s + small, v);
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = half ? 0.25f * v[k] : v[k];
        ew_store<V>(d + big, v);
        ew_store<V>(d + big + c, v);
        ew_store<V>(d + big + row, v);
        ew_store<V>(d + big + row + c, v);
      }
    }
  }
}

template <int V>
__global__ void __launch_bounds__(256) add_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out,
                                                  int64_t n) {
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * V; i < n; i += (int64_t)gridDim.x * blockDim.x * V) {
    float u[V], v[V];
    ew_load<V>(a + i, u);
    ew_load<V>(b + i, v);
#pragma unroll
    for (int k = 0; k < V; ++k) u[k] += v[k];
    ew_store<V>(out + i, u);
  }
}

// db[c] += sum over pixels of dy[p][c]: V channels per thread, the threads of a block over pixels, halved
// in shared memory by all threads down to one sum per channel, which neighbouring threads add to db
// (a warp's atomics are one line; added by the few threads of one pixel, eight strided channels each, they
// took most of the time).  16 x 128^2 pixels of 64 channels 16.3 -> 5.7 us, 256^2 of 256 26.7 -> 6.6 us.
template <int V>
__global__ void __launch_bounds__(256) bias_grad_kernel(const __nv_bfloat16* dy, float* db, int64_t pixels, int c) {
  __shared__ float part[256 * V];
  const int cv = min(c / V, 256);              // channel groups of this block (blockIdx.y: the next 256)
  const int lanes = 256 / cv, g = threadIdx.x % cv, lane = threadIdx.x / cv;
  const int ch = (blockIdx.y * 256 + g) * V;
  float s[V];
#pragma unroll
  for (int k = 0; k < V; ++k) s[k] = 0.f;
  if (lane < lanes && ch < c) {
    const int64_t step = (int64_t)gridDim.x * lanes;
    int64_t p = (int64_t)blockIdx.x * lanes + lane;
    for (; p + 7 * step < pixels; p += 8 * step) {  // eight loads in flight
      float v[8][V];
#pragma unroll
      for (int u = 0; u < 8; ++u) ew_load<V>(dy + (p + u * step) * c + ch, v[u]);
#pragma unroll
      for (int k = 0; k < V; ++k)
        s[k] += ((v[0][k] + v[1][k]) + (v[2][k] + v[3][k])) + ((v[4][k] + v[5][k]) + (v[6][k] + v[7][k]));
    }
    for (; p < pixels; p += step) {
      float v[V];
      ew_load<V>(dy + p * c + ch, v);
#pragma unroll
      for (int k = 0; k < V; ++k) s[k] += v[k];
    }
  }
#pragma unroll
  for (int k = 0; k < V; ++k) part[threadIdx.x * V + k] = s[k];
  const int width = cv * V;  // part: a row of the block's channels per lane
  for (int rows = lanes; rows > 1;) {
    const int half = (rows + 1) / 2;
    __syncthreads();
    for (int i = threadIdx.x; i < (rows - half) * width; i += 256) part[i] += part[i + half * width];
    rows = half;
  }
  __syncthreads();
  const int c0 = blockIdx.y * 256 * V;
  for (int i = threadIdx.x; i < min(width, c - c0); i += 256) atomicAdd(db + c0 + i, part[i]);
}

// MSE loss on channel 0 of an NHWC prediction vs an FP32 target [b][h][w]:
// loss += sum (pred - t)^2 / count; grad = 2 (pred - t) / count written to channel 0 (others 0)
__global__ void mse_kernel(const __nv_bfloat16* pred, const float* target, __nv_bfloat16* grad, double* loss,
                           int64_t pixels, int c) {
  double acc = 0.0;
  const float inv = 1.f / (float)pixels;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < pixels; p += (int64_t)gridDim.x * blockDim.x) {
    const float d = __bfloat162float(pred[p * c]) - target[p];
    acc += (double)d * d;
    grad[p * c] = __float2bfloat16_rn(2.f * d * inv);
    for (int ch = 1; ch < c; ++ch) grad[p * c + ch] = __float2bfloat16_rn(0.f);
  }
  acc = warp_sum_double(acc);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, acc / (double)pixels);
}

// Adam with FP32 master weights; writes the BF16 copy used by the GEMMs
__global__ void adam_kernel(float* p, const float* g, float* m, float* v, __nv_bfloat16* p16, int64_t n, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    if (p16 != nullptr) p16[i] = __float2bfloat16_rn(pi);
  }
}

// weights [co][3][3][ci] -> data-gradient weights [ci][3][3][co] with the taps flipped
__global__ void flip_weights_kernel(const __nv_bfloat16* w, __nv_bfloat16* wf, int cin, int cout) {
  const int64_t n = 9LL * cin * cout;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int co = (int)(i % cout);
    int64_t r = i / cout;
    const int tap = (int)(r % 9);
    const int ci = (int)(r / 9);
    wf[i] = w[((int64_t)co * 9 + (8 - tap)) * cin + ci];
  }
}

// FP32 planar images (channel k of `nch` sources, each [pixels]) -> NHWC bf16 with c channels
// (zero padded), every value divided by the scale of its slice (slices of slice_pixels pixels)
__global__ void pack_nhwc_kernel(const float* const* src, int nch, __nv_bfloat16* dst, int64_t pixels, int c,
                                 const float* slice_scale, int64_t slice_pixels) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < pixels; p += (int64_t)gridDim.x * blockDim.x) {
    const float inv = slice_scale != nullptr ? 1.f / slice_scale[p / slice_pixels] : 1.f;
    for (int ch = 0; ch < c; ++ch) {
      const float v = ch < nch ? src[ch][p] * inv : 0.f;
      dst[p * c + ch] = __float2bfloat16_rn(v);
    }
  }
}

// channel 0 of NHWC bf16 -> FP32 planar.  mode 0: out = max(base + scale_s * v, floor);
// mode 1 (multiplicative): out = max((base + scale_s * floor) * exp(v) - scale_s * floor, floor)
__global__ void unpack_c0_kernel(const __nv_bfloat16* src, int c, const float* base, const float* slice_scale,
                                 int64_t slice_pixels, int mode, float floor_v, float* out, int64_t pixels) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < pixels; p += (int64_t)gridDim.x * blockDim.x) {
    const float sc = slice_scale != nullptr ? slice_scale[p / slice_pixels] : 1.f;
    const float v = __bfloat162float(src[p * c]);
    const float b = base != nullptr ? base[p] : 0.f;
    float r;
    if (mode == 1) {
      const float off = sc * floor_v;
      r = (b + off) * expf(v) - off;
    } else {
      r = b + sc * v;
    }
    out[p] = fmaxf(r, floor_v);
  }
}

// out[i] = a[i] / b[i % b_count] (b broadcast over slices)
__global__ void ratio_kernel(const float* a, const float* b, float* out, int64_t n, int64_t b_count) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = a[i] / b[i % b_count];
}

static inline unsigned ew_blocks(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 4096) b = 4096;
  return (unsigned)(b < 1 ? 1 : b);
}

// 16-byte accesses: every address and the channel count allow them
static bool ew_wide(const void* a, const void* b, const void* d, int64_t c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(d)) & 15) == 0 &&
         c % 8 == 0;
}

// small (h x w) and large (2h x 2w) images of c channels
static void launch_resize2(const void* src, void* dst, int64_t rows, int w, int c, int half, bool to_small,
                           cudaStream_t st) {
  if (rows <= 0 || w <= 0) return;  // empty images: nothing to do
  const bool wide = ew_wide(src, dst, nullptr, c);
  const int per_row = w * (wide ? c / 8 : c);
  const dim3 grid((unsigned)std::min(64, (per_row + 255) / 256), (unsigned)std::min<int64_t>(rows, 65535));
  const __nv_bfloat16* s = reinterpret_cast<const __nv_bfloat16*>(src);
  __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(dst);
  if (wide && to_small) {
    resize2_kernel<8, true><<<grid, 256, 0, st>>>(s, d, rows, w, c, half);
  } else if (wide) {
    resize2_kernel<8, false><<<grid, 256, 0, st>>>(s, d, rows, w, c, half);
  } else if (to_small) {
    resize2_kernel<1, true><<<grid, 256, 0, st>>>(s, d, rows, w, c, half);
  } else {
    resize2_kernel<1, false><<<grid, 256, 0, st>>>(s, d, rows, w, c, half);
  }
}

static void launch_bias_grad(const void* dy, float* db, int64_t pixels, int c, cudaStream_t st) {
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(dy);
  const bool wide = ew_wide(dy, nullptr, nullptr, c);
  const int groups = wide ? c / 8 : c, lanes = 256 / std::min(groups, 256);
  // 8 pixels per thread, or more where that takes over two blocks per SM (every block adds its sums to the
  // same few addresses: 256^2 pixels of 256 channels 6.6 us, 9.1 with four blocks, 11.9 with eight; 64^2 of
  // 256 2.9 us, 3.3 with 16 pixels per thread)
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(2 * net_sms(), pixels / (8 * lanes)));
  const dim3 grid((unsigned)blocks, (unsigned)((groups + 255) / 256));
  if (wide) {
    bias_grad_kernel<8><<<grid, 256, 0, st>>>(p, db, pixels, c);
  } else {
    bias_grad_kernel<1><<<grid, 256, 0, st>>>(p, db, pixels, c);
  }
}

int read_net_timeout(int clear, int* value) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_net_timeout, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  if (clear) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_net_timeout, &zero, sizeof(int));
    if (e != cudaSuccess) return (int)e;
  }
  *value = v;
  return 0;
}

}  // namespace cct

// ------------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------------
static int net_check_conv(const cct_conv_desc* d) {
  CCT_REQUIRE(d != nullptr, "conv descriptor is NULL");
  CCT_REQUIRE(d->batch >= 1 && d->height >= 1 && d->width >= 1, "batch, height and width must be >= 1");
  CCT_REQUIRE(d->cin >= 16 && d->cin <= 512 && (d->cin & (d->cin - 1)) == 0, "cin must be a power of two in [16, 512]");
  CCT_REQUIRE(d->cout >= 16 && d->cout <= 512 && d->cout % 16 == 0, "cout must be a multiple of 16 in [16, 512]");
  return CCT_OK;
}

// TMA reads tensors that start on 16-byte boundaries
static bool net_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static int net_launch_check() {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    cct_set_last_error(cudaGetErrorString(e));
    return CCT_ERR_CUDA;
  }
  return CCT_OK;
}

extern "C" {

int cct_conv3x3_fwd(const cct_conv_desc* desc, const void* x, const void* w, const float* bias, int32_t relu,
                    void* y, void* stream) {
  int rc = net_check_conv(desc);
  if (rc != CCT_OK) return rc;
  CCT_REQUIRE(x != nullptr && w != nullptr && y != nullptr, "x, w and y are required");
  CCT_REQUIRE(net_aligned16(x) && net_aligned16(w) && net_aligned16(y), "x, w and y must be 16-byte aligned");
  cct::ConvArgs a;
  std::memset(&a, 0, sizeof(a));
  a.batch = desc->batch; a.h = desc->height; a.w = desc->width; a.cin = desc->cin; a.cout = desc->cout;
  a.ck = desc->cin < 64 ? desc->cin : 64;
  a.bias = bias;
  a.y = reinterpret_cast<__nv_bfloat16*>(y);
  a.relu = relu;
  a.wide = (reinterpret_cast<uintptr_t>(y) & 31) == 0;
  // weights of one output tile stay in shared memory up to 74 KB (64 x 64 channels); beyond that two
  // pixel tiles share each load of them
  a.resident = desc->cout <= 128 && 9 * desc->cin * desc->cout * 2 <= 9 * 64 * 64 * 2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a.resident) {
    rc = a.ck == 64   ? cct::launch_conv_fwd<1, 64>(a, x, w, st)
         : a.ck == 32 ? cct::launch_conv_fwd<1, 32>(a, x, w, st)
                      : cct::launch_conv_fwd<1, 16>(a, x, w, st);
  } else {
    rc = a.ck == 64   ? cct::launch_conv_fwd<2, 64>(a, x, w, st)
         : a.ck == 32 ? cct::launch_conv_fwd<2, 32>(a, x, w, st)
                      : cct::launch_conv_fwd<2, 16>(a, x, w, st);
  }
  if (rc != CCT_OK) return rc;
  return net_launch_check();
}

int cct_conv3x3_wgrad(const cct_conv_desc* desc, const void* x, const void* dy, float* dw, void* stream) {
  int rc = net_check_conv(desc);
  if (rc != CCT_OK) return rc;
  CCT_REQUIRE(x != nullptr && dy != nullptr && dw != nullptr, "x, dy and dw are required");
  CCT_REQUIRE(net_aligned16(x) && net_aligned16(dy), "x and dy must be 16-byte aligned");
  cct::WgradArgs a;
  std::memset(&a, 0, sizeof(a));
  a.batch = desc->batch; a.h = desc->height; a.w = desc->width; a.cin = desc->cin; a.cout = desc->cout;
  a.dw = dw;
  rc = cct::launch_conv_wgrad(a, x, dy, reinterpret_cast<cudaStream_t>(stream));
  if (rc != CCT_OK) return rc;
  return net_launch_check();
}

int cct_net_flip_weights(const void* w, void* w_flipped, int32_t cin, int32_t cout, void* stream) {
  CCT_REQUIRE(w != nullptr && w_flipped != nullptr && cin > 0 && cout > 0, "bad flip_weights arguments");
  const int64_t n = 9LL * cin * cout;
  cct::flip_weights_kernel<<<cct::ew_blocks(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(w), reinterpret_cast<__nv_bfloat16*>(w_flipped), cin, cout);
  return net_launch_check();
}

int cct_net_relu_bwd(const void* y, const void* dy, void* dx, int64_t count, void* stream) {
  CCT_REQUIRE(y && dy && dx && count > 0, "bad relu_bwd arguments");
  cct::relu_bwd_kernel<<<cct::ew_blocks(count), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(y), reinterpret_cast<const __nv_bfloat16*>(dy),
      reinterpret_cast<__nv_bfloat16*>(dx), count);
  return net_launch_check();
}

int cct_net_avgpool2(const void* x, void* y, int32_t batch, int32_t height, int32_t width, int32_t channels,
                     int32_t backward, void* stream) {
  CCT_REQUIRE(x && y && batch > 0 && height % 2 == 0 && width % 2 == 0 && channels > 0, "bad avgpool2 arguments");
  cct::launch_resize2(x, y, (int64_t)batch * (height / 2), width / 2, channels, 1, !backward,
                      reinterpret_cast<cudaStream_t>(stream));
  return net_launch_check();
}

int cct_net_upsample2(const void* x, void* y, int32_t batch, int32_t height, int32_t width, int32_t channels,
                      int32_t backward, void* stream) {
  CCT_REQUIRE(x && y && batch > 0 && height > 0 && width > 0 && channels > 0, "bad upsample2 arguments");
  cct::launch_resize2(x, y, (int64_t)batch * height, width, channels, 0, backward != 0,
                      reinterpret_cast<cudaStream_t>(stream));
  return net_launch_check();
}

int cct_net_add(const void* a, const void* b, void* out, int64_t count, void* stream) {
  CCT_REQUIRE(a && b && out && count > 0, "bad add arguments");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const __nv_bfloat16 *pa = reinterpret_cast<const __nv_bfloat16*>(a), *pb = reinterpret_cast<const __nv_bfloat16*>(b);
  __nv_bfloat16* po = reinterpret_cast<__nv_bfloat16*>(out);
  if (cct::ew_wide(a, b, out, count)) {
    cct::add_kernel<8><<<cct::ew_blocks(count / 8), 256, 0, st>>>(pa, pb, po, count);
  } else {
    cct::add_kernel<1><<<cct::ew_blocks(count), 256, 0, st>>>(pa, pb, po, count);
  }
  return net_launch_check();
}

int cct_net_bias_grad(const void* dy, float* db, int64_t pixels, int32_t channels, void* stream) {
  CCT_REQUIRE(dy && db && pixels > 0 && channels > 0, "bad bias_grad arguments");
  cct::launch_bias_grad(dy, db, pixels, channels, reinterpret_cast<cudaStream_t>(stream));
  return net_launch_check();
}

int cct_net_mse(const void* pred, const float* target, void* grad, double* loss, int64_t pixels, int32_t channels,
                void* stream) {
  CCT_REQUIRE(pred && target && grad && loss && pixels > 0 && channels > 0, "bad mse arguments");
  cct::mse_kernel<<<cct::ew_blocks(pixels), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(pred), target, reinterpret_cast<__nv_bfloat16*>(grad), loss, pixels,
      channels);
  return net_launch_check();
}

int cct_net_adam(float* p, const float* g, float* m, float* v, void* p_bf16, int64_t count, float lr, float beta1,
                 float beta2, float eps, int32_t step, void* stream) {
  CCT_REQUIRE(p && g && m && v && count > 0 && step >= 1, "bad adam arguments");
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  cct::adam_kernel<<<cct::ew_blocks(count), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      p, g, m, v, reinterpret_cast<__nv_bfloat16*>(p_bf16), count, lr, beta1, beta2, eps, c1, c2);
  return net_launch_check();
}

int cct_net_pack_nhwc(const float* const* src, int32_t n_src, void* dst, int64_t pixels, int32_t channels,
                      const float* slice_scale, int64_t slice_pixels, void* stream) {
  CCT_REQUIRE(src && dst && n_src >= 1 && n_src <= channels && pixels > 0, "bad pack_nhwc arguments");
  CCT_REQUIRE(slice_scale == nullptr || (slice_pixels > 0 && pixels % slice_pixels == 0), "bad slice_pixels");
  cct::pack_nhwc_kernel<<<cct::ew_blocks(pixels), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      src, n_src, reinterpret_cast<__nv_bfloat16*>(dst), pixels, channels, slice_scale, slice_pixels);
  return net_launch_check();
}

int cct_net_unpack_c0(const void* src, int32_t channels, const float* base, const float* slice_scale,
                      int64_t slice_pixels, int32_t mode, float floor_value, float* out, int64_t pixels, void* stream) {
  CCT_REQUIRE(src && out && pixels > 0 && channels > 0 && (mode == 0 || mode == 1), "bad unpack_c0 arguments");
  CCT_REQUIRE(slice_scale == nullptr || (slice_pixels > 0 && pixels % slice_pixels == 0), "bad slice_pixels");
  cct::unpack_c0_kernel<<<cct::ew_blocks(pixels), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(src), channels, base, slice_scale, slice_pixels, mode, floor_value, out,
      pixels);
  return net_launch_check();
}

int cct_net_ratio(const float* a, const float* b, float* out, int64_t count, int64_t b_count, void* stream) {
  CCT_REQUIRE(a && b && out && count > 0 && b_count > 0 && count % b_count == 0, "bad ratio arguments");
  cct::ratio_kernel<<<cct::ew_blocks(count), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a, b, out, count, b_count);
  return net_launch_check();
}

int cct_net_timeout(int32_t clear, int32_t* value) {
  CCT_REQUIRE(value != nullptr, "value is required");
  int v = 0;
  const int e = cct::read_net_timeout(clear, &v);
  if (e != 0) {
    cct_set_last_error(cudaGetErrorString((cudaError_t)e));
    return CCT_ERR_CUDA;
  }
  *value = v;
  return CCT_OK;
}

}  // extern "C"
