// Forward and back projection kernels of the XRF path (sm_100a).
//
// Forward projection (scikit-image radon discretisation, corrct:
// src/corrct/_projector_backends.py:312-333, attenuated form projectors.py:502-531):
//   sino[s][d][a][c] = w[a][d] * sum_r bilin(vol[s] * maps[s][a][d], M_a (c, r))
// One CTA owns (slice, angle, detector, band of 64 detector bins) and walks the
// column band in chunks of 64 rows.  For each chunk the bounding box of the
// rotated chunk is staged in shared memory as z = vol * map (coalesced float4
// loads of both, zero outside the image, a row stride of 100 so lanes on different
// rows hit different banks), then each thread samples 16 rows of one column
// from shared memory.  Column sums stay in registers; the CTA writes final
// values, so the result is deterministic and needs no atomics or partial sums.
// The map of every angle is read from HBM once; the volume is L2-resident.
//
// Back projection (scikit-image iradon, filter None, corrct:
// src/corrct/_projector_backends.py:335-359): one CTA owns a tile of 32 columns and 32 or
// 64 rows and walks its (detector, angle) lines in chunks of 16; each chunk stages, per
// line, the <= 74 detector bins the tile can reach as (value, slope) pairs, and every
// pixel does one shared-memory lookup and one FMA per line.  np.interp's left=0 / right=0
// edges are discontinuous: pixels within 0.01 bin of a detector edge are decided apart,
// exactly as numpy decides them in double.

#include <cstring>

#include "cct_common.cuh"
#include "cct_internal.cuh"

namespace cct {

// Raised (never trapped) if a staged box would exceed its shared-memory bound; valid
// rotation matrices cannot reach it.  Read through cct_device_error().
__device__ int g_box_overflow = 0;

// ------------------------------------------------------------------------------------------
// Forward projection
// ------------------------------------------------------------------------------------------
constexpr int FP_TC = 64;                          // detector bins per CTA
constexpr int FP_TR = 64;                          // rows per staged chunk
constexpr int FP_THREADS = 256;
// Lanes of a warp cover an 8 (columns) x 4 (rows) block of samples: 32 points of a rotated
// lattice patch spread over ~2 wavefronts per shared load at any angle, where a 32 x 1 line
// of lanes hits 32-way bank conflicts at some angles.  Warp w owns columns 8w..8w+7.
constexpr int FP_LC = 8;
constexpr int FP_LR = 4;
constexpr int FP_RPT = FP_TR / FP_LR;              // 16 samples per thread per chunk
// Rotated 64x64 chunk: extent <= 63*sqrt(2) = 89.1, +1/+2 tap margins, +3 for float4
// alignment of the left edge, rounded up to a multiple of 4.
constexpr int FP_BOX_W = 100;
constexpr int FP_BOX_H = 96;
constexpr int FP_STRIDE = FP_BOX_W;                // 16-byte rows: conflict-free float4 fills
constexpr int FP_MAX_CHUNKS = (8192 + FP_TR - 1) / FP_TR;  // row chunks of the largest n
constexpr float FP_SLAB_EPS = 0.01f;               // slab widening of a box row (y)
constexpr float FP_ROW_MARGIN = 0.5f;              // column range widening (x)
static_assert(FP_MAX_CHUNKS <= FP_THREADS, "one thread per chunk box");
constexpr int FP_FILL_BATCH = 3;                   // float4 items whose loads are issued together

template <bool HAS_MAPS, int MAPS_DTYPE>
__device__ __forceinline__ float4 fp_load_item(const float* vol, const MapRef& mref, int n, int gy, int gx) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (gy < 0 || gy >= n || gx + 3 < 0 || gx >= n) return v;
  const int off = gy * n + gx;  // < 2^31 for n <= 8192... n*n <= 2^26
  float e[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int xx = gx + k;
    float val = 0.f;
    if (xx >= 0 && xx < n) {
      val = __ldg(vol + off + k);
      if (HAS_MAPS) val *= map_at<MAPS_DTYPE>(mref, off + k);
    }
    e[k] = val;
  }
  return make_float4(e[0], e[1], e[2], e[3]);
}

// Bounding box of the sample positions of columns [c0, c_last] x rows [r0, r_last] (the corners
// of a rotated rectangle), widened by the bilinear taps; x origin floored to a multiple of 4.
__device__ __forceinline__ void chunk_box(float m00, float m01, float m02, float m10, float m11, float m12, int c0,
                                          int c_last, int r0, int r_last, int& bx0, int& bx1, int& by0, int& by1) {
  const float fc0 = (float)c0, fc1 = (float)c_last, fr0 = (float)r0, fr1 = (float)r_last;
  const float xa = sample_x(m00, m01, m02, fc0, fr0), xb = sample_x(m00, m01, m02, fc1, fr0);
  const float xc = sample_x(m00, m01, m02, fc0, fr1), xd = sample_x(m00, m01, m02, fc1, fr1);
  const float ya = sample_x(m10, m11, m12, fc0, fr0), yb = sample_x(m10, m11, m12, fc1, fr0);
  const float yc = sample_x(m10, m11, m12, fc0, fr1), yd = sample_x(m10, m11, m12, fc1, fr1);
  const float xmin = fminf(fminf(xa, xb), fminf(xc, xd)), xmax = fmaxf(fmaxf(xa, xb), fmaxf(xc, xd));
  const float ymin = fminf(fminf(ya, yb), fminf(yc, yd)), ymax = fmaxf(fmaxf(ya, yb), fmaxf(yc, yd));
  bx0 = ((int)floorf(xmin) - 1) & ~3;  // floor to a multiple of 4 (two's complement)
  bx1 = (int)floorf(xmax) + 2;
  by0 = (int)floorf(ymin) - 1;
  by1 = (int)floorf(ymax) + 2;
}

// Quads (4-column groups counted from the box origin bx0) of box row y that the bilinear taps
// of a chunk can read.  Samples whose floor(py) is y - 1 or y lie in the slab y - 1 <= py < y + 1;
// their x over the chunk's parallelogram (corners (px[k], py[k]) in cyclic order, the positions
// of the corner samples) is the range of its edges clipped to the slab, widened by
// FP_ROW_MARGIN against rounding (the approximate division moves it by far less) and by the
// right tap.  Returns (first, last) clipped to [0, q4 - 1]; first > last when no tap reads it.
__device__ __forceinline__ short2 fp_row_quads(const float (&px)[4], const float (&py)[4], int y, int bx0, int q4) {
  const float ylo = (float)y - 1.f - FP_SLAB_EPS, yhi = (float)y + 1.f + FP_SLAB_EPS;
  float xmin = 3.0e38f, xmax = -3.0e38f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float xa = px[e], ya = py[e], xb = px[(e + 1) & 3], yb = py[(e + 1) & 3];
    float t0 = 0.f, t1 = 1.f;
    const float dy = yb - ya;
    if (fabsf(dy) < 1e-6f) {
      if (ya < ylo || ya > yhi) continue;
    } else {
      float ta = __fdividef(ylo - ya, dy), tb = __fdividef(yhi - ya, dy);
      if (ta > tb) { const float t = ta; ta = tb; tb = t; }
      t0 = fmaxf(ta, 0.f);
      t1 = fminf(tb, 1.f);
      if (t0 > t1) continue;
    }
    const float x0 = fmaf(t0, xb - xa, xa), x1 = fmaf(t1, xb - xa, xa);
    xmin = fminf(xmin, fminf(x0, x1));
    xmax = fmaxf(xmax, fmaxf(x0, x1));
  }
  if (xmin > xmax) return make_short2(1, 0);
  const int lo = (int)floorf(xmin - FP_ROW_MARGIN) - bx0;
  const int hi = (int)floorf(xmax + FP_ROW_MARGIN) + 1 - bx0;
  return make_short2((short)(max(lo, 0) >> 2), (short)min(hi >> 2, q4 - 1));
}

// Positions of the four corner samples of chunk columns [c0, c1] x rows [r0, r1], cyclic order.
__device__ __forceinline__ void chunk_corners(float m00, float m01, float m02, float m10, float m11, float m12, int c0,
                                              int c1, int r0, int r1, float (&px)[4], float (&py)[4]) {
  const float fc0 = (float)c0, fc1 = (float)c1, fr0 = (float)r0, fr1 = (float)r1;
  px[0] = sample_x(m00, m01, m02, fc0, fr0); py[0] = sample_x(m10, m11, m12, fc0, fr0);
  px[1] = sample_x(m00, m01, m02, fc1, fr0); py[1] = sample_x(m10, m11, m12, fc1, fr0);
  px[2] = sample_x(m00, m01, m02, fc1, fr1); py[2] = sample_x(m10, m11, m12, fc1, fr1);
  px[3] = sample_x(m00, m01, m02, fc0, fr1); py[3] = sample_x(m10, m11, m12, fc0, fr1);
}

// CTA sum of one residual partial per thread (FP64, fixed order) into partials[slot]; red
// holds one double per warp.  Every thread of the CTA calls it.
__device__ __forceinline__ void fp_write_partial(double v, double* partials, int64_t slot, double* red, int lane,
                                                 int warp, int tid) {
  v = warp_sum_double(v);
  __syncthreads();  // red may still be read by a previous call
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < FP_TC / FP_LC; ++w) t += red[w];
    partials[slot] = t;
  }
}

// Asks L2 for the map rows of a chunk's box, a 128-byte line per request (the first at the row's start in
// the box, so that every address lies inside the row).  The fill is bound by the latency of its loads
// (the long scoreboard is half of all stalls): issued one chunk ahead, its map loads wait for L2 and not
// for HBM.  MLEM at 512x720, 16 slices: 8.4 -> 7.6 ms an iteration, 8 slices in subsets 7.43 -> 6.70 ms,
// 32 slices with BF16 maps 12.7 -> 11.8 ms a projection.  One bulk request per row
// (cp.async.bulk.prefetch) does the same with more instructions, as its operands are uniform and
// the lanes take turns: 7.9 ms, 6.98 ms and 13.0 ms.  Asking after the fill (2% slower) or two chunks
// ahead (no difference) gains less.  Line-integral fields are not asked for: their planes are shared
// by the channels' CTAs, which already find them in L2 (9.4 -> 10.2 ms a 1024x720 4-channel
// iteration with every channel asking, 9.7 ms with one, both in bulk).
template <int DT>
__device__ __forceinline__ void fp_prefetch_rows(const MapRef& m, int n, const int4 box, int tid) {
  constexpr int ES = DT == CCT_DTYPE_BF16 ? 2 : 4;
  // lines asked for of a row, which has at most 400 (BF16: 200) bytes: the end of a row that reaches into one
  // more line (BF16 rows near 45 degrees, FP32 rows at n % 4 != 0) is left to the fill
  constexpr int LINES = DT == CCT_DTYPE_BF16 ? 2 : 4;
  const int x0 = max(box.x, 0), x1 = min(box.y + 1, n);
  const int line = tid % LINES;
#pragma unroll
  for (int k = 0; k < (FP_BOX_H * LINES + FP_THREADS - 1) / FP_THREADS; ++k) {
    const int y = box.z + tid / LINES + k * (FP_THREADS / LINES);
    if (y > box.w || (unsigned)y >= (unsigned)n) continue;
    const uint64_t row = reinterpret_cast<uint64_t>(m.base) + (uint64_t)(m.off + (int64_t)y * n) * ES;
    const uint64_t b = row + (uint64_t)(x0 * ES), e = row + (uint64_t)(x1 * ES);
    uint64_t at = (b & ~127ull) + 128ull * line;
    if (line == 0) at = b;
    if (at < e && x0 < x1) asm volatile("prefetch.global.L2 [%0];" ::"l"(at) : "memory");
  }
}

// One CTA of the forward projection: detector band `band` of (angle, detector) `ad` of slice
// `s`; `n_bands` and `n_ad` are the batch's band and (angle, detector) counts (the residual
// partials are indexed by them).
template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
__device__ __forceinline__ void fp_cta(const FpArgs& args, const int band, const int ad, const int s, const int n_bands,
                                       const int n_ad) {
  __shared__ __align__(16) float z[FP_BOX_H * FP_STRIDE];
  __shared__ double red_d[FP_TC / FP_LC];
  __shared__ int4 box_sh[FP_MAX_CHUNKS];  // every chunk's box, computed once per CTA

  const int n = args.n;
  if (args.active != nullptr && args.active[s] == 0) return;
  const int a = ad / args.n_det;
  const int d = ad - a * args.n_det;

  const float* M = args.fp_matrix + 6 * a;
  const float m00 = M[0], m01 = M[1], m02 = M[2], m10 = M[3], m11 = M[4], m12 = M[5];

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int lc = lane & (FP_LC - 1);
  const int lr = lane / FP_LC;
  const int c0 = band * FP_TC;
  const int c = c0 + warp * FP_LC + lc;
  const int c_last = min(c0 + FP_TC, n) - 1;

  const float* vol = args.vol + (int64_t)s * n * n;
  const MapRef mref = make_map_ref(args.maps, MAPS_DTYPE, args.maps_slice_stride, args.n_angles, args.n_det, n, s, a,
                                   d, args.n_channels, args.chan_scale);
  const bool vec4 = args.vec4 != 0;
  const float fc = (float)c;
  const float pxc = fmaf(m00, fc, m02);
  const float pyc = fmaf(m10, fc, m12);
  constexpr bool SKIP = HAS_MAPS && MAPS_DTYPE == CCT_DTYPE_FIELDS_F32;
  // fields: three loads an item and the exponentials between them fill the pipe (9.01 ms at 1, 9.76 at
  // 2, 9.11 at 3)
  constexpr int FILL_BATCH = SKIP ? 1 : FP_FILL_BATCH;
  const float idet = SKIP ? 1.f / (m00 * m11 - m01 * m10) : 0.f;  // inverse of the rotation part
  const float i00 = m11 * idet, i01 = -m01 * idet, i10 = -m10 * idet, i11 = m00 * idet;

  // thread t computes the box of row chunk t (n <= 8192: at most FP_MAX_CHUNKS chunks)
  if (tid * FP_TR < n) {
    int4 b;
    chunk_box(m00, m01, m02, m10, m11, m12, c0, c_last, tid * FP_TR, min((tid + 1) * FP_TR, n) - 1, b.x, b.y, b.z,
              b.w);
    box_sh[tid] = b;
  }
  __syncthreads();

  float acc = 0.f;
  for (int r0 = 0; r0 < n; r0 += FP_TR) {
    const int r_last = min(r0 + FP_TR, n) - 1;
    const int4 box = box_sh[r0 / FP_TR];
    const int bx0 = box.x, bx1 = box.y, by0 = box.z, by1 = box.w;
    const int q4 = (bx1 - bx0) / 4 + 1;  // float4 columns
    const int bh = by1 - by0 + 1;
    if (4 * q4 > FP_BOX_W || bh > FP_BOX_H) {  // cannot happen for valid matrices; never trap
      if (tid == 0) atomicExch(&g_box_overflow, 1);
      return;
    }

    if (HAS_MAPS && MAPS_DTYPE != CCT_DTYPE_FIELDS_F32 && r0 + FP_TR < n) fp_prefetch_rows<MAPS_DTYPE>(mref, n, box_sh[r0 / FP_TR + 1], tid);
    // Stage z = vol * map over the box (zeros outside the image); every thread takes items
    // tid, tid + 256, ... of the q4 x bh grid, issuing FILL_BATCH items' loads at once.
    // Line-integral fields pay four expf per quad, so quads that no tap reads are left out: a tap of
    // a sample at (c, r) lies in the quad (columns gx .. gx + 3 of row gy) only if the sample's
    // position is within (2.5, 1) of (gx + 1.5, gy); taken back to lattice coordinates, the quad is
    // needed only if |c - cm| <= hc and |r - rm| <= hr (0.05 for rounding).  About half of a box's
    // quads fail at 45 degrees.  PDHG 1024x720, 4 channels: 9.39 -> 9.10 ms an iteration; with stored
    // maps the test costs more than the loads it saves (MLEM 512x720 15.8 -> 16.9 ms).
    const float cm = 0.5f * (float)(c0 + c_last), rm = 0.5f * (float)(r0 + r_last);
    const float qc0 = fmaf(i00, 1.5f - m02, -i01 * m12) - cm, qr0 = fmaf(i10, 1.5f - m02, -i11 * m12) - rm;
    const float hc = 0.5f * (float)(c_last - c0) + 2.5f * fabsf(i00) + fabsf(i01) + 0.05f;
    const float hr = 0.5f * (float)(r_last - r0) + 2.5f * fabsf(i10) + fabsf(i11) + 0.05f;
    const int items = q4 * bh;
    // it / q4 = (it * ceil(2^20 / q4)) >> 20, exact for it < 2^12 and q4 <= 25 (the error
    // it * (magic - 2^20 / q4) / 2^20 < 2^-8 stays below 1 / q4), and the product fits 32 bits
    const unsigned magic = (1048576u + (unsigned)q4 - 1u) / (unsigned)q4;
    for (int base = tid; base < items; base += FP_THREADS * FILL_BATCH) {
      float4 v[FILL_BATCH];
      int dst[FILL_BATCH];
#pragma unroll
      for (int k = 0; k < FILL_BATCH; ++k) {
        const int it = base + k * FP_THREADS;
        dst[k] = -1;
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (it < items) {
          const int rr = (int)(((unsigned)it * magic) >> 20);
          const int qq = it - rr * q4;
          const int gy = by0 + rr, gx = bx0 + 4 * qq;
          if (SKIP) {
            const float fy = (float)gy, fx = (float)gx;
            const float qc = fmaf(i00, fx, fmaf(i01, fy, qc0)), qr = fmaf(i10, fx, fmaf(i11, fy, qr0));
            if (fabsf(qc) > hc || fabsf(qr) > hr) continue;
          }
          dst[k] = rr * FP_STRIDE + 4 * qq;
          if (vec4) {
            // n % 4 == 0 and gx % 4 == 0: a float4 is either fully inside or fully outside
            if ((unsigned)gy < (unsigned)n && (unsigned)gx < (unsigned)n) {
              const int off = gy * n + gx;
              v[k] = __ldg(reinterpret_cast<const float4*>(vol + off));
              if (HAS_MAPS) {
                const float4 mv = map_at4<MAPS_DTYPE>(mref, off);
                v[k].x *= mv.x; v[k].y *= mv.y; v[k].z *= mv.z; v[k].w *= mv.w;
              }
            }
          } else {
            v[k] = fp_load_item<HAS_MAPS, MAPS_DTYPE>(vol, mref, n, gy, gx);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < FILL_BATCH; ++k) {
        if (dst[k] >= 0) *reinterpret_cast<float4*>(z + dst[k]) = v[k];
      }
    }
    __syncthreads();

    if (c <= c_last) {
      // Sample positions use exactly sample_x()'s expression so that the adjoint kernel (and
      // the box corners) see bit-identical coordinates.  Taps index the __shared__ array with
      // 32-bit offsets (zoff moves the box origin to (by0, bx0)).
      const int zoff = -by0 * FP_STRIDE - bx0;
      float fr = (float)(r0 + lr);
      const int rem = r_last - r0 - lr;                      // rows of this thread left in the chunk
      const int kmax = rem >= 0 ? rem / FP_LR + 1 : 0;       // samples of this thread in the chunk
      if (kmax >= FP_RPT) {
        // two samples (rows r and r + FP_LR) per packed FP32x2 instruction, with the roundings
        // of the scalar loop below
        const float2 mx = make_float2(m01, m01), my = make_float2(m11, m11);
        const float2 cx = make_float2(pxc, pxc), cy = make_float2(pyc, pyc);
        const float2 step2 = make_float2(2.f * FP_LR, 2.f * FP_LR);
        float2 fr2 = make_float2(fr, fr + (float)FP_LR);
#pragma unroll 4
        for (int k = 0; k < FP_RPT; k += 2) {
          acc = bilerp2<FP_STRIDE>(z, zoff, __ffma2_rn(mx, fr2, cx), __ffma2_rn(my, fr2, cy), acc);
          fr2 = __fadd2_rn(fr2, step2);
        }
      } else {
        for (int k = 0; k < kmax; ++k) {
          const FloorSplit fx = floor_split(fmaf(m01, fr, pxc));
          const FloorSplit fy = floor_split(fmaf(m11, fr, pyc));
          const int q = fy.i * FP_STRIDE + fx.i + zoff;
          const float t0 = z[q], t1 = z[q + 1], b0 = z[q + FP_STRIDE], b1 = z[q + FP_STRIDE + 1];
          const float top = fmaf(fx.f, t1 - t0, t0);
          const float bot = fmaf(fx.f, b1 - b0, b0);
          acc += fmaf(fy.f, bot - top, top);
          fr += (float)FP_LR;
        }
      }
    }
    __syncthreads();
  }

  // column sum over the 4 row-lanes of the 8x4 lane block (lanes lc, lc+8, lc+16, lc+24)
  acc += __shfl_xor_sync(0xffffffffu, acc, 8);
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);
  double part = 0.0, ptest = 0.0;
  if (lr == 0 && c <= c_last) {
    float total = acc;
    if (args.weights != nullptr) total *= args.weights[a * args.n_det + d];
    const int64_t idx = (((int64_t)s * args.n_det + d) * args.n_angles + a) * n + c;
    part = fp_epilogue<EPI>(args, idx, total, &ptest);
  }
  // only the MLEM and SIRT epilogues produce residual partials (PDHG passes none)
  if (EPI == FP_EPI_MLEM || EPI == FP_EPI_SIRT) {
    const int64_t slot = (int64_t)s * n_bands * n_ad + (int64_t)ad * n_bands + band;
    fp_write_partial(part, args.partials, slot, red_d, lane, warp, tid);
    if (args.partials_test != nullptr) fp_write_partial(ptest, args.partials_test, slot, red_d, lane, warp, tid);
  }
}

template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
__global__ void __launch_bounds__(FP_THREADS, 5) fp_kernel(FpArgs args) {
  fp_cta<EPI, HAS_MAPS, MAPS_DTYPE>(args, blockIdx.x, blockIdx.y, blockIdx.z, gridDim.x, gridDim.y);
}

// Line-integral fields: the channels of a field slice read the same two planes per angle, so
// they run as neighbouring CTAs (grid x = band * C + channel, z = field slice) and all but the
// first find the planes in L2.  Same per-CTA work as fp_kernel.
template <int EPI>
__global__ void __launch_bounds__(FP_THREADS, 5) fp_fields_kernel(FpArgs args) {
  const int C = args.n_channels;
  const int band = blockIdx.x / C;
  const int ch = blockIdx.x - band * C;
  fp_cta<EPI, true, CCT_DTYPE_FIELDS_F32>(args, band, blockIdx.y, blockIdx.z * C + ch, gridDim.x / C, gridDim.y);
}

// Group g of a ragged launch owns CTAs [start[g], start[g + 1]); binary search over the groups.
__device__ __forceinline__ int ragged_group(const int64_t* __restrict__ start, int n_groups, int64_t cta) {
  int lo = 0, hi = n_groups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(start + mid) <= cta) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Forward projection over groups of slices with different sizes, angle counts and buffers, in
// one launch: group g's CTAs are (band, angle * detector, slice) in band-fastest order.
template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
__global__ void __launch_bounds__(FP_THREADS, 5) fp_ragged_kernel(const FpArgs* __restrict__ groups,
                                                                  const int64_t* __restrict__ start, int n_groups) {
  const int64_t cta = blockIdx.x;
  const int g = ragged_group(start, n_groups, cta);
  const FpArgs& a = groups[g];
  const int n_bands = (a.n + FP_TC - 1) / FP_TC;
  const int n_ad = a.n_angles * a.n_det;
  const int64_t local = cta - start[g];
  const int band = (int)(local % n_bands);
  const int64_t rest = local / n_bands;
  const int ad = (int)(rest % n_ad);
  const int sl = (int)(rest / n_ad);
  fp_cta<EPI, HAS_MAPS, MAPS_DTYPE>(a, band, ad, sl, n_bands, n_ad);
}

// ------------------------------------------------------------------------------------------
// Forward projection, TMA-staged variant (n % 8 == 0)
//
// The chunk's x box and map box (fixed 96 x 104 boxes, zero-filled outside the image) arrive
// through two cp.async.bulk.tensor loads on one mbarrier; one vectorised pass multiplies them
// in place (z = x * map), then the same 8x4-lane sampling as fp_kernel runs on row stride 104.
// No load instruction per element, and the copy overlaps the other resident CTA's sampling.
// The left box edge is a multiple of 8 elements (16 bytes for BF16 maps too), as TMA needs.
// ------------------------------------------------------------------------------------------
constexpr int FPT_BOX_W = 104;
constexpr int FPT_BOX_H = 96;
constexpr int FPT_Q4 = FPT_BOX_W / 4;              // float4 per box row
constexpr uint32_t FPT_WAIT_LIMIT = 1u << 22;      // bounded mbarrier polling (never spins forever)

__device__ int g_tma_timeout = 0;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t phase) {
  for (uint32_t it = 0; it < FPT_WAIT_LIMIT; ++it) {
    if (mbar_try_wait(bar, phase)) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
__global__ void __launch_bounds__(FP_THREADS, 2)
    fp_tma_kernel(FpArgs args, const __grid_constant__ CUtensorMap tm_vol, const __grid_constant__ CUtensorMap tm_maps) {
  extern __shared__ __align__(128) unsigned char fpt_smem[];
  float* zb = reinterpret_cast<float*>(fpt_smem);                                  // [96][104] x, then z
  unsigned char* mraw = fpt_smem + FPT_BOX_H * FPT_BOX_W * sizeof(float);         // [96][104] map
  __shared__ __align__(8) uint64_t bar;
  __shared__ double red_d[FP_TC / FP_LC];
  __shared__ int timed_out;

  const int n = args.n;
  const int band = blockIdx.x;
  const int ad = blockIdx.y;
  const int s = blockIdx.z;
  if (args.active != nullptr && args.active[s] == 0) return;
  const int a = ad / args.n_det;
  const int d = ad - a * args.n_det;

  const float* M = args.fp_matrix + 6 * a;
  const float m00 = M[0], m01 = M[1], m02 = M[2], m10 = M[3], m11 = M[4], m12 = M[5];

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int lc = lane & (FP_LC - 1);
  const int lr = lane / FP_LC;
  const int c0 = band * FP_TC;
  const int c = c0 + warp * FP_LC + lc;
  const int c_last = min(c0 + FP_TC, n) - 1;
  const int map_img = (s * args.n_angles + a) * args.n_det + d;
  const uint32_t box_bytes = FPT_BOX_H * FPT_BOX_W * sizeof(float) +
                             (HAS_MAPS ? FPT_BOX_H * FPT_BOX_W * (MAPS_DTYPE == CCT_DTYPE_BF16 ? 2 : 4) : 0);
  const float fc = (float)c;
  const float pxc = fmaf(m00, fc, m02);
  const float pyc = fmaf(m10, fc, m12);

  if (tid == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    timed_out = 0;
  }
  __syncthreads();

  uint32_t phase = 0;
  float acc = 0.f;
  for (int r0 = 0; r0 < n; r0 += FP_TR) {
    const int r_last = min(r0 + FP_TR, n) - 1;
    const float fc0 = (float)c0, fc1 = (float)c_last, fr0 = (float)r0, fr1 = (float)r_last;
    const float xa = sample_x(m00, m01, m02, fc0, fr0), xb = sample_x(m00, m01, m02, fc1, fr0);
    const float xc = sample_x(m00, m01, m02, fc0, fr1), xd = sample_x(m00, m01, m02, fc1, fr1);
    const float ya = sample_x(m10, m11, m12, fc0, fr0), yb = sample_x(m10, m11, m12, fc1, fr0);
    const float yc = sample_x(m10, m11, m12, fc0, fr1), yd = sample_x(m10, m11, m12, fc1, fr1);
    const float xmin = fminf(fminf(xa, xb), fminf(xc, xd)), xmax = fmaxf(fmaxf(xa, xb), fmaxf(xc, xd));
    const float ymin = fminf(fminf(ya, yb), fminf(yc, yd)), ymax = fmaxf(fmaxf(ya, yb), fmaxf(yc, yd));
    const int bx0 = ((int)floorf(xmin) - 1) & ~7;  // 16-byte aligned TMA x coordinate (BF16 too)
    const int bx1 = (int)floorf(xmax) + 2;
    const int by0 = (int)floorf(ymin) - 1;
    const int by1 = (int)floorf(ymax) + 2;
    const int wq = (bx1 - bx0) / 4 + 1;  // float4 columns used
    const int bh = by1 - by0 + 1;
    if (4 * wq > FPT_BOX_W || bh > FPT_BOX_H) {  // cannot happen for valid matrices; never trap
      if (tid == 0) atomicExch(&g_box_overflow, 1);
      return;
    }

    if (tid == 0) {
      mbar_expect_tx(&bar, box_bytes);
      tma_load_3d(zb, &tm_vol, bx0, by0, s, &bar);
      if (HAS_MAPS) tma_load_3d(mraw, &tm_maps, bx0, by0, map_img, &bar);
    }
    // every thread observes the phase flip itself (acquire of the bulk-copy writes)
    if (!mbar_wait_bounded(&bar, phase)) timed_out = 1;
    __syncthreads();
    if (timed_out) {
      // give the copies in flight one more bounded wait, then leave without touching smem
      if (tid == 0) {
        atomicExch(&g_tma_timeout, 1);
        mbar_wait_bounded(&bar, phase);
      }
      return;
    }
    phase ^= 1u;

    if (HAS_MAPS) {
      float4* z4 = reinterpret_cast<float4*>(zb);
      for (int it = tid; it < bh * FPT_Q4; it += FP_THREADS) {
        const int rr = it / FPT_Q4;
        const int qq = it - rr * FPT_Q4;
        if (qq < wq) {
          float4 v = z4[it];
          if (MAPS_DTYPE == CCT_DTYPE_BF16) {
            const uint2 raw = reinterpret_cast<const uint2*>(mraw)[it];
            const float2 flo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
            const float2 fhi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
            v.x *= flo.x; v.y *= flo.y; v.z *= fhi.x; v.w *= fhi.y;
          } else {
            const float4 mv = reinterpret_cast<const float4*>(mraw)[it];
            v.x *= mv.x; v.y *= mv.y; v.z *= mv.z; v.w *= mv.w;
          }
          z4[it] = v;
        }
      }
      __syncthreads();
    }

    if (c <= c_last) {
      const int zoff = -by0 * FPT_BOX_W - bx0;
      float fr = (float)(r0 + lr);
      const int rem = r_last - r0 - lr;
      const int kmax = rem >= 0 ? rem / FP_LR + 1 : 0;
      if (kmax >= FP_RPT) {
        const float2 mx = make_float2(m01, m01), my = make_float2(m11, m11);
        const float2 cx = make_float2(pxc, pxc), cy = make_float2(pyc, pyc);
        const float2 step2 = make_float2(2.f * FP_LR, 2.f * FP_LR);
        float2 fr2 = make_float2(fr, fr + (float)FP_LR);
#pragma unroll 4
        for (int k = 0; k < FP_RPT; k += 2) {
          acc = bilerp2<FPT_BOX_W>(zb, zoff, __ffma2_rn(mx, fr2, cx), __ffma2_rn(my, fr2, cy), acc);
          fr2 = __fadd2_rn(fr2, step2);
        }
      } else {
        for (int k = 0; k < kmax; ++k) {
          const FloorSplit fx = floor_split(fmaf(m01, fr, pxc));
          const FloorSplit fy = floor_split(fmaf(m11, fr, pyc));
          const int q = fy.i * FPT_BOX_W + fx.i + zoff;
          const float t0 = zb[q], t1 = zb[q + 1], b0 = zb[q + FPT_BOX_W], b1 = zb[q + FPT_BOX_W + 1];
          const float top = fmaf(fx.f, t1 - t0, t0);
          const float bot = fmaf(fx.f, b1 - b0, b0);
          acc += fmaf(fy.f, bot - top, top);
          fr += (float)FP_LR;
        }
      }
    }
    __syncthreads();
    // generic-proxy writes/reads of the boxes are done; order them before the next bulk copy
    if (tid == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }

  acc += __shfl_xor_sync(0xffffffffu, acc, 8);
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);
  double part = 0.0, ptest = 0.0;
  if (lr == 0 && c <= c_last) {
    float total = acc;
    if (args.weights != nullptr) total *= args.weights[a * args.n_det + d];
    const int64_t idx = (((int64_t)s * args.n_det + d) * args.n_angles + a) * n + c;
    part = fp_epilogue<EPI>(args, idx, total, &ptest);
  }
  if (EPI == FP_EPI_MLEM || EPI == FP_EPI_SIRT) {
    const int64_t slot = (int64_t)s * gridDim.x * gridDim.y + (int64_t)blockIdx.y * gridDim.x + blockIdx.x;
    fp_write_partial(part, args.partials, slot, red_d, lane, warp, tid);
    if (args.partials_test != nullptr) fp_write_partial(ptest, args.partials_test, slot, red_d, lane, warp, tid);
  }
}

// ------------------------------------------------------------------------------------------
// Forward projection, two slices per CTA
//
// All slices of a batch share the angle's sample positions, so one CTA owns (band, angle *
// detector, pair of slices): it computes each sample's coordinates and tap offsets once, stages
// z = x * map of both slices interleaved (one float2 element per pixel) and reads every
// bilinear tap of both with one 8-byte shared load.  The arithmetic per sample and slice is
// fp_cta's (bit-identical results).  Chunks are 64 columns x 32 rows so that three CTAs fit per
// SM; like fp_cta, only the quads of each box row that the taps read are staged, and the row
// stride (80 + 2v elements, v in 0..4, even so that 16-byte stores stay aligned) is chosen per angle on
// the host (column 1 of cct_xrf_desc::fp_box_strides).  The fill loads float4 quads of both
// slices, and writes a quad as two 16-byte element pairs; lanes 4-7 of every 8-lane store phase
// write their second pair first, which keeps the 16-byte stores of a phase on distinct banks.
// Four CTAs fit per SM (64 registers, < 56 KB of shared memory each).
// ------------------------------------------------------------------------------------------
constexpr int FP2_TR = 32;                          // rows per staged chunk
constexpr int FP2_RPT = FP2_TR / FP_LR;             // 8 samples per thread per chunk
// 64 x 32 chunk rotated: x extent <= sqrt(63^2 + 31^2) = 70.2 (+ 11 for taps, margins and the
// float4-aligned origin) -> 80; y extent 70.2 + 5 -> 75 rows.
constexpr int FP2_BOX_W = 80;
constexpr int FP2_BOX_H = 75;
constexpr int FP2_STRIDE_MAX = FP2_BOX_W + 8;       // strides 80, 82, ..., 88 elements
constexpr int FP2_MAX_CHUNKS = (8192 + FP2_TR - 1) / FP2_TR;
static_assert(FP2_MAX_CHUNKS <= FP_THREADS, "one thread per chunk box");
constexpr int FP2_FILL_BATCH = 2;
constexpr size_t FP2_SMEM_BYTES = (size_t)FP2_STRIDE_MAX * FP2_BOX_H * sizeof(float2);

template <bool HAS_MAPS, int MAPS_DTYPE>
__device__ __forceinline__ float4 fp2_quad(const float* vol, const MapRef& mref, int n, int gy, int gx, bool vec4,
                                           bool ok) {
  if (!ok) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec4) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((unsigned)gy < (unsigned)n && (unsigned)gx < (unsigned)n) {
      const int off = gy * n + gx;
      v = __ldg(reinterpret_cast<const float4*>(vol + off));
      if (HAS_MAPS) {
        const float4 mv = map_at4<MAPS_DTYPE>(mref, off);
        v.x *= mv.x; v.y *= mv.y; v.z *= mv.z; v.w *= mv.w;
      }
    }
    return v;
  }
  return fp_load_item<HAS_MAPS, MAPS_DTYPE>(vol, mref, n, gy, gx);
}

template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
__global__ void __launch_bounds__(FP_THREADS, 4) fp_pair_kernel(FpArgs args) {
  extern __shared__ __align__(16) float2 z2[];  // [FP2_BOX_H][stride] elements (slice 0, slice 1)
  __shared__ double red_d[FP_TC / FP_LC];
  __shared__ short4 box_sh[FP2_MAX_CHUNKS];  // (bx0, by0, quads, rows) of every chunk's box
  __shared__ short2 quads_sh[FP2_BOX_H];

  const int n = args.n;
  const int band = blockIdx.x;
  const int ad = blockIdx.y;
  const int s0 = 2 * blockIdx.z;
  bool ok[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int s = s0 + g;
    ok[g] = s < args.n_slices && (args.active == nullptr || args.active[s] != 0);
  }
  if (!ok[0] && !ok[1]) return;  // the whole CTA
  const int a = ad / args.n_det;
  const int d = ad - a * args.n_det;

  const float* M = args.fp_matrix + 6 * a;
  const float m00 = M[0], m01 = M[1], m02 = M[2], m10 = M[3], m11 = M[4], m12 = M[5];
  const int sel = args.box_strides != nullptr ? min(max(args.box_strides[2 * a + 1], 0), 4) : 0;
  const int S = FP2_BOX_W + 2 * sel;  // row stride (elements), even

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int lc = lane & (FP_LC - 1);
  const int lr = lane / FP_LC;
  const int c0 = band * FP_TC;
  const int c = c0 + warp * FP_LC + lc;
  const int c_last = min(c0 + FP_TC, n) - 1;
  const bool vec4 = args.vec4 != 0;
  const bool swap = (lane & 4) != 0;  // lanes 4-7 of each store phase write their second pair first

  const float* vol[2];
  MapRef mref[2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int s = ok[g] ? s0 + g : s0 + (ok[0] ? 0 : 1);
    vol[g] = args.vol + (int64_t)s * n * n;
    mref[g] = make_map_ref(args.maps, MAPS_DTYPE, args.maps_slice_stride, args.n_angles, args.n_det, n, s, a, d,
                           args.n_channels, args.chan_scale);
  }
  const float fc = (float)c;
  const float pxc = fmaf(m00, fc, m02);
  const float pyc = fmaf(m10, fc, m12);

  // box coordinates fit 16 bits: |x|, |y| < 1.5 n + 3 for n <= 8192
  if (tid * FP2_TR < n) {
    int bx0, bx1, by0, by1;
    chunk_box(m00, m01, m02, m10, m11, m12, c0, c_last, tid * FP2_TR, min((tid + 1) * FP2_TR, n) - 1, bx0, bx1, by0,
              by1);
    box_sh[tid] = make_short4((short)bx0, (short)by0, (short)((bx1 - bx0) / 4 + 1), (short)(by1 - by0 + 1));
  }
  __syncthreads();
  {
    const short4 b0 = box_sh[0];
    if (tid < b0.w && tid < FP2_BOX_H) {
      float px[4], py[4];
      chunk_corners(m00, m01, m02, m10, m11, m12, c0, c_last, 0, min(FP2_TR, n) - 1, px, py);
      quads_sh[tid] = fp_row_quads(px, py, b0.y + tid, b0.x, b0.z);
    }
  }
  __syncthreads();

  float acc0 = 0.f, acc1 = 0.f;
  for (int r0 = 0; r0 < n; r0 += FP2_TR) {
    const int r_last = min(r0 + FP2_TR, n) - 1;
    const short4 box = box_sh[r0 / FP2_TR];
    const int bx0 = box.x, by0 = box.y, q4 = box.z, bh = box.w;
    if (4 * q4 > FP2_BOX_W || bh > FP2_BOX_H) {  // cannot happen for valid matrices; never trap
      if (tid == 0) atomicExch(&g_box_overflow, 1);
      return;
    }

    const int items = q4 * bh;
    const unsigned magic = (1048576u + (unsigned)q4 - 1u) / (unsigned)q4;  // it / q4 as in fp_cta
    for (int base = tid; base < items; base += FP_THREADS * FP2_FILL_BATCH) {
      float4 v0[FP2_FILL_BATCH], v1[FP2_FILL_BATCH];
      int dst[FP2_FILL_BATCH];
#pragma unroll
      for (int k = 0; k < FP2_FILL_BATCH; ++k) {
        const int it = base + k * FP_THREADS;
        dst[k] = -1;
        v0[k] = v1[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (it < items) {
          const int rr = (int)(((unsigned)it * magic) >> 20);
          const int qq = it - rr * q4;
          const short2 qr = quads_sh[rr];
          if (qq >= qr.x && qq <= qr.y) {
            const int gy = by0 + rr, gx = bx0 + 4 * qq;
            dst[k] = rr * S + 4 * qq;
            v0[k] = fp2_quad<HAS_MAPS, MAPS_DTYPE>(vol[0], mref[0], n, gy, gx, vec4, ok[0]);
            v1[k] = fp2_quad<HAS_MAPS, MAPS_DTYPE>(vol[1], mref[1], n, gy, gx, vec4, ok[1]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < FP2_FILL_BATCH; ++k) {
        if (dst[k] >= 0) {
          // elements 4q, 4q + 1 (lo) and 4q + 2, 4q + 3 (hi); the order of the two stores is
          // selected per lane so that both store instructions run with every lane active
          const float4 lo = make_float4(v0[k].x, v1[k].x, v0[k].y, v1[k].y);
          const float4 hi = make_float4(v0[k].z, v1[k].z, v0[k].w, v1[k].w);
          float4* q = reinterpret_cast<float4*>(z2 + dst[k]);
          const int f = swap ? 1 : 0;
          q[f] = swap ? hi : lo;
          q[1 - f] = swap ? lo : hi;
        }
      }
    }
    __syncthreads();

    if (r0 + FP2_TR < n) {
      const short4 nb = box_sh[r0 / FP2_TR + 1];
      if (tid < nb.w && tid < FP2_BOX_H) {
        float px[4], py[4];
        chunk_corners(m00, m01, m02, m10, m11, m12, c0, c_last, r0 + FP2_TR, min(r0 + 2 * FP2_TR, n) - 1, px, py);
        quads_sh[tid] = fp_row_quads(px, py, nb.y + tid, nb.x, nb.z);
      }
    }

    if (c <= c_last) {
      const int zoff = -by0 * S - bx0;
      float fr = (float)(r0 + lr);
      const int rem = r_last - r0 - lr;
      const int kmax = rem >= 0 ? rem / FP_LR + 1 : 0;
      if (kmax >= FP2_RPT) {
        // both slices' lerps in packed FP32x2 arithmetic, rounding like the scalar loop below
        // (a - b as fma(b, -1, a))
        const float2 neg1 = make_float2(-1.f, -1.f);
        float2 acc2 = make_float2(acc0, acc1);
#pragma unroll 4
        for (int k = 0; k < FP2_RPT; ++k) {
          const FloorSplit fx = floor_split(fmaf(m01, fr, pxc));
          const FloorSplit fy = floor_split(fmaf(m11, fr, pyc));
          const int q = fy.i * S + fx.i + zoff;
          const float2 t0 = z2[q], t1 = z2[q + 1], b0 = z2[q + S], b1 = z2[q + S + 1];
          const float2 fxx = make_float2(fx.f, fx.f), fyy = make_float2(fy.f, fy.f);
          const float2 top = __ffma2_rn(fxx, __ffma2_rn(t0, neg1, t1), t0);
          const float2 bot = __ffma2_rn(fxx, __ffma2_rn(b0, neg1, b1), b0);
          acc2 = __fadd2_rn(acc2, __ffma2_rn(fyy, __ffma2_rn(top, neg1, bot), top));
          fr += (float)FP_LR;
        }
        acc0 = acc2.x;
        acc1 = acc2.y;
      } else {
        for (int k = 0; k < kmax; ++k) {
          const FloorSplit fx = floor_split(fmaf(m01, fr, pxc));
          const FloorSplit fy = floor_split(fmaf(m11, fr, pyc));
          const int q = fy.i * S + fx.i + zoff;
          const float2 t0 = z2[q], t1 = z2[q + 1], b0 = z2[q + S], b1 = z2[q + S + 1];
          const float top0 = fmaf(fx.f, t1.x - t0.x, t0.x), bot0 = fmaf(fx.f, b1.x - b0.x, b0.x);
          const float top1 = fmaf(fx.f, t1.y - t0.y, t0.y), bot1 = fmaf(fx.f, b1.y - b0.y, b0.y);
          acc0 += fmaf(fy.f, bot0 - top0, top0);
          acc1 += fmaf(fy.f, bot1 - top1, top1);
          fr += (float)FP_LR;
        }
      }
    }
    __syncthreads();
  }

  const int n_bands = gridDim.x;
  const int n_ad = gridDim.y;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    if (!ok[g]) continue;  // uniform across the CTA
    const int s = s0 + g;
    float col = g == 0 ? acc0 : acc1;
    col += __shfl_xor_sync(0xffffffffu, col, 8);
    col += __shfl_xor_sync(0xffffffffu, col, 16);
    double part = 0.0, ptest = 0.0;
    if (lr == 0 && c <= c_last) {
      float total = col;
      if (args.weights != nullptr) total *= args.weights[a * args.n_det + d];
      const int64_t idx = (((int64_t)s * args.n_det + d) * args.n_angles + a) * n + c;
      part = fp_epilogue<EPI>(args, idx, total, &ptest);
    }
    if (EPI == FP_EPI_MLEM || EPI == FP_EPI_SIRT) {
      const int64_t slot = (int64_t)s * n_bands * n_ad + (int64_t)ad * n_bands + band;
      fp_write_partial(part, args.partials, slot, red_d, lane, warp, tid);
      if (args.partials_test != nullptr) fp_write_partial(ptest, args.partials_test, slot, red_d, lane, warp, tid);
    }
  }
}

// ------------------------------------------------------------------------------------------
// Back projection (reference iradon discretisation, optional maps x weights)
//
// A CTA owns a 32-column tile of TI = 32 or 64 rows (bp_tile_rows); a warp holds TI / 8 whole rows of it.
//
// Bound: an 8-byte lookup is two shared-memory wavefronts whatever the lanes' pixels (0.40 ms of
// them for 8 slices of 512^2 x 720), next the ~8 instructions per pixel and line.  What else
// the time went on was the rare case: the FP64 edge decision, inlined per pixel or called, cost
// registers and branches on every line (1.20 ms with the call, 0.99 ms with no edge at all, 1.13 ms
// as below, for 16 slices), and the three barriers per chunk of lines.  Measured on 512^2 x 720
// (before -> now): 1 slice 281 -> 99 us, 8 slices 880 -> 621 us, 16 slices 1519 -> 1134 us; 256^2 x
// 360 161 -> 23 us, 128^2 x 180 77 -> 11 us; with maps (512^2 x 360, 2 slices) 1577 -> 278 us.  (Values at
// the edges in FP64 cost four spilled registers where one CTA walks all segments: 8 slices 600 us without.)
//
// The lines are summed in up to eight fixed segments, whose sums are added in order (which also
// shortens the FP32 sums: the error against FP64 falls from 3.9e-7 to 1e-7 at 722 lines).  One CTA
// walks all of them, or, where the batch has few tiles, the CTAs of a cluster take one each and
// combine them through distributed shared memory; both give the same bits.
// ------------------------------------------------------------------------------------------
constexpr int BP_TJ = 32;                                // tile columns
constexpr int BP_BLOCK_ROWS = 64;                        // rows of the blocks whose bins are staged
constexpr int BP_MAX_RANKS = 8;                          // CTAs of a cluster, at most, and in a ragged launch
constexpr int BP_THREADS = 256;
constexpr int BP_LINES = 16;                             // lines staged per chunk
constexpr int BP_KW = 80;                                // staged pairs per line (>= 74 needed)
constexpr float BP_EDGE_GUARD = 0.01f;

enum : int { LINE_FAST = 0, LINE_CHECKED = 1, LINE_EMPTY = 2 };

// Tiles of a slice with tiles of `rows` rows.
__host__ __device__ inline int bp_tiles(int n, int rows) {
  return ((n + BP_TJ - 1) / BP_TJ) * ((n + rows - 1) / rows);
}
// log2 of the segments of the line sum (at least eight lines each); segment g of n_lines <= 65535
// lines starts at (g * n_lines) >> log2.
__host__ __device__ inline int bp_log2_segments(int n_lines) {
  return n_lines >= 64 ? 3 : n_lines >= 32 ? 2 : n_lines >= 16 ? 1 : 0;
}

__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();  // .aligned takes whole warps, also after stores that depend on the pixel
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The float at shared address p of this CTA's layout in CTA `rank` of the cluster.
__device__ __forceinline__ float cluster_load(const float* p, int rank) {
  uint32_t a;
  float v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

struct __align__(16) BpLine {
  float cs, sn, off;      // cos, sin, K - kbase
  int kind;
  float mid, half;        // centre and half length of the detector in bins from kbase
  float w;                // weight of the line
  int kbase;
};

struct BpShared {
  float2 pairs[2][BP_LINES][BP_KW];  // chunk being looked up, chunk being staged
  BpLine line[3][BP_LINES];          // and the chunk after those
};

// np.interp(t, k - K, line, left=0, right=0) for a pixel (jc, ic from the centre) whose FP32 position
// is within BP_EDGE_GUARD of a detector edge.  numpy decides the edge on t = jc cos - ic sin in
// double, where both products are exact; here the distance d past the edge is formed from the
// products' FP32 halves, the exact error of their difference and a difference with the edge that
// is exact too (Sterbenz), so that only the sum of the errors rounds: at |d| < 0.02 by less than 1e-11, with
// the sign of a d that is exactly 0 (angles of 0 and 90 degrees) intact.  The value is interpolated in
// FP64.  A pixel on the edge itself takes the
// edge bin as it is, like np.interp: the pair of bins n - 2 and n - 1 gives the latter only to the
// rounding of their difference (0 for 3e7 and 0.5).  bins points at the staged pair of bin 0, line at the
// unstaged bins and w is their weight.
__device__ __forceinline__ float bp_edge_value(const float2* bins, const float* line, float w, float cs, float sn, int n,
                                               float jc, float ic) {
  const int K = n / 2;
  const float p = jc * cs, pe = fmaf(jc, cs, -p);
  const float q = -ic * sn, qe = fmaf(-ic, sn, -q);
  const float s = p + q, b = s - p;
  const float se = (p - (s - b)) + (q - b);  // p + q = s + se exactly
  const bool left = s < -0.5f;
  const double d = (double)(s + (left ? (float)K : -(float)(n - 1 - K))) + (double)(se + (pe + qe));
  if (left ? d < 0.0 : d > 0.0) return 0.f;
  if (!left && d == 0.0) return w * __ldg(line + (n - 1));
  const float2 v = bins[left ? 0 : n - 2];
  if (d == 0.0) return v.x;
  return (float)fma(left ? d : 1.0 + d, (double)v.y, (double)v.x);
}

// Values of a staged line at two positions (bins from kbase), in packed FP32x2 arithmetic that rounds
// like floor_split; `row` is the byte offset of the line's bin 0 in pairs, less the exponent bits
// of the floors.
__device__ __forceinline__ float2 bp_lerp2(const float2 (*pairs)[BP_KW], unsigned row, float2 u) {
  const float2 magic = make_float2(12582912.0f, 12582912.0f);  // 1.5 * 2^23, see floor_split
  const float2 nmagic = make_float2(-12582912.0f, -12582912.0f);
  const float2 t = __fadd2_rd(u, magic);
  const float2 f = __ffma2_rn(__fadd2_rn(t, nmagic), make_float2(-1.f, -1.f), u);  // u - floor(u), exact
  const char* base = reinterpret_cast<const char*>(pairs);
  const float2 p0 = *reinterpret_cast<const float2*>(base + ((__float_as_uint(t.x) << 3) + row));
  const float2 p1 = *reinterpret_cast<const float2*>(base + ((__float_as_uint(t.y) << 3) + row));
  return make_float2(fmaf(f.x, p0.y, p0.x), fmaf(f.y, p1.y, p1.x));
}

// Sum of lines [l0, l1) at the PPT pixels (rows i0 + k, column j) of this thread; ti0, tj0 is the
// tile's first row and column.  ONE: all lines are one chunk and nothing is fetched ahead, which with few lines
// is most of a CTA's instructions (512^2, 64 slices: 1 line 45 -> 37 us, 4 lines 64 -> 56, 12 lines 103 -> 97).
template <bool SYM, int MAPS_DTYPE, int PPT, bool ONE>
__device__ __forceinline__ void bp_segment(const BpArgs& args, BpShared& sh, int s, int ti0, int tj0, int i0, int j,
                                           int l0, int l1, float (&acc)[PPT]) {
  static_assert(PPT % 2 == 0 && BP_LINES <= 32, "pixels go in pairs, lines in one mask");
  const int n = args.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = n / 2;  // detector offset (img_shape // 2) and output radius (output_size // 2)
  const float* sino = args.sino + (int64_t)s * args.n_det * args.n_angles * n;
  const float fj = (float)(j - K);
  float2 nfi[PPT / 2];
  int pix[PPT];  // SYM: map offsets of the pixels (clamped into the image)
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const float v = -(float)(i0 + k - K);
    if (k & 1) nfi[k / 2].y = v; else nfi[k / 2].x = v;
    if (SYM) pix[k] = min(i0 + k, n - 1) * n + min(j, n - 1);
    acc[k] = 0.f;
  }
  // centre of the warp's pixels
  const float wj = (float)(tj0 - K) + 0.5f * (float)(BP_TJ - 1);
  const float wi = -((float)(i0 - K) + 0.5f * (float)(PPT - 1));

  // While chunk c is looked up, the lines of chunk c + 2 are described (one warp, a lane per line) and
  // those of chunk c + 1 loaded, to be written as pairs at its end: one barrier per chunk.
  constexpr int PER_WARP = BP_LINES / (BP_THREADS / 32);
  float held[PER_WARP][3];
  auto describe = [&](int lc, int ll, int slot) {
    const int l = lc + ll;
    if (l >= l1) return;
    const int d = l / args.n_angles;
    const int a = l - d * args.n_angles;
    // full tile (also pixels beyond n, which are computed and discarded) so every thread's lookup
    // stays inside the staged range: t = (j - K) cos - (i - K) sin at the four corners (of the block of 64
    // rows, whatever the tile's: a pixel's bin is rounded from there, and so the same in both)
    const int b0 = ti0 & ~(BP_BLOCK_ROWS - 1);
    const float cj0 = (float)(tj0 - K), cj1 = (float)(tj0 + BP_TJ - 1 - K);
    const float ci0 = (float)(b0 - K), ci1 = (float)(b0 + BP_BLOCK_ROWS - 1 - K);
    BpLine li;
    li.cs = args.bp_trig[2 * a];
    li.sn = args.bp_trig[2 * a + 1];
    const float t00 = fmaf(cj0, li.cs, -ci0 * li.sn), t01 = fmaf(cj1, li.cs, -ci0 * li.sn);
    const float t10 = fmaf(cj0, li.cs, -ci1 * li.sn), t11 = fmaf(cj1, li.cs, -ci1 * li.sn);
    const float tmin = fminf(fminf(t00, t01), fminf(t10, t11));
    const float tmax = fmaxf(fmaxf(t00, t01), fmaxf(t10, t11));
    const float t_left = (float)(-K), t_right = (float)(n - 1 - K);
    li.kind = LINE_FAST;
    if (tmax < t_left - BP_EDGE_GUARD || tmin > t_right + BP_EDGE_GUARD) {
      li.kind = LINE_EMPTY;
    } else if (tmin < t_left + BP_EDGE_GUARD || tmax > t_right - BP_EDGE_GUARD) {
      li.kind = LINE_CHECKED;
    }
    li.kbase = (int)floorf(tmin + (float)K) - 1;
    li.off = (float)(K - li.kbase);
    li.w = 1.f;
    if (SYM && args.weights != nullptr) li.w = args.weights[a * args.n_det + d];
    if (!SYM && args.line_scale != nullptr) li.w = args.line_scale[a];
    li.half = 0.5f * (float)(n - 1);
    li.mid = li.half - (float)li.kbase;
    sh.line[slot][ll] = li;
  };
  // A warp loads and writes lines warp, warp + 8, ... of a chunk.
  auto load_chunk = [&](int lc, int slot) {
#pragma unroll
    for (int p = 0; p < PER_WARP; ++p) {
      const int ll = warp + (BP_THREADS / 32) * p;
      if (lc + ll >= l1) break;
      const int kk = sh.line[slot][ll].kind != LINE_EMPTY ? sh.line[slot][ll].kbase + lane : n;
      const float* line = sino + (int64_t)(lc + ll) * n;
#pragma unroll
      for (int q = 0; q < 3; ++q) held[p][q] = (unsigned)(kk + 32 * q) < (unsigned)n ? __ldg(line + kk + 32 * q) : 0.f;
    }
  };
  // (value, slope) pairs, zero outside [0, n - 1)
  auto store_chunk = [&](int lc, int slot, int buf) {
#pragma unroll
    for (int p = 0; p < PER_WARP; ++p) {
      const int ll = warp + (BP_THREADS / 32) * p;
      if (lc + ll >= l1) break;
      const int kbase = sh.line[slot][ll].kbase;
      const float w = sh.line[slot][ll].w;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        float vn = __shfl_down_sync(0xffffffffu, held[p][q], 1);
        const float v32 = q < 2 ? __shfl_sync(0xffffffffu, held[p][q < 2 ? q + 1 : q], 0) : 0.f;
        if (lane == 31) vn = v32;
        const int b = lane + 32 * q;
        const bool in = (unsigned)(kbase + b) < (unsigned)(n - 1);
        if (b < BP_KW) sh.pairs[buf][ll][b] = in ? make_float2(w * held[p][q], w * (vn - held[p][q])) : make_float2(0.f, 0.f);
      }
    }
  };

  // (the previous segment's last barrier is behind every thread)
  if (lane < PER_WARP) describe(l0, warp + (BP_THREADS / 32) * lane, 0);
  if (!ONE && warp == BP_THREADS / 32 - 1 && lane < BP_LINES) describe(l0 + BP_LINES, lane, 1);
  __syncwarp();
  load_chunk(l0, 0);
  store_chunk(l0, 0, 0);
  __syncthreads();
  int slot = 0, buf = 0;
  for (int lc = l0, c = 0; lc < l1; lc += BP_LINES, buf ^= 1, ++c) {
    const int count = min(BP_LINES, l1 - lc);
    const bool more = !ONE && lc + BP_LINES < l1;
    const int next = slot == 2 ? 0 : slot + 1;
    if (!ONE && warp == (c & 7) && lane < BP_LINES) describe(lc + 2 * BP_LINES, lane, next == 2 ? 0 : next + 1);
    if (!SYM && more) load_chunk(lc + BP_LINES, next);  // SYM keeps the registers for its maps
    const float2 (*pairs)[BP_KW] = sh.pairs[buf];
    const BpLine* lines = sh.line[slot];
    unsigned near_edge = 0u;  // lines of the chunk with a pixel of this thread at a detector edge
    for (int ll = 0; ll < count; ++ll) {
      const float4 li = *reinterpret_cast<const float4*>(&lines[ll]);
      const int kind = __float_as_int(li.w);
      if (kind == LINE_EMPTY) continue;
      bool edge = false;
      if (kind == LINE_CHECKED) {
        // does a detector edge cross this warp's 32 x PPT pixels?
        const float uc = fmaf(wi, li.y, fmaf(wj, li.x, li.z));
        const float reach =
            fmaf(0.5f * (float)(BP_TJ - 1), fabsf(li.x), 0.5f * (float)(PPT - 1) * fabsf(li.y)) + 2.f * BP_EDGE_GUARD;
        edge = fabsf(fabsf(uc - lines[ll].mid) - lines[ll].half) < reach;
      }
      const float base = fmaf(fj, li.x, li.z);
      const float2 base2 = make_float2(base, base), sn2 = make_float2(li.y, li.y);
      // byte offset of the line's bin 0, less the exponent bits of the floors
      const unsigned row = (unsigned)ll * (unsigned)sizeof(sh.pairs[0][0]) - (0x4B400000u << 3);
      float m[PPT];
      if (SYM) {
        const int l = lc + ll;
        const int d = l / args.n_angles;
        const MapRef mr = make_map_ref(args.maps, MAPS_DTYPE, args.maps_slice_stride, args.n_angles, args.n_det, n, s,
                                       l - d * args.n_angles, d, args.n_channels, args.chan_scale);
#pragma unroll
        for (int k = 0; k < PPT; ++k) m[k] = map_at<MAPS_DTYPE>(mr, pix[k]);
      }
      if (!edge) {
#pragma unroll
        for (int k = 0; k < PPT; k += 2) {
          const float2 r = bp_lerp2(pairs, row, __ffma2_rn(nfi[k / 2], sn2, base2));
          acc[k] = SYM ? acc[k] + r.x * m[k] : acc[k] + r.x;
          acc[k + 1] = SYM ? acc[k + 1] + r.y * m[k + 1] : acc[k + 1] + r.y;
        }
      } else {
        // np.interp's left = right = 0 make the detector edges discontinuous; the FP32 position is
        // within ~1e-4 of its exact value, so only pixels this close to an edge need more: they are
        // left out here and added after the chunk
        const float mid = lines[ll].mid, half = lines[ll].half;
        bool any = false;
#pragma unroll
        for (int k = 0; k < PPT; k += 2) {
          const float2 u = __ffma2_rn(nfi[k / 2], sn2, base2);
          const float2 r = bp_lerp2(pairs, row, u);
          const bool e0 = fabsf(fabsf(u.x - mid) - half) < BP_EDGE_GUARD;
          const bool e1 = fabsf(fabsf(u.y - mid) - half) < BP_EDGE_GUARD;
          any = any || e0 || e1;
          if (!e0) acc[k] = SYM ? acc[k] + r.x * m[k] : acc[k] + r.x;
          if (!e1) acc[k + 1] = SYM ? acc[k + 1] + r.y * m[k + 1] : acc[k + 1] + r.y;
        }
        if (any) near_edge |= 1u << ll;
      }
    }
    for (; near_edge != 0u; near_edge &= near_edge - 1u) {
      const int ll = __ffs(near_edge) - 1;
      const BpLine li = lines[ll];
      const float base = fmaf(fj, li.cs, li.off);
#pragma unroll
      for (int k = 0; k < PPT; ++k) {
        const float u = fmaf(k & 1 ? nfi[k / 2].y : nfi[k / 2].x, li.sn, base);
        if (fabsf(fabsf(u - li.mid) - li.half) >= BP_EDGE_GUARD) continue;
        float v = bp_edge_value(pairs[ll] - li.kbase, sino + (int64_t)(lc + ll) * n, li.w, li.cs, li.sn, n, fj,
                                -(k & 1 ? nfi[k / 2].y : nfi[k / 2].x));
        if (SYM) {
          const int l = lc + ll;
          const int d = l / args.n_angles;
          const MapRef mr = make_map_ref(args.maps, MAPS_DTYPE, args.maps_slice_stride, args.n_angles, args.n_det, n, s,
                                         l - d * args.n_angles, d, args.n_channels, args.chan_scale);
          v *= map_at<MAPS_DTYPE>(mr, pix[k]);
        }
        acc[k] += v;
      }
    }
    if (SYM && more) load_chunk(lc + BP_LINES, next);
    if (more) store_chunk(lc + BP_LINES, next, buf ^ 1);
    if (ONE) break;
    slot = next;
    __syncthreads();
  }
}

template <int EPI, int PPT>
__device__ __forceinline__ void bp_epilogue_tile(const BpArgs& args, int s, int i0, int j, const float (&v)[PPT]) {
  if constexpr (EPI == BP_EPI_MLEM || EPI == BP_EPI_SIRT) {
    bp_epilogue_rows<EPI, PPT>(args, s, i0, 1, j, v);
  } else {
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int i = i0 + k;
      if (i < args.n && j < args.n) bp_epilogue<EPI>(args, s, i, j, v[k]);
    }
  }
}

// One CTA of the back projection: pixel tile `tile` of slice `s`; with CLUSTER, segment `rank` of the
// cluster's tile, else all segments.
template <int EPI, bool SYM, int MAPS_DTYPE, int PPT, bool CLUSTER, bool ONE>
__device__ __forceinline__ void bp_tile(const BpArgs& args, BpShared& sh, int tile, int s, int rank, int ranks) {
  constexpr int TI = 8 * PPT;
  const int n = args.n;
  if (args.active != nullptr && args.active[s] == 0) return;  // every CTA of the cluster
  const int tiles_j = (n + BP_TJ - 1) / BP_TJ;
  const int ti = tile / tiles_j;
  const int ti0 = ti * TI, tj0 = (tile - ti * tiles_j) * BP_TJ;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j = tj0 + lane;
  const int i0 = ti0 + PPT * warp;
  const int n_lines = args.n_det * args.n_angles;
  const int log2_segs = bp_log2_segments(n_lines), segs = 1 << log2_segs;
  float acc[PPT];
  if constexpr (ONE) {
    bp_segment<SYM, MAPS_DTYPE, PPT, true>(args, sh, s, ti0, tj0, i0, j, 0, n_lines, acc);
    bp_epilogue_tile<EPI, PPT>(args, s, i0, j, acc);
  } else if constexpr (!CLUSTER) {
    float total[PPT];
    for (int g = 0; g < segs; ++g) {
      bp_segment<SYM, MAPS_DTYPE, PPT, false>(args, sh, s, ti0, tj0, i0, j, (g * n_lines) >> log2_segs,
                                       ((g + 1) * n_lines) >> log2_segs, acc);
#pragma unroll
      for (int k = 0; k < PPT; ++k) total[k] = g == 0 ? acc[k] : total[k] + acc[k];
    }
    bp_epilogue_tile<EPI, PPT>(args, s, i0, j, total);
  } else {
    if (rank < segs) {
      bp_segment<SYM, MAPS_DTYPE, PPT, false>(args, sh, s, ti0, tj0, i0, j, (rank * n_lines) >> log2_segs,
                                       ((rank + 1) * n_lines) >> log2_segs, acc);
    }
    __syncthreads();
    float* part = reinterpret_cast<float*>(sh.pairs[0]);  // [TI][32] of this segment
    if (rank < segs) {
#pragma unroll
      for (int k = 0; k < PPT; ++k) part[(i0 - ti0 + k) * BP_TJ + lane] = acc[k];
    }
    cluster_sync_all();
    const int per_rank = TI * BP_TJ / ranks;
    for (int p = rank * per_rank + tid; p < (rank + 1) * per_rank; p += BP_THREADS) {
      float v = cluster_load(part + p, 0);
      for (int g = 1; g < segs; ++g) v += cluster_load(part + p, g);
      const int pi = ti0 + p / BP_TJ, pj = tj0 + p % BP_TJ;
      if (pi < n && pj < n) bp_epilogue<EPI>(args, s, pi, pj, v);
    }
    cluster_sync_all();  // the others may still read this CTA's sums
  }
}

template <int EPI, bool SYM, int MAPS_DTYPE, bool CLUSTER, bool ONE = false>
__device__ __forceinline__ void bp_cta(const BpArgs& args, int tile, int s, int rank, int ranks) {
  __shared__ __align__(16) BpShared sh;
  if (args.tile_rows == BP_BLOCK_ROWS) {
    bp_tile<EPI, SYM, MAPS_DTYPE, 8, CLUSTER, ONE>(args, sh, tile, s, rank, ranks);
  } else {
    bp_tile<EPI, SYM, MAPS_DTYPE, 4, CLUSTER, ONE>(args, sh, tile, s, rank, ranks);
  }
}

template <int EPI, bool SYM, int MAPS_DTYPE, bool ONE>
__global__ void __launch_bounds__(BP_THREADS, 4) bp_kernel(BpArgs args) {
  bp_cta<EPI, SYM, MAPS_DTYPE, false, ONE>(args, blockIdx.x, blockIdx.y, 0, 1);
}

// The same over clusters of `ranks` CTAs along x.
template <int EPI, bool SYM, int MAPS_DTYPE>
__global__ void __launch_bounds__(BP_THREADS, 4) bp_cluster_kernel(BpArgs args, int ranks) {
  const int tile = blockIdx.x / ranks;
  bp_cta<EPI, SYM, MAPS_DTYPE, true>(args, tile, blockIdx.y, blockIdx.x - tile * ranks, ranks);
}

// Back projection over groups of slices in one launch: group g's tiles are (tile, slice), tile
// fastest, each one CTA or one cluster of BP_MAX_RANKS CTAs (CLUSTER).
template <int EPI, bool SYM, int MAPS_DTYPE, bool CLUSTER>
__global__ void __launch_bounds__(BP_THREADS, 4) bp_ragged_kernel(const BpArgs* __restrict__ groups,
                                                                  const int64_t* __restrict__ start, int n_groups) {
  constexpr int RANKS = CLUSTER ? BP_MAX_RANKS : 1;
  const int64_t cta = blockIdx.x / RANKS;
  const int g = ragged_group(start, n_groups, cta);
  const BpArgs& a = groups[g];
  const int tiles = bp_tiles(a.n, a.tile_rows);
  const int64_t local = cta - start[g];
  bp_cta<EPI, SYM, MAPS_DTYPE, CLUSTER>(a, (int)(local % tiles), (int)(local / tiles), blockIdx.x % RANKS, RANKS);
}

// ------------------------------------------------------------------------------------------
// Exact adjoint of the forward projection (gather form; no reference counterpart)
// bp[p] = sum_a sum_{(r,c)} w_a hat(col_in(r,c) - p_x) hat(row_in(r,c) - p_y) y[a][c] (* map[a][p])
// For a pixel p and angle a the samples that reach it lie within distance < 1 (per axis) of p, so within
// sqrt(2) < 1.42 of its inverse-rotated lattice position along r and along c: at most three
// values of each, ceil(position - 1.42) and the next two.
//
// Bound: issue (~110 instructions per pixel and line for the nine candidates).  With few pixels a CTA holds 64
// of them and four threads of each take every fourth line, since one thread per pixel leaves most of the
// chip's warps empty at 256^2; batches that fill the chip, and a few lines, take one thread per pixel.  Positions and hats are FP32 like the forward's; the products of two
// hats and all sums are FP64 (253 us; with FP32 products and column sums 230 us, with their errors
// carried along in FP32 279 us).  256^2 x 360 with 36 candidates per thread and line: 1170 us.
// ------------------------------------------------------------------------------------------
constexpr int ADJ_THREADS = 256;
// Pixels of a batch below which four threads share one: 1.5 waves of CTAs of 256 pixels (256^2 x 60: 40 us
// with four, 50 with one at 1 slice, 138 and 137 at 4, 588 and 550 at 16), and less for lines that
// four threads cannot share (256^2 x 1: 5.7 and 4.1 us at 1 slice, 983 and 301 at 256; 128^2 x 3: 4.1 and 5.3).
constexpr int64_t ADJ_FEW_PIXELS = 227328, ADJ_FEW_LINES_PIXELS = 32768;
constexpr int ADJ_CHUNK = 32;       // lines whose geometry is staged together
constexpr float ADJ_REACH = 1.42f;  // > sqrt(2), by more than the FP32 error of the inverse position

struct AdjLine {
  float m00, m01, m02, m10, m11, m12;  // the forward map
  float cx, cy, c0, rx, ry, r0;        // lattice column and row of a pixel: cx x + cy y + c0, ...
  float w;
  int angle, det;
};

template <bool HAS_MAPS, int MAPS_DTYPE, int SPLIT>
__global__ void __launch_bounds__(ADJ_THREADS) bp_adjoint_kernel(BpArgs args) {
  constexpr int PIXELS = ADJ_THREADS / SPLIT;
  __shared__ AdjLine lines[ADJ_CHUNK];
  __shared__ double part[SPLIT][PIXELS];
  const int n = args.n;
  const int64_t total = (int64_t)n * n;
  const int s = blockIdx.y;
  const int tid = threadIdx.x, t = tid % PIXELS, g = tid / PIXELS;
  const int64_t pix = (int64_t)blockIdx.x * PIXELS + t;
  const bool in = pix < total;
  const int pi = in ? (int)(pix / n) : 0, pj = in ? (int)(pix - (int64_t)pi * n) : 0;
  const float fi = (float)pi, fj = (float)pj;
  const int n_lines = args.n_det * args.n_angles;
  const float* sino = args.sino + (int64_t)s * n_lines * n;
  double acc = 0.0;
  for (int l0 = 0; l0 < n_lines; l0 += ADJ_CHUNK) {
    const int count = min(ADJ_CHUNK, n_lines - l0);
    __syncthreads();
    if (tid < count) {
      const int l = l0 + tid;
      const int d = l / args.n_angles;
      const int a = l - d * args.n_angles;
      const float* M = args.fp_matrix + 6 * a;
      AdjLine al;
      al.m00 = M[0]; al.m01 = M[1]; al.m02 = M[2]; al.m10 = M[3]; al.m11 = M[4]; al.m12 = M[5];
      const double det = (double)M[0] * M[4] - (double)M[1] * M[3];
      al.cx = (float)(M[4] / det);
      al.cy = (float)(-M[1] / det);
      al.c0 = (float)(((double)M[1] * M[5] - (double)M[4] * M[2]) / det);
      al.rx = (float)(-M[3] / det);
      al.ry = (float)(M[0] / det);
      al.r0 = (float)(((double)M[3] * M[2] - (double)M[0] * M[5]) / det);
      al.w = args.weights != nullptr ? args.weights[a * args.n_det + d] : 1.f;
      al.angle = a;
      al.det = d;
      lines[tid] = al;
    }
    __syncthreads();
    for (int ll = g; in && ll < count; ll += SPLIT) {
      const AdjLine al = lines[ll];
      const float cb = ceilf(fmaf(al.cx, fj, fmaf(al.cy, fi, al.c0)) - ADJ_REACH);
      const float rb = ceilf(fmaf(al.rx, fj, fmaf(al.ry, fi, al.r0)) - ADJ_REACH);
      const float* y = sino + (int64_t)(l0 + ll) * n;
      // rows outside the lattice go far away, where the hat of the axis that r moves is zero
      float2 fr[3];
#pragma unroll
      for (int dr = 0; dr < 3; ++dr) {
        const float r = rb + (float)dr;
        fr[dr].x = fr[dr].y = r >= 0.f && r <= (float)(n - 1) ? r : 1.0e9f;
      }
      double lsum = 0.0;
#pragma unroll
      for (int dc = 0; dc < 3; ++dc) {
        const float fc = cb + (float)dc;
        const int c = (int)fc;
        if ((unsigned)c >= (unsigned)n) continue;
        const float yc = __ldg(y + c);
        const float2 pc = make_float2(fmaf(al.m00, fc, al.m02), fmaf(al.m10, fc, al.m12));
        double h = 0.0;
#pragma unroll
        for (int dr = 0; dr < 3; ++dr) {
          // same float arithmetic as the forward kernel's sample position (sample_x)
          const float2 d = __fadd2_rn(__ffma2_rn(make_float2(al.m01, al.m11), fr[dr], pc), make_float2(-fj, -fi));
          h = fma((double)fmaxf(1.f - fabsf(d.x), 0.f), (double)fmaxf(1.f - fabsf(d.y), 0.f), h);
        }
        // a bin that does not reach the pixel adds nothing, whatever it holds
        lsum = fma(h, h > 0.0 ? (double)yc : 0.0, lsum);
      }
      double contrib = lsum * al.w;
      if (HAS_MAPS) {
        const MapRef mr = make_map_ref(args.maps, MAPS_DTYPE, args.maps_slice_stride, args.n_angles, args.n_det, n, s,
                                       al.angle, al.det, args.n_channels, args.chan_scale);
        contrib *= map_at<MAPS_DTYPE>(mr, pix);
      }
      acc += contrib;
    }
  }
  if constexpr (SPLIT > 1) {
    part[g][t] = acc;
    __syncthreads();
    acc = 0.0;
#pragma unroll
    for (int k = 0; k < SPLIT; k += 2) acc += part[k][t] + part[k + 1][t];
  }
  if (g == 0 && in) bp_epilogue<BP_EPI_STORE>(args, s, pi, pj, (float)acc);
}

// ------------------------------------------------------------------------------------------
// Detector PSF: out[i] = sum_j in[clamp(i + (L-1)/2 - j)] * k[j] along each sinogram line (the
// reference pads with edge values, convolves with scipy 'same' and crops), followed by the same
// fused solver epilogue as the fp.  One CTA per line; args.vol holds the unconvolved sinogram.
// ------------------------------------------------------------------------------------------
constexpr int PSF_THREADS = 256;

template <int EPI>
__global__ void __launch_bounds__(PSF_THREADS) psf_kernel(FpArgs args, const float* __restrict__ k, int len) {
  extern __shared__ float line_sh[];
  __shared__ double red_d[PSF_THREADS / 32];
  const int n = args.n;
  const int64_t line = blockIdx.x;  // ((s * D + d) * A + a)
  const int s = (int)(line / ((int64_t)args.n_det * args.n_angles));
  if (args.active != nullptr && args.active[s] == 0) return;
  const float* in = args.vol + line * n;
  for (int i = threadIdx.x; i < n; i += PSF_THREADS) line_sh[i] = in[i];
  __syncthreads();
  const int p = (len - 1) / 2;
  double part = 0.0, ptest = 0.0;
  for (int i = threadIdx.x; i < n; i += PSF_THREADS) {
    float acc = 0.f;
    for (int j = 0; j < len; ++j) {
      int q = i + p - j;
      q = q < 0 ? 0 : (q >= n ? n - 1 : q);
      acc = fmaf(line_sh[q], __ldg(k + j), acc);
    }
    part += fp_epilogue<EPI>(args, line * n + i, acc, &ptest);
  }
  if (EPI == FP_EPI_MLEM || EPI == FP_EPI_SIRT) {
    // one partial per (detector, angle) line of the slice
    for (int which = 0; which < 2; ++which) {
      double* dst = which == 0 ? args.partials : args.partials_test;
      if (dst == nullptr) continue;  // uniform across the CTA
      double v = warp_sum_double(which == 0 ? part : ptest);
      __syncthreads();
      if ((threadIdx.x & 31) == 0) red_d[threadIdx.x >> 5] = v;
      __syncthreads();
      if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < PSF_THREADS / 32; ++w) t += red_d[w];
        dst[line] = t;
      }
    }
  }
}

void launch_psf(const FpArgs& a, const float* psf, int psf_len, cudaStream_t st) {
  const unsigned lines = (unsigned)((int64_t)a.n_slices * a.n_det * a.n_angles);
  const size_t smem = (size_t)a.n * sizeof(float);
  switch (a.epi) {
    case FP_EPI_MLEM: psf_kernel<FP_EPI_MLEM><<<lines, PSF_THREADS, smem, st>>>(a, psf, psf_len); break;
    case FP_EPI_SIRT: psf_kernel<FP_EPI_SIRT><<<lines, PSF_THREADS, smem, st>>>(a, psf, psf_len); break;
    case FP_EPI_PDHG: psf_kernel<FP_EPI_PDHG><<<lines, PSF_THREADS, smem, st>>>(a, psf, psf_len); break;
    default: psf_kernel<FP_EPI_STORE><<<lines, PSF_THREADS, smem, st>>>(a, psf, psf_len); break;
  }
}

// ------------------------------------------------------------------------------------------
// Launchers
// ------------------------------------------------------------------------------------------

// 3-D tiled map over `images` row-major n x n images with a 96 x 104 box.
static bool make_box_map(CUtensorMap* map, const void* base, int n, int64_t images, bool bf16) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (enc == nullptr) return false;
  const uint64_t esz = bf16 ? 2 : 4;
  const cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)images};
  const cuuint64_t strides[2] = {(cuuint64_t)(n * esz), (cuuint64_t)((uint64_t)n * n * esz)};
  const cuuint32_t box[3] = {(cuuint32_t)FPT_BOX_W, (cuuint32_t)FPT_BOX_H, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
static bool launch_fp_tma_inst(const FpArgs& a, const dim3& grid, cudaStream_t st) {
  CUtensorMap tv, tm;
  std::memset(&tm, 0, sizeof(tm));
  if (!make_box_map(&tv, a.vol, a.n, a.n_slices, false)) return false;
  if (HAS_MAPS &&
      !make_box_map(&tm, a.maps, a.n, (int64_t)a.n_slices * a.n_angles * a.n_det, MAPS_DTYPE == CCT_DTYPE_BF16)) {
    return false;
  }
  const size_t smem = FPT_BOX_H * FPT_BOX_W * sizeof(float) +
                      (HAS_MAPS ? FPT_BOX_H * FPT_BOX_W * (MAPS_DTYPE == CCT_DTYPE_BF16 ? 2 : 4) : 0);
  if (!ensure_dynamic_smem<fp_tma_kernel<EPI, HAS_MAPS, MAPS_DTYPE>>((int)smem)) return false;
  fp_tma_kernel<EPI, HAS_MAPS, MAPS_DTYPE><<<grid, FP_THREADS, smem, st>>>(a, tv, tm);
  return launched_ok();
}

template <int EPI, bool HAS_MAPS, int MAPS_DTYPE>
static bool launch_fp_pair_inst(const FpArgs& a, cudaStream_t st) {
  const dim3 grid((a.n + FP_TC - 1) / FP_TC, a.n_angles * a.n_det, (a.n_slices + 1) / 2);
  if (!ensure_dynamic_smem<fp_pair_kernel<EPI, HAS_MAPS, MAPS_DTYPE>>((int)FP2_SMEM_BYTES)) return false;
  fp_pair_kernel<EPI, HAS_MAPS, MAPS_DTYPE><<<grid, FP_THREADS, FP2_SMEM_BYTES, st>>>(a);
  return launched_ok();
}

template <int EPI>
static bool launch_fp_pair(const FpArgs& a, cudaStream_t st) {
  if (a.maps == nullptr) return launch_fp_pair_inst<EPI, false, CCT_DTYPE_F32>(a, st);
  if (a.maps_dtype == CCT_DTYPE_BF16) return launch_fp_pair_inst<EPI, true, CCT_DTYPE_BF16>(a, st);
  if (a.maps_dtype == CCT_DTYPE_FIELDS_F32) return launch_fp_pair_inst<EPI, true, CCT_DTYPE_FIELDS_F32>(a, st);
  return launch_fp_pair_inst<EPI, true, CCT_DTYPE_F32>(a, st);
}

// 16-byte staging loads need a 16-byte aligned volume, maps at 16 (FP32) or 8 (BF16) bytes and
// map images that stay aligned (n % 4 == 0, slice stride a multiple of 4 elements)
bool fp_vec4_ok(const FpArgs& a) {
  const uintptr_t map_align = a.maps_dtype == CCT_DTYPE_BF16 ? 8 : 16;
  return (a.n % 4) == 0 && (reinterpret_cast<uintptr_t>(a.vol) % 16) == 0 &&
         (a.maps == nullptr || ((reinterpret_cast<uintptr_t>(a.maps) % map_align) == 0 && a.maps_slice_stride % 4 == 0));
}

template <int EPI>
static void launch_fp_epi(const FpArgs& a, cudaStream_t st) {
  const dim3 grid((a.n + FP_TC - 1) / FP_TC, a.n_angles * a.n_det, a.n_slices);
  // two slices per CTA: any n, maps stride and storage type; the plain kernel if refused
  if ((a.variant & CCT_VARIANT_FP_SLICES2) && a.n_slices >= 2) {
    FpArgs v = a;
    v.vec4 = fp_vec4_ok(a) ? 1 : 0;
    if (launch_fp_pair<EPI>(v, st)) return;
  }
  // TMA path: rows and images must be 16-byte multiples for both FP32 and BF16 boxes
  const int64_t dense = (int64_t)a.n_angles * a.n_det * a.n * a.n;
  const bool aligned = (a.n % 8) == 0 && (reinterpret_cast<uintptr_t>(a.vol) % 16) == 0 &&
                       (a.maps == nullptr || (reinterpret_cast<uintptr_t>(a.maps) % 16) == 0) &&
                       a.maps_slice_stride == dense && a.maps_dtype != CCT_DTYPE_FIELDS_F32;
  if (aligned && (a.variant & CCT_VARIANT_FP_TMA)) {
    bool ok;
    if (a.maps == nullptr) {
      ok = launch_fp_tma_inst<EPI, false, CCT_DTYPE_F32>(a, grid, st);
    } else if (a.maps_dtype == CCT_DTYPE_BF16) {
      ok = launch_fp_tma_inst<EPI, true, CCT_DTYPE_BF16>(a, grid, st);
    } else {
      ok = launch_fp_tma_inst<EPI, true, CCT_DTYPE_F32>(a, grid, st);
    }
    if (ok) return;
  }
  FpArgs v = a;
  v.vec4 = fp_vec4_ok(a) ? 1 : 0;
  if (a.maps == nullptr) {
    fp_kernel<EPI, false, CCT_DTYPE_F32><<<grid, FP_THREADS, 0, st>>>(v);
  } else if (a.maps_dtype == CCT_DTYPE_BF16) {
    fp_kernel<EPI, true, CCT_DTYPE_BF16><<<grid, FP_THREADS, 0, st>>>(v);
  } else if (a.maps_dtype == CCT_DTYPE_FIELDS_F32) {
    const dim3 fgrid(grid.x * a.n_channels, grid.y, a.n_slices / a.n_channels);
    fp_fields_kernel<EPI><<<fgrid, FP_THREADS, 0, st>>>(v);
  } else {
    fp_kernel<EPI, true, CCT_DTYPE_F32><<<grid, FP_THREADS, 0, st>>>(v);
  }
}

void launch_fp(const FpArgs& a, cudaStream_t st) {
  switch (a.epi) {
    case FP_EPI_MLEM: launch_fp_epi<FP_EPI_MLEM>(a, st); break;
    case FP_EPI_SIRT: launch_fp_epi<FP_EPI_SIRT>(a, st); break;
    case FP_EPI_PDHG: launch_fp_epi<FP_EPI_PDHG>(a, st); break;
    default: launch_fp_epi<FP_EPI_STORE>(a, st); break;
  }
}

// A kernel over clusters of `ranks` CTAs along x.
template <typename Kernel, typename... Args>
static void launch_cluster(Kernel kernel, const dim3& grid, int ranks, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(BP_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)ranks;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, args...);  // a refused launch is the entry point's sticky error
}

// Tiles of a batch below which the CTAs of a cluster share each tile's lines: the crossing lies between
// two and four tiles per SM (512^2 x 720: 327 us in clusters, 333 without at 3 slices = 384 tiles, 422
// and 414 at 4; 256^2 x 360: 144 and 157 at 8 slices = 256 tiles, 203 and 182 at 12; 128^2 x 180: 64 and 72
// at 32 slices = 256 tiles, 118 and 119 at 64).
constexpr int64_t BP_FEW_TILES = 352;

// Rows of a batch's tiles (one CTA or, with `segs` > 1, a cluster of as many for each).  A tile of 64 rows
// stages a line for twice the pixels; tiles of 32 rows pay while their CTAs leave most of the chip idle
// and a tile's own time counts: up to two per SM in clusters (128^2 x 180: 10.8 us with 32 rows, 12.1 with 64
// at 1 slice = 128 CTAs, 15.5 and 14.3 at 4 slices = 512), up to four per SM with one segment (192^2 x 4:
// 5.6 and 6.6 us at 16 slices = 576 CTAs, 9.0 and 8.5 at 32).  Large batches gain most from 64 rows
// (128^2 x 180, 1024 slices: 2020 and 1338 us).
static int bp_tile_rows(int64_t tiles32, int segs) { return tiles32 * segs <= (segs > 1 ? 296 : 592) ? 32 : BP_BLOCK_ROWS; }

template <int EPI, bool SYM, int MAPS_DTYPE>
static void launch_bp_inst(BpArgs a, cudaStream_t st) {
  const int segs = 1 << bp_log2_segments(a.n_det * a.n_angles);
  a.tile_rows = bp_tile_rows((int64_t)bp_tiles(a.n, 32) * a.n_slices, segs);
  const int tiles = bp_tiles(a.n, a.tile_rows);
  if (segs > 1 && (int64_t)tiles * a.n_slices < BP_FEW_TILES) {
    launch_cluster(bp_cluster_kernel<EPI, SYM, MAPS_DTYPE>, dim3(tiles * segs, a.n_slices), segs, st, a, segs);
  } else if (segs == 1) {  // at most 15 lines
    bp_kernel<EPI, SYM, MAPS_DTYPE, true><<<dim3(tiles, a.n_slices), BP_THREADS, 0, st>>>(a);
  } else {
    bp_kernel<EPI, SYM, MAPS_DTYPE, false><<<dim3(tiles, a.n_slices), BP_THREADS, 0, st>>>(a);
  }
}

template <int EPI>
static void launch_bp_epi(const BpArgs& a, cudaStream_t st) {
  if (a.mode != CCT_BP_SYMMETRIC) {
    launch_bp_inst<EPI, false, CCT_DTYPE_F32>(a, st);
  } else if (a.maps_dtype == CCT_DTYPE_BF16) {
    launch_bp_inst<EPI, true, CCT_DTYPE_BF16>(a, st);
  } else if (a.maps_dtype == CCT_DTYPE_FIELDS_F32) {
    launch_bp_inst<EPI, true, CCT_DTYPE_FIELDS_F32>(a, st);
  } else {
    launch_bp_inst<EPI, true, CCT_DTYPE_F32>(a, st);
  }
}

template <int EPI>
static void launch_fp_ragged_epi(const FpArgs* g, const int64_t* start, int ng, int64_t ctas, bool has_maps, int dt,
                                 cudaStream_t st) {
  const dim3 grid((unsigned)ctas);
  if (!has_maps) {
    fp_ragged_kernel<EPI, false, CCT_DTYPE_F32><<<grid, FP_THREADS, 0, st>>>(g, start, ng);
  } else if (dt == CCT_DTYPE_BF16) {
    fp_ragged_kernel<EPI, true, CCT_DTYPE_BF16><<<grid, FP_THREADS, 0, st>>>(g, start, ng);
  } else if (dt == CCT_DTYPE_FIELDS_F32) {
    fp_ragged_kernel<EPI, true, CCT_DTYPE_FIELDS_F32><<<grid, FP_THREADS, 0, st>>>(g, start, ng);
  } else {
    fp_ragged_kernel<EPI, true, CCT_DTYPE_F32><<<grid, FP_THREADS, 0, st>>>(g, start, ng);
  }
}

void launch_fp_ragged(const FpArgs* groups, const int64_t* start, int n_groups, int64_t ctas, int epi, bool has_maps,
                      int maps_dtype, cudaStream_t st) {
  if (epi == FP_EPI_SIRT) {
    launch_fp_ragged_epi<FP_EPI_SIRT>(groups, start, n_groups, ctas, has_maps, maps_dtype, st);
  } else {
    launch_fp_ragged_epi<FP_EPI_MLEM>(groups, start, n_groups, ctas, has_maps, maps_dtype, st);
  }
}

template <int EPI, bool SYM, int DT>
static void launch_bp_ragged_inst(const BpArgs* g, const int64_t* start, int ng, int64_t tiles, cudaStream_t st) {
  if (tiles < BP_FEW_TILES) {
    launch_cluster(bp_ragged_kernel<EPI, SYM, DT, true>, dim3((unsigned)tiles * BP_MAX_RANKS), BP_MAX_RANKS, st, g, start,
                   ng);
  } else {
    bp_ragged_kernel<EPI, SYM, DT, false><<<(unsigned)tiles, BP_THREADS, 0, st>>>(g, start, ng);
  }
}

template <int EPI>
static void launch_bp_ragged_epi(const BpArgs* g, const int64_t* start, int ng, int64_t tiles, bool sym, int dt,
                                 cudaStream_t st) {
  if (!sym) {
    launch_bp_ragged_inst<EPI, false, CCT_DTYPE_F32>(g, start, ng, tiles, st);
  } else if (dt == CCT_DTYPE_BF16) {
    launch_bp_ragged_inst<EPI, true, CCT_DTYPE_BF16>(g, start, ng, tiles, st);
  } else if (dt == CCT_DTYPE_FIELDS_F32) {
    launch_bp_ragged_inst<EPI, true, CCT_DTYPE_FIELDS_F32>(g, start, ng, tiles, st);
  } else {
    launch_bp_ragged_inst<EPI, true, CCT_DTYPE_F32>(g, start, ng, tiles, st);
  }
}

int64_t bp_tile_count(int n, int rows) { return bp_tiles(n, rows); }

// A ragged launch ends with its longest tiles: up to four waves of tiles of 64 rows (4 x 592) the small sides,
// which often have the most lines, keep 32 (eight groups of 128^2 x 360 to 512^2 x 90, 2 slices each: SIRT
// step 1038 us, 1124 with 64 rows); with more the rows' own cost counts, as above.
int bp_ragged_tile_rows(int n, int64_t tiles64) { return n <= 192 && tiles64 < 2368 ? 32 : BP_BLOCK_ROWS; }

void launch_bp_ragged(const BpArgs* groups, const int64_t* start, int n_groups, int64_t ctas, int epi, bool sym,
                      int maps_dtype, cudaStream_t st) {
  if (epi == BP_EPI_SIRT) {
    launch_bp_ragged_epi<BP_EPI_SIRT>(groups, start, n_groups, ctas, sym, maps_dtype, st);
  } else {
    launch_bp_ragged_epi<BP_EPI_MLEM>(groups, start, n_groups, ctas, sym, maps_dtype, st);
  }
}

template <int SPLIT>
static void launch_adjoint(const BpArgs& a, cudaStream_t st) {
  constexpr int pixels = ADJ_THREADS / SPLIT;
  const dim3 grid((unsigned)(((int64_t)a.n * a.n + pixels - 1) / pixels), a.n_slices);
  if (a.maps == nullptr) {
    bp_adjoint_kernel<false, CCT_DTYPE_F32, SPLIT><<<grid, ADJ_THREADS, 0, st>>>(a);
  } else if (a.maps_dtype == CCT_DTYPE_BF16) {
    bp_adjoint_kernel<true, CCT_DTYPE_BF16, SPLIT><<<grid, ADJ_THREADS, 0, st>>>(a);
  } else if (a.maps_dtype == CCT_DTYPE_FIELDS_F32) {
    bp_adjoint_kernel<true, CCT_DTYPE_FIELDS_F32, SPLIT><<<grid, ADJ_THREADS, 0, st>>>(a);
  } else {
    bp_adjoint_kernel<true, CCT_DTYPE_F32, SPLIT><<<grid, ADJ_THREADS, 0, st>>>(a);
  }
}

void launch_bp(const BpArgs& a, cudaStream_t st) {
  if (a.mode == CCT_BP_ADJOINT) {
    const int64_t pixels = (int64_t)a.n * a.n * a.n_slices;
    if (pixels < (a.n_det * a.n_angles < 4 ? ADJ_FEW_LINES_PIXELS : ADJ_FEW_PIXELS)) {
      launch_adjoint<4>(a, st);
    } else {
      launch_adjoint<1>(a, st);
    }
    return;
  }
  switch (a.epi) {
    case BP_EPI_MLEM: launch_bp_epi<BP_EPI_MLEM>(a, st); break;
    case BP_EPI_SIRT: launch_bp_epi<BP_EPI_SIRT>(a, st); break;
    case BP_EPI_PDHG: launch_bp_epi<BP_EPI_PDHG>(a, st); break;
    default: launch_bp_epi<BP_EPI_STORE>(a, st); break;
  }
}

}  // namespace cct

namespace cct {
int read_scan_error(int clear, int* value);  // cct_maps.cu

int read_device_error(int clear, int* value) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_box_overflow, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  int t = 0;
  e = cudaMemcpyFromSymbol(&t, g_tma_timeout, sizeof(int));
  if (e != cudaSuccess) return (int)e;
  if (clear) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_box_overflow, &zero, sizeof(int));
    if (e != cudaSuccess) return (int)e;
    e = cudaMemcpyToSymbol(g_tma_timeout, &zero, sizeof(int));
    if (e != cudaSuccess) return (int)e;
  }
  int m = 0;
  const int rc = read_scan_error(clear, &m);
  if (rc != 0) return rc;
  *value = v | (t << 1) | (m << 2);
  return 0;
}
}  // namespace cct
