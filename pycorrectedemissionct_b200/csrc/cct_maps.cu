// Attenuation maps of the XRF path (sm_100a).
//
// The reference (corrct: src/corrct/_projector_backends.py:43-99) computes, per angle and
// direction, on the image zero-padded to P = n + 2e (e = ceil((ceil(sqrt(2) n) - n) / 2)):
//   U = rotate(V, -phi)                       (scikit-image bilinear, zero outside)
//   W[r] = sum_{k<r} U[k] + U[r]/2 + U[P-1]/2  (roll + cumsum of halves along rows)
//   L = rotate(W, +phi)[e:e+n, e:e+n]
//   factor = exp(-L)
// and AttenuationVolume (corrct: src/corrct/physics/attenuation.py:105-180) multiplies the
// incident factor by the mean over sub-angles of the emitted factor of every detector.
//
// Phase 1 (maps_scan_kernel): CTAs of 64 rotated-frame columns c' of one rotation job walk the
// rows r' where the columns cross the image (elsewhere U is exactly 0), sampling U from staged
// boxes of mu and keeping the running sums in FP64, and write W (FP32) to the workspace.
// Phase 2 (maps_resample_kernel): one thread per four map pixels samples W of the incident job
// and of every emitted (detector, sub-angle) job at the rotated-back position, and writes
// exp(-L_in) * mean_k exp(-L_out,k) as FP32 or BF16.  Angles are processed in passes sized
// to the caller's workspace.
// Half-turn pairs: for angles phi and phi + pi every rotation of the second is the first's turned
// by 180 degrees about the frame centre, a permutation of the lattice.  Its W at the first's
// (r', c') is then K[c'] - W[r'][c'] with the per-column constant K = sum U + U[0]/2 + U[P-1]/2,
// and its rotate-back samples sit at the same positions; one scan and one resample per direction
// give both angles' maps.

#include <algorithm>
#include <cmath>

#include "cct_common.cuh"
#include "cct_internal.cuh"

namespace cct {

struct MapsPass {
  int n, P, e, n_det, n_sub, has_in, has_out, maps_dtype, n_angles;
  int a0, na;                 // first entry (first quad with quads) and scanned entries of this pass
  int n_entries;              // entries of `pairs` (angles without)
  int jobs_per_angle;         // has_in + has_out * n_det * n_sub
  const double* rot_in;       // [A][2][6]
  const double* rot_out;      // [A][D][n_sub][2][6]
  const int* pairs;           // [entries][2] (angle, partner) or NULL
  const int* quads;           // [quads][6] (entry, entry', emitted source of the 4 angles) or NULL
  float emitted_scale;        // quads: mu_out = emitted_scale * mu_in
  const float* mu_in;         // [S][n][n]
  const float* mu_out;
  const float* mu_in_t;       // [S][n][pitch] transposed copies (mu_t[s][x][y] = mu[s][y][x]) or NULL
  const float* mu_out_t;
  const float* mu_in_p;       // [S][n][pitch] row-major copies with rows on 16 bytes (n % 4 != 0) or NULL
  const float* mu_out_p;
  int pitch;                  // row pitch of the copies: n rounded up to 4, zeros past n
  float* work;                // [S][na][jobs_per_angle][P][P]
  float* kcol;                // [S][na][jobs_per_angle][P] per-column constants of the partner scans
  void* maps;                 // [S][A][D][n][n]
};

// Entry scanned in slot ai of the pass: with quads, slots 2q and 2q + 1 are quad (a0 + q)'s two
// entries (a0 counts quads); otherwise slot ai is entry a0 + ai.
__device__ __forceinline__ int slot_entry(const MapsPass& p, int ai) {
  if (p.quads == nullptr) return p.a0 + ai;
  return p.quads[6 * (p.a0 + (ai >> 1)) + (ai & 1)];
}

// Angle of entry e and its half-turn partner (-1: none); a = -1 for an out-of-range entry.
__device__ __forceinline__ void entry_angles(const MapsPass& p, int e, int* a, int* b) {
  if (e < 0 || e >= p.n_entries) {
    *a = *b = -1;
    return;
  }
  if (p.pairs == nullptr) {
    *a = e;
    *b = -1;
    return;
  }
  const int aa = p.pairs[2 * e], bb = p.pairs[2 * e + 1];
  *a = (aa >= 0 && aa < p.n_angles) ? aa : -1;
  *b = (bb >= 0 && bb < p.n_angles && bb != aa) ? bb : -1;
}

__device__ __forceinline__ const double* job_matrix(const MapsPass& p, int a, int job, int which) {
  // job 0 = incident (if has_in); then emitted jobs d * n_sub + k
  if (p.has_in) {
    if (job == 0) return p.rot_in + ((int64_t)a * 2 + which) * 6;
    job -= 1;
  }
  return p.rot_out + ((((int64_t)a * p.n_det * p.n_sub) + job) * 2 + which) * 6;
}

// Bilinear sample of an (h x w) FP32 image with zero outside (scikit-image constant mode).
__device__ __forceinline__ float bilin_zero(const float* img, int h, int w, float x, float y) {
  const FloorSplit fx = floor_split(x), fy = floor_split(y);
  const int x0 = fx.i, y0 = fy.i;
  const bool xin0 = x0 >= 0 && x0 < w, xin1 = x0 + 1 >= 0 && x0 + 1 < w;
  const bool yin0 = y0 >= 0 && y0 < h, yin1 = y0 + 1 >= 0 && y0 + 1 < h;
  const float v00 = (yin0 && xin0) ? __ldg(img + (int64_t)y0 * w + x0) : 0.f;
  const float v01 = (yin0 && xin1) ? __ldg(img + (int64_t)y0 * w + x0 + 1) : 0.f;
  const float v10 = (yin1 && xin0) ? __ldg(img + (int64_t)(y0 + 1) * w + x0) : 0.f;
  const float v11 = (yin1 && xin1) ? __ldg(img + (int64_t)(y0 + 1) * w + x0 + 1) : 0.f;
  const float top = fmaf(fx.f, v01 - v00, v00);
  const float bot = fmaf(fx.f, v11 - v10, v10);
  return fmaf(fy.f, bot - top, top);
}

// The position (x, y) in packed FP32x2 arithmetic, split like floor_split: fractions, and the index
// floor(y) * pitch + floor(x) (TR: floor(x) * pitch + floor(y)) of its first tap.
struct TapSplit {
  float2 f;
  unsigned q;
};
template <bool TR>
__device__ __forceinline__ TapSplit tap_split(float2 xy, unsigned pitch) {
  const float2 t = __fadd2_rd(xy, make_float2(12582912.0f, 12582912.0f));  // 1.5 * 2^23, see floor_split
  TapSplit r;
  r.f = __ffma2_rn(__fadd2_rn(t, make_float2(-12582912.0f, -12582912.0f)), make_float2(-1.f, -1.f), xy);
  const unsigned major = __float_as_uint(TR ? t.x : t.y), minor = __float_as_uint(TR ? t.y : t.x);
  r.q = major * pitch + (minor - 0x4B400000u * (pitch + 1u));
  return r;
}

// Bilinear sample at xy of a (P x P) image W, and with PAIR of the partner field K[c] - W[r][c]: the
// x-interpolated column constant minus the sample (bilinear interpolation is linear and K does not vary
// along rows).  A map pixel rotated about the frame's centre stays 0.2 pixels inside the frame
// (P >= sqrt(2) n), so its four taps are there; the minimum keeps the loads of pixels past the image
// edge, which are not stored, in bounds.
template <bool PAIR>
__device__ __forceinline__ void bilin_frame(const float* img, const float* K, unsigned P, float2 xy, float* La, float* Lb) {
  const TapSplit t = tap_split<false>(xy, P);
  const float *p = img + min(t.q, P * P - P - 2u), *q = p + P;
  const float v00 = __ldg(p), v01 = __ldg(p + 1), v10 = __ldg(q), v11 = __ldg(q + 1);
  const float top = fmaf(t.f.x, v01 - v00, v00);
  const float bot = fmaf(t.f.x, v11 - v10, v10);
  *La = fmaf(t.f.y, bot - top, top);
  if constexpr (PAIR) {
    const unsigned c = min((unsigned)floor_split(xy.x).i, P - 2u);
    const float k0 = __ldg(K + c), k1 = __ldg(K + c + 1);
    *Lb = fmaf(t.f.x, k1 - k0, k0) - *La;
  }
}

// Range of r' (inclusive) where the column c' samples inside (-1, n) x (-1, n) of mu, widened
// by one row each side; outside it every bilinear tap is zero padding.
__device__ __forceinline__ void column_support(double ax, double bx, double ay, double by, int n, int P,
                                               int* lo, int* hi) {
  double tlo = -1e300, thi = 1e300;
  const double lim0 = -1.0, lim1 = (double)n;
  // x(r) = ax + r bx in (lim0, lim1)
  if (fabs(bx) < 1e-12) {
    if (!(ax > lim0 && ax < lim1)) { *lo = 1; *hi = 0; return; }
  } else {
    double t0 = (lim0 - ax) / bx, t1 = (lim1 - ax) / bx;
    if (t0 > t1) { double t = t0; t0 = t1; t1 = t; }
    tlo = fmax(tlo, t0); thi = fmin(thi, t1);
  }
  if (fabs(by) < 1e-12) {
    if (!(ay > lim0 && ay < lim1)) { *lo = 1; *hi = 0; return; }
  } else {
    double t0 = (lim0 - ay) / by, t1 = (lim1 - ay) / by;
    if (t0 > t1) { double t = t0; t0 = t1; t1 = t; }
    tlo = fmax(tlo, t0); thi = fmin(thi, t1);
  }
  if (tlo > thi) { *lo = 1; *hi = 0; return; }
  *lo = max(0, (int)floor(tlo) - 1);
  *hi = min(P - 1, (int)ceil(thi) + 1);
}

// ------------------------------------------------------------------------------------------
// Scan
//
// A CTA owns 64 rotated-frame columns of one job and walks their support rows in chunks of 64.  The
// bounding box of a chunk in mu (at most 94 rows of 103 pixels, zeros outside the image) is staged in
// shared memory; each of 256 threads then samples 16 consecutive rows of one column, the column's four
// threads exchange their FP64 sums, and each writes its rows.  A warp is 32 neighbouring columns at
// one row, so the stores of W are coalesced; where the columns run closer to y than to x the box comes
// from the transposed copy of mu, and the row stride of 128 floats makes a tap's bank its
// position along the columns (1.6 wavefronts per load on average).
//
// Bound: sampling mu directly, a warp's load touched ~10 cache lines and the tag stage of L1, not its
// data, set the pace; staged, a row costs ~12 data wavefronts.  (8 slices of 512^2, 14 jobs per
// slice: 188 us per launch sampling directly, 121 us so.)  Staging needs rows on 16-byte boundaries:
// with n % 4 != 0 the row-major side also comes from a copy with padded rows (301^2: 187 us per launch
// with 4-byte staging, 117 us so).
// ------------------------------------------------------------------------------------------
constexpr int SCAN_COLS = 64;
constexpr int SCAN_ROWS = 64;
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_PER_THREAD = SCAN_ROWS / (SCAN_THREADS / SCAN_COLS);  // rows of one thread per chunk
constexpr int SCAN_STRIDE = 128;
constexpr int SCAN_BOX_W = 100, SCAN_BOX_H = 94;
constexpr size_t SCAN_SMEM = SCAN_BOX_H * SCAN_STRIDE * sizeof(float) + 4 * SCAN_COLS * sizeof(double);

// Raised (never trapped) if a chunk's box would exceed its bound; rotation matrices cannot reach it.
__device__ int g_scan_overflow = 0;

// Stage a box in items of W pixels (W = 4: pitch, bu and the address allow 16-byte loads, and the
// pitch's pixels past n are zeros), BATCH items' loads in flight per thread.
template <int W, int BATCH>
__device__ __forceinline__ void scan_stage(float* z, const float* mu, int n, int pitch, int bu, int bv, int bw, int bh,
                                           int tid) {
  const int per_row = (bw + W - 1) / W, items = per_row * bh;
  // it / per_row = (it * ceil(2^20 / per_row)) >> 20, exact while it * per_row < 2^20
  const unsigned magic = (1048576u + (unsigned)per_row - 1u) / (unsigned)per_row;
  for (int base = tid; base < items; base += SCAN_THREADS * BATCH) {
    float v[BATCH][W];
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int it = base + k * SCAN_THREADS;
      const int row = (int)(((unsigned)it * magic) >> 20);
      const int gv = bv + row, gu = bu + W * (it - row * per_row);
#pragma unroll
      for (int q = 0; q < W; ++q) v[k][q] = 0.f;
      if (it < items && (unsigned)gv < (unsigned)n && (unsigned)gu < (unsigned)n) {
        const float* src = mu + (gv * pitch + gu);
        if constexpr (W == 4) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(src));
          v[k][0] = t.x; v[k][1] = t.y; v[k][2] = t.z; v[k][3] = t.w;
        } else {
          v[k][0] = __ldg(src);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int it = base + k * SCAN_THREADS;
      const int row = (int)(((unsigned)it * magic) >> 20);
      if (it >= items) break;
      float* dst = z + (row * SCAN_STRIDE + W * (it - row * per_row));
      if constexpr (W == 4) {
        *reinterpret_cast<float4*>(dst) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
      } else {
        *dst = v[k][0];
      }
    }
  }
}

// The walk of one band.  (u, v) = (x, y), or (y, x) with TR: u runs along the staged rows.
template <bool PAIRS, bool TR>
__device__ __forceinline__ void scan_band(const MapsPass& p, float* z, double* sums, const float* mu, int pitch, const float* mu_row,
                                          float m00, float m01, float m02, float m10, float m11, float m12, int c0,
                                          int blo, int bhi, float* W, float* kcol) {
  const int n = p.n, P = p.P;
  const int tid = threadIdx.x;
  const int col = tid & (SCAN_COLS - 1), quarter = tid / SCAN_COLS;
  const int c = min(c0 + col, P - 1);
  const bool valid = c0 + col < P;  // lanes past the frame shadow the last column, store nothing
  const float fc = (float)c, fc1 = (float)min(c0 + SCAN_COLS - 1, P - 1);
  const float xc = fmaf(m00, fc, m02), yc = fmaf(m10, fc, m12);
  // wrap-around term U[P-1] / 2 of roll + cumsum (0 unless the support reaches the last row)
  double wrap = 0.0;
  if (bhi == P - 1) {
    const float fr = (float)(P - 1);
    wrap = 0.5 * (double)bilin_zero(mu_row, n, n, fmaf(m01, fr, xc), fmaf(m11, fr, yc));
  }
  const bool vec4 = pitch % 4 == 0 && (reinterpret_cast<uintptr_t>(mu) & 15) == 0;
  double carry = 0.0;
  for (int r0 = blo; r0 <= bhi; r0 += SCAN_ROWS) {
    const int r_last = min(r0 + SCAN_ROWS - 1, bhi);
    // box of the chunk's samples, widened by the taps; u origin a multiple of 4
    const float fr0 = (float)r0, fr1 = (float)r_last;
    const float xa = fmaf(m00, (float)c0, m02), xb = fmaf(m00, fc1, m02);
    const float ya = fmaf(m10, (float)c0, m12), yb = fmaf(m10, fc1, m12);
    const float x0 = fmaf(m01, fr0, xa), x1 = fmaf(m01, fr0, xb), x2 = fmaf(m01, fr1, xa), x3 = fmaf(m01, fr1, xb);
    const float y0 = fmaf(m11, fr0, ya), y1 = fmaf(m11, fr0, yb), y2 = fmaf(m11, fr1, ya), y3 = fmaf(m11, fr1, yb);
    const float xmin = fminf(fminf(x0, x1), fminf(x2, x3)), xmax = fmaxf(fmaxf(x0, x1), fmaxf(x2, x3));
    const float ymin = fminf(fminf(y0, y1), fminf(y2, y3)), ymax = fmaxf(fmaxf(y0, y1), fmaxf(y2, y3));
    const int bu = ((int)floorf(TR ? ymin : xmin) - 1) & ~3, bu1 = (int)floorf(TR ? ymax : xmax) + 2;
    const int bv = (int)floorf(TR ? xmin : ymin) - 1, bv1 = (int)floorf(TR ? xmax : ymax) + 2;
    const int bw = bu1 - bu + 1, bh = bv1 - bv + 1;
    if (bw > SCAN_BOX_W + 3 || bh > SCAN_BOX_H) {  // uniform; never trap
      if (tid == 0) atomicExch(&g_scan_overflow, 1);
      return;
    }
    if (vec4) {
      scan_stage<4, 3>(z, mu, n, pitch, bu, bv, bw, bh, tid);
    } else {
      scan_stage<1, 10>(z, mu, n, pitch, bu, bv, bw, bh, tid);
    }
    __syncthreads();

    // this thread's rows: samples as bilin_zero forms them (taps outside mu are staged zeros)
    const int rb = r0 + SCAN_PER_THREAD * quarter;
    const int rows = min(max(r_last - rb + 1, 0), SCAN_PER_THREAD);
    const unsigned zoff = (unsigned)(-bv * SCAN_STRIDE - bu);
    const float2 m = make_float2(m01, m11), c2 = make_float2(xc, yc);
    float u[SCAN_PER_THREAD];
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; ++k) {
      u[k] = 0.f;
      if (k < rows) {  // uniform in a warp
        const float fr = (float)(rb + k);
        const TapSplit t = tap_split<TR>(__ffma2_rn(m, make_float2(fr, fr), c2), SCAN_STRIDE);
        const float* q = z + (int)(t.q + zoff);
        const float v00 = q[0], v01 = TR ? q[SCAN_STRIDE] : q[1], v10 = TR ? q[1] : q[SCAN_STRIDE], v11 = q[SCAN_STRIDE + 1];
        const float top = fmaf(t.f.x, v01 - v00, v00);
        const float bot = fmaf(t.f.x, v11 - v10, v10);
        u[k] = fmaf(t.f.y, bot - top, top);
        sum += (double)u[k];
      }
    }
    sums[quarter * SCAN_COLS + col] = sum;
    __syncthreads();
    // W[r] = sum_{k<r} U[k] + U[r]/2 + wrap in FP64
    double acc = carry;
#pragma unroll
    for (int q = 0; q < SCAN_THREADS / SCAN_COLS; ++q) {
      const double sq = sums[q * SCAN_COLS + col];
      if (q < quarter) acc += sq;
      carry += sq;
    }
    float* w = W + (int64_t)rb * P + c;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; ++k) {
      if (k < rows) {
        const double d = (double)u[k];
        if (valid) *w = (float)(fma(0.5, d, acc) + wrap);
        acc += d;
        w += P;
      }
    }
  }
  if (PAIRS && kcol != nullptr && quarter == 0 && valid) {
    // the partner angle (phi + pi) rotates by a half turn more: its frame is this one turned
    // about the centre, and its W at this frame's (r', c') is K[c'] - W[r'][c'] with
    // K = sum_k U[k] + U[0]/2 + U[P-1]/2 (the reverse roll + cumsum of the same column)
    const double first = blo == 0 ? 0.5 * (double)bilin_zero(mu_row, n, n, xc, yc) : 0.0;
    kcol[c] = (float)(carry + first + wrap);
  }
}

template <bool PAIRS>
__global__ void __launch_bounds__(SCAN_THREADS, 4) maps_scan_kernel(MapsPass p) {
  extern __shared__ __align__(16) float scan_z[];
  double* sums = reinterpret_cast<double*>(scan_z + SCAN_BOX_H * SCAN_STRIDE);
  const int P = p.P, n = p.n;
  const int c0 = blockIdx.x * SCAN_COLS;
  const int job_lin = blockIdx.y;  // (angle in pass, job)
  const int s = blockIdx.z;
  const int ai = job_lin / p.jobs_per_angle;
  const int job = job_lin - ai * p.jobs_per_angle;
  int a, b;
  entry_angles(p, slot_entry(p, ai), &a, &b);
  if (a < 0) return;  // the whole CTA
  const double* Md = job_matrix(p, a, job, 0);  // rotate(-phi)
  const bool incident = p.has_in && job == 0;
  // neighbouring columns step along (m00, m10) in mu
  const float* mu_t = incident ? p.mu_in_t : p.mu_out_t;
  const bool tr = mu_t != nullptr && fabs(Md[3]) > fabs(Md[0]);
  const float* mu_row = (incident ? p.mu_in : p.mu_out) + (int64_t)s * n * n;
  // mu coordinates = padded coordinates - e
  const float m00 = (float)Md[0], m01 = (float)Md[1], m02 = (float)(Md[2] - p.e);
  const float m10 = (float)Md[3], m11 = (float)Md[4], m12 = (float)(Md[5] - p.e);
  // support rows of the band: outside them W is constant per column and the resample, whose positions
  // all map back into the image, never reads it
  // (tests/test_host.py::test_maps_resample_reads_only_scanned_rows mirrors that arithmetic)
  int lo = P, hi = -1;
  if ((int)threadIdx.x < SCAN_COLS && c0 + (int)threadIdx.x < P) {
    const int c = c0 + threadIdx.x;
    column_support(Md[0] * c + Md[2] - p.e, Md[1], Md[3] * c + Md[5] - p.e, Md[4], n, P, &lo, &hi);
    if (lo > hi) {
      lo = P;
      hi = -1;
    }
  }
  __shared__ int range_sh[2];
  if (threadIdx.x == 0) {
    range_sh[0] = P;
    range_sh[1] = -1;
  }
  __syncthreads();
  if (threadIdx.x < SCAN_COLS) {
    atomicMin(&range_sh[0], lo);
    atomicMax(&range_sh[1], hi);
  }
  __syncthreads();
  const int64_t slot = ((int64_t)s * p.na + ai) * p.jobs_per_angle + job;
  float* W = p.work + slot * (int64_t)P * P;
  float* kcol = PAIRS && b >= 0 ? p.kcol + slot * P : nullptr;
  const float* mu_p = incident ? p.mu_in_p : p.mu_out_p;
  const int64_t copy = (int64_t)s * n * p.pitch;
  if (tr) {
    scan_band<PAIRS, true>(p, scan_z, sums, mu_t + copy, p.pitch, mu_row, m00, m01, m02, m10, m11, m12, c0, range_sh[0],
                           range_sh[1], W, kcol);
  } else {
    scan_band<PAIRS, false>(p, scan_z, sums, mu_p != nullptr ? mu_p + copy : mu_row, mu_p != nullptr ? p.pitch : n, mu_row,
                            m00, m01, m02, m10, m11, m12, c0, range_sh[0], range_sh[1], W, kcol);
  }
}

// One CTA = a 32 x 32 pixel tile of one (slice, angle); thread t owns the four pixels
// (x, y + 8k), k < 4, so that each warp instruction covers an 8-wide, 4-tall block whose taps
// fall in a compact patch of the rotated frame.  The rotate(+phi) matrices of the angle's jobs
// are converted to FP32 once per CTA into shared memory.
constexpr int RS_TILE = 32;
constexpr int RS_PIX = 4;

template <bool PAIRS>
__global__ void __launch_bounds__(256, PAIRS ? 5 : 1) maps_resample_kernel(MapsPass p) {
  extern __shared__ float rs_mats[];  // [jobs_per_angle][6]
  const int n = p.n, P = p.P;
  const int ai = blockIdx.y;
  const int s = blockIdx.z;
  int a, b;
  entry_angles(p, p.a0 + ai, &a, &b);
  if (a < 0) return;  // the whole CTA
  const bool paired = PAIRS && b >= 0;
  const int J = p.jobs_per_angle;
  for (int t = threadIdx.x; t < 6 * J; t += blockDim.x) {
    const int job = t / 6;
    rs_mats[t] = (float)job_matrix(p, a, job, 1)[t - job * 6];
  }
  __syncthreads();
  const int tiles_x = (n + RS_TILE - 1) / RS_TILE;
  const int ty = blockIdx.x / tiles_x, tx = blockIdx.x - ty * tiles_x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = tx * RS_TILE + (warp & 3) * 8 + (lane & 7);
  const int i0 = ty * RS_TILE + (warp >> 2) * 4 + (lane >> 3);
  if (j >= n || i0 >= n) return;
  const float X = (float)(j + p.e);  // padded coordinates of the pixels
  const float* wbase = p.work + ((int64_t)s * p.na + ai) * J * (int64_t)P * P;
  const int64_t n2 = (int64_t)n * n;

  const float* kbase = p.kcol + ((int64_t)s * p.na + ai) * J * (int64_t)P;

  // L of job `job` at the four pixels, and with a partner its L at the same pixels (pixels
  // past the image edge are sampled, in bounds, and not stored)
  auto sample4 = [&](int job, float* L, float* Lb) {
    const float* m = rs_mats + job * 6;
    const float* w = wbase + (int64_t)job * P * P;
    const float* kc = kbase + (int64_t)job * P;
    const float2 my = make_float2(m[1], m[4]);
    const float2 c0 = make_float2(fmaf(m[0], X, m[2]), fmaf(m[3], X, m[5]));
#pragma unroll
    for (int k = 0; k < RS_PIX; ++k) {
      const float Y = (float)(i0 + 8 * k + p.e);
      bilin_frame<PAIRS>(w, kc, (unsigned)P, __ffma2_rn(my, make_float2(Y, Y), c0), &L[k], &Lb[k]);
    }
  };
  auto store4 = [&](int64_t plane, const float* v) {
#pragma unroll
    for (int k = 0; k < RS_PIX; ++k) {
      const int i = i0 + 8 * k;
      if (i >= n) break;
      const int64_t off = plane * n2 + (int64_t)i * n + j;
      if (p.maps_dtype == CCT_DTYPE_BF16) {
        reinterpret_cast<__nv_bfloat16*>(p.maps)[off] = __float2bfloat16_rn(v[k]);
      } else {
        reinterpret_cast<float*>(p.maps)[off] = v[k];
      }
    }
  };

  float L[RS_PIX], Lb[RS_PIX];
  if (p.maps_dtype == CCT_DTYPE_FIELDS_F32) {
    // line-integral fields: plane 0 = L_in, plane 1 + d = L_out of detector d (n_sub == 1)
    const int64_t plane0 = ((int64_t)s * p.n_angles + a) * (1 + p.n_det);
    const int64_t plane0b = ((int64_t)s * p.n_angles + b) * (1 + p.n_det);
    if (p.has_in) {
      sample4(0, L, Lb);
    } else {
#pragma unroll
      for (int k = 0; k < RS_PIX; ++k) L[k] = Lb[k] = 0.f;
    }
    store4(plane0, L);
    if (paired) store4(plane0b, Lb);
    for (int d = 0; d < p.n_det; ++d) {
      if (p.has_out) {
        sample4((p.has_in ? 1 : 0) + d, L, Lb);
      } else {
#pragma unroll
        for (int k = 0; k < RS_PIX; ++k) L[k] = Lb[k] = 0.f;
      }
      store4(plane0 + 1 + d, L);
      if (paired) store4(plane0b + 1 + d, Lb);
    }
    return;
  }
  // exp(-L_in) mean exp(-L_out): with one emitted direction the exponent is summed first
  float l_in[RS_PIX], l_inb[RS_PIX];
  int job = 0;
  if (p.has_in) {
    sample4(0, l_in, l_inb);
    job = 1;
  } else {
#pragma unroll
    for (int k = 0; k < RS_PIX; ++k) l_in[k] = l_inb[k] = 0.f;
  }
  for (int d = 0; d < p.n_det; ++d) {
    float f[RS_PIX], fb[RS_PIX];
    if (p.has_out && p.n_sub > 1) {
      float sum[RS_PIX] = {0.f, 0.f, 0.f, 0.f}, sumb[RS_PIX] = {0.f, 0.f, 0.f, 0.f};
      for (int q = 0; q < p.n_sub; ++q) {
        sample4(job + d * p.n_sub + q, L, Lb);
#pragma unroll
        for (int k = 0; k < RS_PIX; ++k) {
          sum[k] += __expf(-L[k]);
          if (paired) sumb[k] += __expf(-Lb[k]);
        }
      }
      const float ns = (float)p.n_sub;
#pragma unroll
      for (int k = 0; k < RS_PIX; ++k) {
        f[k] = __expf(-l_in[k]) * (sum[k] / ns);
        if (paired) fb[k] = __expf(-l_inb[k]) * (sumb[k] / ns);
      }
    } else {
      if (p.has_out) {
        sample4(job + d, L, Lb);
      } else {
#pragma unroll
        for (int k = 0; k < RS_PIX; ++k) L[k] = Lb[k] = 0.f;
      }
#pragma unroll
      for (int k = 0; k < RS_PIX; ++k) {
        f[k] = __expf(-(l_in[k] + L[k]));
        if (paired) fb[k] = __expf(-(l_inb[k] + Lb[k]));
      }
    }
    store4(((int64_t)s * p.n_angles + a) * p.n_det + d, f);
    if (paired) store4(((int64_t)s * p.n_angles + b) * p.n_det + d, fb);
  }
}

// Quarter-turn quads (one point detector whose emitted direction is the incident direction of
// another angle of the set, mu_out = emitted_scale * mu_in): the pass scanned only incident
// fields, two per quad (slots 2q, 2q + 1), each a half-turn pair of angles.  At every pixel the two
// pair samples give the incident line integrals L[0..3] of the quad's four angles (entry e's angle
// and partner, entry e''s angle and partner); the map of angle k is
// exp(-L[k]) * exp(-emitted_scale * L[src[k]]), src[k] naming which of the four angles the
// emitted direction of angle k is (its rotation angle differs from the reference's emitted angle
// only by the float32 rounding of the angles, like a half-turn partner's).  Four maps from two
// gathers per pixel, where the per-pair resample needs two gathers for two maps.  Bound: the L1 pipe
// (16 taps of W per pixel), then issue: 56 (slice, quad)s of 512^2 took 158 us with 64-bit index
// arithmetic, range tests that a pixel of the image cannot fail and two exps per map, 125 us so.
__global__ void __launch_bounds__(256, 5) maps_resample_quad_kernel(MapsPass p) {
  __shared__ float qm[2][6];  // rotate(+phi) matrices of the two entries' angles
  __shared__ int qa[4];       // the four angles
  __shared__ int qs[4];       // emitted sources
  const int n = p.n, P = p.P;
  const int qi = blockIdx.y;
  const int s = blockIdx.z;
  const int* row = p.quads + 6 * (p.a0 + qi);
  if (threadIdx.x < 2) {
    int a, b;
    entry_angles(p, slot_entry(p, 2 * qi + threadIdx.x), &a, &b);
    qa[2 * threadIdx.x] = a;
    qa[2 * threadIdx.x + 1] = b;
  }
  if (threadIdx.x >= 32 && threadIdx.x < 36) qs[threadIdx.x - 32] = row[2 + threadIdx.x - 32];
  __syncthreads();
  bool ok = true;
#pragma unroll
  for (int k = 0; k < 4; ++k) ok = ok && qa[k] >= 0 && qs[k] >= 0 && qs[k] < 4;
  if (!ok) return;  // the whole CTA (only complete quads are valid)
  if (threadIdx.x < 12) {
    const int w = threadIdx.x / 6;
    qm[w][threadIdx.x - 6 * w] = (float)job_matrix(p, qa[2 * w], 0, 1)[threadIdx.x - 6 * w];
  }
  __syncthreads();
  const int tiles_x = (n + RS_TILE - 1) / RS_TILE;
  const int ty = blockIdx.x / tiles_x, tx = blockIdx.x - ty * tiles_x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = tx * RS_TILE + (warp & 3) * 8 + (lane & 7);
  const int i0 = ty * RS_TILE + (warp >> 2) * 4 + (lane >> 3);
  if (j >= n || i0 >= n) return;
  const float X = (float)(j + p.e);
  const int64_t n2 = (int64_t)n * n;
  const float sc = p.emitted_scale;
  float L[4][RS_PIX];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const float* m = qm[w];
    const int slot = 2 * qi + w;
    const float* wf = p.work + ((int64_t)s * p.na + slot) * (int64_t)P * P;
    const float* kc = p.kcol + ((int64_t)s * p.na + slot) * (int64_t)P;
    const float2 my = make_float2(m[1], m[4]);
    const float2 c0 = make_float2(fmaf(m[0], X, m[2]), fmaf(m[3], X, m[5]));
#pragma unroll
    for (int k = 0; k < RS_PIX; ++k) {
      const float Y = (float)(i0 + 8 * k + p.e);
      bilin_frame<true>(wf, kc, (unsigned)P, __ffma2_rn(my, make_float2(Y, Y), c0), &L[2 * w][k], &L[2 * w + 1][k]);
    }
  }
  // exp(-L[q]) exp(-scale L[source]) with the exponents summed first (one exp per map and pixel)
  auto emit = [&](int q, const float (&lq)[RS_PIX], const float (&le)[RS_PIX]) {
    const int64_t off = ((int64_t)s * p.n_angles + qa[q]) * n2 + (int64_t)i0 * n + j;  // n_det == 1
#pragma unroll
    for (int k = 0; k < RS_PIX; ++k) {
      if (i0 + 8 * k >= n) break;
      const float v = __expf(-fmaf(sc, le[k], lq[k]));
      if (p.maps_dtype == CCT_DTYPE_BF16) {
        reinterpret_cast<__nv_bfloat16*>(p.maps)[off + (int64_t)8 * k * n] = __float2bfloat16_rn(v);
      } else {
        reinterpret_cast<float*>(p.maps)[off + (int64_t)8 * k * n] = v;
      }
    }
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int src = qs[q];
    if (src == 0) {
      emit(q, L[q], L[0]);
    } else if (src == 1) {
      emit(q, L[q], L[1]);
    } else if (src == 2) {
      emit(q, L[q], L[2]);
    } else {
      emit(q, L[q], L[3]);
    }
  }
}

int padded_edge(int n) {
  // edges = ceil((ceil(sqrt(2 n^2)) - n) / 2)  (corrct: src/corrct/_projector_backends.py:75-77)
  const double min_size = ceil(sqrt(2.0 * (double)n * (double)n));
  return (int)ceil((min_size - n) / 2.0);
}

// mu_t[s][x][y] = mu[s][y][x] for the scan's transposed reads (32 x 32 tiles through shared
// memory, coalesced on both sides), rows of `pitch` with zeros past n.
__global__ void __launch_bounds__(256) maps_transpose_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                             int n, int pitch) {
  __shared__ float t[32][33];
  src += (int64_t)blockIdx.z * n * n;
  dst += (int64_t)blockIdx.z * n * pitch;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int y = y0 + k, x = x0 + threadIdx.x;
    t[k][threadIdx.x] = y < n && x < n ? src[(int64_t)y * n + x] : 0.f;
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += 8) {
    const int x = x0 + k, y = y0 + threadIdx.x;
    if (x < n && y < pitch) dst[(int64_t)x * pitch + y] = t[threadIdx.x][k];
  }
}

// Row-major copy with rows of `pitch`, zeros past n.
__global__ void __launch_bounds__(256) maps_pad_kernel(const float* __restrict__ src, float* __restrict__ dst, int n,
                                                       int pitch) {
  const int64_t row = blockIdx.y + (int64_t)blockIdx.z * n;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x < pitch) dst[row * pitch + x] = x < n ? src[row * n + x] : 0.f;
}

static int copy_pitch(int n) { return (n + 3) & ~3; }

// One copy of mu in the workspace's prefix: transposed, or (n % 4 != 0) with padded rows.
static size_t copy_bytes(const cct_maps_desc* d) {
  const size_t b = (size_t)d->n * copy_pitch(d->n) * sizeof(float) * d->n_slices;
  return (b + 255) & ~(size_t)255;
}

// Transposed (and padded) copies of mu at *work, which moves past them.
static void launch_copies(const cct_maps_desc* d, const float* mu, char** work, const float** mu_t, const float** mu_p,
                          cudaStream_t st) {
  const int n = d->n, pitch = copy_pitch(n), t = (n + 31) / 32;
  float* dst = reinterpret_cast<float*>(*work);
  maps_transpose_kernel<<<dim3(t, t, d->n_slices), dim3(32, 8), 0, st>>>(mu, dst, n, pitch);
  *mu_t = dst;
  *work += copy_bytes(d);
  if (pitch != n) {
    dst = reinterpret_cast<float*>(*work);
    maps_pad_kernel<<<dim3((pitch + 255) / 256, n, d->n_slices), 256, 0, st>>>(mu, dst, n, pitch);
    *mu_p = dst;
    *work += copy_bytes(d);
  }
}

// Copies take two or four launches of ~2 us each, which small sets do not repay: one angle of 33^2 x 4 slices
// 16.4 us (40 with the host's launches) with copies and 11.9 (29) in place, 16 angles of 64^2 18.4 (37) and 20.1
// (31), one angle of 128^2 19.2 (35) and 29.1 (33), of 256^2 26.6 and 50.
constexpr int COPIES_PAY_N = 128;
constexpr int64_t COPIES_PAY_ELEMENTS = 262144;  // of W, over all entries

// Entries per pass and whether the workspace also holds the copies of `volumes` attenuation volumes at
// its start: they are used when, after them, at least half the entries of a pass without them fit.
static int plan_pass(const cct_maps_desc* d, size_t work_bytes, int64_t per_entry, int entries, int volumes,
                     size_t* prefix) {
  const bool pay = d->n >= COPIES_PAY_N || per_entry / (int64_t)sizeof(float) * entries >= COPIES_PAY_ELEMENTS;
  const int copies = pay ? volumes * (copy_pitch(d->n) != d->n ? 2 : 1) : 0;
  const int64_t plain = std::min<int64_t>((int64_t)work_bytes / per_entry, entries);
  const size_t tb = (size_t)copies * copy_bytes(d);
  const int64_t with_t = work_bytes > tb ? std::min<int64_t>((int64_t)(work_bytes - tb) / per_entry, entries) : 0;
  if (copies > 0 && with_t >= 1 && 2 * with_t >= plain) {
    *prefix = tb;
    return (int)with_t;
  }
  *prefix = 0;
  return (int)plain;
}

int64_t maps_bytes_per_angle(const cct_maps_desc* d) {
  const int e = padded_edge(d->n);
  const int64_t P = d->n + 2 * e;
  const int64_t jobs = (d->has_in ? 1 : 0) + (d->has_out ? (int64_t)d->n_det * d->n_sub : 0);
  return jobs * (P * P + P) * (int64_t)sizeof(float) * d->n_slices;  // W planes + partner constants
}

template <bool PAIRS>
static void launch_scan(const MapsPass& p, int jobs, int slices, cudaStream_t st) {
  (void)ensure_dynamic_smem<maps_scan_kernel<PAIRS>>((int)SCAN_SMEM);  // without it the launch fails and reports
  maps_scan_kernel<PAIRS><<<dim3((p.P + SCAN_COLS - 1) / SCAN_COLS, jobs, slices), SCAN_THREADS, SCAN_SMEM, st>>>(p);
}

// Quarter-turn quads: per pass, the incident fields of 2 entries per quad (one job each, so a quad
// takes the workspace of one entry with incident and emitted jobs), then one quad resample.
static int launch_maps_quads(const cct_maps_desc* d, const float* mu_in, void* maps, void* work, size_t work_bytes,
                             cudaStream_t st) {
  const int e = padded_edge(d->n);
  const int P = d->n + 2 * e;
  const int64_t per_quad = 2 * ((int64_t)P * P + P) * (int64_t)sizeof(float) * d->n_slices;
  size_t prefix = 0;
  int per_pass = plan_pass(d, work_bytes, per_quad, d->n_quads, 1, &prefix);
  if (per_pass < 1) return CCT_ERR_VALUE;
  per_pass = std::min(per_pass, 65535 / 2);
  MapsPass p;
  p.mu_in_t = p.mu_out_t = p.mu_in_p = p.mu_out_p = nullptr;
  p.pitch = copy_pitch(d->n);
  if (prefix > 0) {
    char* w = reinterpret_cast<char*>(work);
    launch_copies(d, mu_in, &w, &p.mu_in_t, &p.mu_in_p, st);
    work = w;
  }
  p.n = d->n; p.P = P; p.e = e; p.n_det = 1; p.n_sub = 1;
  p.has_in = 1; p.has_out = 0; p.maps_dtype = d->maps_dtype; p.n_angles = d->n_angles;
  p.jobs_per_angle = 1;
  p.rot_in = d->rot_in; p.rot_out = d->rot_out; p.pairs = d->pairs; p.mu_in = mu_in; p.mu_out = nullptr;
  p.quads = d->quads; p.emitted_scale = d->emitted_scale; p.n_entries = d->n_entries;
  p.work = reinterpret_cast<float*>(work); p.maps = maps;
  p.kcol = p.work + (int64_t)2 * per_pass * (int64_t)P * P * d->n_slices;
  const int tiles = (d->n + RS_TILE - 1) / RS_TILE;
  for (int q0 = 0; q0 < d->n_quads; q0 += per_pass) {
    const int nq = std::min(per_pass, d->n_quads - q0);
    p.a0 = q0;
    p.na = 2 * nq;
    launch_scan<true>(p, p.na, d->n_slices, st);
    maps_resample_quad_kernel<<<dim3((unsigned)(tiles * tiles), nq, d->n_slices), 256, 0, st>>>(p);
  }
  return CCT_OK;
}

int launch_maps(const cct_maps_desc* d, const float* mu_in, const float* mu_out, void* maps, void* work,
                size_t work_bytes, cudaStream_t st) {
  const int e = padded_edge(d->n);
  const int P = d->n + 2 * e;
  const int64_t per_angle = maps_bytes_per_angle(d);
  const int entries = d->pairs != nullptr ? d->n_entries : d->n_angles;
  if (entries < 1 || entries > d->n_angles) return CCT_ERR_VALUE;
  if (d->quads != nullptr) return launch_maps_quads(d, mu_in, maps, work, work_bytes, st);
  // copies of mu_in and of a distinct mu_out
  const bool out_own = d->has_out && (!d->has_in || mu_out != mu_in);
  const int copies = (d->has_in ? 1 : 0) + (out_own ? 1 : 0);
  size_t prefix = 0;
  int per_pass = plan_pass(d, work_bytes, per_angle, entries, copies, &prefix);
  if (per_pass < 1) return CCT_ERR_VALUE;
  // the scan grid's y dimension is entries x jobs (at most 65535): small slices with a large
  // workspace take more passes instead
  const int jobs = (d->has_in ? 1 : 0) + (d->has_out ? d->n_det * d->n_sub : 0);
  per_pass = std::max(1, std::min(per_pass, 65535 / std::max(1, jobs)));
  if ((int64_t)jobs > 65535) return CCT_ERR_VALUE;
  MapsPass p;
  p.mu_in_t = p.mu_out_t = p.mu_in_p = p.mu_out_p = nullptr;
  p.pitch = copy_pitch(d->n);
  if (prefix > 0) {
    char* w = reinterpret_cast<char*>(work);
    if (d->has_in) launch_copies(d, mu_in, &w, &p.mu_in_t, &p.mu_in_p, st);
    if (out_own) {
      launch_copies(d, mu_out, &w, &p.mu_out_t, &p.mu_out_p, st);
    } else if (d->has_out) {
      p.mu_out_t = p.mu_in_t;
      p.mu_out_p = p.mu_in_p;
    }
    work = w;
  }
  p.n = d->n; p.P = P; p.e = e; p.n_det = d->n_det; p.n_sub = d->n_sub;
  p.has_in = d->has_in; p.has_out = d->has_out; p.maps_dtype = d->maps_dtype; p.n_angles = d->n_angles;
  p.jobs_per_angle = (d->has_in ? 1 : 0) + (d->has_out ? d->n_det * d->n_sub : 0);
  p.rot_in = d->rot_in; p.rot_out = d->rot_out; p.pairs = d->pairs; p.mu_in = mu_in; p.mu_out = mu_out;
  p.quads = nullptr; p.emitted_scale = 0.f; p.n_entries = entries;
  p.work = reinterpret_cast<float*>(work); p.maps = maps;
  p.kcol = p.work + (int64_t)per_pass * p.jobs_per_angle * (int64_t)P * P * d->n_slices;
  for (int a0 = 0; a0 < entries; a0 += per_pass) {
    p.a0 = a0;
    p.na = std::min(per_pass, entries - a0);
    if (p.pairs != nullptr) {
      launch_scan<true>(p, p.na * p.jobs_per_angle, d->n_slices, st);
    } else {
      launch_scan<false>(p, p.na * p.jobs_per_angle, d->n_slices, st);
    }
    const int tiles = (d->n + RS_TILE - 1) / RS_TILE;
    const dim3 g2((unsigned)(tiles * tiles), p.na, d->n_slices);
    const size_t smem = 6 * p.jobs_per_angle * sizeof(float);
    if (p.pairs != nullptr) {
      maps_resample_kernel<true><<<g2, 256, smem, st>>>(p);
    } else {
      maps_resample_kernel<false><<<g2, 256, smem, st>>>(p);
    }
  }
  return CCT_OK;
}

int read_scan_error(int clear, int* value) {
  cudaError_t e = cudaMemcpyFromSymbol(value, g_scan_overflow, sizeof(int));
  if (e == cudaSuccess && clear) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_scan_overflow, &zero, sizeof(int));
  }
  return (int)e;
}

}  // namespace cct
