// IPM deposition: each lens-plane cell maps to two source-plane triangles whose
// image-plane area is spread over the pixels they overlap, in proportion to the
// overlap area.
//
// Semantics of the reference (ipm_functions.cuh:168-216 and
// Polygon::allocate_area_among_pixels, polygon.cuh:349-467): triangles
// (y0,y1,y2) and (y2,y3,y0) from the cell corners; skip |A| >= 1e4 * cell
// area; route by the sign of A to the minima (A < 0) or saddle map when
// parities are kept; every pixel of the map receives
// factor * |A ∩ pixel| / |A|.
//
// How, differently by design:
//   * the overlap of a triangle with a pixel is computed directly from
//     Green's theorem instead of by successive polygon clips: the edges are
//     clipped once per row strip, and the pixels of the row are then visited
//     column line by column line, each edge and the top chord being clamped to
//     the next line only once (deposit_row): register-only arithmetic, no
//     polygon arrays;
//   * rows of a triangle are independent work items; a warp expands the rows
//     of its 64 triangles and shares them out 32 at a time;
//   * pixels inside both the bottom and the top chord of a row strip are fully
//     covered (area exactly 1) and are added as a run through a per-row
//     difference array;
//   * coordinates are relative to an integer origin at the triangle's
//     lower-left pixel; the map accumulates unsigned 64-bit fixed point (2^32
//     per unit) with integer atomics, so the result does not depend on thread
//     order: given the same corner positions the map is bit-exact.
// Every floating-point operation is an explicitly rounded intrinsic (fused
// multiply-adds only where written, no contraction by the compiler), so a host
// implementation with the same operation sequence reproduces the map bit for
// bit.
#pragma once
#include "common.cuh"

#include <algorithm>
#include <limits>

namespace irsb {

template <typename D>
struct RN;
template <>
struct RN<float> {
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float div(float a, float b) { return __fdiv_rn(a, b); }
  static __device__ __forceinline__ float rcp(float a) { return __frcp_rn(a); }
  static __device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
  static __device__ __forceinline__ float min(float a, float b) { return fminf(a, b); }
  static __device__ __forceinline__ float max(float a, float b) { return fmaxf(a, b); }
  // clamped to [0, 1], NaN to 0 (the multiplication's saturating form)
  static __device__ __forceinline__ float mul_sat(float a, float b) { return __saturatef(__fmul_rn(a, b)); }
  static __device__ __forceinline__ int floor_int(float a) { return __float2int_rd(a); }
  static __device__ __forceinline__ int ceil_int(float a) { return __float2int_ru(a); }
  static __device__ __forceinline__ unsigned long long to_fix(float a) {
    return (unsigned long long)__float2ll_rn(a);
  }
};
template <>
struct RN<double> {
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
  static __device__ __forceinline__ double rcp(double a) { return __drcp_rn(a); }
  static __device__ __forceinline__ double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
  static __device__ __forceinline__ double min(double a, double b) { return a < b ? a : b; }
  static __device__ __forceinline__ double max(double a, double b) { return a > b ? a : b; }
  static __device__ __forceinline__ double mul_sat(double a, double b) {
    const double v = __dmul_rn(a, b);
    return v > 0.0 ? (v < 1.0 ? v : 1.0) : 0.0;
  }
  static __device__ __forceinline__ int floor_int(double a) { return __double2int_rd(a); }
  static __device__ __forceinline__ int ceil_int(double a) { return __double2int_ru(a); }
  static __device__ __forceinline__ unsigned long long to_fix(double a) {
    return (unsigned long long)__double2ll_rn(a);
  }
};

// Fire-and-forget add to a map word in global memory (PTX red): the adding
// thread never reads the word back, so no old value has to travel back to it
// (a plain atomicAdd on these generic pointers compiles to a returning atom).
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v) {
  asm volatile("red.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(v) : "memory");
}

template <typename D>
__device__ __forceinline__ D dabs(D a) {
  return a < D(0) ? -a : a;
}

// Output of the deposition: per-pixel fixed-point pieces plus a per-row
// difference array for runs of fully covered pixels (row stride npx + 1).
struct DepositMaps {
  unsigned long long* acc;   // [npy][npx] boundary pieces
  unsigned long long* diff;  // [npy][npx + 1] span starts (+q) and ends (-q), modulo 2^64
};

// A triangle prepared for deposition: CCW vertices relative to the integer
// origin (ox, oy), per-edge reciprocals, fixed-point scale and target map.
template <typename D>
struct Tri {
  D x[3], y[3];     // CCW, relative to (ox, oy)
  D idy[3];         // 1 / (y[k+1] - y[k]) (infinite for a zero difference)
  D sl[3];          // (y[k+1] - y[k]) * (1 / |x[k+1] - x[k]|); 0 for a vertical edge or an overflow
  D scale;          // factor * 2^32 / |area|
  int ox, oy;
  int rlo, nrows;   // first row (relative) and number of rows to visit
  int map;          // 0 total, 1 minima, 2 saddles
  int single;       // 1: the triangle lies inside one map pixel, (ox, oy)
};

template <typename D>
__device__ __forceinline__ D rcp_or_zero(D v) {
  return v != D(0) ? RN<D>::rcp(v) : D(0);  // correctly rounded 1 / v
}

// Integer part (floor) of a pixel coordinate: the sum v + 1.5 * 2^52, rounded
// down, has it in its low word while |v| < 2^31 (two FP64 additions' worth of
// work where floor and the conversion to int take the slow conversion pipe).
// `far` collects the coordinates beyond that, and NaN.
constexpr double kFloorMagic = 6755399441055744.0;
__device__ __forceinline__ int floor_low(double v, unsigned& far) {
  const double t = __dadd_rd(v, kFloorMagic);
  const int n = __double2loint(t);
  far |= unsigned(__double2hiint(t) ^ (0x43380000 + (n >> 31)));
  return n;
}
// The same for any value: beyond the range of int its end, NaN as +inf.
__device__ __forceinline__ int floor_clamped(double v) {
  return v < -2.0e9 ? -2000000000 : (v < 2.0e9 ? __double2int_rd(v) : 2000000000);
}
// n as a double, exactly (the low word of n + 1.5 * 2^52).
__device__ __forceinline__ double int_as_double(int n) {
  return __dsub_rn(__hiloint2double(0x43380000 + (n >> 31), n), kFloorMagic);
}

// A cell corner in absolute pixel coordinates (row axis flipped) and the
// integer parts of its coordinates.
struct Corner {
  double2 p;
  int nx, ny;
};

// Triangle (a, b, c) -> Tri without its reciprocals and scale (setup_tail), or
// nrows = 0 when it deposits nothing; scale holds the triangle's area. Tests
// of the reference (ipm_functions.cuh:170-193, polygon.cuh:351-372): NaN
// corner and |A| >= 1e4 * factor (both fail the comparison of A), zero area,
// entirely outside the map.
template <typename D>
__device__ __forceinline__ Tri<D> setup_head(const Corner& a, const Corner& b, const Corner& c, D factor, int npx,
                                             int npy, bool parities) {
  Tri<D> t;
  t.nrows = 0;
  t.rlo = 0;
  t.ox = t.oy = 0;
  t.map = 0;
  t.single = 0;
  t.scale = D(0);
  for (int k = 0; k < 3; k++) t.x[k] = t.y[k] = t.sl[k] = t.idy[k] = D(0);
  const int ox = min(a.nx, min(b.nx, c.nx)), oy = min(a.ny, min(b.ny, c.ny));
  if (!(ox > -1000000000 && ox < 1000000000 && oy > -1000000000 && oy < 1000000000)) return t;
  const double fx = int_as_double(ox), fy = int_as_double(oy);
  D x0 = D(a.p.x - fx), y0 = D(a.p.y - fy), x1 = D(b.p.x - fx), y1 = D(b.p.y - fy), x2 = D(c.p.x - fx),
    y2 = D(c.p.y - fy);
  // shoelace, as Poly::area
  D s = D(0);
  s = RN<D>::add(s, RN<D>::fma(RN<D>::sub(y1, y0), x0, -RN<D>::mul(RN<D>::sub(x1, x0), y0)));
  s = RN<D>::add(s, RN<D>::fma(RN<D>::sub(y2, y1), x1, -RN<D>::mul(RN<D>::sub(x2, x1), y1)));
  s = RN<D>::add(s, RN<D>::fma(RN<D>::sub(y0, y2), x2, -RN<D>::mul(RN<D>::sub(x0, x2), y2)));
  D A = RN<D>::mul(s, D(0.5));  // the correctly rounded s / 2, as a division gives
  const D whole = dabs(A);
  if (!(whole < RN<D>::mul(D(10000), factor)) || whole == D(0)) return t;
  // x and y are >= 0 and one of each is 0 up to rounding, so the triangle's
  // lowest column and row are ox and oy
  if (ox >= npx || oy >= npy) return t;
  const D mxx = RN<D>::max(RN<D>::max(x0, x1), x2), mxy = RN<D>::max(RN<D>::max(y0, y1), y2);
  if (ox < 0 && mxx <= D(-ox)) return t;
  if (oy < 0 && mxy <= D(-oy)) return t;
  t.map = parities ? (A < D(0) ? 1 : 2) : 0;
  if (A < D(0)) {  // make counter-clockwise
    D tx = x1, ty = y1;
    x1 = x2;
    y1 = y2;
    x2 = tx;
    y2 = ty;
  }
  t.x[0] = x0;
  t.y[0] = y0;
  t.x[1] = x1;
  t.y[1] = y1;
  t.x[2] = x2;
  t.y[2] = y2;
  t.scale = whole;  // setup_tail turns it into the fixed-point scale
  t.ox = ox;
  t.oy = oy;
  const int rlo = oy < 0 ? -oy : 0;
  const int rhi = min(RN<D>::floor_int(mxy), npy - 1 - oy);
  t.rlo = rlo;
  t.nrows = rhi >= rlo ? rhi - rlo + 1 : 0;
  // inside one pixel of the map: all its area goes there
  t.single = (t.nrows == 1 && mxx < D(1) && mxy < D(1) && ox >= 0) ? 1 : 0;
  return t;
}

// Edge reciprocals, slopes and the fixed-point scale of a triangle that
// deposits row by row (nrows > 0, not single).
template <typename D>
__device__ __forceinline__ void setup_tail(Tri<D>& t, D factor) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int j = k == 2 ? 0 : k + 1;
    const D dx = RN<D>::sub(t.x[j], t.x[k]), dy = RN<D>::sub(t.y[j], t.y[k]);
    t.idy[k] = RN<D>::rcp(dy);
    const D g = RN<D>::mul(dy, rcp_or_zero(dabs(dx)));
    t.sl[k] = dabs(g) <= std::numeric_limits<D>::max() ? g : D(0);
  }
  t.scale = RN<D>::div(RN<D>::mul(factor, D(kFixScale)), t.scale);
}

// Shared-memory staging of the 64 triangles of a warp's 32 cells that go row
// by row (one array per field: lane k touches word k, no bank conflicts).
template <typename D>
struct TriSlots {
  D x[3][64], y[3][64], scale[64];  // scale: the area until setup_tail
  D idy[3][64], sl[3][64];          // from setup_tail
  int ox[64], oy[64], rlo[64], nrows[64], map[64];
  __device__ __forceinline__ void put(int k, const Tri<D>& t) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      x[q][k] = t.x[q];
      y[q][k] = t.y[q];
    }
    scale[k] = t.scale;
    ox[k] = t.ox;
    oy[k] = t.oy;
    rlo[k] = t.rlo;
    nrows[k] = t.nrows;
    map[k] = t.map;
  }
  __device__ __forceinline__ void put_tail(int k, const Tri<D>& t) {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      idy[q][k] = t.idy[q];
      sl[q][k] = t.sl[q];
    }
    scale[k] = t.scale;
  }
  __device__ __forceinline__ void get_head(int k, Tri<D>& t) const {
#pragma unroll
    for (int q = 0; q < 3; q++) {
      t.x[q] = x[q][k];
      t.y[q] = y[q][k];
    }
    t.scale = scale[k];
    t.ox = ox[k];
    t.oy = oy[k];
    t.rlo = rlo[k];
    t.map = map[k];
  }
  __device__ __forceinline__ void get(int k, Tri<D>& t) const {
    get_head(k, t);
#pragma unroll
    for (int q = 0; q < 3; q++) {
      t.idy[q] = idy[q][k];
      t.sl[q] = sl[q][k];
    }
  }
};
constexpr int kDepositWarps = 2;  // warps per CTA of the deposition kernels
constexpr int kDepositThreads = kDepositWarps * 32;
// Order of the deposition's work units (32-cell chunks, or blocks of them) over
// at most 256 CTAs per SM. CTAs start in order, so about kWave warps are at work
// at a time; the warps of such a wave share one stretch of the lattice, striding
// through it (neighbouring warps on neighbouring units, each warp's units spread
// over the stretch, which evens out the cells' cost). The stretch's images share
// a part of the map, so that most adds meet their words in L2 (a middle band of the
// lattice below takes 15 % of the memory bandwidth, corners included).
// With the warps striding over the whole lattice every wave swept it end to end,
// and its adds missed L2 where the fixed-point map is larger: 1.0e9 cells into
// 4096^2 pixels (268 MB of map words) took 168 ms, now 81.5 (B200; 84 to 85 in
// other fields, where it was 175); with consecutive units per warp 92 ms, but 5.3
// against 4.9 ms for 8.8e7 cells into 2000^2 pixels. Small CTAs retire as soon as
// their two warps are done, which keeps the SMs full to the end.
struct DepositOrder {
  long long first, stride;  // this warp's first unit and the step to its next
  int count;                // units (those past the last unit are absent)
};
template <typename D>
__device__ __forceinline__ DepositOrder deposit_order(long long nunits) {
  constexpr long long kWave = 148LL * (sizeof(D) == 4 ? 16 : 8) * kDepositWarps;  // resident warps
  const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long count = (nunits + nwarps - 1) / nwarps, wave = w / kWave, in = w - wave * kWave;
  const long long size = nwarps - wave * kWave < kWave ? nwarps - wave * kWave : kWave;
  return {wave * kWave * count + in, size, int(count)};
}
inline int deposit_grid(long long nchunks) {
  const long long ctas = (nchunks + kDepositWarps - 1) / kDepositWarps, cap = 148LL * 256;
  return int(ctas < 1 ? 1 : (ctas > cap ? cap : ctas));
}

// One row of a triangle, the strip y in [rb, rt = rb + 1]: the run of fully
// covered pixels goes to the difference array, the other overlapped pixels get
// their coverage from Green's theorem, area = -(sum over the boundary of the
// integral of (y - rb) dx).
//
//   Strip segments: edge k runs from (x1, y1) to (x2, y2); its parameters at
//   y = rb and y = rt, clamped to [0, 1] (saturating multiplications), bound
//   the piece inside the strip. An edge that misses the strip is clamped to one
//   parameter and becomes a point, which adds nothing. A horizontal edge has an
//   infinite reciprocal: the products are -inf, NaN (clamped to 0) or +inf and
//   give (0, 1) for y1 in [rb, rt) and a point elsewhere, so an edge lying on
//   the line between two rows is counted once (by the top chord of the row
//   below).
//   Chords: x-extent of the triangle on the lines y = rb and y = rt (an edge
//   reaching the line contributes its crossing, x1 + ((y - y1) / dy) dx, or
//   both ends when it lies on the line). The top chord matters only when the
//   triangle reaches rt, the bottom one only when it spans the strip.
//   Pixels: for every column line c the position P = c clamped to the segment
//   and the (signed) height V there; the pixel between two lines adds the
//   trapezoid (P' - P)(V + V') of every segment and the top chord's length
//   between the lines. A line's values serve the pixels on both sides, so a
//   pixel costs one clamp and one height per edge. ya and sl carry the sign of
//   the edge's direction, so that P never decreases.
//
// Every value is the one that clamping both ends of each segment to each
// pixel gives (the earlier form and the host restatement): the products with
// -1/2 are exact, a sum of two heights does not depend on their order, and a
// sign carried through a rounded product or sum is exact.
//
// Bound by instruction issue (FP32 and ALU pipes). Against the form that
// clamped both segment ends for every pixel and computed both chords of every
// row: 8.76e7 cells of a 2000^2 map 6.36 -> 4.91 ms (FP32), 4.1e7 cells 2.61 ->
// 2.45 ms (FP64), maps bit-identical (B200); 4.63 and 2.28 ms with the triangles
// read back from the slots (deposit_rows_warp) and deposit_order.
template <typename D>
__device__ __forceinline__ void deposit_row(const Tri<D>& t, int r, int npx, const DepositMaps& M) {
  const D rb = D(r), rt = D(r + 1);
  D lo[3], hi[3], xa[3], ya[3];
  D xlo = std::numeric_limits<D>::infinity(), xhi = -xlo;
  bool any = false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int j = k == 2 ? 0 : k + 1;
    const D x1 = t.x[k], y1 = t.y[k];
    const D dx = RN<D>::sub(t.x[j], x1), dy = RN<D>::sub(t.y[j], y1);
    const D sa = RN<D>::mul_sat(RN<D>::sub(rb, y1), t.idy[k]), sb = RN<D>::mul_sat(RN<D>::sub(rt, y1), t.idy[k]);
    const D t0 = RN<D>::min(sa, sb), t1 = RN<D>::max(sa, sb);
    const D a = RN<D>::fma(t0, dx, x1), b = RN<D>::fma(t1, dx, x1);
    const D y = RN<D>::sub(RN<D>::fma(t0, dy, y1), rb);
    xa[k] = a;
    ya[k] = dx < D(0) ? -y : y;
    lo[k] = RN<D>::min(a, b);
    hi[k] = RN<D>::max(a, b);
    if (t0 < t1) {
      any = true;
      xlo = RN<D>::min(xlo, lo[k]);
      xhi = RN<D>::max(xhi, hi[k]);
    }
  }
  if (!any) return;
  const int cmap_lo = -t.ox, cmap_hi = npx - 1 - t.ox;  // columns inside the map (relative)
  const int cmin = max(RN<D>::floor_int(xlo), cmap_lo), cmax = min(RN<D>::floor_int(xhi), cmap_hi);
  if (cmin > cmax) return;
  D ct0 = D(0), ct1 = D(0);  // top chord
  int fa = 1, fb = 0;        // full run [fa, fb)
  if (RN<D>::max(RN<D>::max(t.y[0], t.y[1]), t.y[2]) >= rt) {
    auto chord = [&](D yk, D& c0, D& c1) {
      c0 = std::numeric_limits<D>::infinity();
      c1 = -c0;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int j = k == 2 ? 0 : k + 1;
        const D x1 = t.x[k], y1 = t.y[k], x2 = t.x[j], y2 = t.y[j];
        if ((y1 <= yk && yk <= y2) || (y2 <= yk && yk <= y1)) {
          D p = x1, q = x2;
          if (y1 != y2) p = q = RN<D>::fma(RN<D>::mul(RN<D>::sub(yk, y1), t.idy[k]), RN<D>::sub(x2, x1), x1);
          c0 = RN<D>::min(c0, RN<D>::min(p, q));
          c1 = RN<D>::max(c1, RN<D>::max(p, q));
        }
      }
    };
    chord(rt, ct0, ct1);
    if (RN<D>::min(RN<D>::min(t.y[0], t.y[1]), t.y[2]) <= rb) {
      D cb0, cb1;
      chord(rb, cb0, cb1);
      fa = max(RN<D>::ceil_int(RN<D>::max(cb0, ct0)), cmap_lo);
      fb = min(RN<D>::floor_int(RN<D>::min(cb1, ct1)), cmap_hi + 1);
    }
  }
  const long long row = (long long)t.oy + r;
  unsigned long long* acc = M.acc + row * npx + t.ox;
  const bool run = fa < fb;
  if (run) {
    const unsigned long long q = RN<D>::to_fix(t.scale);
    unsigned long long* diff = M.diff + row * ((long long)npx + 1) + t.ox;
    red_add(diff + fa, q);
    red_add(diff + fb, (unsigned long long)(0ULL - q));
  }
  D P[3], V[3], T;
  auto line = [&](int c) {
    const D x = D(c);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      P[k] = RN<D>::min(RN<D>::max(x, lo[k]), hi[k]);
      V[k] = RN<D>::fma(RN<D>::sub(P[k], xa[k]), t.sl[k], ya[k]);
    }
    T = RN<D>::min(RN<D>::max(x, ct0), ct1);
  };
  line(cmin);
  for (int c = cmin; c <= cmax; c++) {
    if (run && c == fa) {
      c = fb;
      if (c > cmax) break;
      line(c);
    }
    const D x = D(c + 1);
    D s = D(0);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const D Pn = RN<D>::min(RN<D>::max(x, lo[k]), hi[k]);
      const D Vn = RN<D>::fma(RN<D>::sub(Pn, xa[k]), t.sl[k], ya[k]);
      s = RN<D>::fma(RN<D>::sub(Pn, P[k]), RN<D>::add(V[k], Vn), s);
      P[k] = Pn;
      V[k] = Vn;
    }
    const D Tn = RN<D>::min(RN<D>::max(x, ct0), ct1);
    const D a = RN<D>::fma(s, D(-0.5), RN<D>::sub(Tn, T));
    T = Tn;
    if (a > D(0)) {
      const unsigned long long q = RN<D>::to_fix(RN<D>::mul(a, t.scale));
      if (q) red_add(acc + c, q);
    }
  }
}

// The rows of the staged triangles [k0, k0 + 32) of a warp, one triangle per lane
// (n staged in all): each lane finishes its own triangle (setup_tail) and
// deposits its first row; the warp then scans the counts of the remaining rows
// and works through those (triangle, row) items 32 at a time, each lane finding
// its item's owner by a binary search over the scan and reading the triangle
// from the slots (consecutive words: no bank conflicts), so a triangle with many
// rows is spread over the warp instead of holding one lane, and no triangle is
// held in registers across the rows.
template <typename D>
__device__ __forceinline__ void deposit_rows_warp(TriSlots<D>& stage, int k0, int n, D factor, int npx,
                                                  const DepositMaps& m_total, const DepositMaps& m_min,
                                                  const DepositMaps& m_sad) {
  const int lane = threadIdx.x & 31;
  int extra = 0;
  if (k0 + lane < n) {
    Tri<D> t;
    stage.get_head(k0 + lane, t);
    setup_tail(t, factor);
    extra = stage.nrows[k0 + lane] - 1;
    if (extra > 0) stage.put_tail(k0 + lane, t);
    deposit_row<D>(t, t.rlo, npx, t.map == 0 ? m_total : (t.map == 1 ? m_min : m_sad));
  }
  int incl = extra;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  __syncwarp();
  for (int it0 = 0; it0 < total; it0 += 32) {
    const int item = it0 + lane;
    int lo = 0, hi = 31;  // owner: first lane whose inclusive count exceeds item
#pragma unroll
    for (int step = 0; step < 5; step++) {
      int mid = (lo + hi) >> 1;
      int v = __shfl_sync(0xffffffffu, incl, mid);
      if (v > item) hi = mid;
      else lo = mid + 1;
    }
    const int owner = lo & 31;
    const int before = __shfl_sync(0xffffffffu, incl - extra, owner);
    if (item < total) {
      Tri<D> t;
      stage.get(k0 + owner, t);
      deposit_row<D>(t, t.rlo + 1 + (item - before), npx, t.map == 0 ? m_total : (t.map == 1 ? m_min : m_sad));
    }
  }
}

// The 32 cells [base, base + 32) of an ncx-wide lattice whose corner rows are
// vx apart (whole warp; lanes past ncells idle).
template <typename D>
__device__ __forceinline__ void deposit_warp_cells(const double2* __restrict__ verts, long long ncx, long long vx,
                                                   long long ncells, long long base, D factor, int npx, int npy,
                                                   const DepositMaps& m_total, const DepositMaps& m_min,
                                                   const DepositMaps& m_sad, int parities, TriSlots<D>& stage,
                                                   long long vstep = 1, double ox = 0.0, double oy = 0.0,
                                                   double inv_scale = 1.0) {
  const int lane = threadIdx.x & 31;
  const long long c = base + lane;
  double2 y0 = make_double2(0, 0), y1 = y0, y2 = y0, y3 = y0;
  if (c < ncells) {
    long long j, i;
    if (((c | ncx) >> 31) == 0) {  // 32-bit division where it suffices
      const unsigned jj = unsigned(c) / unsigned(ncx);
      j = jj;
      i = unsigned(c) - jj * unsigned(ncx);
    } else {
      j = c / ncx;
      i = c - j * ncx;
    }
    y0 = verts[((j + 1) * vx + (i + 1)) * vstep];  // z + rhs
    y1 = verts[((j + 1) * vx + i) * vstep];        // z - conj(rhs)
    y2 = verts[(j * vx + i) * vstep];              // z - rhs
    y3 = verts[(j * vx + (i + 1)) * vstep];        // z + conj(rhs)
    if (ox != 0.0 || oy != 0.0) {  // origin of the piece's map in the positions' pixel frame
      y0.x -= ox, y1.x -= ox, y2.x -= ox, y3.x -= ox;
      y0.y -= oy, y1.y -= oy, y2.y -= oy, y3.y -= oy;
    }
    if (inv_scale != 1.0) {  // the piece's map has pixels 1 / inv_scale wide
      y0.x *= inv_scale, y1.x *= inv_scale, y2.x *= inv_scale, y3.x *= inv_scale;
      y0.y *= inv_scale, y1.y *= inv_scale, y2.y *= inv_scale, y3.y *= inv_scale;
    }
  }
  // a cell whose four corners all lie beyond one edge of the map deposits
  // nothing (setup_head would reject both its triangles); the high words decide
  // (a corner within 2^-20 of the far edge counts as inside)
  const int hx0 = __double2hiint(y0.x), hx1 = __double2hiint(y1.x), hx2 = __double2hiint(y2.x),
            hx3 = __double2hiint(y3.x);
  const int hy0 = __double2hiint(y0.y), hy1 = __double2hiint(y1.y), hy2 = __double2hiint(y2.y),
            hy3 = __double2hiint(y3.y);
  const bool live = c < ncells && (hx0 & hx1 & hx2 & hx3) >= 0 && (hy0 & hy1 & hy2 & hy3) >= 0 &&
                    min(min(hx0, hx1), min(hx2, hx3)) <= __double2hiint(double(npx)) &&
                    min(min(hy0, hy1), min(hy2, hy3)) <= __double2hiint(double(npy));
  if (__ballot_sync(0xffffffffu, live) == 0u) return;
  Corner k0, k1, k2, k3;
  k0.p = y0, k1.p = y1, k2.p = y2, k3.p = y3;
  {
    unsigned far = 0;
    k0.nx = floor_low(y0.x, far), k1.nx = floor_low(y1.x, far), k2.nx = floor_low(y2.x, far),
    k3.nx = floor_low(y3.x, far);
    k0.ny = floor_low(y0.y, far), k1.ny = floor_low(y1.y, far), k2.ny = floor_low(y2.y, far),
    k3.ny = floor_low(y3.y, far);
    if (far) {
      k0.nx = floor_clamped(y0.x), k1.nx = floor_clamped(y1.x), k2.nx = floor_clamped(y2.x),
      k3.nx = floor_clamped(y3.x);
      k0.ny = floor_clamped(y0.y), k1.ny = floor_clamped(y1.y), k2.ny = floor_clamped(y2.y),
      k3.ny = floor_clamped(y3.y);
    }
  }
  // each half's head: a triangle inside one pixel deposits at once, the
  // others are staged in the warp's slots, compacted in lane order
  const unsigned lt = (1u << lane) - 1u;
  int n = 0;
#pragma unroll 1
  for (int half = 0; half < 2; half++) {
    Tri<D> h;
    h.nrows = 0;  // idle lanes (past the last cell) deposit nothing
    h.single = 0;
    if (live) {
      h = half == 0 ? setup_head<D>(k0, k1, k2, factor, npx, npy, parities != 0)
                    : setup_head<D>(k2, k3, k0, factor, npx, npy, parities != 0);
    }
    {
      // lanes in a row whose triangles fall in the same pixel add once for
      // all of them (adjacent cells of a fine lattice share pixels)
      unsigned long long* a = nullptr;
      if (h.single) a = (h.map == 0 ? m_total : (h.map == 1 ? m_min : m_sad)).acc + (long long)h.oy * npx + h.ox;
      const unsigned long long key = (unsigned long long)a;
      const unsigned long long prev = __shfl_up_sync(0xffffffffu, key, 1);
      const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || prev != key);
      if (h.single && (starts >> lane & 1u)) {
        const unsigned later = starts & ~((2u << lane) - 1u);  // lane 31: mask of all bits, none later
        const int end = later ? __ffs(later) - 1 : 32;
        red_add(a, (unsigned long long)(end - lane) * RN<D>::to_fix(RN<D>::mul(factor, D(kFixScale))));
      }
    }
    const bool cx = h.nrows > 0 && !h.single;
    const unsigned b = __ballot_sync(0xffffffffu, cx);
    if (cx) stage.put(n + __popc(b & lt), h);
    n += __popc(b);
  }
  __syncwarp();
  // the staged ones go row by row, one per lane: one round when at most 32
  // of the warp's 64 triangles need it (fine lattices), else two
  for (int k0 = 0; k0 < n; k0 += 32) deposit_rows_warp<D>(stage, k0, n, factor, npx, m_total, m_min, m_sad);
  __syncwarp();  // slots free for the warp's next cells
}

// Cells of an ncx x ncy lattice whose (ncx+1) x (ncy+1) corner positions are in
// `verts`. A warp takes 32 consecutive cells at a time (deposit_order); each lane classifies the two
// triangles of its cell (setup_head); a triangle inside one pixel is
// deposited at once; the others are staged in shared memory, compacted, and
// then get their reciprocals and scale (setup_tail) and go row by row
// (deposit_rows_warp), one per lane: one round when at most 32 of the warp's
// 64 triangles need it (fine lattices), else two.
template <typename D>
__global__ void __launch_bounds__(kDepositThreads, sizeof(D) == 4 ? 16 : 8)
    ipm_deposit_cells(const double2* __restrict__ verts, long long ncx, long long ncy, D factor, int npx, int npy,
                      DepositMaps m_total, DepositMaps m_min, DepositMaps m_sad, int parities) {
  const long long ncells = ncx * ncy;
  __shared__ TriSlots<D> slots[kDepositWarps];
  TriSlots<D>& stage = slots[threadIdx.x >> 5];
  const DepositOrder o = deposit_order<D>((ncells + 31) / 32);
  long long base = o.first * 32;
  for (int i = 0; i < o.count && base < ncells; i++, base += o.stride * 32)
    deposit_warp_cells<D>(verts, ncx, ncx + 1, ncells, base, factor, npx, npy, m_total, m_min, m_sad, parities, stage);
}

// A block of cells inside a pass of the batched (or adaptive) deposition: its
// corner rows start at `voff` in the pass's corner buffer, vstride apart.
template <typename D>
struct DepositPiece {
  long long voff;
  long long vstride;   // corner row stride (ncx + 1 for a whole lattice row)
  long long vstep;     // corner (i, j) is at (j * vstride + i) * vstep (a coarser view of a finer grid)
  double ox, oy;       // origin of the piece's map in the positions' pixel frame
  double inv_scale;    // 1 / width of the piece's map pixels in the positions' pixels
  long long ncx, ncy;  // cells
  long long chunk0;    // first 32-cell chunk of the piece in the pass
  D factor;
  int r;               // realization (map index)
};

// Batched deposition over the 32-cell chunks of all pieces of the pass, in blocks
// of 8 consecutive ones (deposit_order): a block's first piece is found by a
// binary search over chunk0 and the next chunks advance from it (one search per
// 8 chunks). Realization r accumulates into the maps at r * map_stride /
// r * diff_stride.
template <typename D>
__global__ void __launch_bounds__(kDepositThreads, sizeof(D) == 4 ? 16 : 8)
    ipm_deposit_batch(const double2* __restrict__ verts, const DepositPiece<D>* __restrict__ pieces, int npieces,
                      long long nchunks, int npx, int npy, DepositMaps maps, long long map_stride,
                      long long diff_stride) {
  __shared__ TriSlots<D> slots[kDepositWarps];
  TriSlots<D>& stage = slots[threadIdx.x >> 5];
  constexpr int K = 8;
  const DepositOrder o = deposit_order<D>((nchunks + K - 1) / K);
  long long g0 = o.first * K;
  for (int i = 0; i < o.count && g0 < nchunks; i++, g0 += o.stride * K) {
    int lo = 0, hi = npieces - 1;  // last piece with chunk0 <= g0
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (pieces[mid].chunk0 <= g0) lo = mid;
      else hi = mid - 1;
    }
    const long long gend = g0 + K < nchunks ? g0 + K : nchunks;
    for (long long g = g0; g < gend; g++) {
      while (lo + 1 < npieces && pieces[lo + 1].chunk0 <= g) lo++;
      const DepositPiece<D> pc = pieces[lo];
      const DepositMaps M{maps.acc + pc.r * map_stride, maps.diff + pc.r * diff_stride};
      deposit_warp_cells<D>(verts + pc.voff, pc.ncx, pc.vstride, pc.ncx * pc.ncy, (g - pc.chunk0) * 32, pc.factor,
                            npx, npy, M, M, M, 0, stage, pc.vstep, pc.ox, pc.oy, pc.inv_scale);
    }
  }
}

// Row prefix sum of the difference array added to the pieces: one warp per
// row, 32 columns per step with a carried running sum (integer, exact).
__global__ void ipm_resolve_rows(int npx, int npy, DepositMaps m) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int y = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; y < npy; y += warps) {
    unsigned long long carry = 0;
    const long long rs = (long long)npx + 1;
    for (int x0 = 0; x0 < npx; x0 += 32) {
      int x = x0 + lane;
      unsigned long long v = x < npx ? m.diff[y * rs + x] : 0ULL;
      for (int o = 1; o < 32; o <<= 1) {
        unsigned long long u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      v += carry;
      if (x < npx) m.acc[(long long)y * npx + x] += v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  }
}

// The row resolve and the conversion to T in one pass, for a run without
// parity maps: one warp per row, each lane 4 consecutive pixels (a
// 2000-pixel row in 16 dependent steps). The fixed-point map is still written
// (the resolved accumulators); integer sums, so both maps are those of
// ipm_resolve_rows followed by ipm_finalize.
template <typename T>
__global__ void ipm_resolve_rows_out(int npx, int npy, DepositMaps m, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const long long rs = (long long)npx + 1;
  for (int y = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; y < npy; y += warps) {
    unsigned long long carry = 0;
    for (int x0 = 0; x0 < npx; x0 += 128) {
      const int x = x0 + 4 * lane;
      unsigned long long d[4];
#pragma unroll
      for (int i = 0; i < 4; i++) d[i] = x + i < npx ? m.diff[y * rs + x + i] : 0ULL;
      d[1] += d[0];
      d[2] += d[1];
      d[3] += d[2];
      unsigned long long incl = d[3];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      const unsigned long long base = carry + (incl - d[3]);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (x + i < npx) {
          const long long k = (long long)y * npx + x + i;
          const unsigned long long v = m.acc[k] + (base + d[i]);
          m.acc[k] = v;
          out[k] = T(double(v) * kFixInv);
        }
      }
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}

// map (fixed point) -> magnification in T; with parities total = min + sad.
template <typename T>
__global__ void ipm_finalize(long long n, const unsigned long long* __restrict__ acc_total,
                             const unsigned long long* __restrict__ acc_min,
                             const unsigned long long* __restrict__ acc_sad, T* __restrict__ out_total,
                             T* __restrict__ out_min, T* __restrict__ out_sad, int parities) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    if (parities) {
      unsigned long long a = acc_min[k], b = acc_sad[k];
      out_min[k] = T(double(a) * kFixInv);
      out_sad[k] = T(double(b) * kFixInv);
      out_total[k] = T(double(a + b) * kFixInv);
    } else {
      out_total[k] = T(double(acc_total[k]) * kFixInv);
    }
  }
}

}  // namespace irsb
