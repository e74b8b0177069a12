// line.cuh -- the row-by-row walk of a ray's line (LineRay), shared by the
// forward projectors that gather through L1 (project.cu) and from shared
// memory (slab.cu).  Both run exactly these operations per row and fold the
// row sums at the same rows, so their sums agree bit for bit.
#pragma once

#include "epilogue.cuh"

namespace medimg {

// one pixel of G scans projected together (three scans take the float4 form)
template <int G>
struct Elem;
template <>
struct Elem<1> {
  using T = float;
};
template <>
struct Elem<2> {
  using T = float2;
};
template <>
struct Elem<4> {
  using T = float4;
};

// two fmaf side by side in one instruction (the same rounding)
__device__ __forceinline__ void fma_pair(float &x, float &y, float w, float a, float b) {
  uint64_t s, v, ww;
  asm("mov.b64 %0, {%1, %2};" : "=l"(s) : "f"(x), "f"(y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
  asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s) : "l"(ww), "l"(v));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(s));
}

template <int G>
__device__ __forceinline__ void fma_elem(float (&part)[G], float wt, const typename Elem<G>::T &v) {
  if constexpr (G == 1) {
    part[0] = fmaf(wt, v, part[0]);
  } else if constexpr (G == 2) {
    fma_pair(part[0], part[1], wt, v.x, v.y);
  } else {
    fma_pair(part[0], part[1], wt, v.x, v.y);
    fma_pair(part[2], part[3], wt, v.z, v.w);
  }
}

template <int G>
__device__ __forceinline__ typename Elem<G>::T zero_elem() {
  if constexpr (G == 1) return 0.f;
  else if constexpr (G == 2) return make_float2(0.f, 0.f);
  else return make_float4(0.f, 0.f, 0.f, 0.f);
}

// A ray's walk over the rows of its copy, in blocks of 32 steps (steps 0..31 of
// the copy, 32..63, ...).  A block's state depends on the ray and the block
// alone (enter()), and the block sums are folded in order into a Kahan total
// (LineTotal), so a ray's blocks may be walked by one thread after another or
// by several threads: the sums are the same bit for bit.  Row coordinates are
// relative to the middle of the kSub rows around the step (at(), called before
// each step, moves on; exact, as it only takes away from a larger number).
template <int G>
struct LineWalk {
  float e_ref, inv, slope, kv0;
  int first, last;  // steps
  float e;          // the next crossing
  float part[G];

  __device__ __forceinline__ void load(const LineRay &r) {
    e_ref = r.e_ref;
    inv = r.inv;
    slope = inv > 0.f ? __frcp_rn(inv) : 0.f;
    kv0 = r.kv0;
    first = (int)(r.rows & 0xffffu);
    last = (int)(r.rows >> 16);
  }
  __device__ __forceinline__ bool empty() const { return first > last; }
  __device__ __forceinline__ bool in_block(int blk) const { return first <= last && first >> 5 <= blk && blk <= last >> 5; }
  static constexpr int kSub = 8;
  // begins the block of steps from step0, in column c0 + the returned number
  // (negative where the line has yet to reach c0)
  __device__ __forceinline__ int enter(int step0, int n) {
    constexpr float kHalf = kSub / 2;
#pragma unroll
    for (int m = 0; m < G; m++) part[m] = 0.f;
    const float rel = e_ref - ((float)(step0 + kSub / 2) - 0.5f * (float)n);
    float k = ceilf(fmaf(-kHalf - rel, slope, -kv0));
    e = fmaf(kv0 + k, inv, rel);
    // the estimate is one off where a crossing nearly meets the block's start
    const float d = e < -kHalf ? 1.f : inv > 0.f && e - inv >= -kHalf ? -1.f : 0.f;
    k += d;
    if (d != 0.f) e = fmaf(kv0 + k, inv, rel);
    return (int)k;
  }
  // Step b of the block: the part of the row before the crossing, whether the
  // ray crosses into the next column (and, if so, the crossing after that),
  // and the sums, with a and c the pixels of the current and the next column.
  // A crossing adds inv to e: |e| stays below 4 + inv, so that up to 32 sums
  // round less than e_ref does.  Crossings' share of the error against 64 bits
  // (sinograms of noise) relative to the middle of 32 rows, 8 rows, and with
  // every crossing an fmaf of its own: 32^2 2.0e-7, 1.1e-7, 1.0e-7; 64^2
  // 1.5e-7, 9.3e-8, 8.8e-8; 512^2 1.38e-7, 1.32e-7, 1.32e-7.
  __device__ __forceinline__ void at(int b) {
    if (b > 0 && b % kSub == 0) e -= (float)kSub;
  }
  __device__ __forceinline__ float before(int b) const { return __saturatef(e - (float)(b % kSub - kSub / 2)); }
  __device__ __forceinline__ bool crosses(int b) {
    const bool x = e < (float)(b % kSub + 1 - kSub / 2);
    if (x) e += inv;
    return x;
  }
  __device__ __forceinline__ void add(float f, bool x, const typename Elem<G>::T &a, const typename Elem<G>::T &c) {
    fma_elem<G>(part, f, a);
    if (x) fma_elem<G>(part, 1.f - f, c);
  }
  __device__ __forceinline__ bool row(int b, const typename Elem<G>::T &a, const typename Elem<G>::T &c) {
    const float f = before(b);
    const bool x = crosses(b);
    add(f, x, a, c);
    return x;
  }
  // a block's step of any number: enter() or at(), as it needs; col: the column,
  // which enter() sets
  __device__ __forceinline__ void to(int step, int n, int c0, int &col) {
    if (step % kSub != 0) return;
    if ((step & 31) == 0) col = c0 + enter(step, n);
    else at(step & 31);
  }
};

// the Kahan total of a ray's block sums for one scan
struct LineTotal {
  float acc = 0.f, comp = 0.f;
  __device__ __forceinline__ void fold(float part) { kahan_add(acc, comp, part); }
};

// column c0, and the first element of a step's row in its copy
__device__ __forceinline__ int line_c0(const LineRay &r, int n, int pitch) {
  return r.off - ((r.flags & kLineSwap) ? n * pitch : 0) - kLinePad;
}
__device__ __forceinline__ int line_row_of(const LineRay &r, int step, int n) {
  return (r.flags & kLineDown) ? n - 1 - step : step;
}
// no ray: it never crosses
__device__ __forceinline__ LineRay line_none() {
  LineRay r;
  r.e_ref = 1e30f;
  r.inv = r.kv0 = r.len = 0.f;
  r.off = r.corr0 = 0;
  r.rows = 1u;
  r.flags = 0u;
  return r;
}

__device__ __forceinline__ LineRay load_line(const LineRay *p) {
  const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p)), b = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
  LineRay r;
  r.e_ref = __uint_as_float(a.x);
  r.inv = __uint_as_float(a.y);
  r.kv0 = __uint_as_float(a.z);
  r.len = __uint_as_float(a.w);
  r.off = (int)b.x;
  r.rows = b.y;
  r.corr0 = (int)b.z;
  r.flags = b.w;
  return r;
}

template <int G>
__device__ __forceinline__ float elem_of(const typename Elem<G>::T &v, int m) {
  if constexpr (G == 1) return v;
  else if constexpr (G == 2) return m == 0 ? v.x : v.y;
  else return m == 0 ? v.x : m == 1 ? v.y : m == 2 ? v.z : v.w;
}

// The sum along a line without the pixels of its corrections, from one scan's
// values (every stride-th float of the copies at pk): the walk again, pixel by
// pixel, of the rows in the grid and the parts that are not empty.
__device__ __forceinline__ float line_sum_without(const float *pk, int stride, const LineRay *rayp, const LineCorr *corr,
                                                  int n, int pitch) {
  const LineRay r = load_line(rayp);
  const bool swap = (r.flags & kLineSwap) != 0;
  const int nc = (int)(r.flags >> 8), col0 = line_c0(r, n, pitch);
  LineWalk<1> w;
  w.load(r);
  LineTotal tot;
  int col = 0;
  for (int step = w.first & ~31; step <= w.last; step++) {
    w.to(step, n, col0, col);
    const float f = w.before(step & 31);
    const bool x = w.crosses(step & 31);
    const int u = line_row_of(r, step, n);
    for (int k = 0; k < 2 && step >= w.first; k++) {
      const int c = col + k;
      const float part = k == 0 ? f : x ? 1.f - f : 0.f;
      bool use = part > 0.f && (unsigned)c < (unsigned)n;
      for (int i = 0; i < nc; i++) use = use && corr[r.corr0 + i].pix != (swap ? c * n + u : u * n + c);
      if (use) w.part[0] = fmaf(part, pk[(size_t)stride * ((swap ? n * pitch : 0) + u * pitch + kLinePad + c)], w.part[0]);
    }
    col += x ? 1 : 0;
    if (step == w.last || (step & 31) == 31) tot.fold(w.part[0]);
  }
  return (tot.acc - tot.comp) * r.len;
}

// The G scans' line integrals of a warp's rays, with their corrections, from the
// padded copies at pk.  All lanes of the warp take part.
// A ray that is no line is its corrections, hundreds of them: the warp takes
// each such ray together (512^2, 360 x 888, of whose rays 5.5 % end inside the
// grid: 224 us a projection with a lane each, 97 us so, 157 us by segments).
// A line's corrections are the last pieces that the traversal leaves out, as
// minus what the line had: where that leaves little or nothing of the sum
// (their pixels not finite, or far above the others), the line is walked again
// without them (inlined: a call cost every walk 2 % of its registers' schedule).
template <int G>
__device__ __forceinline__ void line_finish(const LineRay *rayp, bool valid, const LineCorr *__restrict__ corr,
                                            const LineTotal (&tot)[G],
                                            const typename Elem<G>::T *__restrict__ pk, int n, int pitch,
                                            float (&out)[G]) {
  const LineRay r = valid ? load_line(rayp) : line_none();
  const int lane = threadIdx.x & 31, nc = (int)(r.flags >> 8);
  const bool whole = (r.rows & 0xffffu) > r.rows >> 16;
  // pixel x*n + y in the row-major copy: x rows' padding further on
  const float rcp = __frcp_rn((float)n);
  auto value = [&](int pix) {
    const int p = pix & ~kCorrForwardOnly;
    int x = (int)((float)p * rcp);
    const int y = p - x * n;  // (x is one off at most: p is below 2^26)
    x += y >= n ? 1 : y < 0 ? -1 : 0;
    return __ldg(pk + p + x * (pitch - n) + kLinePad);
  };
  bool again = false;
#pragma unroll
  for (int m = 0; m < G; m++) out[m] = (tot[m].acc - tot[m].comp) * r.len;
  if (!whole && nc > 0) {
    float line[G];
#pragma unroll
    for (int m = 0; m < G; m++) line[m] = out[m];
    for (int k = 0; k < nc; k++) {
      const LineCorr c = corr[r.corr0 + k];
      const typename Elem<G>::T v = value(c.pix);
#pragma unroll
      for (int m = 0; m < G; m++) out[m] = fmaf(c.w, elem_of<G>(v, m), out[m]);
    }
#pragma unroll
    for (int m = 0; m < G; m++) again |= !(fabsf(line[m]) <= 1024.f * fabsf(out[m]));
    if (again)
#pragma unroll 1
      for (int m = 0; m < G; m++) {
        const float o = m == 0 ? out[0] : m == 1 ? out[G > 1 ? 1 : 0] : m == 2 ? out[G > 2 ? 2 : 0] : out[G - 1];
        const float l = m == 0 ? line[0] : m == 1 ? line[G > 1 ? 1 : 0] : m == 2 ? line[G > 2 ? 2 : 0] : line[G - 1];
        if (fabsf(l) <= 1024.f * fabsf(o)) continue;
        const float s = line_sum_without(reinterpret_cast<const float *>(pk) + m, G, rayp, corr, n, pitch);
#pragma unroll
        for (int j = 0; j < G; j++) out[j] = j == m ? s : out[j];
      }
  }
  for (unsigned left = __ballot_sync(0xffffffffu, whole && nc > 0); left; left &= left - 1) {
    const int src = __ffs(left) - 1;
    const int first = __shfl_sync(0xffffffffu, r.corr0, src), count = __shfl_sync(0xffffffffu, nc, src);
    LineTotal s[G];
    constexpr int kAtOnce = 4;
    for (int k = lane; k < count; k += 32 * kAtOnce) {
      LineCorr c[kAtOnce];
      typename Elem<G>::T v[kAtOnce];
#pragma unroll
      for (int i = 0; i < kAtOnce; i++) c[i] = k + 32 * i < count ? corr[first + k + 32 * i] : LineCorr{0, 0.f};
#pragma unroll
      for (int i = 0; i < kAtOnce; i++) v[i] = value(c[i].pix);
#pragma unroll
      for (int i = 0; i < kAtOnce; i++)
#pragma unroll
        for (int m = 0; m < G; m++)
          if (k + 32 * i < count) s[m].fold(c[i].w * elem_of<G>(v[i], m));
    }
#pragma unroll
    for (int m = 0; m < G; m++) {
      float sum = s[m].acc - s[m].comp;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == src) out[m] = sum;
    }
  }
}

}  // namespace medimg
