// strip.cu -- fan-beam / ray-table back projection along the rays' lines
// (LineRay): the transpose of the row-by-row forward walk.
//
// Rays are walked row by row along the axis they run closer to, as forward.
// A CTA owns a strip of that axis (up to 32 rows and 512 columns of 32-bit
// fixed-point sums in shared memory) and a range of at most kBpViewBlock views;
// each lane of a warp takes one ray of a view through the strip, every row
// adding the ray's two parts of it to their pixels.  A plan has two sets of
// strips, of rows along x and along y; a ray belongs to one.  The strips' sums
// and the rays' corrections meet as exact 64-bit integers in global memory, and
// a per-pixel pass turns them into the image and runs the epilogue.  Integer
// sums do not depend on the order or the split (deterministic, and a member of
// a group gets exactly the sums it gets alone).
//
// Against the walk over (ray, 16x16 tile) runs in project.cu: no run list to
// stream (288 MB at 512^2, 720 x 888), no decision bits, and the lanes of a
// warp, neighbouring rays in the same row, add side by side instead of in a
// dozen rows of a small tile (two wavefronts an add for almost four).  512^2,
// 720 x 888: one slice 287 -> 181 us, sixteen slices 2.51 -> 1.73 ms; 1024^2,
// 1440 x 1536: 1.70 -> 1.02 ms; error against 64 bits 5.9e-7 -> 1.9e-7 (a
// crossing is rounded as a row number, not as a distance from the source).
// The forward walk takes a line up every 32 rows, the strips every 16, so that
// the two sides' weights agree to the rounding of a crossing.
// Bound: the L1 data pipe (78 % while CTAs run, 93 % with four members; two
// wavefronts an add, because 32 neighbouring rays cover either more or fewer
// than 32 columns), then issue (77 %, 72 %).
// Measured and left: 16-row strips for one member (more loads of rays), the
// gather by pixel of every ray that can cross it (340 us one slice, 571 us four
// slices against 190 and 552: address arithmetic and 16-byte shared loads).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>

#include "epilogue.cuh"
#include "launch.h"
#include "line.cuh"
#include "smem_optin.h"
#include "solver.h"

namespace medimg {

cudaError_t launch_max(const unsigned *v, size_t n, unsigned *out, cudaStream_t st);

namespace {

// Strip of G members' sums.  About 66 KB: three CTAs per SM.
template <int G>
struct StripShape;
template <>
struct StripShape<1> {
  static constexpr int rows = 32, cols = 512;
};
template <>
struct StripShape<2> {
  static constexpr int rows = 32, cols = 256;
};
template <>
struct StripShape<4> {
  static constexpr int rows = 16, cols = 256;
};
constexpr int kStripThreads = 512;
// odd, so that strips along y flush without bank conflicts; one member's walk
// adds zeros to the column behind its last one
template <int G>
constexpr int strip_pitch() {
  return StripShape<G>::cols + 3;
}
template <int G>
constexpr int strip_plane() {
  return StripShape<G>::rows * strip_pitch<G>();
}
template <int G>
constexpr size_t strip_smem() {
  return (size_t)G * strip_plane<G>() * sizeof(int) + 256;  // (room past the last row)
}

// cells of columns in one strip of a scan, and strips along its columns
__host__ __device__ inline int strip_tile_cells(int ncc, int cols) {
  const int most = cols / kStripCellCols, tiles = (ncc + most - 1) / most;
  return (ncc + tiles - 1) / tiles;
}
template <int G>
__host__ __device__ inline int strip_cells_of(int n, int ncc) {
  const int tc = strip_tile_cells(ncc, StripShape<G>::cols);
  return ((n + StripShape<G>::rows - 1) / StripShape<G>::rows) * ((ncc + tc - 1) / tc);
}

__device__ __forceinline__ void red_global_add(unsigned long long *p, int v) {
  asm volatile("red.global.add.u64 [%0], %1;" ::"l"(p), "l"((long long)v) : "memory");
}

__device__ __forceinline__ void red_shared(unsigned at, int v) {
  asm volatile("red.shared.add.s32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: rounds to an integer in the low mantissa bits
constexpr int kMagicBits = 0x4B400000;

// power of two that brings a member's terms (|w r| <= 1.5 pixel max|r|) below 2^bp_term_bits
__device__ __forceinline__ int strip_scale_exp(const ScanDev &S, float mx) {
  int ex = 0;
  frexpf(fmaxf(1.5f * S.pixel_mm * mx, 1e-30f), &ex);
  return min(S.bp_term_bits - ex, 120);
}

// One row of a ray for M members (LineWalk's at(), before() and crosses()): the part
// before the crossing to the pixel at addr, rounded by kMagic, and where the
// ray crosses the rest of the rounded whole to the next pixel; then on to the
// next row.  Without a crossing the rest is zero: one member adds it all the
// same, because a predicated add compiles to a branch of its own (512^2, 720 x
// 888: 204 us a back projection against 221); several take one branch for all
// their second adds, which the lanes that cross (two in five) make in fewer
// wavefronts (four slices 612 us against 682).  kChecked: adds to columns
// outside the strip (col, of ncols) are left out.
template <int M, int kPlane, bool kChecked>
__device__ __forceinline__ void strip_row(float &e, unsigned &addr, int &col, int ncols, float inv, int step, int b,
                                          const float (&rs)[M], const int (&whole)[M]) {
  constexpr int kSub = LineWalk<1>::kSub;
  if (b > 0 && b % kSub == 0) e -= (float)kSub;
  const float f = __saturatef(e - (float)(b % kSub - kSub / 2));
  const bool x = e < (float)(b % kSub + 1 - kSub / 2);
  int bits[M];
#pragma unroll
  for (int m = 0; m < M; m++) bits[m] = __float_as_int(fmaf(f, rs[m], kMagic));
  if (!kChecked || (unsigned)col < (unsigned)ncols)
#pragma unroll
    for (int m = 0; m < M; m++) red_shared(addr + m * kPlane * 4, bits[m] - kMagicBits);
  if (M == 1 && !kChecked) {
    red_shared(addr + 4, whole[0] - bits[0]);
  } else if (x && (!kChecked || (unsigned)(col + 1) < (unsigned)ncols)) {
#pragma unroll
    for (int m = 0; m < M; m++) red_shared(addr + m * kPlane * 4 + 4, whole[m] - bits[m]);
  }
  if (x) {
    e += inv;
    addr += 4;
    if (kChecked) col++;
  }
  addr += step;
}

// Lane's ray through a cell's rows: addr is the shared byte address of its
// pixel of the first row, step the bytes to the next row.  rs: scaled residuals
// times the length of a row; whole: the bits of rs rounded by kMagic.
template <int M, int kPlane, bool kChecked>
__device__ __forceinline__ void strip_walk(const LineWalk<1> &w, unsigned addr, int step, const float (&rs)[M],
                                           const int (&whole)[M], int col, int ncols) {
  float e = w.e;
#pragma unroll
  for (int b = 0; b < kStripCellRows; b++)
    strip_row<M, kPlane, kChecked>(e, addr, col, ncols, w.inv, step, b, rs, whole);
}

template <int G>
__device__ __forceinline__ void strip_load_r(const ScanDev &S, const Launch &L, int bin, float (&r)[G]) {
  if constexpr (G == 1) {
    r[0] = __ldg(S.buf[L.in_buf] + bin);
  } else if constexpr (G == 2) {
    const float2 v = __ldg(reinterpret_cast<const float2 *>(S.pack) + bin);
    r[0] = v.x;
    r[1] = v.y;
  } else {
    const float4 v = __ldg(S.pack + bin);
    r[0] = v.x;
    r[1] = v.y;
    r[2] = v.z;
    r[3] = v.w;
  }
}

}  // namespace

// One CTA per (block of views and ray direction, strip): see the top of the
// file.  A warp's item is 32 rays, strip_k detectors apart, of one view.
// strip_k > 1 where detectors are finer than the pixels: lanes that add to the
// same pixel in one instruction serialise.
template <int G>
__device__ __forceinline__ void strip_bp_body(const Launch &L, const int scan, const ScanDev &S, int *const acc,
                                              int *const s_lo, int *const s_hi, int *const s_first) {
  constexpr int kRows = StripShape<G>::rows, kPitch = strip_pitch<G>(), kPlane = strip_plane<G>();
  constexpr int kCellRows = kRows / kStripCellRows;
  static_assert(kRows % kStripCellRows == 0 && StripShape<G>::cols % kStripCellCols == 0, "strips are whole cells");
  __shared__ float s_max[G];
  const int n = S.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned act = group_active<G>(L, S);
  if (!act) return grid_dependency_wait();
  // this CTA's views, direction and strip
  const int tcells = strip_tile_cells(S.strip_ncc, StripShape<G>::cols), ntile = (S.strip_ncc + tcells - 1) / tcells;
  const int ncell = strip_cells_of<G>(n, S.strip_ncc);
  const int local = blockIdx.x - (L.scans ? __ldg(L.prefix + scan) : 0);
  // strips from the middle outwards: the light ones at the edges end the launch
  const int nstrip = ncell / ntile, rank = local / S.strip_npart / ntile;
  const int strip = nstrip / 2 + ((rank & 1) ? -((rank + 1) >> 1) : rank >> 1);
  const int cell = strip * ntile + local / S.strip_npart % ntile;
  const int2 part = __ldg(S.strip_parts + local % S.strip_npart);
  const int dir = part.x & 1, v0 = part.x >> 1, nv = part.y;
  const int u0 = strip * kRows;
  const int cc0 = (cell - strip * ntile) * tcells, col0 = cc0 * kStripCellCols;
  const int ncols = min(n - col0, tcells * kStripCellCols);
  for (int r = warp; r < G * kRows; r += kStripThreads / 32)
    for (int c = lane; c < ncols + 2; c += 32) acc[r * kPitch + c] = 0;
  // the detectors of each view that meet the strip, and the items they make:
  // eight threads a view, a cell each
  static_assert(kStripThreads == 8 * kBpViewBlock && kCellRows * (StripShape<G>::cols / kStripCellCols) <= 8, "");
  {
    const int v = threadIdx.x >> 3, r = strip * kCellRows + (threadIdx.x & 7) % kCellRows, c = (threadIdx.x & 7) / kCellRows;
    int2 e = make_int2(INT_MAX, -1);
    if (v < nv && r < S.strip_ncr && c < tcells && cc0 + c < S.strip_ncc)
      e = __ldg(S.strip_rng + (((size_t)(v0 + v) * 2 + dir) * S.strip_ncr + r) * S.strip_ncc + cc0 + c);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      e.x = min(e.x, __shfl_xor_sync(0xffffffffu, e.x, o));
      e.y = max(e.y, __shfl_xor_sync(0xffffffffu, e.y, o));
    }
    if ((threadIdx.x & 7) == 0) {
      const int span = 32 * S.strip_k;
      s_lo[v] = e.x;
      s_hi[v] = e.y;
      s_first[v + 1] = e.y >= e.x ? (e.y - e.x + span) / span * S.strip_k : 0;
    }
  }
  // up to here the kernel may run beside the one before it
  grid_dependency_wait();
#pragma unroll
  for (int m = 0; m < G; m++) {
    if (warp != 1 + m || !((act >> m) & 1u)) continue;
    const ScanDev &M = L.scans ? L.scans[S.mem[m]] : L.single;
    float mx = fmaxf(M.bpmax[lane], M.bpmax[lane + 32]);
    static_assert(kBpMaxParts == 64, "two parts a lane");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) s_max[m] = mx;
  }
  __syncthreads();
  if (warp == 0) {  // two views a lane
    static_assert(kBpViewBlock == 64, "two views a lane");
    const int a = s_first[2 * lane + 1], b = a + s_first[2 * lane + 2];
    int sum = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 0) s_first[0] = 0;
    s_first[2 * lane + 1] = sum - b + a;
    s_first[2 * lane + 2] = sum;
  }
  __syncthreads();
  float scale[G];
  unsigned use = 0;
#pragma unroll
  for (int m = 0; m < G; m++) {
    scale[m] = 0.f;
    if ((act >> m) & 1u) {
      scale[m] = ldexpf(1.f, strip_scale_exp(S, s_max[m]));
      use |= s_max[m] > 0.f ? 1u << m : 0u;
    }
  }
  if (!use) return;
  // the member of each plane of sums
  const int nuse = __popc(use);
  unsigned member = 0;
  for (unsigned u = use, c = 0; u; u &= u - 1, c += 4) member |= (unsigned)(__ffs(u) - 1) << c;
  // this CTA's share of what the rays' traversals have besides their lines (a
  // gather by pixel took 20 us at 512^2: the pieces end at the image's border)
  {
    const int ctas = S.strip_npart * ncell;
    const int c1 = (int)((int64_t)S.strip_ncorr * (local + 1) / ctas);
    for (int c = (int)((int64_t)S.strip_ncorr * local / ctas) + threadIdx.x; c < c1; c += kStripThreads) {
      const uint4 e = __ldg(reinterpret_cast<const uint4 *>(S.strip_corr) + c);
      float r[G];
      strip_load_r<G>(S, L, (int)e.x, r);
#pragma unroll
      for (int m = 0; m < G; m++) {
        if (!((use >> m) & 1u)) continue;
        const ScanDev &M = L.scans ? L.scans[S.mem[m]] : L.single;
        const int v = __float_as_int(fmaf(__uint_as_float(e.z) * scale[m], r[m], kMagic)) - kMagicBits;
        red_global_add(M.bp_acc + e.y, v);
      }
    }
  }
  const int total = s_first[nv];
  if (total == 0) return;
  const unsigned acc0 = (unsigned)__cvta_generic_to_shared(acc);
  int vi = 0;
  for (int i = warp; i < total; i += kStripThreads / 32) {
    while (s_first[vi + 1] <= i) vi++;
    const int j = i - s_first[vi], k = S.strip_k;
    const int det = s_lo[vi] + j / k * (32 * k) + j % k + lane * k;
    const int bin = (v0 + vi) * S.ndets + min(det, S.ndets - 1);
    const LineRay ray = load_line(S.line + bin);
    LineWalk<1> w;
    w.load(ray);
    const bool down = (ray.flags & kLineDown) != 0;
    const int step0 = down ? n - u0 - kRows : u0;
    // (a row around the ones in the grid is harmless: its columns are outside)
    const bool on = det <= s_hi[vi] && ((ray.flags & kLineSwap) != 0) == (dir != 0) && !w.empty() &&
                    w.last >= step0 && w.first < step0 + kRows;
    float r[G];
    strip_load_r<G>(S, L, bin, r);
    // the members in use, side by side
    const float *const rm = r;
    auto cells = [&](auto count) {
      constexpr int M = decltype(count)::value;
      float rs[M];
      int whole[M];
#pragma unroll
      for (int c = 0; c < M; c++) {
        float v = rm[0], sc = scale[0];
#pragma unroll
        for (int m = 1; m < G; m++)
          if (M < G && ((member >> (4 * c)) & 15u) == m) {
            v = rm[m];
            sc = scale[m];
          }
        if (M == G) {
          v = rm[c];
          sc = scale[c];
        }
        rs[c] = v * (ray.len * sc);
        whole[c] = __float_as_int(__fadd_rn(rs[c], kMagic));
      }
      const int step = down ? -kPitch * 4 : kPitch * 4, c0 = line_c0(ray, n, S.lpitch) - col0;
      // cell by cell, so that a ray's parts do not depend on the strip's height
#pragma unroll 1
      for (int c = 0; c < kCellRows; c++) {
        const int col = c0 + w.enter(step0 + c * kStripCellRows, n);
        const int row = down ? kRows - 1 - c * kStripCellRows : c * kStripCellRows;
        const unsigned addr = acc0 + (unsigned)((row * kPitch + col) * 4);
        // at most one crossing a row, and inv rows between two of them
        const bool inside = col >= 0 && col + min(kStripCellRows, (int)(kStripCellRows * w.slope) + 2) < ncols;
        if (__all_sync(0xffffffffu, inside || !on)) {
          if (on) strip_walk<M, kPlane, false>(w, addr, step, rs, whole, col, ncols);
        } else if (on && col < ncols) {
          strip_walk<M, kPlane, true>(w, addr, step, rs, whole, col, ncols);
        }
      }
    };
    if (G == 1 || nuse == 1) cells(std::integral_constant<int, 1>{});
    else if (G == 2 || nuse == 2) cells(std::integral_constant<int, G >= 2 ? 2 : 1>{});
    else if (nuse == 3) cells(std::integral_constant<int, G >= 4 ? 3 : 1>{});
    else cells(std::integral_constant<int, G >= 4 ? 4 : 1>{});
  }
  __syncthreads();
  // the strip's sums into the members' 64-bit pixels; in a strip along y the
  // lanes run along its rows, which are the image's columns
  for (int m = 0; m < nuse; m++) {
    const ScanDev &M = L.scans ? L.scans[S.mem[(member >> (4 * m)) & 15u]] : L.single;
    unsigned long long *out = M.bp_acc;
    const int nr = min(kRows, n - u0);
    if (dir == 0) {
      for (int row = warp; row < nr; row += kStripThreads / 32)
        for (int c = lane; c < ncols; c += 32) {
          const int v = acc[m * kPlane + row * kPitch + c];
          if (v) red_global_add(out + (size_t)(u0 + row) * n + col0 + c, v);
        }
    } else {
      for (int i = threadIdx.x; i < kRows * ncols; i += kStripThreads) {
        const int row = i % kRows, c = i / kRows;
        const int v = row < nr ? acc[m * kPlane + row * kPitch + c] : 0;
        if (v) red_global_add(out + (size_t)(col0 + c) * n + u0 + row, v);
      }
    }
  }
}

__global__ void __launch_bounds__(kStripThreads, 3) strip_bp_kernel(const Launch L) {
  extern __shared__ __align__(16) int acc[];
  __shared__ int s_lo[kBpViewBlock], s_hi[kBpViewBlock], s_first[kBpViewBlock + 1];
  const int scan = L.scans ? find_scan(L.prefix, L.nscans, blockIdx.x) : 0;
  const ScanDev &S = scan_of(L, scan);
  if (!S.strip) return grid_dependency_wait();  // (a kernel's end means the end of those before it)
  const int nm = L.scans ? S.nmem : 1;
  if (nm >= 3) strip_bp_body<4>(L, scan, S, acc, s_lo, s_hi, s_first);
  else if (nm == 2) strip_bp_body<2>(L, scan, S, acc, s_lo, s_hi, s_first);
  else strip_bp_body<1>(L, scan, S, acc, s_lo, s_hi, s_first);
}

// The sums as pixels, through the solver's epilogue; leaves zeros.  Over the
// pixel-pass CTAs.
__global__ void __launch_bounds__(256) strip_finish_kernel(const Launch L) {
  chain_begin();
  const int scan = L.scans ? find_scan(L.prefix, L.nscans, blockIdx.x) : 0;
  const ScanDev &S = scan_of(L, scan);
  if (!S.strip || !flow_active(S, L.flow)) return;
  const int cta0 = L.scans ? __ldg(L.prefix + scan) : 0;
  const int ncta = L.scans ? __ldg(L.prefix + scan + 1) - cta0 : gridDim.x;
  const int local = blockIdx.x - cta0, n = S.n, nt = (n + 31) / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float mx = fmaxf(S.bpmax[lane], S.bpmax[lane + 32]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float unit = ldexpf(1.f, -strip_scale_exp(S, mx));  // (a power of two: one rounding, the conversion's)
  const int y = (local % nt) * 32 + lane, x0 = (local / nt) * kPixRows + warp;
  constexpr int kRowsEach = kPixRows / 8;
  long long t[kRowsEach];
#pragma unroll
  for (int r = 0; r < kRowsEach; r++) {
    const int x = x0 + r * 8;
    t[r] = x < n && y < n ? (long long)S.bp_acc[x * n + y] : 0;
  }
  FF s0[1] = {ff_zero()};
#pragma unroll
  for (int r = 0; r < kRowsEach; r++) {
    const int x = x0 + r * 8;
    if (x >= n || y >= n) continue;
    if (t[r]) S.bp_acc[x * n + y] = 0ull;
    bp_epilogue(S, L, 0, x, y, __ll2float_rn(t[r]) * unit, s0[0]);
  }
  if (stage_reduces(L.stage)) reduce_and_finalize<1>(S, L, s0, local, ncta);
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
namespace {
constexpr size_t kStripSmem = std::max({strip_smem<1>(), strip_smem<2>(), strip_smem<4>()});

// parts of a direction's rays in each division of the views (small ones are
// raised to whole blocks of views)
constexpr int kStripParts[kStripDivs] = {1, 2, 3, 4, 6, 8, 11, 14, 18, 22, 28, 36, 48, 64, 96, 128};

int strip_cells(const ScanDev &S, int nmem) {
  return nmem >= 3 ? strip_cells_of<4>(S.n, S.strip_ncc)
                   : nmem == 2 ? strip_cells_of<2>(S.n, S.strip_ncc) : strip_cells_of<1>(S.n, S.strip_ncc);
}
}  // namespace

cudaError_t launch_strip_bp(const Launch &L, int nctas, cudaStream_t st) {
  static SmemOptIn optin;
  const cudaError_t e = optin.ensure(kStripSmem, [](int *dev) { return cudaGetDevice(dev); }, [](size_t bytes) {
    return cudaFuncSetAttribute(strip_bp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  });
  if (e != cudaSuccess) return e;
  return launch_dependent(strip_bp_kernel, nctas, kStripThreads, kStripSmem, st, L);
}

cudaError_t launch_strip_finish(const Launch &Lpix, int pix_nctas, cudaStream_t st) {
  return launch_dependent(strip_finish_kernel, pix_nctas, 256, 0, st, Lpix);
}

// CTAs of a scan (or the group it leads)
int strip_ctas(const ScanDev &S) { return S.strip_npart * strip_cells(S, std::max(1, S.nmem)); }

// Chooses the division of the views for a launch, by an estimate of the items
// (32 rays through a strip) that the busiest SM goes through: its CTAs' items
// and what each CTA's own passes over its sums are worth.  Up to three CTAs on
// every SM run at once: their own passes overlap (12 items), the strips'
// differences stay (1.75), and an SM with fewer of them waits more.  Beyond,
// CTAs follow as others end (30 items), and the last ones leave SMs idle for
// three of them.  Fitted to sweeps over the divisions (one slice of 100^2: 144
// CTAs 18 us, 288 16 us; 217^2: 392 CTAs 34 us, 672 38 us; 512^2: 448 CTAs 198
// us, 1536 187 us; 1024^2: 2944 CTAs 1.08 ms, 6144 1.00 ms; sixteen slices of
// 512^2: 6144 CTAs 1.82 ms, 14336 1.97 ms).  Results do not depend on it.
void strip_choose(ScanDev *scans, int n) {
  constexpr double kOwn = 30.0, kOwnBeside = 12.0, kSms = 152.0;
  // what a scan (or the group it leads) has to do, and its division so far
  struct Work {
    ScanDev *S;
    double items;
    int cells, div;
    int ctas(int q) const { return (S->strip_poff[q + 1] - S->strip_poff[q]) * cells; }
  };
  std::vector<Work> work;
  work.reserve(n);
  bool groups = false;
  size_t most = 0;  // the scan with the most work
  for (int s = 0; s < n; s++) {
    ScanDev &S = scans[s];
    groups |= S.nmem > 1;
    if (!S.strip || !S.nmem) continue;
    const int cells = strip_cells(S, S.nmem);
    work.push_back(Work{&S, (double)S.nbins / 32.0 * cells / 1.5, cells, 0});
    if (work.back().items > work[most].items) most = work.size() - 1;
  }
  if (work.empty()) return;
  // division q for that scan, and for the others the coarsest whose CTAs have
  // no more work than its (scans of 241^2 and 160^2: 56 -> 47 us); with groups,
  // whose items cost more than a single scan's, q for all (302^2, a pair and
  // one alone: 111 us against 202).  The work of its CTAs only falls with q, so
  // the others' divisions only rise (sixteen times as many steps, one division
  // at a time from the coarsest: 17 us of a call for 64 scans)
  auto set = [&](int q) {
    const double each = 1.15 * work[most].items / work[most].ctas(q);
    for (size_t s = 0; s < work.size(); s++) {
      Work &w = work[s];
      if (groups || s == most) w.div = q;
      else while (w.div < q && w.items > each * w.ctas(w.div)) w.div++;
    }
  };
  double best = 1e300;
  int pick = 0;
  for (int q = 0; q < kStripDivs; q++) {
    set(q);
    double ctas = 0.0, items = 0.0;
    for (const Work &w : work) {
      ctas += w.ctas(w.div);
      items += w.items;
    }
    const double per = std::ceil(ctas / kSms);
    const double t = per <= 3.0 ? per * (1.75 * items / ctas + kOwnBeside) / (per == 1.0 ? 0.55 : per == 2.0 ? 0.75 : 1.0)
                                : (ctas / kSms + 3.0) * (items / ctas + kOwn);
    if (t < best) {
      best = t;
      pick = q;
    }
  }
  for (Work &w : work) w.div = 0;
  set(pick);
  for (const Work &w : work) {
    w.S->strip_parts = w.S->strip_part0 + w.S->strip_poff[w.div];
    w.S->strip_npart = w.S->strip_poff[w.div + 1] - w.S->strip_poff[w.div];
  }
}

// ---------------------------------------------------------------------------
// plan tables
// ---------------------------------------------------------------------------
// The detectors of each view whose rays meet each cell of each direction
// (every column the walk adds to, cells as tall as kStripCellRows), and the
// number of each view's rays in each direction.
__global__ void strip_range_kernel(int n, int nviews, int ndets, int ncr, int ncc, const LineRay *line, int2 *rng,
                                   unsigned *count) {
  const int ray = blockIdx.x * blockDim.x + threadIdx.x;
  if (ray >= nviews * ndets) return;
  const LineRay r = load_line(line + ray);
  LineWalk<1> w;
  w.load(r);
  if (w.empty()) return;
  const int view = ray / ndets, det = ray % ndets, dir = (r.flags & kLineSwap) ? 1 : 0;
  const int col0 = line_c0(r, n, line_pitch(n));
  int2 *mine = rng + ((size_t)view * 2 + dir) * ncr * ncc;
  bool any = false;
  for (int cr = 0; cr < ncr; cr++) {
    const int u0 = cr * kStripCellRows;
    const int step0 = (r.flags & kLineDown) ? n - u0 - kStripCellRows : u0;
    if (w.last < step0 || w.first >= step0 + kStripCellRows) continue;
    const int c0 = col0 + w.enter(step0, n);
    int c1 = c0;
    for (int b = 0; b < kStripCellRows; b++) {
      w.at(b);
      c1 += w.crosses(b) ? 1 : 0;
    }
    // one more on either side: a taller strip's walk enters at its own first row
    const int lo = max(c0 - 1, 0), hi = min(c1 + 2, n - 1);
    if (lo > hi) continue;
    any = true;
    for (int c = lo / kStripCellCols; c <= hi / kStripCellCols; c++) {
      int *e = &mine[cr * ncc + c].x;
      const volatile int *ev = e;
      if (ev[0] > det) atomicMin(e, det);
      if (ev[1] < det) atomicMax(e + 1, det);
    }
  }
  if (any) atomicAdd(count + 2 * view + dir, 1u);
}

// What the strips add to each pixel in the views [view0, view1), in 1/64 of a
// whole row of a ray (each part rounded up): the same steps as strip_row.
constexpr unsigned kHitsUnit = 64;
__global__ void strip_hits_kernel(int n, int view0, int view1, int ndets, int ncr, const LineRay *line,
                                  unsigned *hits) {
  const int ray = view0 * ndets + blockIdx.x * blockDim.x + threadIdx.x;
  if (ray >= view1 * ndets) return;
  const LineRay r = load_line(line + ray);
  LineWalk<1> w;
  w.load(r);
  if (w.empty()) return;
  const bool swap = (r.flags & kLineSwap) != 0, down = (r.flags & kLineDown) != 0;
  const int col0 = line_c0(r, n, line_pitch(n));
  auto add = [&](int u, int c, float part) {
    if ((unsigned)u < (unsigned)n && (unsigned)c < (unsigned)n && part > 0.f)
      atomicAdd(hits + (swap ? (size_t)c * n + u : (size_t)u * n + c), (unsigned)ceilf(part * kHitsUnit));
  };
  for (int cr = 0; cr < ncr; cr++) {
    const int u0 = cr * kStripCellRows;
    const int step0 = down ? n - u0 - kStripCellRows : u0;
    if (w.last < step0 || w.first >= step0 + kStripCellRows) continue;
    int c = col0 + w.enter(step0, n);
    for (int b = 0; b < kStripCellRows; b++) {
      w.at(b);
      const float f = w.before(b);
      const bool x = w.crosses(b);
      const int u = line_row_of(r, step0 + b, n);
      add(u, c, f);
      if (x) add(u, ++c, 1.f - f);
    }
  }
}

// Whether the strips' 32-bit sums hold whatever kBpViewBlock views add to a
// pixel.  A term is at most part * (len / 1.5 pixel) * 2^bp_term_bits, len at
// most sqrt(2) pixels, and rounded by half a unit, so the parts' sum bounds the
// terms' in units of 2^bp_term_bits.  Fan beams: the geometric bound that
// bp_term_bits comes from covers every ray through a pixel.  Ray tables: it
// counts the segments of the traversal, which leaves out the last 0.05 mm of
// each ray; the strips add those too (and take them back in 64 bits), so what
// they add is counted here.
int strips_fit(const Plan &p, int ncr, cudaStream_t st, bool *fit) {
  *fit = true;
  if (p.kind == AT_GEOM_FAN) return AT_OK;
  const size_t cells = (size_t)p.n * p.n;
  unsigned *hits = nullptr;
  const auto free_hits = scope_exit([&] { cudaFree(hits); });
  AT_CUDA_TRY(dev_malloc(&hits, sizeof(unsigned) * (cells + 1)));
  unsigned *const mx = hits + cells;
  AT_CUDA_TRY(cudaMemsetAsync(mx, 0, sizeof(unsigned), st));
  for (int v0 = 0; v0 < p.nviews; v0 += kBpViewBlock) {
    const int v1 = std::min(p.nviews, v0 + kBpViewBlock);
    AT_CUDA_TRY(cudaMemsetAsync(hits, 0, sizeof(unsigned) * cells, st));
    strip_hits_kernel<<<((v1 - v0) * p.ndets + 127) / 128, 128, 0, st>>>(p.n, v0, v1, p.ndets, ncr, p.line_d, hits);
    AT_CUDA_TRY(cudaGetLastError());
    AT_CUDA_TRY(launch_max(hits, cells, mx, st));
  }
  unsigned most = 0;
  AT_CUDA_TRY(cudaMemcpyAsync(&most, mx, sizeof(most), cudaMemcpyDeviceToHost, st));
  AT_CUDA_TRY(cudaStreamSynchronize(st));
  *fit = (uint64_t)most << p.bp_term_bits < (uint64_t)kHitsUnit << 31;
  return AT_OK;
}

__global__ void strip_none_kernel(int2 *rng, size_t cells) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < cells) rng[i] = make_int2(INT_MAX, -1);
}

// The tables of the strip back projector; none where its sums might not fit
// (bp_term_bits is known by now).  `off`: first correction of each ray and, at
// the end, how many there are; `corr` the corrections.
int build_strips(Plan &p, const std::vector<int> &off, const std::vector<LineCorr> &corr, cudaStream_t st) {
  const int n = p.n, nrays = p.nviews * p.ndets;
  const int ncr = (n + kStripCellRows - 1) / kStripCellRows, ncc = (n + kStripCellCols - 1) / kStripCellCols;
  bool fit;
  if (const int rc = strips_fit(p, ncr, st, &fit)) return rc;
  if (!fit) return AT_OK;  // (tile runs keep the scale, and with it the precision)
  const size_t cells = (size_t)p.nviews * 2 * ncr * ncc;
  unsigned *count_d = nullptr;
  const auto free_temps = scope_exit([&] { cudaFree(count_d); });
  auto alloc = [&](auto **q, size_t count) {
    const size_t bytes = std::max<size_t>(16, count * sizeof(**q));
    p.device_bytes += (int64_t)bytes;
    return dev_malloc(q, bytes);
  };
  AT_CUDA_TRY(dev_malloc(&count_d, sizeof(unsigned) * 2 * p.nviews));
  AT_CUDA_TRY(cudaMemsetAsync(count_d, 0, sizeof(unsigned) * 2 * p.nviews, st));
  AT_CUDA_TRY(alloc(&p.strip_rng_d, cells));
  strip_none_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(p.strip_rng_d, cells);
  AT_CUDA_TRY(cudaGetLastError());
  strip_range_kernel<<<(nrays + 127) / 128, 128, 0, st>>>(n, p.nviews, p.ndets, ncr, ncc, p.line_d, p.strip_rng_d,
                                                         count_d);
  AT_CUDA_TRY(cudaGetLastError());
  std::vector<unsigned> count(2 * (size_t)p.nviews);
  AT_CUDA_TRY(cudaMemcpyAsync(count.data(), count_d, sizeof(unsigned) * 2 * p.nviews, cudaMemcpyDeviceToHost, st));
  AT_CUDA_TRY(cudaStreamSynchronize(st));
  // The CTAs' ranges of views: about 1/kStripParts[q] of a direction's rays
  // each, so that CTAs of one strip have like work, and none across two blocks
  // of kBpViewBlock views (what the fixed-point scale is made for).
  std::vector<int2> parts;
  for (int q = 0; q < kStripDivs; q++) {
    p.strip_poff[q] = (int)parts.size();
    for (int d = 0; d < 2; d++) {
      int64_t all = 0;
      for (int v = 0; v < p.nviews; v++) all += count[2 * v + d];
      for (int b0 = 0; b0 < p.nviews; b0 += kBpViewBlock) {
        const int b1 = std::min(p.nviews, b0 + kBpViewBlock);
        int64_t mine = 0;
        for (int v = b0; v < b1; v++) mine += count[2 * v + d];
        if (mine == 0) continue;
        const int64_t pieces = std::max<int64_t>(1, (mine * kStripParts[q] + all / 2) / all);
        int first = b0;
        int64_t done = 0, cut = 1;
        for (int v = b0; v < b1; v++) {
          done += count[2 * v + d];
          if (done * pieces < mine * cut) continue;
          if (v + 1 > first) parts.push_back(make_int2(first << 1 | d, v + 1 - first));
          first = v + 1;
          while (done * pieces >= mine * cut) cut++;
        }
      }
    }
    // corrections alone (no ray is a line): somebody adds them
    if ((int)parts.size() == p.strip_poff[q]) parts.push_back(make_int2(0, 1));
  }
  p.strip_poff[kStripDivs] = (int)parts.size();
  AT_CUDA_TRY(alloc(&p.strip_part_d, parts.size()));
  if (!parts.empty())
    AT_CUDA_TRY(cudaMemcpyAsync(p.strip_part_d, parts.data(), sizeof(int2) * parts.size(), cudaMemcpyHostToDevice, st));
  // the corrections, in ray order
  std::vector<StripCorr> list;
  for (int r = 0; r < nrays; r++)
    for (int k = off[r]; k < off[r + 1]; k++)
      if (!(corr[k].pix & kCorrForwardOnly)) list.push_back(StripCorr{r, corr[k].pix, corr[k].w, 0});
  AT_CUDA_TRY(alloc(&p.strip_corr_d, list.size()));
  if (!list.empty())
    AT_CUDA_TRY(cudaMemcpyAsync(p.strip_corr_d, list.data(), sizeof(StripCorr) * list.size(), cudaMemcpyHostToDevice, st));
  AT_CUDA_TRY(cudaStreamSynchronize(st));
  p.strip_ncorr = (int)list.size();
  p.strip_ncr = ncr;
  p.strip_ncc = ncc;
  // rays of a view per pixel of a row, on average
  const double density = (double)p.segments / 1.5 / ((double)p.nviews * n * n);
  p.strip_k = std::max(1, std::min((int)std::lround(0.8 * density), (p.ndets + 31) / 32));
  p.strip_ok = 1;
  return AT_OK;
}

}  // namespace medimg
