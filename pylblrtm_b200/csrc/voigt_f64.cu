// Float64 Voigt summation over reference tiles (pylblrtm/forward.py:295-315).
//
// od[row, p] = R(nu_p, T_row) * sum over the lines admitted by the reference's tile window
// of amp * Re w(x + iy), x = (nu_p - nuc) sqrt(ln 2)/alpha_D, everything in float64.
//
// A line's profile far from a set of points is analytic there, so it is summed at 16
// Chebyshev nodes instead of at every point. A line is "far" of an interval when its
// centre lies more than D_FAR = 6 half-widths from the interval's centre: the nodes'
// Bernstein ellipse then has rho >= 6 + sqrt(35) = 11.9 and the interpolation error of the
// line's own value is below 16 * 11.9^-16 ~ 1e-16 (its slope in a 1/x^2 wing included), so
// the sums keep float64 accuracy; interpolants are evaluated at the rounded grid values
// themselves. Three interval sizes share the work of one CTA (256 threads, one chunk of at
// most 512 points of one tile of one row):
//   level 1  the chunk: one thread takes one line and adds it at the 16 nodes;
//   level 2  256-point sub-chunks, one after the other: the lines that are not far of the
//            chunk, again one per thread; those not far of the sub-chunk go to a list;
//   level 3  32-point segments, one per warp: far lines of the list at 16 nodes, one per
//            lane; the remaining lines directly, one point per lane.
// A far line also needs |z|^2 >= ASYM_Z2 at its nearest node and a width that is not
// negative, so every node value is the asymptotic series in its real-part form with one
// reciprocal; what fails that test is summed directly at each point (faddeeva.cuh has the
// forms by distance). Every
// sum is formed in a fixed order (no floating-point atomics), so results are bit-reproducible.
//
// Bound by float64 issue and latency (two CTAs per SM at 128 registers): about 240 node
// values and 20 direct values per point and layer at 105 lines per cm^-1, 0.001 cm^-1 steps
// and a 25 cm^-1 cut-off, where evaluating every line at every point by the Gautschi method
// takes 5,500. Kernel times on B200, before (every line at every point) and now: 20 cm^-1 of
// a 200,000-line list at 60 layers 91.9 -> 0.92 ms, 20 cm^-1 of a 2,000-line band at 20
// layers 14.6 -> 0.147 ms (0.84 and 0.142 without the quadrature next to the real axis, which
// keeps the accuracy of the former method for lines of small width). Chunks of 512, 1,024 and
// 2,048 points measure the same on the former (0.84, 0.86, 0.9 ms without the quadrature) and
// 0.135, 0.16, 0.3 ms on the latter (too few CTAs); D_FAR of 5 or 8 instead of 6 changes less
// than 5 %.
#include <math.h>

#include "cheb_tables.h"
#include "faddeeva.cuh"
#include "lbl_common.cuh"
#include "sum_common.cuh"

namespace lbl {

constexpr int D_K = 16;            // Chebyshev nodes per interval
constexpr int D_THREADS = 256;
constexpr int D_WARPS = D_THREADS / 32;
constexpr int D_SEG = 32;          // points per warp segment (level 3)
constexpr int D_SUB = D_WARPS * D_SEG;
constexpr int D_CHUNK = 512;      // max points per CTA: a 2,000-point tile gives four chunks of 500
constexpr int D_LIST = 768;        // listed lines per sub-chunk between two passes of the warps
constexpr int D_FEW = 16;          // a chunk of at most D_K points takes every line at every point
constexpr double D_FAR = 6.0;

static __constant__ double c_ddct16[D_K * D_K] = {LBL_DCT16};
// node k (fraction of the half-width): cos((2k+1) pi/32), row 1 of the DCT table
#define D_NODE(k) c_ddct16[D_K + (k)]

// The forms of the core and the reflection below the axis, out of line (registers, code size).
static __device__ __noinline__ double core_f64(double x, double y) { return re_w_f64_core(x, y); }
static __device__ __noinline__ double lower_f64(double x, double ay, double v) { return re_w_f64_lower(x, ay, v); }

// Re w at one point, any z. All 32 lanes of a warp call it together: outside the core the warp
// takes one form, the longest that one of its lanes needs, so at most two run and the choice
// depends on the lanes' arguments alone.
__device__ __forceinline__ double voigt_re_f64(double x, double y) {
  const double ay = fabs(y), y2 = ay * ay, z2 = fma(x, x, y2);
  double v;
  if (!__any_sync(0xffffffffu, !wing_only_f64(ay, z2))) {
    v = INV_SQRT_PI * ay * wing_f64<7>(x, y2);
  } else {
    const bool s22 = __any_sync(0xffffffffu, z2 >= CORE_F64_Z2 && z2 < ASYM13_Z2);
    v = z2 >= CORE_F64_Z2 ? re_w_f64_series(x, ay, s22) : core_f64(x, ay);
  }
  return y >= 0.0 ? v : lower_f64(x, ay, v);
}

template <int N>
__device__ __forceinline__ void nodes_add_n(double (&f)[D_K], double xc, double ha, double y2, double af) {
#pragma unroll
  for (int k = 0; k < D_K / 2; ++k) {
    const double off = D_NODE(k) * ha;
    f[k] = fma(af, wing_f64<N>(xc + off, y2), f[k]);
    f[D_K - 1 - k] = fma(af, wing_f64<N>(xc - off, y2), f[D_K - 1 - k]);
  }
}

// An interval of grid values: centre and half-width in cm^-1.
struct Span64 {
  double c, h;
};

// Adds a far line at the interval's nodes; false when the line is not far of it. The test
// uses the same operations wherever a line meets the same interval.
__device__ __forceinline__ bool far_nodes_add(double (&f)[D_K], const LineF64& L, const Span64& s, bool add) {
  const double d = __dsub_rn(s.c, L.nuc), ad = fabs(d);
  const double xm = __dmul_rn(__dsub_rn(ad, s.h), L.inv_ad);         // |x| at the interval's near end
  const double y2 = __dmul_rn(L.y, L.y), zm = __dadd_rn(__dmul_rn(xm, xm), y2);
  if (!(ad > __dmul_rn(D_FAR, s.h) && wing_only_f64(L.y, zm))) return false;
  if (add) {
    const double xc = d * L.inv_ad, ha = s.h * L.inv_ad, af = L.amp * L.y * INV_SQRT_PI;
    if (zm >= ASYM2_Z2) nodes_add_n<2>(f, xc, ha, y2, af);
    else if (zm >= ASYM4_Z2) nodes_add_n<4>(f, xc, ha, y2, af);
    else nodes_add_n<7>(f, xc, ha, y2, af);
  }
  return true;
}

__device__ __forceinline__ double shfl_xor_f64(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }

// Sum over the 32 lanes of f[16]: afterwards lanes 2j and 2j+1 hold the total of node j.
__device__ __forceinline__ double reduce16_f64(const double (&f)[D_K], int lane) {
  double g[8], h[4], u[2];
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
#pragma unroll
  for (int k = 0; k < 8; ++k) g[k] = (b4 ? f[k + 8] : f[k]) + shfl_xor_f64(b4 ? f[k] : f[k + 8], 16);
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = (b3 ? g[k + 4] : g[k]) + shfl_xor_f64(b3 ? g[k] : g[k + 4], 8);
#pragma unroll
  for (int k = 0; k < 2; ++k) u[k] = (b2 ? h[k + 2] : h[k]) + shfl_xor_f64(b2 ? h[k] : h[k + 2], 4);
  const double v = (b1 ? u[1] : u[0]) + shfl_xor_f64(b1 ? u[0] : u[1], 2);
  return v + shfl_xor_f64(v, 1);
}

// p(t) = c0/2 + sum_{k>=1} c_k T_k(t).
__device__ __forceinline__ double clenshaw_f64(const double* c, double t) {
  double b1 = 0.0, b2 = 0.0;
  const double t2 = 2.0 * t;
#pragma unroll
  for (int k = D_K - 1; k >= 1; --k) {
    const double b0 = fma(t2, b1, c[k] - b2);
    b2 = b1;
    b1 = b0;
  }
  return fma(t, b1, 0.5 * c[0] - b2);
}

// Chebyshev coefficient k of the node values v[16].
__device__ __forceinline__ double dct_f64(const double* v, int k) {
  double c = 0.0;
#pragma unroll
  for (int j = 0; j < D_K; ++j) c = fma(v[j], c_ddct16[k * D_K + j], c);
  return c * (2.0 / D_K);
}

__global__ void __launch_bounds__(D_THREADS, 2)
tau_f64_kernel(const LineF64* __restrict__ prep, int n_lines, const int2* __restrict__ ranges,
               const double* __restrict__ t_layer, double nu_min, double step, long long n_nu,
               int tile_samples, int chunks_per_tile, int chunk_pts, double cutoff, int n_grp,
               double* __restrict__ od, int* err, unsigned long long* evals) {
  __shared__ LineF64 s_list[D_LIST];
  __shared__ double s_part[D_WARPS][D_K];            // per-warp node sums
  __shared__ double s_val[D_K], s_c1[D_K], s_c2[D_K];
  __shared__ double s_seg[D_WARPS][D_K];             // level-3 node sums, then the segment's series
  __shared__ int s_cnt[D_WARPS], s_lo, s_hi;
  __shared__ unsigned s_pass;

  const int row = blockIdx.y;
  const int tile = blockIdx.x / chunks_per_tile, chunk = blockIdx.x % chunks_per_tile;
  const long long t0 = (long long)tile * tile_samples;
  const long long t1 = min(t0 + (long long)tile_samples, n_nu);
  long long c0;
  int n_c;
  if (!tile_chunk(t0, t1, chunk, chunk_pts, c0, n_c)) return;
  const double wlo = __dsub_rn(grid_nu(nu_min, step, t0), cutoff);
  const double whi = __dadd_rn(grid_nu(nu_min, step, t1 - 1), cutoff);
  const int2 rng = ranges[tile];
  const LineF64* lp = prep + (long long)row * n_lines;
  const double T = t_layer[row];
  double* out = od + (long long)row * n_nu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool bad = false;

  auto span = [&](int p, int n) {                    // points [p, p + n) of the chunk
    const double a = grid_nu(nu_min, step, c0 + p), b = grid_nu(nu_min, step, c0 + p + n - 1);
    return Span64{0.5 * (a + b), 0.5 * (b - a)};
  };
  auto load = [&](int li, LineF64& L) {              // the reference's window test (NaN centres fail)
    if (li >= rng.y) return false;
    L = lp[li];
    return L.nuc >= wlo && L.nuc <= whi;
  };

  if (n_c <= D_FEW) {
    // The one-point tile at a grid's end and other slivers: every line at every point, a
    // line per thread and a point at a time (a warp per point would walk the window alone).
    unsigned np = 0;
    for (int p = 0; p < n_c; ++p) {
      const double nu = grid_nu(nu_min, step, c0 + p);
      double acc = 0.0;
      np = 0;
      for (int base = rng.x; base < rng.y; base += D_THREADS) {   // whole warps, absent lines as zeros
        LineF64 L;
        const bool on = load(base + tid, L);
        np += on;
        const double v = voigt_re_f64(on ? (nu - L.nuc) * L.inv_ad : 100.0, on ? L.y : 1.0);
        acc = fma(on ? L.amp : 0.0, v, acc);
      }
      for (int o = 16; o > 0; o >>= 1) acc += shfl_xor_f64(acc, o);
      if (lane == 0) s_part[warp][0] = acc;
      __syncthreads();
      if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < D_WARPS; ++w) s += s_part[w][0];
        const double v = __dmul_rn(s, radiation_term_grid(nu, T));
        if (!isfinite(v)) flag_error(err, row * (n_grp + 1) + n_grp);
        out[c0 + p] = v;
      }
      __syncthreads();
    }
    np = __reduce_add_sync(0xffffffffu, np);
    if (lane == 0 && evals && np) atomicAdd(evals, (unsigned long long)np * n_c);
    return;
  }

  // ---- level 1: every line of the window, one per thread
  const Span64 sp1 = span(0, n_c);
  if (tid == 0) {
    s_lo = 0x7fffffff;
    s_hi = -1;
    s_pass = 0u;
  }
  double f[D_K];
#pragma unroll
  for (int k = 0; k < D_K; ++k) f[k] = 0.0;
  __syncthreads();
  {
    unsigned np = 0;
    int lo = 0x7fffffff, hi = -1;
    for (int li = rng.x + tid; li < rng.y; li += D_THREADS) {
      LineF64 L;
      if (!load(li, L)) continue;
      ++np;
      if (!far_nodes_add(f, L, sp1, true)) {
        lo = min(lo, li);
        hi = max(hi, li);
      }
    }
    np = __reduce_add_sync(0xffffffffu, np);
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      atomicAdd(&s_pass, np);
      atomicMin(&s_lo, lo);
      atomicMax(&s_hi, hi);
    }
    const double v = reduce16_f64(f, lane);
    if (!(lane & 1)) s_part[warp][lane >> 1] = v;
  }
  __syncthreads();
  if (tid < D_K) {
    double v = 0.0;
    for (int w = 0; w < D_WARPS; ++w) v += s_part[w][tid];
    s_val[tid] = v;
  }
  __syncthreads();
  if (tid < D_K) s_c1[tid] = dct_f64(s_val, tid);
  if (tid == 0 && evals && s_pass) atomicAdd(evals, (unsigned long long)s_pass * n_c);
  __syncthreads();
  const int in_lo = s_lo, in_hi = s_hi;              // the lines that are not far of the chunk lie here

  // ---- levels 2 and 3, one sub-chunk after the other
  for (int w0 = 0; w0 < n_c; w0 += D_SUB) {
    const int n_w = min(D_SUB, n_c - w0);
    const Span64 sp2 = span(w0, n_w);
    const int g0 = w0 + warp * D_SEG, n_g = max(0, min(D_SEG, n_c - g0));   // this warp's segment
    const Span64 sp3 = n_g > 0 ? span(g0, n_g) : Span64{0.0, 0.0};
    const bool use3 = n_g > D_K;
    const double nu = grid_nu(nu_min, step, c0 + g0 + min(lane, max(n_g - 1, 0)));
    double acc = 0.0;
    if (lane < D_K) {
      s_seg[warp][lane] = 0.0;
      s_part[warp][lane] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < D_K; ++k) f[k] = 0.0;
    int n_list = 0;

    // the warps' pass over the listed lines: far lines at the segment's nodes (a line per
    // lane), the others at every point (a point per lane)
    auto pass_list = [&]() {
      if (n_g <= 0) return;
      double f3[D_K];
#pragma unroll
      for (int k = 0; k < D_K; ++k) f3[k] = 0.0;
      for (int i0 = 0; i0 < n_list; i0 += 32) {
        const int i = i0 + lane;
        bool near = i < n_list;
        if (near && use3) near = !far_nodes_add(f3, s_list[i], sp3, true);
        unsigned m = __ballot_sync(0xffffffffu, near);
        while (m) {
          const int l = i0 + __ffs(m) - 1;
          m &= m - 1;
          const LineF64 L = s_list[l];
          acc = fma(L.amp, voigt_re_f64((nu - L.nuc) * L.inv_ad, L.y), acc);
        }
      }
      const double v = reduce16_f64(f3, lane);
      if (!(lane & 1)) s_seg[warp][lane >> 1] += v;
      __syncwarp();
    };

    for (int base = in_lo; base <= in_hi; base += D_THREADS) {
      LineF64 L;
      bool list = base + tid <= in_hi && load(base + tid, L);
      if (list && (far_nodes_add(f, L, sp1, false) || far_nodes_add(f, L, sp2, true))) list = false;
      const unsigned b = __ballot_sync(0xffffffffu, list);
      if (lane == 0) s_cnt[warp] = __popc(b);
      __syncthreads();
      int off = n_list, total = 0;
      for (int w = 0; w < D_WARPS; ++w) {
        off += w < warp ? s_cnt[w] : 0;
        total += s_cnt[w];
      }
      if (list) s_list[off + __popc(b & ((1u << lane) - 1u))] = L;
      n_list += total;
      __syncthreads();
      if (n_list > D_LIST - D_THREADS || base + D_THREADS > in_hi) {
        const double v = reduce16_f64(f, lane);      // node sums leave the registers first
        if (!(lane & 1)) s_part[warp][lane >> 1] += v;
#pragma unroll
        for (int k = 0; k < D_K; ++k) f[k] = 0.0;
        pass_list();
        n_list = 0;
        __syncthreads();
      }
    }
    // the sub-chunk's series: its node sums plus the chunk's series at its nodes
    __syncthreads();
    if (tid < D_K) {
      double v = 0.0;
      for (int w = 0; w < D_WARPS; ++w) v += s_part[w][tid];
      s_val[tid] = v + clenshaw_f64(s_c1, ((sp2.c - sp1.c) + sp2.h * D_NODE(tid)) / sp1.h);
    }
    __syncthreads();
    if (tid < D_K) s_c2[tid] = dct_f64(s_val, tid);
    __syncthreads();
    if (n_g > 0) {
      double v;
      if (use3) {
        if (lane < D_K)
          s_seg[warp][lane] += clenshaw_f64(s_c2, ((sp3.c - sp2.c) + sp3.h * D_NODE(lane)) / sp2.h);
        __syncwarp();
        const double c = lane < D_K ? dct_f64(s_seg[warp], lane) : 0.0;
        __syncwarp();
        if (lane < D_K) s_seg[warp][lane] = c;
        __syncwarp();
        v = clenshaw_f64(s_seg[warp], (nu - sp3.c) / sp3.h);
      } else {
        v = n_w > 1 ? clenshaw_f64(s_c2, (nu - sp2.c) / sp2.h) : s_val[0];
      }
      if (lane < n_g) {
        const double o = __dmul_rn(acc + v, radiation_term_grid(nu, T));
        bad |= !isfinite(o);
        out[c0 + g0 + lane] = o;
      }
    }
    __syncthreads();                                 // s_c2, s_part and s_list are rewritten
  }
  if (bad) flag_error(err, row * (n_grp + 1) + n_grp);
}

}  // namespace lbl

using namespace lbl;

extern "C" int lbl_tau_tiles_f64(const LineF64* prep, int n_lines, const int* ranges, const double* t_layer,
                                 int n_rows, double nu_min, double step, long long n_nu, int tile_samples,
                                 double cutoff, int n_grp, double* od, int* err, unsigned long long* evals,
                                 void* stream) {
  if (!prep || !ranges || !t_layer || !od || n_lines < 1 || n_rows < 1 || n_rows > 65535 || n_nu < 1 ||
      tile_samples < 1 || !(step > 0) || !(cutoff >= 0) || n_grp < 1)
    return lbl_set_error(LBL_EINVAL, "lbl_tau_tiles_f64: bad arguments");
  const long long n_tiles = (n_nu + tile_samples - 1) / tile_samples;
  const long long chunks = (tile_samples + D_CHUNK - 1) / D_CHUNK;
  if (n_tiles * chunks > 0x7fffffffLL) return lbl_set_error(LBL_EINVAL, "lbl_tau_tiles_f64: grid too large");
  dim3 grid((unsigned)(n_tiles * chunks), (unsigned)n_rows);
  tau_f64_kernel<<<grid, D_THREADS, 0, (cudaStream_t)stream>>>(prep, n_lines, (const int2*)ranges, t_layer, nu_min,
                                                                step, n_nu, tile_samples, (int)chunks, D_CHUNK,
                                                                cutoff, n_grp, od, err, evals);
  return lbl_check_launch("lbl_tau_tiles_f64");
}
