// Line cells of the level-1 kernels (tau_far_kernel, jac_far_kernel): stretches of the sorted
// lines between every wp-th grid point, whose far wings are summed through moments about the
// cell's centre (voigt_ml.cu for the expansion).
#pragma once

#include "lbl_common.cuh"

namespace lbl {

constexpr float CELL_RATIO = 1.0f / 6.5f;
constexpr int CELL_MIN = 4;                    // fewer lines are cheaper one by one
constexpr int CELL_MIN_CHUNKS = 16;            // fewer chunks on the grid: no cells
constexpr int CELL_MIN_PTS = 64;               // smallest cell (bounds the records to 1 byte per point and row)
constexpr int LINE_CELLS = 512;                // most cells of a tile's window (more: every line by itself)

struct CellGeom {
  int wp, n;            // points per cell, cells (0: none)
  long long off;        // cell q starts at grid index q * wp - off
};

// A quarter of a chunk per cell: far cells (beyond four half-widths) then have |zeta| / |D| of
// about 1/13. No cells where no line can be that far, for chunks shorter than two cells, for a
// grid of few chunks (each cell serves them all), or where a full tile's window holds more
// cells than split_lines takes, since their moments would be formed and never used (25 cm^-1
// cut-off: tiles below 0.4 cm^-1 at 0.001 cm^-1; 2 cm^-1 tiles at 0.0002 cm^-1 and finer, the
// Jacobian's shorter chunks at 0.0004). The rule looks at the grid alone and split_lines at
// what lies inside the tile's window, so a shard takes the same cells as the full job, bit for
// bit.
static inline CellGeom cell_geometry(long long n_nu, int tile_samples, double step, double cutoff, int chunk_max) {
  const long long nch = (tile_samples + chunk_max - 1) / chunk_max;
  const long long n_c = tile_samples / nch;
  CellGeom g = {0, 0, 0};
  const double reach = cutoff / step;
  if (n_c < 2 * CELL_MIN_PTS || !(reach > 2.0 * (double)n_c) || reach > 1.0e9 ||
      (n_nu + tile_samples - 1) / tile_samples * nch < CELL_MIN_CHUNKS)
    return g;
  g.wp = (int)(n_c / 4 > CELL_MIN_PTS ? n_c / 4 : CELL_MIN_PTS);
  const long long tile = tile_samples < n_nu ? tile_samples : n_nu;
  if ((tile + 2 * (long long)reach) / g.wp + 6 > LINE_CELLS) return CellGeom{0, 0, 0};   // qe - qa of split_lines
  g.off = ((long long)reach / g.wp + 2) * g.wp;
  const long long n = (n_nu + 2 * g.off + g.wp - 1) / g.wp;
  if (n > 0x3fffffff) return CellGeom{0, 0, 0};
  g.n = (int)n;
  return g;
}

// idx[q] = first sorted line whose unshifted centre is at or beyond the start of cell q (q <= n).
static __global__ void cell_bounds_kernel(const LineIn* __restrict__ lines, const int* __restrict__ n_kept, double nu_min,
                                   double step, CellGeom cg, int* __restrict__ idx) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q > cg.n) return;
  const double x = grid_nu(nu_min, step, (long long)q * cg.wp - cg.off);
  int a = 0, b = *n_kept;
  while (a < b) {
    const int m = (a + b) >> 1;
    if (lines[m].nu0 < x) a = m + 1; else b = m;
  }
  idx[q] = a;
}

// Layout of a cell buffer: cell bounds (int, n + 1, padded to 4), then the records, whose last
// four floats are e_min, e_max (the lines' extent about the cell's centre, points), a_min and
// the number of active lines (-1: a line too broad or of negative width).
static inline long long cell_head(const CellGeom& g) { return ((long long)g.n + 1 + 3) / 4 * 4; }

template <int T>
struct LineSplit {
  int use[LINE_CELLS];                             // cells evaluated through their moments
  int dir[LINE_CELLS], pre[LINE_CELLS + 1];        // stretches of the other lines: start, lines before
  int wu[T / 32], wd[T / 32], wl[T / 32];          // per-warp scan totals
};

// Splits the lines rng of the tile [t0, t1) for the chunk at c0 of half-width H1 into n_use cells
// (sh.use) that lie, with every line, beyond four half-widths, inside the window and within
// their series' radius, and n_direct other lines in n_dir stretches. All threads of the CTA
// call it. False: no cells considered, the lines are rng itself. REC: floats per record, GMAX:
// the slot of g_max.
template <int T, int REC, int GMAX>
__device__ __forceinline__ bool split_lines(LineSplit<T>& sh, const CellGeom& cg, const int* __restrict__ cell_idx,
                                            const float* __restrict__ rec_row, int2 rng, long long t0, long long t1,
                                            long long c0, float H1, double cutoff, double step, int& n_use, int& n_dir,
                                            int& n_direct) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float C1 = H1;
  bool split = false;
  if (cg.n > 0 && n_direct > 0) {
    // the window in cells, with two cells on either side for shifted lines (checked below)
    const double win0 = cutoff / step;
    const int qa = (int)max(0LL, (t0 - (long long)win0 + cg.off) / cg.wp - 3);
    const int qe = (int)min((long long)cg.n, (t1 + (long long)win0 + cg.off) / cg.wp + 3);
    if (qe - qa <= LINE_CELLS && cell_idx[qa] <= rng.x && cell_idx[qe] >= rng.y) {
      const double wl = (double)(t0 - c0) - win0 + 1.0, wr = (double)(t1 - 1 - c0) + win0 - 1.0;   // a point of margin
      const float half = 0.5f * (float)cg.wp;
      n_dir = 0;
      n_direct = 0;
      split = true;
      for (int q0 = qa; q0 < qe; q0 += T) {
        const int q = q0 + tid;
        int i0 = 0, len = 0;
        bool use = false;
        if (q < qe) {
          const int a = cell_idx[q], b = cell_idx[q + 1];
          i0 = max(a, rng.x);
          len = max(0, min(b, rng.y) - i0);
          if (len > 0) {
            const float4 m = *reinterpret_cast<const float4*>(rec_row + (long long)q * REC + REC - 4);
            const float g_max = rec_row[(long long)q * REC + GMAX];
            const float pc = (float)((long long)q * cg.wp - cg.off - c0) + half;
            // the cell itself inside the window, so that its choice cannot depend on lines
            // beyond it, which a job of this tile's lines only does not hold
            const bool inside = (double)(pc - half) >= wl && (double)(pc + half) <= wr && i0 == a && len == b - a;
            if (inside && m.w == 0.f) len = 0;             // only inactive lines
            const float lo = pc + m.x, hi = pc + m.y;
            // all lines beyond four half-widths on one side, inside the window, in the far-wing
            // regime at the nearest node and well inside the series' radius
            const float gap = fmaxf(lo - (C1 + H1), (C1 - H1) - hi);
            const float z = fmaxf(fabsf(m.x), fabsf(m.y)) + g_max, D = fabsf(pc - C1) - H1;
            use = inside && m.w >= (float)CELL_MIN && gap > 3.f * H1 + 2.f && (double)lo >= wl && (double)hi <= wr &&
                  m.z * gap >= 50.f && z <= CELL_RATIO * D;
          }
        }
        const unsigned bu = __ballot_sync(0xffffffffu, use), bd = __ballot_sync(0xffffffffu, len > 0 && !use);
        int pl = len > 0 && !use ? len : 0;                // inclusive scan of the other lines
        const int own = pl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, pl, o);
          if (lane >= o) pl += u;
        }
        if (lane == 31) {
          sh.wu[warp] = __popc(bu);
          sh.wd[warp] = __popc(bd);
          sh.wl[warp] = pl;
        }
        __syncthreads();
        int ou = n_use, od = n_dir, ol = n_direct;
        for (int w = 0; w < T / 32; ++w) {
          if (w < warp) {
            ou += sh.wu[w];
            od += sh.wd[w];
            ol += sh.wl[w];
          }
          n_use += sh.wu[w];
          n_dir += sh.wd[w];
          n_direct += sh.wl[w];
        }
        const unsigned lt = (1u << lane) - 1u;
        if (use) sh.use[ou + __popc(bu & lt)] = q;
        if (own > 0) {
          const int o = od + __popc(bd & lt);
          sh.dir[o] = i0;
          sh.pre[o] = ol + pl - own;
        }
        __syncthreads();
      }
      if (tid == 0) sh.pre[n_dir] = n_direct;
    }
  }
  __syncthreads();
  return split;
}

// Line of slot `slot` (< n_direct) of the other lines.
template <int T>
__device__ __forceinline__ int split_line(const LineSplit<T>& sh, int n_dir, int slot) {
  int a = 0, b = n_dir - 1;
  while (a < b) {
    const int m = (a + b + 1) >> 1;
    if (sh.pre[m] <= slot) a = m; else b = m - 1;
  }
  return sh.dir[a] + (slot - sh.pre[a]);
}

}  // namespace lbl
