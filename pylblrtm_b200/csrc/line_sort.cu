// Band mask, sort by centre and gather of the candidate lines (pylblrtm/forward.py:190-220)
// as one entry point, and every tile's line ranges in one launch.
//
// Keys are nu0 of the lines the reference masks in and +inf otherwise; ties break on the
// input index, so the order, and every sum built on it, is deterministic. Blocks of 512
// lines are sorted in registers and shared memory (bitonic), then groups of eight sorted runs
// are merged by rank: every element finds how many elements of the seven other runs precede
// it (seven independent binary searches, so their loads overlap) and writes itself to its
// place. 512 -> 4,096 -> 32,768 -> 262,144 lines: two to four launches where the stages of a
// global bitonic sort took 2 (2,048 lines) to 38 (200,000). The last pass writes the sorted
// records directly. Latency-bound. On B200: 16,000 lines 23 us (58 by the
// mask, bitonic sort and gather kernels of prep.cu), 200,000 lines 80 us (270).
#include <float.h>
#include <limits.h>
#include <math.h>

#include "lbl_common.cuh"

namespace lbl {

constexpr int LS_BLOCK = 512;     // lines sorted per CTA
constexpr int LS_RUNS = 8;        // runs merged per pass
constexpr int LS_THREADS = 256;   // threads of the merge pass

struct LineColumns {
  const double *nu0, *sref, *g_air, *g_self, *elow, *n_air, *shift;
  const int* gid;
};

__device__ __forceinline__ bool before(double ka, int va, double kb, int vb) {
  return ka < kb || (ka == kb && va < vb);
}

// Record `rank` of the sorted lines; slots past the kept lines get an inactive record
// (nu0 = NaN, group 0, src = -1).
__device__ __forceinline__ void write_record(const LineColumns& L, int rank, int i, int kept, int n_out, LineIn* out) {
  if (rank >= n_out) return;
  LineIn r;
  if (rank < kept) {
    r.nu0 = L.nu0[i]; r.sref = L.sref[i]; r.g_air = L.g_air[i]; r.g_self = L.g_self[i];
    r.elow = L.elow[i]; r.n_air = L.n_air[i]; r.shift = L.shift[i]; r.gid = L.gid[i]; r.src = i;
  } else {
    r.nu0 = CUDART_NAN; r.sref = 0.0; r.g_air = 0.0; r.g_self = 0.0;
    r.elow = 0.0; r.n_air = 0.0; r.shift = 0.0; r.gid = 0; r.src = -1;
  }
  out[rank] = r;
}

// Masks and sorts 512 lines; counts[block] = kept lines among them. A list of one block is
// written out at once.
__global__ void __launch_bounds__(LS_BLOCK)
line_block_sort_kernel(LineColumns L, int n_lines, double mask_lo, double mask_hi, double p_max,
                       double* __restrict__ keys, int* __restrict__ vals, int* __restrict__ counts, int single, int n_out,
                       LineIn* __restrict__ out, int* __restrict__ n_kept) {
  __shared__ double s_k[2][LS_BLOCK];
  __shared__ int s_v[2][LS_BLOCK];
  const int t = threadIdx.x, i = blockIdx.x * LS_BLOCK + t;
  double key = CUDART_INF;
  int val = i;
  if (i < n_lines && L.gid[i] >= 0) {
    const double sb = __dmul_rn(fabs(L.shift[i]), p_max);      // forward.py:191
    const double v = L.nu0[i];
    // a non-finite centre never lies in a tile window, so it can be dropped here
    if (isfinite(v) && v >= __dsub_rn(mask_lo, sb) && v <= __dadd_rn(mask_hi, sb)) key = v;
  }
  const int kept = __syncthreads_count(key < CUDART_INF);
  int buf = 0;
  for (int k = 2; k <= LS_BLOCK; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      double ok;
      int ov;
      if (j >= 32) {                                           // partner in another warp
        s_k[buf][t] = key;
        s_v[buf][t] = val;
        __syncthreads();                                       // buffers alternate: one barrier per stage
        ok = s_k[buf][t ^ j];
        ov = s_v[buf][t ^ j];
        buf ^= 1;
      } else {
        ok = __shfl_xor_sync(0xffffffffu, key, j);
        ov = __shfl_xor_sync(0xffffffffu, val, j);
      }
      const bool lower = (t & j) == 0, asc = (t & k) == 0;
      if (before(ok, ov, key, val) == (lower == asc)) {
        key = ok;
        val = ov;
      }
    }
  }
  if (single) {
    write_record(L, t, val, kept, n_out, out);
    if (t == 0) *n_kept = kept;
    return;
  }
  keys[i] = key;
  vals[i] = val;
  if (t == 0) counts[blockIdx.x] = kept;
}

// Merges groups of eight sorted runs of `run` elements (n = whole blocks; the last runs of
// the list may be short or empty). Runs hold consecutive stretches of the input, so among
// equal keys those of an earlier run come first and the values need no look. STAGED: runs of
// 512, whose group of 4,096 keys goes to shared memory first (2,000 lines: 9.2 -> 7.0 us). The
// last pass (out != NULL) writes the records.
template <bool STAGED>
__global__ void __launch_bounds__(LS_THREADS)
line_merge_kernel(const double* __restrict__ keys, const int* __restrict__ vals, int n, int run,
                  double* __restrict__ keys_out, int* __restrict__ vals_out, LineColumns L,
                  const int* __restrict__ counts, int n_blocks, int n_out, LineIn* __restrict__ out,
                  int* __restrict__ n_kept) {
  constexpr int GROUP = LS_BLOCK * LS_RUNS;
  static_assert(GROUP % LS_THREADS == 0, "a CTA's elements lie in one group");
  __shared__ double s_key[STAGED ? GROUP : 1];
  __shared__ int s_kept;
  const int e = blockIdx.x * LS_THREADS + threadIdx.x;         // n <= 2^30: whole blocks fit an int
  const long long group = (long long)run * LS_RUNS;
  const int base = (int)(e / group * group);
  if (STAGED)
#pragma unroll                                                  // all 16 loads of a thread in flight
    for (int i = threadIdx.x; i < GROUP; i += LS_THREADS) s_key[i] = base + i < n ? keys[base + i] : CUDART_INF;
  if (out && threadIdx.x == 0) s_kept = 0;
  if (STAGED || out) __syncthreads();
  if (out) {                                                   // kept lines of the whole list
    int c = 0;
    for (int b = threadIdx.x; b < n_blocks; b += LS_THREADS) c += counts[b];
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_kept, c);
    __syncthreads();
    if (e == 0) *n_kept = s_kept;
  }
  if (e >= n) return;
  const double* kg = STAGED ? s_key : keys + base;             // the group's keys
  const int left = n - base;                                   // elements of the list from the group on
  const double key = kg[e - base];
  const int val = vals[e];
  const int own = (e - base) / run;
  int at[LS_RUNS - 1], end[LS_RUNS - 1];                       // elements of run q before this one: [.., at)
#pragma unroll
  for (int q = 0; q < LS_RUNS - 1; ++q) {
    const long long f = (long long)run * (q + (q >= own ? 1 : 0));
    at[q] = (int)min(f, (long long)left);
    end[q] = (int)min(f + run, (long long)left);
  }
  int rank = e - base - own * run;
#pragma unroll
  for (int q = 0; q < LS_RUNS - 1; ++q) rank -= at[q];
  for (int s = run; s >= 1; s >>= 1) {
    double k[LS_RUNS - 1];
#pragma unroll
    for (int q = 0; q < LS_RUNS - 1; ++q) k[q] = at[q] + s <= end[q] ? kg[at[q] + s - 1] : CUDART_NAN;
#pragma unroll
    for (int q = 0; q < LS_RUNS - 1; ++q)
      if (q < own ? k[q] <= key : k[q] < key) at[q] += s;      // NaN: past the run's end
  }
#pragma unroll
  for (int q = 0; q < LS_RUNS - 1; ++q) rank += at[q];
  if (out) {
    write_record(L, base + rank, val, s_kept, n_out, out);
  } else {
    keys_out[base + rank] = key;
    vals_out[base + rank] = val;
  }
}

// First line (of n) whose centre is >= x (strict: > x), by a whole warp: 32 probes a step, so
// 200,000 lines take four dependent loads instead of eighteen.
__device__ __forceinline__ int warp_bound(const LineIn* __restrict__ lines, int n, double x, bool strict, int lane) {
  int lo = 0, hi = n;                                          // the answer lies in [lo, hi]
  while (hi > lo) {
    const int step = (hi - lo + 31) / 32;
    const int p = lo + lane * step;                            // probe p: does line p precede the bound?
    bool less = false;
    if (p < hi) {
      const double v = lines[p].nu0;
      less = strict ? v <= x : v < x;
    }
    const int k = __popc(__ballot_sync(0xffffffffu, less));    // probes that precede it: a prefix
    if (k == 0) return lo;
    const int last = lo + (k - 1) * step;                      // precedes; the next probe does not
    hi = min(hi, lo + k * step);
    lo = last + 1;
  }
  return lo;
}

// Ranges of sorted lines per tile: set s of tile t holds the lines within reach[s] + pad of
// the tile's first and last grid values; a warp per bound (pylblrtm/forward.py:295-301 for
// the window, narrower reaches for the inner lines of the multi-level sums).
struct RangeSets {
  double reach[3];
  int2* out[3];
};
__global__ void __launch_bounds__(256)
line_ranges_kernel(const LineIn* __restrict__ lines, const int* __restrict__ n_kept, double nu_min, double step,
                   long long n_nu, int tile_samples, double pad, int n_tiles, const __grid_constant__ RangeSets sets,
                   int n_sets) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= 2LL * n_sets * n_tiles) return;
  const int side = (int)(w & 1), s = (int)((w >> 1) % n_sets), t = (int)((w >> 1) / n_sets);
  const long long i0 = (long long)t * tile_samples;
  const long long i1 = min(i0 + tile_samples, n_nu) - 1;
  const double x = side == 0 ? __dsub_rn(__dsub_rn(grid_nu(nu_min, step, i0), sets.reach[s]), pad)
                             : __dadd_rn(__dadd_rn(grid_nu(nu_min, step, i1), sets.reach[s]), pad);
  const int b = warp_bound(lines, *n_kept, x, side == 1, lane);
  if (lane == 0) {
    if (side == 0) sets.out[s][t].x = b;
    else sets.out[s][t].y = b;
  }
}

}  // namespace lbl

using namespace lbl;

extern "C" size_t lbl_sort_gather_workspace_bytes(int n_lines) {
  if (n_lines < 1 || n_lines > (1 << 30)) return 0;
  const size_t blocks = ((size_t)n_lines + LS_BLOCK - 1) / LS_BLOCK, n = blocks * LS_BLOCK;
  return 2 * n * (sizeof(double) + sizeof(int)) + blocks * sizeof(int);
}

extern "C" int lbl_sort_gather(const double* nu0, const double* sref, const double* g_air, const double* g_self,
                               const double* elow, const double* n_air, const double* shift, const int* gid,
                               int n_lines, double mask_lo, double mask_hi, double p_max, void* workspace,
                               size_t workspace_bytes, int n_out, LineIn* out, int* n_kept, void* stream) {
  if (n_lines < 1 || n_lines > (1 << 30) || !nu0 || !sref || !g_air || !g_self || !elow || !n_air || !shift || !gid ||
      !workspace || n_out < 1 || !out || !n_kept || ((uintptr_t)workspace) % 8)
    return lbl_set_error(LBL_EINVAL, "lbl_sort_gather: bad arguments");
  if (workspace_bytes < lbl_sort_gather_workspace_bytes(n_lines))
    return lbl_set_error(LBL_EINVAL, "lbl_sort_gather: workspace too small");
  const LineColumns L = {nu0, sref, g_air, g_self, elow, n_air, shift, gid};
  const cudaStream_t st = (cudaStream_t)stream;
  const int blocks = (n_lines + LS_BLOCK - 1) / LS_BLOCK, n = blocks * LS_BLOCK;
  if (n_out > n) return lbl_set_error(LBL_EINVAL, "lbl_sort_gather: more output slots than lines");
  double* k[2] = {(double*)workspace, (double*)workspace + n};
  int* v[2] = {(int*)(k[1] + n), (int*)(k[1] + n) + n};
  int* counts = v[1] + n;
  line_block_sort_kernel<<<blocks, LS_BLOCK, 0, st>>>(L, n_lines, mask_lo, mask_hi, p_max, k[0], v[0], counts,
                                                      blocks == 1, n_out, out, n_kept);
  int from = 0;
  for (long long run = LS_BLOCK; blocks > 1 && run < n; run *= LS_RUNS, from ^= 1) {
    const bool last = run * LS_RUNS >= n;
    auto* merge = run == LS_BLOCK ? line_merge_kernel<true> : line_merge_kernel<false>;
    merge<<<(n + LS_THREADS - 1) / LS_THREADS, LS_THREADS, 0, st>>>(
        k[from], v[from], n, (int)run, k[from ^ 1], v[from ^ 1], L, counts, blocks, n_out, last ? out : nullptr, n_kept);
  }
  return lbl_check_launch("lbl_sort_gather");
}

extern "C" int lbl_line_ranges(const LineIn* lines, const int* n_kept, double nu_min, double step, long long n_nu,
                               int tile_samples, double cutoff, double pad, int n_tiles, int* ranges, int* inner,
                               int* near, void* stream) {
  if (n_nu < 1 || tile_samples < 1 || n_tiles < 1 || !lines || !n_kept || !ranges || !(step > 0))
    return lbl_set_error(LBL_EINVAL, "lbl_line_ranges: bad arguments");
  RangeSets s = {};
  int n = 0;
  s.reach[n] = cutoff;
  s.out[n++] = (int2*)ranges;
  if (inner) {
    s.reach[n] = lbl_ml_inner_reach(tile_samples, step);
    s.out[n++] = (int2*)inner;
  }
  if (near) {
    s.reach[n] = lbl_jac_near_reach(tile_samples, step);
    s.out[n++] = (int2*)near;
  }
  const long long warps = 2LL * n * n_tiles;
  line_ranges_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>(lines, n_kept, nu_min, step, n_nu,
                                                                                    tile_samples, pad, n_tiles, s, n);
  return lbl_check_launch("lbl_line_ranges");
}
