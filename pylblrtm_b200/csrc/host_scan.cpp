// One host pass over the line list for the group selection of pylblrtm/forward.py:189-245
// (liblblio.so): the distinct (mol_id, iso_id) pairs, how many lines of each fall inside
// the band mask of forward.py:190-191, and the pair index of every line. The band test
// is evaluated in the reference's operation order,
//     sb = |shift| * p_max;  in = (nu0 >= (nu_first - cutoff) - sb) & (nu0 <= (nu_last + cutoff) + sb)
// and this file is compiled with floating-point contraction off, so every comparison
// sees the same doubles as NumPy's.
#include <float.h>
#include <math.h>
#include <string.h>

#include <thread>
#include <vector>

#include "../../include/lblio.h"

// Runs fn(part, begin, end) over [0, n) in `parts` contiguous parts, the first one on the calling
// thread (threads cost ~20 us each to start; a list of 200,000 lines is scanned in 0.2 instead of
// 0.6 ms). A thread that cannot be started has its part run by the caller.
template <typename F>
static void in_parts(long long n, int parts, F fn) {
  std::vector<std::thread> pool;
  int started = 1;
  try {
    pool.reserve(parts);
    for (; started < parts; ++started)
      pool.emplace_back(fn, started, n * started / parts, n * (started + 1) / parts);
  } catch (...) {
  }
  for (int p = started; p < parts; ++p) fn(p, n * p / parts, n * (p + 1) / parts);
  fn(0, 0ll, n / parts);
  for (std::thread& t : pool) t.join();
}

static int part_count(long long n, long long grain, int cap) {
  long long p = n / grain, hw = (long long)std::thread::hardware_concurrency();
  if (p > cap) p = cap;
  if (hw > 0 && p > hw) p = hw;
  return p < 1 ? 1 : (int)p;
}

extern "C" int lbl_line_pairs(const int* mol, const int* iso, const double* nu0, const double* shift, long long n,
                              double lo_edge, double hi_edge, double p_max, int max_pairs, int* pair_mol,
                              int* pair_iso, long long* pair_band, int* n_pairs, int* pair_index,
                              double* max_abs_shift) {
  if (n < 0 || max_pairs < 1 || !n_pairs || (n > 0 && (!mol || !iso || !nu0 || !shift || !pair_index)) ||
      !pair_mol || !pair_iso || !pair_band || !max_abs_shift)
    return LBL_EINVAL;
  int np_ = 0, last = -1;
  double smax = -1.0;                               // largest finite |shift| (-1: none)
  for (long long i = 0; i < n; ++i) {
    const int m = mol[i], s = iso[i];
    int k = last;
    if (k < 0 || pair_mol[k] != m || pair_iso[k] != s) {
      k = -1;
      for (int j = 0; j < np_; ++j)
        if (pair_mol[j] == m && pair_iso[j] == s) {
          k = j;
          break;
        }
      if (k < 0) {
        if (np_ >= max_pairs) return LBL_EINVAL;
        k = np_++;
        pair_mol[k] = m;
        pair_iso[k] = s;
        pair_band[k] = 0;
      }
      last = k;
    }
    pair_index[i] = k;
    const double as = fabs(shift[i]);
    if (isfinite(as) && as > smax) smax = as;
    const double sb = as * p_max;
    const double v = nu0[i];
    if ((v >= lo_edge - sb) & (v <= hi_edge + sb)) ++pair_band[k];
  }
  *n_pairs = np_;
  *max_abs_shift = smax;
  return LBL_OK;
}

extern "C" int lbl_map_index(const int* index, long long n, const int* lut, int n_lut, int* out) {
  if (n < 0 || n_lut < 0 || (n > 0 && (!index || !lut || !out))) return LBL_EINVAL;
  unsigned bad = 0;
  for (long long i = 0; i < n; ++i) {
    const int k = index[i];
    const bool ok = k >= 0 && k < n_lut;
    bad |= !ok;
    out[i] = lut[ok ? k : 0];
  }
  return bad ? LBL_EINVAL : LBL_OK;
}

// Host count of the lines the device sort keeps (lbl_sort_lines): gid >= 0, finite nu0
// inside [lo_edge - |shift| p_max, hi_edge + |shift| p_max], the same comparisons in the
// same order, so the count equals the device's. Sizes a wavenumber shard's buffers when
// the band edges are narrowed to the shard's line window.
extern "C" long long lbl_count_band(const double* nu0, const double* shift, const int* gid, long long n,
                                    double lo_edge, double hi_edge, double p_max) {
  if (n < 0 || (n > 0 && (!nu0 || !shift || !gid))) return -1;
  long long c = 0;
  for (long long i = 0; i < n; ++i) {
    if (gid[i] < 0) continue;
    const double sb = fabs(shift[i]) * p_max;
    const double v = nu0[i];
    c += isfinite(v) && (v >= lo_edge - sb) && (v <= hi_edge + sb);
  }
  return c;
}

// lbl_line_pairs that also lists the lines inside the band mask: band_line[i], band_pair[i]
// (i < *n_band, input order; both of capacity n). Each part of the list fills its own stretch
// of the outputs, which are then closed up.
extern "C" int lbl_band_scan(const int* mol, const int* iso, const double* nu0, const double* shift, long long n,
                             double lo_edge, double hi_edge, double p_max, int max_pairs, int* pair_mol,
                             int* pair_iso, long long* pair_band, int* n_pairs, int* band_line, int* band_pair,
                             long long* n_band, double* max_abs_shift) {
  if (n < 0 || n > 0x7fffffffLL || max_pairs < 1 || !n_pairs || !n_band || !max_abs_shift || !pair_mol ||
      !pair_iso || !pair_band || (n > 0 && (!mol || !iso || !nu0 || !shift || !band_line || !band_pair)))
    return LBL_EINVAL;
  struct Part {
    std::vector<int> mol, iso;
    std::vector<long long> band;
    long long begin = 0, kept = 0;
    double smax = -1.0;
    bool full = false;
  };
  const int parts = part_count(n, 16384, 6);
  std::vector<Part> part;
  try {
    part.resize(parts);
    for (Part& q : part) {
      q.mol.resize(max_pairs);
      q.iso.resize(max_pairs);
      q.band.assign(max_pairs, 0);
    }
  } catch (...) {
    return LBL_EINVAL;
  }
  in_parts(n, parts, [&](int p, long long a, long long b) {
    Part& q = part[p];
    q.begin = a;
    int* pm = q.mol.data();
    int* pi = q.iso.data();
    int np_ = 0, last = -1;
    long long kept = a;
    double sm[4] = {-1.0, -1.0, -1.0, -1.0};
    unsigned char in[1024];
    for (long long i = a; i < b;) {
      const int m = mol[i], s = iso[i];
      int k = last;
      if (k < 0 || pm[k] != m || pi[k] != s) {
        for (k = 0; k < np_ && (pm[k] != m || pi[k] != s); ++k) {
        }
        if (k == np_) {
          if (np_ >= max_pairs) {
            q.full = true;
            return;
          }
          pm[np_] = m;
          pi[np_] = s;
          ++np_;
        }
        last = k;
      }
      long long e = i + 1;                           // the run of lines of this pair (at most 1,024)
      const long long stop = b - i > 1024 ? i + 1024 : b;
      while (e < stop && mol[e] == m && iso[e] == s) ++e;
      const int len = (int)(e - i);
      const double* vs = nu0 + i;
      const double* ss = shift + i;
      for (int j = 0; j < len; ++j) {
        const double sb = fabs(ss[j]) * p_max;
        in[j] = (unsigned char)((vs[j] >= lo_edge - sb) & (vs[j] <= hi_edge + sb));
      }
      for (int j = 0; j < len; ++j) {                // four chains: the comparison's latency
        const double as = fabs(ss[j]), fin = as <= DBL_MAX ? as : -1.0;
        sm[j & 3] = fin > sm[j & 3] ? fin : sm[j & 3];
      }
      const long long before = kept;
      for (int j = 0; j < len; ++j) {
        band_line[kept] = (int)(i + j);              // kept <= i + j: no branch on the outcome
        band_pair[kept] = k;
        kept += in[j];
      }
      q.band[k] += kept - before;
      i = e;
    }
    q.mol.resize(np_);
    q.iso.resize(np_);
    q.kept = kept - a;
    q.smax = fmax(fmax(sm[0], sm[1]), fmax(sm[2], sm[3]));
  });
  int np_ = 0;
  long long out = 0;
  double smax = -1.0;
  std::vector<int> to;
  for (Part& q : part) {                             // parts in order: pairs come in first-seen order
    if (q.full) return LBL_EINVAL;
    try {
      to.assign(q.mol.size(), 0);
    } catch (...) {
      return LBL_EINVAL;
    }
    for (size_t j = 0; j < q.mol.size(); ++j) {
      int k = 0;
      while (k < np_ && (pair_mol[k] != q.mol[j] || pair_iso[k] != q.iso[j])) ++k;
      if (k == np_) {
        if (np_ >= max_pairs) return LBL_EINVAL;
        pair_mol[k] = q.mol[j];
        pair_iso[k] = q.iso[j];
        pair_band[k] = 0;
        ++np_;
      }
      to[j] = k;
      pair_band[k] += q.band[j];
    }
    if (q.smax > smax) smax = q.smax;
    if (out != q.begin && q.kept > 0) memmove(band_line + out, band_line + q.begin, sizeof(int) * (size_t)q.kept);
    bool same = out == q.begin;
    for (size_t j = 0; j < to.size(); ++j) same &= to[j] == (int)j;
    if (!same)
      for (long long i = 0; i < q.kept; ++i) band_pair[out + i] = to[band_pair[q.begin + i]];
    out += q.kept;
  }
  *n_pairs = np_;
  *n_band = out;
  *max_abs_shift = smax;
  return LBL_OK;
}

// The listed lines whose group lut[band_pair[i]] is not negative and, with `narrowed`, that lie
// inside the band [lo_edge - |shift| p_max, hi_edge + |shift| p_max] (lbl_count_band's
// comparisons): their seven columns, one after the other with stride `stride`, into out and
// their groups into gid, in list order. out may be NULL (count only). Returns how many, -1
// for bad arguments or when they exceed `stride`.
extern "C" long long lbl_pack_band(const double* const* cols, const int* band_line, const int* band_pair,
                                   long long n_band, const int* lut, int n_lut, int narrowed, double lo_edge,
                                   double hi_edge, double p_max, double* out, long long stride, int* gid) {
  if (!cols || n_band < 0 || n_lut < 0 || (n_band > 0 && (!band_line || !band_pair || !lut)) || (out && !gid))
    return -1;
  const int parts = part_count(n_band, 4096, 3);     // a cache miss per value where the list is unsorted;
                                                     // more threads' cores make the upload's reads slow
  long long first[9] = {0}, kept[8] = {0};
  bool bad[8] = {false};
  auto group = [&](long long i) {                    // -1: not kept
    const int g = lut[band_pair[i]];
    if (g < 0 || !narrowed) return g;
    const double v = cols[0][band_line[i]], sb = fabs(cols[6][band_line[i]]) * p_max;
    return isfinite(v) && v >= lo_edge - sb && v <= hi_edge + sb ? g : -1;
  };
  auto count = [&](int p, long long a, long long b) {
    long long c = 0;
    for (long long i = a; i < b; ++i) {
      if (band_pair[i] < 0 || band_pair[i] >= n_lut) {
        bad[p] = true;
        return;
      }
      c += group(i) >= 0;
    }
    kept[p] = c;
  };
  for (int p = 0; p < parts; ++p) count(p, n_band * p / parts, n_band * (p + 1) / parts);
  for (int p = 0; p < parts; ++p) {
    if (bad[p]) return -1;
    first[p + 1] = first[p] + kept[p];
  }
  const long long total = first[parts];
  if (!out) return total;
  if (total > stride) return -1;
  in_parts(n_band, parts, [&](int p, long long a, long long b) {
    long long o = first[p];
    for (long long i = a; i < b; ++i) {
      const int g = group(i);
      if (g < 0) continue;
      const long long l = band_line[i];
      for (int c = 0; c < 7; ++c) out[c * stride + o] = cols[c][l];
      gid[o++] = g;
    }
  });
  return total;
}
