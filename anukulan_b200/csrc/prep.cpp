// Host-side preparation: CSR copy/validation, transpose, diagonal scaling and
// the row-block schedule of the staged SpMV.
#include "prep.hpp"

#include <algorithm>
#include <chrono>
#include <cmath>

namespace anu {

double now_seconds() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch())
      .count();
}

std::string validate_csr(int32_t rows, int32_t cols, int32_t nnz, const int32_t* start,
                         const int32_t* index) {
  if (rows < 0 || cols < 0 || nnz < 0) return "negative dimensions";
  if (rows > 0 && start == nullptr) return "null row starts";
  if (nnz > 0 && index == nullptr) return "null column indices";
  if (start != nullptr) {
    if (start[0] != 0) return "start does not begin at 0";
    if (start[rows] != nnz) return "start does not end at nnz";
    for (int32_t r = 0; r < rows; ++r)
      if (start[r + 1] < start[r]) return "start is not monotone at row " + std::to_string(r);
  }
  for (int32_t k = 0; k < nnz; ++k)
    if (index[k] < 0 || index[k] >= cols) return "column index out of range";
  return "";
}

HostCsr copy_csr(int32_t rows, int32_t cols, int32_t nnz, const int32_t* start,
                 const int32_t* index, const double* value) {
  HostCsr a;
  a.rows = rows;
  a.cols = cols;
  a.start.assign(start, start + rows + 1);
  a.index.assign(index, index + nnz);
  a.value.assign(value, value + nnz);
  return a;
}

HostCsr transpose(const HostCsr& a) { return transpose(a, nullptr); }

HostCsr transpose(const HostCsr& a, std::vector<int32_t>* pos) {
  HostCsr t;
  t.rows = a.cols;
  t.cols = a.rows;
  t.start.assign(static_cast<std::size_t>(a.cols) + 1, 0);
  t.index.resize(a.index.size());
  t.value.resize(a.value.size());
  for (const int32_t c : a.index) t.start[static_cast<std::size_t>(c) + 1]++;
  for (std::size_t i = 1; i < t.start.size(); ++i) t.start[i] += t.start[i - 1];
  std::vector<int32_t> cursor(t.start.begin(), t.start.end() - 1);
  if (pos != nullptr) pos->resize(a.index.size());
  for (int32_t r = 0; r < a.rows; ++r) {
    for (int32_t k = a.start[r]; k < a.start[r + 1]; ++k) {
      const int32_t dest = cursor[a.index[k]]++;
      t.index[dest] = r;
      t.value[dest] = a.value[k];
      if (pos != nullptr) (*pos)[dest] = k;
    }
  }
  return t;
}

void multiply(const HostCsr& a, const double* x, double* y) {
  for (int32_t r = 0; r < a.rows; ++r) {
    double sum = 0.0;
    for (int32_t k = a.start[r]; k < a.start[r + 1]; ++k) sum += a.value[k] * x[a.index[k]];
    y[r] = sum;
  }
}

namespace {

void row_norms(const HostCsr& a, bool one_norm, std::vector<double>* out) {
  out->assign(static_cast<std::size_t>(a.rows), 0.0);
  for (int32_t r = 0; r < a.rows; ++r) {
    double acc = 0.0;
    for (int32_t k = a.start[r]; k < a.start[r + 1]; ++k) {
      const double v = std::fabs(a.value[k]);
      acc = one_norm ? acc + v : std::fmax(acc, v);
    }
    (*out)[r] = acc;
  }
}

void col_norms(const HostCsr& a, bool one_norm, std::vector<double>* out) {
  out->assign(static_cast<std::size_t>(a.cols), 0.0);
  for (std::size_t k = 0; k < a.value.size(); ++k) {
    const double v = std::fabs(a.value[k]);
    double& acc = (*out)[a.index[k]];
    acc = one_norm ? acc + v : std::fmax(acc, v);
  }
}

double spread(const std::vector<double>& norms) {
  double lo = kInf, hi = 0.0;
  for (const double v : norms) {
    if (v <= 0.0) continue;
    lo = std::fmin(lo, v);
    hi = std::fmax(hi, v);
  }
  return hi == 0.0 ? 1.0 : hi / lo;
}

}  // namespace

double norm_spread(const std::vector<double>& norms) { return spread(norms); }

Scaling scale_matrix_sweeps(HostCsr* k, int ruiz_iterations, bool pock_chambolle,
                            ScalingSweeps* sweeps) {
  Scaling s;
  s.row_scale.assign(static_cast<std::size_t>(k->rows), 1.0);
  s.col_scale.assign(static_cast<std::size_t>(k->cols), 1.0);
  std::vector<double> rn, cn;
  row_norms(*k, false, &rn);
  col_norms(*k, false, &cn);
  s.row_spread_before = spread(rn);
  s.col_spread_before = spread(cn);
  const int total = ruiz_iterations + (pock_chambolle ? 1 : 0);
  sweeps->d1.clear();
  sweeps->d2.clear();
  for (int sweep = 0; sweep < total; ++sweep) {
    const bool one = sweep >= ruiz_iterations;
    row_norms(*k, one, &rn);
    col_norms(*k, one, &cn);
    std::vector<double> d1(rn.size()), d2(cn.size());
    for (std::size_t i = 0; i < rn.size(); ++i) d1[i] = rn[i] > 0.0 ? 1.0 / std::sqrt(rn[i]) : 1.0;
    for (std::size_t j = 0; j < cn.size(); ++j) d2[j] = cn[j] > 0.0 ? 1.0 / std::sqrt(cn[j]) : 1.0;
    for (int32_t r = 0; r < k->rows; ++r)
      for (int32_t e = k->start[r]; e < k->start[r + 1]; ++e) k->value[e] *= d1[r];
    for (std::size_t e = 0; e < k->value.size(); ++e) k->value[e] *= d2[k->index[e]];
    for (std::size_t i = 0; i < d1.size(); ++i) s.row_scale[i] *= d1[i];
    for (std::size_t j = 0; j < d2.size(); ++j) s.col_scale[j] *= d2[j];
    sweeps->d1.push_back(std::move(d1));
    sweeps->d2.push_back(std::move(d2));
  }
  row_norms(*k, false, &rn);
  col_norms(*k, false, &cn);
  s.row_spread_after = spread(rn);
  s.col_spread_after = spread(cn);
  return s;
}

void scale_vectors(const ScalingSweeps& sw, int32_t m, int32_t n, double* c, double* q,
                   double* lower, double* upper) {
  for (std::size_t s = 0; s < sw.d1.size(); ++s) {
    const std::vector<double>& d1 = sw.d1[s];
    const std::vector<double>& d2 = sw.d2[s];
    for (int32_t i = 0; i < m; ++i) q[i] *= d1[i];
    for (int32_t j = 0; j < n; ++j) {
      c[j] *= d2[j];
      lower[j] /= d2[j];
      upper[j] /= d2[j];
    }
  }
}

std::vector<RowBlock> row_blocks(const HostCsr& a, int32_t block_nnz, int32_t block_rows,
                                 int32_t long_row) {
  std::vector<RowBlock> blocks;
  int32_t r = 0;
  while (r < a.rows) {
    const int32_t len = a.start[r + 1] - a.start[r];
    if (len > long_row || len > block_nnz) {
      blocks.push_back({r, r + 1});
      ++r;
      continue;
    }
    const int32_t r0 = r;
    int32_t nnz = 0;
    while (r < a.rows && r - r0 < block_rows) {
      const int32_t l = a.start[r + 1] - a.start[r];
      if (l > long_row || l > block_nnz || nnz + l > block_nnz) break;
      nnz += l;
      ++r;
    }
    blocks.push_back({r0, r});
  }
  // Longest blocks first: a block of one long row runs longest, so starting it
  // in the first wave keeps it off the tail.
  std::stable_sort(blocks.begin(), blocks.end(), [&](const RowBlock& x, const RowBlock& y) {
    const int32_t nx = a.start[x.row_end] - a.start[x.row_begin];
    const int32_t ny = a.start[y.row_end] - a.start[y.row_begin];
    const bool lx = nx > block_nnz || (x.row_end - x.row_begin == 1 && nx > long_row);
    const bool ly = ny > block_nnz || (y.row_end - y.row_begin == 1 && ny > long_row);
    if (lx != ly) return lx;
    if (lx) return nx > ny;
    return false;
  });
  return blocks;
}

namespace {

// Nonzeros per segment of a row of `len`: seg_nnz, or more where the row would
// not fit a CTA's segments.
int32_t segment_step(int32_t len, int32_t seg_nnz, int32_t seg_per_cta) {
  return len > seg_nnz * seg_per_cta ? (len + seg_per_cta - 1) / seg_per_cta : seg_nnz;
}

// parts + 1 row bounds, cut where the running cost (a row's nonzeros plus
// kClusterRowCost) crosses each part's even share.
std::vector<int32_t> cluster_bounds(const HostCsr& a, int32_t parts) {
  std::vector<int32_t> bounds(static_cast<size_t>(parts) + 1, a.rows);
  bounds[0] = 0;
  const int64_t total = a.nnz() + static_cast<int64_t>(kClusterRowCost) * a.rows;
  int32_t part = 1;
  for (int32_t r = 0; r < a.rows && part < parts; ++r) {
    // Part `part` starts at the first row whose cost begins at or past its
    // share; a row never splits.
    const int64_t before = a.start[r] + static_cast<int64_t>(kClusterRowCost) * r;
    while (part < parts && before * parts >= total * part) bounds[part++] = r;
  }
  return bounds;
}

}  // namespace

SegmentSchedule segment_schedule(const HostCsr& a, int32_t seg_nnz, int32_t seg_per_cta,
                                 int32_t row_max) {
  SegmentSchedule s;
  s.row_seg.assign(static_cast<size_t>(a.rows) + 1, 0);
  for (int32_t r = 0; r < a.rows; ++r) {
    const int32_t b = a.start[r], e = a.start[r + 1];
    const int32_t step = segment_step(e - b, seg_nnz, seg_per_cta);
    s.row_seg[r] = static_cast<int32_t>(s.seg_begin.size());
    for (int32_t k = b; k < e; k += step) s.seg_begin.push_back(k);
  }
  s.row_seg[a.rows] = static_cast<int32_t>(s.seg_begin.size());
  s.seg_begin.push_back(a.nnz());
  s.cta_row.push_back(0);
  s.cta_seg.push_back(0);
  int32_t r = 0;
  while (r < a.rows) {
    const int32_t r0 = r;
    int32_t count = 0;
    while (r < a.rows && r - r0 < row_max) {
      const int32_t c = s.row_seg[r + 1] - s.row_seg[r];
      if (count + c > seg_per_cta && r > r0) break;
      count += c;
      ++r;
    }
    s.cta_row.push_back(r);
    s.cta_seg.push_back(s.row_seg[r]);
  }
  return s;
}

ClusterShape cluster_shape(const HostCsr& a, int32_t parts, int32_t serial_row, int32_t seg_nnz,
                           int32_t seg_per_cta) {
  ClusterShape s;
  const std::vector<int32_t> bounds = cluster_bounds(a, parts);
  for (int32_t q = 0; q < parts; ++q) {
    int32_t apart = 0;
    for (int32_t r = bounds[q]; r < bounds[q + 1]; ++r) {
      const int32_t len = a.start[r + 1] - a.start[r];
      s.max_row = std::max(s.max_row, len);
      if (seg_nnz == 0) {
        apart += len > serial_row ? 1 : 0;
      } else {
        const int32_t step = segment_step(len, seg_nnz, seg_per_cta);
        if (len > step) apart += (len + step - 1) / step;
      }
    }
    s.max_rows = std::max(s.max_rows, bounds[q + 1] - bounds[q]);
    s.max_nnz = std::max(s.max_nnz, a.start[bounds[q + 1]] - a.start[bounds[q]]);
    s.max_parts = std::max(s.max_parts, apart);
  }
  return s;
}

ClusterSchedule cluster_schedule(const HostCsr& a, int32_t parts, int32_t serial_row,
                                 const SegmentSchedule* seg) {
  ClusterSchedule c;
  c.bounds = cluster_bounds(a, parts);
  c.part_start.push_back(0);
  c.row.reserve(a.rows);
  c.entry.resize(a.index.size());
  constexpr int32_t kLanes = 32;
  for (int32_t q = 0; q < parts; ++q) {
    const int32_t rb = c.bounds[q], re = c.bounds[q + 1];
    const size_t p0 = c.part.size();
    int32_t slots = 0;
    // Here `first` is the sum's first nonzero; the layout below replaces it.
    for (int32_t r = rb; r < re; ++r) {
      const int32_t b = a.start[r], len = a.start[r + 1] - b;
      const int32_t g0 = seg != nullptr ? seg->row_seg[r] : 0;
      const int32_t g1 = seg != nullptr ? seg->row_seg[r + 1] : (len > serial_row ? 2 : 1);
      if (g1 - g0 <= 1) {
        c.row.push_back({r, b, len, 0});
      } else if (seg == nullptr) {
        c.row.push_back({r, slots, 1, 1});
        c.part.push_back({b, len, slots++});
      } else {
        c.row.push_back({r, slots, g1 - g0, 1});
        for (int32_t g = g0; g < g1; ++g) {
          const int32_t e = g + 1 < g1 ? seg->seg_begin[g + 1] : a.start[r + 1];
          c.part.push_back({seg->seg_begin[g], e - seg->seg_begin[g], slots++});
        }
      }
    }
    std::stable_sort(c.row.begin() + rb, c.row.begin() + re,
                     [](const ClusterSchedule::Row& x, const ClusterSchedule::Row& y) {
                       return (x.apart ? 0 : x.count) > (y.apart ? 0 : y.count);
                     });
    int32_t entries = 0;
    auto lay_out = [&](int32_t* first, int32_t count, int32_t at, int32_t step) {
      for (int32_t k = 0; k < count; ++k) c.entry[*first + k] = at + k * step;
      *first = at;
    };
    // Thread-summed: the i-th row (or segment) in lane i % 32 of its group.
    auto lanes = [&](auto&& get, int32_t count) {
      for (int32_t i0 = 0; i0 < count; i0 += kLanes) {
        int32_t longest = 0;
        for (int32_t i = i0; i < std::min(count, i0 + kLanes); ++i) {
          auto* d = get(i);
          if (d == nullptr) continue;
          longest = std::max(longest, d->count);
          lay_out(&d->first, d->count, entries + i - i0, kLanes);
        }
        entries += longest * kLanes;
      }
    };
    lanes([&](int32_t i) { return c.row[rb + i].apart ? nullptr : &c.row[rb + i]; }, re - rb);
    if (seg != nullptr) {
      lanes([&](int32_t i) { return &c.part[p0 + i]; }, static_cast<int32_t>(c.part.size() - p0));
    } else {
      for (size_t i = p0; i < c.part.size(); ++i) {
        lay_out(&c.part[i].first, c.part[i].count, entries, 1);
        entries += c.part[i].count;
      }
    }
    c.part_start.push_back(static_cast<int32_t>(c.part.size()));
    c.max_rows = std::max(c.max_rows, re - rb);
    c.max_entries = std::max(c.max_entries, entries);
    c.max_parts = std::max(c.max_parts, slots);
  }
  c.stride = (c.max_rows + 3) / 4 * 4;
  c.place.resize(a.rows);
  for (int32_t q = 0; q < parts; ++q)
    for (int32_t r = c.bounds[q]; r < c.bounds[q + 1]; ++r)
      c.place[c.row[r].row] = q * c.stride + (r - c.bounds[q]);
  return c;
}

}  // namespace anu
