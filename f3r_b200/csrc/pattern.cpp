// pattern.cpp -- finds the row patterns of an offset-aligned SELL matrix and
// lays them out for k_sell_pattern (pattern.cuh).  Host work over the stored
// form (slices, slot bases, values), so that a row's pattern is exactly what
// the streamed kernels would read for it, padding and clamped columns included.
#include <cstring>
#include <map>
#include <numeric>

#include "objects.cuh"

namespace f3r {

namespace {

struct Row {
  std::vector<int32_t> d;  // column - row
  std::vector<double> v;
  bool operator==(const Row &o) const {
    return d == o.d && v.size() == o.v.size() && std::memcmp(v.data(), o.v.data(), v.size() * 8) == 0;
  }
  uint64_t hash() const {
    uint64_t h = 1469598103934665603ull ^ d.size();
    for (size_t k = 0; k < d.size(); k++) {
      uint64_t b;
      std::memcpy(&b, &v[k], 8);
      h = (h ^ (uint32_t)d[k]) * 1099511628211ull;
      h = (h ^ b ^ (b >> 29)) * 1099511628211ull;
    }
    return h;
  }
};

// storage row r as the kernels read it
void read_row(const SellHost &h, int64_t r, Row &o) {
  const int32_t H = h.height, s = (int32_t)(r / H), q = (int32_t)(r % H), w = h.sptr[s + 1] - h.sptr[s];
  const bool explicit_cols = !h.xoff.empty() && h.xoff[s] >= 0, clamp = h.aligned_all && (h.cbptr[s] & 1);
  const int32_t chunk = h.aligned_all ? kAllAlignedChunk : kAlignedChunk;
  o.d.resize(w);
  o.v.resize(w);
  for (int32_t k = 0; k < w; k++) {
    int32_t c;
    if (explicit_cols) {
      c = h.col[h.xoff[s] + (int64_t)k * 32 + q];
    } else {
      c = h.cbase[(h.cbptr[s] & ~3) + k] + q;
      if (clamp) c = std::min(std::max(c, 0), h.ncols - 1);
    }
    const int32_t k0 = k / chunk * chunk, kw = std::min(chunk, w - k0);
    o.d[k] = c - (int32_t)r;
    o.v[k] = h.val[(int64_t)h.sptr[s] * H + (int64_t)k0 * H + (int64_t)q * kw + (k - k0)];
  }
}

struct Run {
  int32_t d, len;
  double v[3];
};
struct Pattern {
  Row row;
  std::vector<Run> runs;
  bool pad = false;
};

// what k_sell_pattern reads, on the host
struct Layout {
  PatArgs a{};
  int warps = 0;
  PatArgs ab{};  // tiles of one block
  std::vector<Pattern> pats;
  std::vector<int32_t> soff, soffb;  // of every run, pattern by pattern
  std::vector<uint8_t> blk, live;
  std::vector<int32_t> irow, iptr, icol;
  std::vector<double> ival;
  int32_t listed = 0;  // rows off their block's pattern
};

// the runs of a pattern; false where its offsets do not increase or are too many
bool make_runs(Pattern &p) {
  int32_t w = (int32_t)p.row.d.size();
  const std::vector<int32_t> &d = p.row.d;
  while (w > 1 && d[w - 1] == d[w - 2] && p.row.v[w - 1] == 0.0 && !std::signbit(p.row.v[w - 1])) {
    p.pad = true;  // zeros times the last x again: one stands for all
    w--;
  }
  for (int32_t k = 1; k < w; k++)
    if (d[k] <= d[k - 1]) return false;
  for (int32_t k = 0; k < w;) {
    const int32_t len = k + 2 < w && d[k + 1] == d[k] + 1 && d[k + 2] == d[k] + 2 ? 3 : 1;
    Run r{d[k], len, {0, 0, 0}};
    for (int32_t j = 0; j < len; j++) r.v[j] = p.row.v[k + j];
    p.runs.push_back(r);
    k += len;
  }
  return w > 0 && (int)p.runs.size() <= kPatRuns;
}

// The windows of x that tiles of a.tile rows read, and every run's place in the
// stage; offsets less than a tile apart share a window (the rows between cost
// less than a window of their own).
bool windows(const std::vector<Pattern> &pats, PatArgs &a, std::vector<int32_t> &soff) {
  std::vector<int32_t> offs;
  for (const Pattern &q : pats)
    for (const Run &r : q.runs) {
      offs.push_back(r.d);
      offs.push_back(r.d + r.len - 1);
    }
  std::sort(offs.begin(), offs.end());
  auto down = [](int64_t v) { return (int32_t)((v >= 0 ? v : v - (kPatUnit - 1)) / kPatUnit * kPatUnit); };
  std::vector<std::pair<int32_t, int32_t>> win;
  for (const int32_t e : offs) {
    if (!win.empty() && (int64_t)e - win.back().second < a.tile) win.back().second = e;
    else win.emplace_back(e, e);
  }
  if ((int)win.size() > kPatWindows) return false;
  a.nwin = (int32_t)win.size();
  int64_t elems = 0;
  for (int w = 0; w < a.nwin; w++) {
    const int32_t lo = down(win[w].first);
    // up to 8 elements past the last row's last one are read (and not used)
    const int64_t len = cdiv((int64_t)a.tile + win[w].second - lo + 9, kPatUnit) * kPatUnit;
    if (elems + len >= kPatLong) return false;
    a.win[w] = PatWindow{lo, (int32_t)len, (int32_t)elems};
    elems += len;
  }
  a.elems = (int32_t)elems;
  for (const Pattern &q : pats)
    for (const Run &r : q.runs)
      for (int w = 0; w < a.nwin; w++)
        if (r.d >= win[w].first && r.d <= win[w].second) {
          soff.push_back(a.win[w].base + r.d - a.win[w].lo);
          break;
        }
  return true;
}

template <typename T> Status put(Context &c, DevPattern &p, T **d, const T *h, size_t count) {
  F3R_TRY(c.alloc((void **)d, std::max<size_t>(count, 1) * sizeof(T)));
  p.allocs.push_back((void *)*d);
  if (count) CUDA_TRY(cudaMemcpyAsync(*d, h, count * sizeof(T), cudaMemcpyHostToDevice, c.stream));
  return F3R_SUCCESS;
}

struct Temp {
  void *p = nullptr;
  ~Temp() { cudaFree(p); }
};

// v in type T as the device rounds the matrix's values
template <typename T> Status rounded(Context &c, const std::vector<double> &v, std::vector<T> &o) {
  Temp a, b;
  o.resize(v.size());
  F3R_TRY(c.alloc(&a.p, v.size() * 8));
  F3R_TRY(c.alloc(&b.p, v.size() * sizeof(T)));
  double *d = static_cast<double *>(a.p);
  T *t = static_cast<T *>(b.p);
  CUDA_TRY(cudaMemcpyAsync(d, v.data(), v.size() * 8, cudaMemcpyHostToDevice, c.stream));
  launch_k(c, k_convert_vals<T>, c.ew_grid((int64_t)v.size()), kEwThreads, 0, c.stream, (const double *)d, t,
           (int64_t)v.size());
  CUDA_TRY(cudaMemcpyAsync((void *)o.data(), t, v.size() * sizeof(T), cudaMemcpyDeviceToHost, c.stream));
  CUDA_TRY(cudaStreamSynchronize(c.stream));
  return F3R_SUCCESS;
}

// the pattern table and the other rows' values in type V
template <typename V>
Status put_values(Context &c, DevPattern &p, const Layout &o, PatRun<V> *(&tab)[2], V **val) {
  const std::vector<Pattern> &pats = o.pats;
  const std::vector<double> &ival = o.ival;
  std::vector<double> flat;
  for (const Pattern &q : pats)
    for (const Run &r : q.runs) flat.insert(flat.end(), r.v, r.v + 3);
  std::vector<V> rv;
  F3R_TRY(rounded<V>(c, flat, rv));
  for (int i = 0; i < (o.ab.ntiles > 0 ? 2 : 1); i++) {
    const std::vector<int32_t> &soff = i ? o.soffb : o.soff;
    std::vector<PatRun<V>> t((size_t)p.a.np * p.a.stride);
    std::memset((void *)t.data(), 0, t.size() * sizeof(PatRun<V>));
    size_t at = 0;
    for (size_t q = 0; q < pats.size(); q++) {
      PatRun<V> *r = t.data() + q * p.a.stride;
      bool lng = true;
      for (const Run &e : pats[q].runs) lng = lng && e.len == 3;
      r[0].at = (int32_t)pats[q].runs.size() | (pats[q].pad ? kPatPadded : 0) | (lng ? kPatAllLong : 0);
      for (size_t k = 0; k < pats[q].runs.size(); k++, at++) {
        r[k + 1].at = soff[at] | (pats[q].runs[k].len == 3 ? kPatLong : 0);
        for (int j = 0; j < 3; j++) r[k + 1].v[j] = rv[3 * at + j];
      }
    }
    F3R_TRY(put(c, p, &tab[i], t.data(), t.size()));
    CUDA_TRY(cudaStreamSynchronize(c.stream));  // t is read until then
  }
  F3R_TRY(c.alloc((void **)val, std::max<size_t>(ival.size(), 1) * sizeof(V)));
  p.allocs.push_back((void *)*val);
  if (!ival.empty()) {
    Temp a;
    F3R_TRY(c.alloc(&a.p, ival.size() * 8));
    double *d = static_cast<double *>(a.p);
    CUDA_TRY(cudaMemcpyAsync(d, ival.data(), ival.size() * 8, cudaMemcpyHostToDevice, c.stream));
    launch_k(c, k_convert_vals<V>, c.ew_grid((int64_t)ival.size()), kEwThreads, 0, c.stream, (const double *)d, *val,
             (int64_t)ival.size());
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(c.stream));
  }
  return F3R_SUCCESS;
}

}  // namespace

// Set up for offset-aligned storage in natural order, rows longer than the
// thread-a-row kernels', matrices large enough (pattern_rows), and only where at
// least half of the rows follow at most kPatMax patterns (each block's most
// frequent row); the other rows cost about 2.5 times as much as those that do.
static bool layout(const SellHost &h, int sm_count, Layout &o) {
  const int64_t n = h.n;
  const bool aligned = h.aligned_all || !h.xoff.empty();
  if (!aligned || h.sigma != 1 || h.max_width <= kDirectShort || 
      n < pattern_rows(sm_count, 32, 8))
    return false;
  {  // a matrix of varying coefficients shows in a few rows
    std::map<uint64_t, int> seen;
    Row row;
    int most = 0;
    constexpr int kSample = 512;
    for (int i = 0; i < kSample; i++) {
      read_row(h, n * i / kSample, row);
      most = std::max(most, ++seen[row.hash()]);
    }
    if (most * 8 < kSample) return false;
  }
  // every block's leading pattern: its most frequent row (a majority vote)
  const int32_t nblk = (int32_t)cdiv(n, kPatBlock);
  std::vector<int64_t> lead(nblk);
  std::vector<uint64_t> lead_hash(nblk);
#pragma omp parallel for schedule(dynamic, 64)
  for (int32_t b = 0; b < nblk; b++) {
    Row row;
    int64_t cand = 0;
    uint64_t ch = 0;
    int votes = 0;
    for (int64_t r = (int64_t)b * kPatBlock; r < std::min<int64_t>(n, (int64_t)(b + 1) * kPatBlock); r++) {
      read_row(h, r, row);
      const uint64_t x = row.hash();
      if (votes == 0) {
        cand = r;
        ch = x;
      }
      votes += x == ch ? 1 : -1;
    }
    lead[b] = cand;
    lead_hash[b] = ch;
  }
  std::map<uint64_t, std::pair<int64_t, int64_t>> count;  // hash -> blocks, one row
  for (int32_t b = 0; b < nblk; b++) {
    auto &e = count[lead_hash[b]];
    e.first++;
    e.second = lead[b];
  }
  std::vector<std::pair<int64_t, int64_t>> order;
  for (auto &kv : count) order.push_back(kv.second);
  std::sort(order.begin(), order.end(), [](const auto &x, const auto &y) { return x.first > y.first; });
  std::vector<Pattern> &pats = o.pats;
  for (auto &e : order) {
    if ((int)pats.size() == kPatMax) break;
    Pattern p;
    read_row(h, e.second, p.row);
    if (make_runs(p)) pats.push_back(std::move(p));
  }
  if (pats.empty()) return false;
  std::map<uint64_t, int> index;
  for (size_t q = 0; q < pats.size(); q++) index[pats[q].row.hash()] = (int)q;
  // which rows follow their block's pattern, value for value
  std::vector<uint8_t> &blk = o.blk, &live = o.live;
  blk.assign(nblk, 0);
  live.assign((size_t)nblk * 32, 0);
  std::vector<uint8_t> off(n, 1);
  int64_t regular = 0;
#pragma omp parallel for schedule(dynamic, 64) reduction(+ : regular)
  for (int32_t b = 0; b < nblk; b++) {
    const auto it = index.find(lead_hash[b]);
    if (it == index.end()) continue;
    blk[b] = (uint8_t)it->second;
    Row row;
    for (int64_t r = (int64_t)b * kPatBlock; r < std::min<int64_t>(n, (int64_t)(b + 1) * kPatBlock); r++) {
      read_row(h, r, row);
      if (!(row == pats[it->second].row)) continue;
      const int q = (int)(r % kPatBlock);
      live[(size_t)b * 32 + q % 128 / 4] |= (uint8_t)(1 << (q / 128 * 4 + q % 4));
      off[r] = 0;
      regular++;
    }
  }
  if (regular * 2 < n) return false;
  PatArgs &a = o.a;
  // tiles of 2,048 rows, half of that on smaller systems so that every SM gets several
  o.warps = n >= (int64_t)sm_count * 4096 ? kPatWarps : kPatWarps / 2;
  a.n = (int32_t)n;
  a.ncols = h.ncols;
  a.nblk = nblk;
  a.tile = o.warps * kPatBlock;
  a.ntiles = (int32_t)cdiv(n, a.tile);
  a.np = (int32_t)pats.size();
  a.stride = 1;
  for (const Pattern &q : pats) a.stride = std::max<int32_t>(a.stride, (int32_t)q.runs.size() + 1);
  o.ab = a;
  o.ab.tile = kPatBlock;
  o.ab.ntiles = nblk;
  if (!windows(pats, a, o.soff)) return false;
  if (pattern_shape(a, o.warps, 2, sizeof(PatRun<__half>)).stages == 0) return false;
  // offsets a block or more apart take a window each there (a 27-point stencil on lines of 258 rows and
  // more has 9): the K-column products then stream the matrix, the others keep their 3
  if (!windows(pats, o.ab, o.soffb)) o.ab.ntiles = 0;
  // the other rows, grouped by width
  std::vector<int32_t> rest;
  for (int64_t r = 0; r < n; r++)
    if (off[r]) rest.push_back((int32_t)r);
  o.listed = (int32_t)rest.size();
  auto width = [&](int32_t r) { return h.sptr[r / h.height + 1] - h.sptr[r / h.height]; };
  std::stable_sort(rest.begin(), rest.end(), [&](int32_t x, int32_t y) { return width(x) < width(y); });
  std::vector<int32_t> &irow = o.irow, &iptr = o.iptr;
  iptr.assign(1, 0);
  for (size_t i = 0; i < rest.size();) {
    const int32_t w = width(rest[i]);
    for (int l = 0; l < 32; l++) {
      const bool in = i < rest.size() && width(rest[i]) == w;
      irow.push_back(in ? rest[i] : -1);
      if (in) i++;
    }
    if ((int64_t)iptr.back() + w > INT32_MAX / 32) return false;
    iptr.push_back(iptr.back() + w);
  }
  a.ngroups = (int32_t)iptr.size() - 1;
  std::vector<int32_t> &icol = o.icol;
  std::vector<double> &ival = o.ival;
  icol.assign((size_t)iptr.back() * 32, 0);
  ival.assign((size_t)iptr.back() * 32, 0.0);
#pragma omp parallel for schedule(static)
  for (int32_t g = 0; g < a.ngroups; g++) {
    Row row;
    for (int l = 0; l < 32; l++) {
      const int32_t r = irow[(size_t)g * 32 + l];
      if (r < 0) continue;
      read_row(h, r, row);
      for (int32_t k = 0; k < iptr[g + 1] - iptr[g]; k++) {
        icol[((size_t)iptr[g] + k) * 32 + l] = r + row.d[k];
        ival[((size_t)iptr[g] + k) * 32 + l] = row.v[k];
      }
    }
  }
  return true;
}

static Status upload_pattern(Context &c, const Layout &o, int dtype_mask, DeviceSell &d) {
  auto dp = std::make_unique<DevPattern>();
  DevPattern &p = *dp;
  p.a = o.a;
  p.warps = o.warps;
  p.listed_rows = o.listed;
  p.listed_entries = (int64_t)o.icol.size();
  uint8_t *bd = nullptr, *ld = nullptr;
  int32_t *rd = nullptr, *pd = nullptr, *cd = nullptr;
  F3R_TRY(put(c, p, &bd, o.blk.data(), o.blk.size()));
  F3R_TRY(put(c, p, &ld, o.live.data(), o.live.size()));
  F3R_TRY(put(c, p, &rd, o.irow.data(), o.irow.size()));
  F3R_TRY(put(c, p, &pd, o.iptr.data(), o.iptr.size()));
  F3R_TRY(put(c, p, &cd, o.icol.data(), o.icol.size()));
  p.a.blk = bd;
  p.a.live = ld;
  p.a.irow = rd;
  p.a.iptr = pd;
  p.a.icol = cd;
  p.ab = o.ab;
  p.ab.ngroups = p.a.ngroups;
  p.ab.blk = bd;
  p.ab.live = ld;
  p.ab.irow = rd;
  p.ab.iptr = pd;
  p.ab.icol = cd;
  if (dtype_mask & (1 << F3R_F64)) F3R_TRY(put_values<double>(c, p, o, p.t64, &p.v64));
  if (dtype_mask & (1 << F3R_F32)) F3R_TRY(put_values<float>(c, p, o, p.t32, &p.v32));
  if (dtype_mask & (1 << F3R_F16)) F3R_TRY(put_values<__half>(c, p, o, p.t16, &p.v16));
  CUDA_TRY(cudaStreamSynchronize(c.stream));
  d.pat = dp.release();
  return F3R_SUCCESS;
}

// A matrix works without its patterns: where the device has no room for them, it does.
Status make_pattern(Context &c, const SellHost &h, int dtype_mask, DeviceSell &d) {
  Layout o;
  if (!layout(h, c.sm_count, o)) return F3R_SUCCESS;
  const Status s = upload_pattern(c, o, dtype_mask, d);
  if (s != F3R_ERROR_OUT_OF_MEMORY) return s;
  clear_stale_error();
  return F3R_SUCCESS;
}

}  // namespace f3r
