// Diagonal phase layers (b): RZ / U1 / Z / S / T, CZ / CPHASE / CRZ, ZZ and
// any mix of them, in ONE streaming pass.
//
// Replaces diag_pair_layer / diag_weighted_layer (shaders/diag.py:19-217),
// zz_chain_layer / zz_weighted_layer (shaders/zz.py:16-185) and the per-gate
// apply_diagonal passes of the CPU path (sim.py:94-138, device.py:1154-1211).
//
// The reference multiplies one unit phase per equal-angle group inside the
// kernel (zz.py:40-71); here the host factors the whole diagonal into at most
// eight lookup tables, each indexed by a window of <= 10 index bits (or by a
// short list of scattered bits for far-apart pairs).  Every term's phase is
// folded into exactly one table in double precision, so a 29-bond chain with
// all-different angles costs four table reads and four complex products per
// amplitude, independent of the number of bonds.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <initializer_list>
#include <vector>

#include "mq_internal.cuh"

namespace mq {

struct DiagLut {
  uint16_t off;
  uint8_t nbits;
  uint8_t contig;
  uint8_t shift;
  uint8_t pos[11];
};

constexpr int kMaxLuts = 8;
template <typename R> struct DiagCap;
template <> struct DiagCap<float> { static constexpr int v = 2048; };
template <> struct DiagCap<double> { static constexpr int v = 1024; };

template <typename R>
struct DiagParams {
  uint32_t n_pairs;  // 2^(n-1) element pairs
  int32_t n_luts;
  uint32_t n_entries;
  int32_t n_low;     // tables [0, n_low) read index bit 0
  int32_t pair_lut0; // table 0 is a contiguous window starting at bit 0
  int32_t pad[3];
  DiagLut lut[kMaxLuts];
  V2<R> e[DiagCap<R>::v];
};

__device__ __forceinline__ uint32_t lut_index(const DiagLut& L, uint32_t i) {
  if (L.contig) return (i >> L.shift) & ((1u << L.nbits) - 1u);
  uint32_t x = 0;
  for (int k = 0; k < L.nbits; ++k) x |= ((i >> L.pos[k]) & 1u) << k;
  return x;
}

// Each thread handles amplitude pairs (2p, 2p+1), four independent pairs per
// iteration, with 16-byte (complex64) accesses that are contiguous across the
// warp.  Tables [0, n_low) read index bit 0: when table 0 is a window starting
// at bit 0 (pair_lut0) the pair's two entries are adjacent and read as one
// 16-byte value; the other tables give one factor per pair.
template <typename R>
__global__ void __launch_bounds__(256) k_diag(V2<R>* __restrict__ st, const __grid_constant__ DiagParams<R> P) {
  using T = V2<R>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* lut = reinterpret_cast<T*>(smem_raw);
  for (uint32_t j = threadIdx.x; j < P.n_entries; j += blockDim.x) lut[j] = P.e[j];
  __syncthreads();
  constexpr int U = 4;
  const uint32_t stride = gridDim.x * blockDim.x;
  const int n_low = P.n_low;
  const bool pair0 = P.pair_lut0;
  for (uint32_t p0 = blockIdx.x * blockDim.x + threadIdx.x; p0 < P.n_pairs; p0 += U * stride) {
    T a0[U], a1[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t p = p0 + (uint32_t)u * stride;
      if (p < P.n_pairs) {
        if constexpr (sizeof(R) == 4) {
          const float4 x = reinterpret_cast<const float4*>(st)[p];
          a0[u] = make_float2(x.x, x.y);
          a1[u] = make_float2(x.z, x.w);
        } else {
          a0[u] = st[2 * p];
          a1[u] = st[2 * p + 1];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t p = p0 + (uint32_t)u * stride;
      if (p >= P.n_pairs) continue;
      const uint32_t i0 = 2 * p;
      T hi = mk<R>(1, 0);
      for (int l = n_low; l < P.n_luts; ++l) hi = cmul(hi, lut[P.lut[l].off + lut_index(P.lut[l], i0)]);
      T f0 = hi, f1 = hi;
      int l = 0;
      if (pair0 && n_low > 0) {
        const uint32_t k = P.lut[0].off + lut_index(P.lut[0], i0);
        f0 = cmul(f0, lut[k]);
        f1 = cmul(f1, lut[k + 1]);
        l = 1;
      }
      for (; l < n_low; ++l) {
        f0 = cmul(f0, lut[P.lut[l].off + lut_index(P.lut[l], i0)]);
        f1 = cmul(f1, lut[P.lut[l].off + lut_index(P.lut[l], i0 + 1)]);
      }
      const T b0 = cmul(a0[u], f0), b1 = cmul(a1[u], f1);
      if constexpr (sizeof(R) == 4) {
        reinterpret_cast<float4*>(st)[p] = make_float4(b0.x, b0.y, b1.x, b1.y);
      } else {
        st[i0] = b0;
        st[i0 + 1] = b1;
      }
    }
  }
}

// ---------------------------------------------------------------- planner
// at most N values in place (terms are copied while a plan is sought)
template <typename T, int N>
struct Few {
  int n = 0;
  T v[N];
  void push_back(T x) { v[n++] = x; }
  Few& operator=(std::initializer_list<T> l) {
    n = 0;
    for (const T& x : l) push_back(x);
    return *this;
  }
  const T* begin() const { return v; }
  const T* end() const { return v + n; }
  size_t size() const { return (size_t)n; }
  T& operator[](size_t i) { return v[i]; }
  const T& operator[](size_t i) const { return v[i]; }
};
struct Term {
  Few<int, 2> bits;                    // global index bits, first = MSB of table index
  Few<std::complex<double>, 4> tab;    // 2^|bits| values
  int lo = 0, hi = 0;                  // lowest and highest bit
};

struct PlannedLut {
  std::vector<int> pos;  // index bit k of the table <- global bit pos[k]
  bool contig = false;
  std::vector<const Term*> members;          // terms the table holds
  std::vector<std::complex<double>> vals;    // filled by realize() once a plan is chosen
};
static size_t lut_size(const PlannedLut& L) { return L.vals.empty() ? (size_t(1) << L.pos.size()) : L.vals.size(); }

static std::complex<double> cis(double t) { return {std::cos(t), std::sin(t)}; }

static int build_terms(int n, int n_terms, const int32_t* kinds, const int32_t* wires, const double* params,
                       std::vector<Term>& terms, std::complex<double>& scalar) {
  scalar = 1.0;
  for (int t = 0; t < n_terms; ++t) {
    const int kind = kinds[t];
    const int a = wires[2 * t], b = wires[2 * t + 1];
    const double* p = params + 8 * t;
    const bool two = (kind == MQ_DIAG_ZZ || kind == MQ_DIAG_CPHASE || kind == MQ_DIAG_CRZ || kind == MQ_DIAG_2Q);
    const bool one = (kind == MQ_DIAG_RZ || kind == MQ_DIAG_PHASE || kind == MQ_DIAG_1Q);
    if (kind == MQ_DIAG_GLOBAL) { scalar *= cis(p[0]); continue; }
    if (!one && !two) return fail(MQ_EINVAL, "unknown diagonal term kind " + std::to_string(kind));
    if (a < 0 || a >= n) return fail(MQ_EINVAL, "diagonal term wire out of range");
    if (two && (b < 0 || b >= n || b == a)) return fail(MQ_EINVAL, "invalid bond (" + std::to_string(a) + ", " + std::to_string(b) + ")");
    Term tm;
    const double th = p[0];
    switch (kind) {
      case MQ_DIAG_ZZ: tm.tab = {cis(-th), cis(th), cis(th), cis(-th)}; break;
      case MQ_DIAG_CPHASE: tm.tab = {1.0, 1.0, 1.0, cis(th)}; break;
      case MQ_DIAG_CRZ: tm.tab = {1.0, 1.0, cis(-th / 2), cis(th / 2)}; break;
      case MQ_DIAG_2Q:
        tm.tab = {{p[0], p[1]}, {p[2], p[3]}, {p[4], p[5]}, {p[6], p[7]}};
        break;
      case MQ_DIAG_RZ: tm.tab = {cis(-th / 2), cis(th / 2)}; break;
      case MQ_DIAG_PHASE: tm.tab = {1.0, cis(th)}; break;
      case MQ_DIAG_1Q: tm.tab = {{p[0], p[1]}, {p[2], p[3]}}; break;
    }
    // CZ is CPHASE(pi): use exact -1 (diag.py:89-98 keeps +-1 exact too)
    if (kind == MQ_DIAG_CPHASE && std::fabs(th - M_PI) < 1e-15) tm.tab[3] = -1.0;
    if (kind == MQ_DIAG_PHASE && std::fabs(th - M_PI) < 1e-15) tm.tab[1] = -1.0;
    tm.bits.push_back(n - 1 - a);
    if (two) tm.bits.push_back(n - 1 - b);
    tm.lo = *std::min_element(tm.bits.begin(), tm.bits.end());
    tm.hi = *std::max_element(tm.bits.begin(), tm.bits.end());
    terms.push_back(std::move(tm));
  }
  return MQ_OK;
}

// v[x] *= the term's value at x, where bit p of x is the global bit pos[p], for
// every x.  Term by term over the whole table: an entry's factors multiply up
// in the order of the terms, and a run of entries takes one factor.  (The
// products are written out: std::complex checks each for infinities.)
static void multiply_term(std::vector<std::complex<double>>& v, const Term& tm, const std::vector<int>& pos) {
  auto at = [&](int bit) { return (int)(std::find(pos.begin(), pos.end(), bit) - pos.begin()); };
  const int hi = at(tm.bits[0]), lo = tm.bits.size() == 2 ? at(tm.bits[1]) : -1;  // table index: bits[0] first
  const size_t run = size_t(1) << (lo < 0 ? hi : std::min(hi, lo));
  for (size_t x = 0; x < v.size(); x += run) {
    const size_t i = lo < 0 ? (x >> hi) & 1u : (((x >> hi) & 1u) << 1) | ((x >> lo) & 1u);
    const double fr = tm.tab[i].real(), fi = tm.tab[i].imag();
    for (size_t k = x; k < x + run; ++k) {
      const double re = v[k].real(), im = v[k].imag();
      v[k] = {re * fr - im * fi, re * fi + im * fr};
    }
  }
}

static void finalize_lut(PlannedLut& L) {
  L.vals.assign(size_t(1) << L.pos.size(), 1.0);
  for (const Term* tm : L.members) multiply_term(L.vals, *tm, L.pos);
}
// Table values of a chosen plan (planning itself only sizes the tables).
static void realize(std::vector<PlannedLut>& luts) {
  for (auto& L : luts)
    if (L.vals.empty()) finalize_lut(L);
}

// Greedy factorisation with windows of width <= W.
static std::vector<PlannedLut> plan_luts(const std::vector<Term>& terms, int W) {
  std::vector<PlannedLut> luts;
  std::vector<int> local, far;
  for (size_t t = 0; t < terms.size(); ++t) {
    (terms[t].hi - terms[t].lo < W ? local : far).push_back((int)t);
  }
  std::vector<bool> done(terms.size(), false);
  while (true) {
    int s = 1 << 30;
    for (int t : local)
      if (!done[t]) s = std::min(s, terms[t].lo);
    if (s == (1 << 30)) break;
    std::vector<const Term*> members;
    int hi = s;
    for (int t : local) {
      if (done[t]) continue;
      if (terms[t].lo >= s && terms[t].hi < s + W) { done[t] = true; members.push_back(&terms[t]); hi = std::max(hi, terms[t].hi); }
    }
    PlannedLut L;
    for (int b = s; b <= hi; ++b) L.pos.push_back(b);
    L.contig = true;
    L.members = std::move(members);
    luts.push_back(std::move(L));
  }
  // far pairs: scattered-bit tables
  size_t i = 0;
  while (i < far.size()) {
    PlannedLut L;
    std::vector<const Term*> members;
    while (i < far.size()) {
      std::vector<int> pos = L.pos;
      for (int b : terms[far[i]].bits)
        if (std::find(pos.begin(), pos.end(), b) == pos.end()) pos.push_back(b);
      if ((int)pos.size() > W && !members.empty()) break;
      L.pos = pos;
      members.push_back(&terms[far[i]]);
      ++i;
    }
    std::sort(L.pos.begin(), L.pos.end());
    L.contig = true;
    for (size_t k = 1; k < L.pos.size(); ++k)
      if (L.pos[k] != L.pos[0] + (int)k) L.contig = false;
    L.members = std::move(members);
    luts.push_back(std::move(L));
  }
  return luts;
}

// Whether plan_luts(terms, W) would exceed `most` table entries or kMaxLuts
// tables, where that shows without building it (no term wider than a window).
static bool too_large(const std::vector<Term>& terms, int W, size_t most) {
  std::vector<bool> done(terms.size(), false);
  size_t entries = 0;
  for (const Term& t : terms)
    if (t.hi - t.lo >= W) return false;
  for (int tables = 0;; ++tables) {
    int s = 1 << 30;
    for (size_t t = 0; t < terms.size(); ++t)
      if (!done[t]) s = std::min(s, terms[t].lo);
    if (s == (1 << 30)) return entries > most;
    if (tables == kMaxLuts) return true;
    int hi = s;
    for (size_t t = 0; t < terms.size(); ++t)
      if (!done[t] && terms[t].hi < s + W) {
        done[t] = true;
        hi = std::max(hi, terms[t].hi);
      }
    entries += size_t(1) << (hi - s + 1);
  }
}

template <typename R>
static int launch_diag_pass(mq_state* h, const std::vector<PlannedLut>& in_luts) {
  using T = V2<R>;
  std::vector<PlannedLut> luts;
  auto has0 = [](const PlannedLut& L) { return std::find(L.pos.begin(), L.pos.end(), 0) != L.pos.end(); };
  for (const auto& L : in_luts)
    if (has0(L) && L.contig && L.pos[0] == 0) luts.push_back(L);
  const bool pair0 = !luts.empty();
  for (const auto& L : in_luts)
    if (has0(L) && !(L.contig && L.pos[0] == 0)) luts.push_back(L);
  const int n_low = (int)luts.size();
  for (const auto& L : in_luts)
    if (!has0(L)) luts.push_back(L);
  auto* P = new DiagParams<R>();
  std::memset(P, 0, sizeof(DiagParams<R>));
  P->n_pairs = (uint32_t)(h->dim() >> 1);
  P->n_luts = (int32_t)luts.size();
  P->n_low = n_low;
  P->pair_lut0 = pair0 ? 1 : 0;
  uint32_t off = 0;
  for (size_t l = 0; l < luts.size(); ++l) {
    const PlannedLut& L = luts[l];
    DiagLut& d = P->lut[l];
    d.off = (uint16_t)off;
    d.nbits = (uint8_t)L.pos.size();
    d.contig = L.contig ? 1 : 0;
    d.shift = (uint8_t)(L.pos.empty() ? 0 : L.pos[0]);
    for (size_t k = 0; k < L.pos.size(); ++k) d.pos[k] = (uint8_t)L.pos[k];
    for (auto v : L.vals) P->e[off++] = mk<R>((R)v.real(), (R)v.imag());
  }
  P->n_entries = off;
  const size_t smem = sizeof(T) * std::max<uint32_t>(off, 1);
  const uint32_t pairs = P->n_pairs;
  const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((pairs + 255) / 256, (uint64_t)h->num_sms * 8));
  k_diag<R><<<grid, 256, smem, h->stream>>>(reinterpret_cast<T*>(h->cur_buf()), *P);
  delete P;
  MQ_LAUNCHED("k_diag");
  h->launches += 1;
  h->sweeps += 1;
  return MQ_OK;
}

int check_diag_terms(const mq_state* h, int n_terms, const int32_t* kinds, const int32_t* wires, const double* params) {
  std::vector<Term> terms;
  std::complex<double> scalar;
  return build_terms(h->n, n_terms, kinds, wires, params, terms, scalar);
}

// The diagonal as contiguous-window tables for a tile-sweep epilogue (the
// fused layer of mq_tile.cu): same factorisation as launch_diag_terms, with
// the global phase folded into the first table.  out.n = -1 when no plan with
// <= 8 contiguous windows and <= max_entries entries exists.
int plan_diag_windows(mq_state* h, int n_terms, const int32_t* kinds, const int32_t* wires, const double* params,
                      int max_entries, DiagWindows& out) {
  std::vector<Term> terms;
  std::complex<double> scalar;
  int rc = build_terms(h->n, n_terms, kinds, wires, params, terms, scalar);
  if (rc) return rc;
  out = DiagWindows();
  out.n = -1;
  for (int W = 10; W >= 1; --W) {
    if (too_large(terms, W, (size_t)std::max(max_entries, 0))) continue;
    std::vector<PlannedLut> luts = plan_luts(terms, W);
    size_t entries = 0;
    bool contig = true;
    for (auto& L : luts) {
      entries += lut_size(L);
      contig = contig && L.contig && !L.pos.empty();
    }
    if (!contig || (int)luts.size() > kMaxLuts) continue;
    if (luts.empty()) {
      PlannedLut L;
      L.pos = {0};
      L.contig = true;
      L.vals = {1.0, 1.0};
      luts.push_back(L);
      entries = 2;
    }
    if ((int)entries > max_entries) continue;
    realize(luts);
    for (auto& v : luts[0].vals) v *= scalar;
    out.n = (int)luts.size();
    uint32_t off = 0;
    for (int l = 0; l < out.n; ++l) {
      out.shift[l] = luts[l].pos[0];
      out.nbits[l] = (int)luts[l].pos.size();
      out.off[l] = (int)off;
      for (auto v : luts[l].vals) {
        out.vals.push_back(v.real());
        out.vals.push_back(v.imag());
      }
      off += (uint32_t)luts[l].vals.size();
    }
    break;
  }
  return MQ_OK;
}

// The diagonal split for a register phase whose register bits are rbits[4]
// (ascending): phase(x) = W(x) * T[c(x)][r(x)] (row c at entry 17c) with r(x) the four register
// bits, c(x) the values of the (at most 3) other bits that share a term with
// a register bit, T the product of those terms, and W the remaining terms as
// contiguous windows that do not read the register bits (so W can be taken
// at the register group's base index).  out.n = -1 when this does not fit.
int plan_diag_register(mq_state* h, int n_terms, const int32_t* kinds, const int32_t* wires, const double* params,
                       const int* rbits, int max_entries, DiagRegister& out) {
  std::vector<Term> terms;
  std::complex<double> scalar;
  int rc = build_terms(h->n, n_terms, kinds, wires, params, terms, scalar);
  if (rc) return rc;
  out = DiagRegister();
  out.win.n = -1;
  auto is_reg = [&](int b) { return b == rbits[0] || b == rbits[1] || b == rbits[2] || b == rbits[3]; };
  std::vector<Term> group, reg;
  std::vector<int> cross;
  for (const Term& t : terms) {
    bool touches = false;
    for (int b : t.bits) touches = touches || is_reg(b);
    if (!touches) { group.push_back(t); continue; }
    reg.push_back(t);
    for (int b : t.bits)
      if (!is_reg(b) && std::find(cross.begin(), cross.end(), b) == cross.end()) cross.push_back(b);
  }
  if (cross.size() > 3) return MQ_OK;
  std::sort(cross.begin(), cross.end());
  // T[c][r]: value bit k of r = global bit rbits[k], bit j of c = cross[j]
  std::vector<int> pos = {rbits[0], rbits[1], rbits[2], rbits[3]};
  for (int b : cross) pos.push_back(b);
  const uint32_t nt = 1u << pos.size();
  std::vector<std::complex<double>> T(nt, scalar);
  for (const Term& t : reg) multiply_term(T, t, pos);
  // W: contiguous windows over the group terms
  std::vector<PlannedLut> luts;
  bool ok = false;
  for (int W = 10; W >= 1 && !ok; --W) {
    size_t entries = (nt / 16) * 17;
    if ((int)entries > max_entries || too_large(group, W, (size_t)max_entries - entries)) continue;
    luts = plan_luts(group, W);
    bool contig = true;
    for (auto& L : luts) {
      entries += lut_size(L);
      contig = contig && L.contig && !L.pos.empty();
    }
    ok = contig && (int)luts.size() <= kMaxLuts && (int)entries <= max_entries;
  }
  if (!ok) return MQ_OK;
  realize(luts);
  out.nc = (int)cross.size();
  for (int j = 0; j < out.nc; ++j) out.cbit[j] = cross[j];
  out.win.n = (int)luts.size();
  uint32_t off = 0;
  for (int l = 0; l < out.win.n; ++l) {
    out.win.shift[l] = luts[l].pos[0];
    out.win.nbits[l] = (int)luts[l].pos.size();
    out.win.off[l] = (int)off;
    for (auto v : luts[l].vals) {
      out.win.vals.push_back(v.real());
      out.win.vals.push_back(v.imag());
    }
    off += (uint32_t)luts[l].vals.size();
  }
  // rows of 16 at a stride of 17 entries: lanes that read rows c and c' of
  // the same register pattern hit different shared-memory banks
  out.t_off = (int)off;
  for (uint32_t c = 0; c < nt / 16; ++c) {
    for (uint32_t r = 0; r < 16; ++r) {
      out.win.vals.push_back(T[c * 16 + r].real());
      out.win.vals.push_back(T[c * 16 + r].imag());
    }
    out.win.vals.push_back(1.0);
    out.win.vals.push_back(0.0);
  }
  return MQ_OK;
}

// ------------------------------------------------- tiles of the index space
// The window tables above pay one look-up (for far bonds, one bit at a time)
// and one complex product per table and amplitude, and a graph with many far
// bonds needs eight of them.  This kernel uses that a term touches at most two
// bits.  With t[b_a][b_b] = c u_a^{b_a} u_b^{b_b} w^{b_a b_b} the whole diagonal is
//   c * prod_j u_j^{b_j} * prod_{i<j} w_ij^{b_i b_j},
// and for a tile of 2^M consecutive amplitudes (high bits H fixed) the pairs of
// low bits are the same in every tile (a thread keeps its 16 or 8 factors in
// shared memory), the pairs of high bits are one scalar, and the mixed pairs leave
// one factor f_l = u_l prod_{h in H} w_lh per low bit.  One warp forms the f_l
// and the scalar in float64 while the tile's loads are in flight, and 48
// threads turn them into three tables over four bits, so an amplitude costs
// three complex products whatever the graph.  Bound by memory: 26 qubits, a
// ring and a random matching (38 bonds): 553 us with eight tables, 177 us
// this way (6.1 TB/s).
template <typename R> struct DiagTile;
template <> struct DiagTile<float> { static constexpr int M = 12, CB = 1; };
template <> struct DiagTile<double> { static constexpr int M = 11, CB = 0; };
constexpr int kDiagLT = 8;  // 256 threads: index bits [CB, CB + 8)
constexpr int kDiagCtas = 4;   // resident CTAs per SM: 64 registers a thread
constexpr int kDiagHigh = 20;

template <typename R>
struct DiagTileParams {
  static constexpr int M = DiagTile<R>::M;
  uint32_t n_tiles;
  int32_t n;
  double2 c;
  double2 u[32];
  double2 wl[M][M];            // w of low pairs (symmetric)
  double2 wh[kDiagHigh][32];   // wh[h - M][j]: w of (j, h) for low j, and for high j with h < j (else 1)
};

template <typename R>
__global__ void __launch_bounds__(1 << kDiagLT, kDiagCtas) k_diag_tile(V2<R>* __restrict__ st,
                                                            const __grid_constant__ DiagTileParams<R> P) {
  using T = V2<R>;
  constexpr int M = DiagTile<R>::M, CB = DiagTile<R>::CB;
  constexpr int NT = 1 << kDiagLT;
  constexpr int KB = M - kDiagLT;      // register bits: [0, CB) and [CB + 8, M)
  constexpr int NK = 1 << KB;
  __shared__ double2 wh[kDiagHigh][32];
  __shared__ double2 f[32];
  __shared__ double2 scal;
  __shared__ T tabA[16], tabB[16], tabK[16];
  // a thread's static factors: two complex64 or one complex128 per 16 bytes
  constexpr int SV = 1 << CB;
  __shared__ __align__(16) T S[NK / SV][NT][SV];
  const int tid = threadIdx.x;
  const int nh = P.n - M;
  for (int j = tid; j < nh * 32; j += NT) wh[j >> 5][j & 31] = P.wh[j >> 5][j & 31];
  auto reg_bit = [](int k) { return k < CB ? k : kDiagLT + k; };
  // the static factors: pairs of low bits
  {
    double2 base = make_double2(1.0, 0.0), cr[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) cr[k] = make_double2(1.0, 0.0);
    for (int a = 0; a < kDiagLT; ++a) {
      if (!((tid >> a) & 1)) continue;
      for (int b = 0; b < a; ++b)
        if ((tid >> b) & 1) base = cmul(base, P.wl[CB + a][CB + b]);
#pragma unroll
      for (int k = 0; k < KB; ++k) cr[k] = cmul(cr[k], P.wl[CB + a][reg_bit(k)]);
    }
#pragma unroll
    for (int x = 0; x < NK; ++x) {
      double2 v = base;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        if (!((x >> k) & 1)) continue;
        v = cmul(v, cr[k]);
#pragma unroll
        for (int i = 0; i < k; ++i)
          if ((x >> i) & 1) v = cmul(v, P.wl[reg_bit(k)][reg_bit(i)]);
      }
      S[x / SV][tid][x % SV] = mk<R>((R)v.x, (R)v.y);
    }
  }
  __syncthreads();
  for (uint32_t t = blockIdx.x; t < P.n_tiles; t += gridDim.x) {
    T* at = st + ((size_t)t << M);
    T a[NK];
#pragma unroll
    for (int k = 0; k < (NK >> CB); ++k) {
      if constexpr (CB == 1) {
        const float4 v = reinterpret_cast<const float4*>(at)[tid + k * NT];
        a[2 * k] = mk<R>(v.x, v.y);
        a[2 * k + 1] = mk<R>(v.z, v.w);
      } else {
        a[k] = at[tid + k * NT];
      }
    }
    if (tid < 32) {
      const int j = tid;
      double2 g = j < P.n ? P.u[j] : make_double2(1.0, 0.0);
      for (int h = 0; h < nh; ++h)
        if ((t >> h) & 1u) g = cmul(g, wh[h][j]);
      f[j] = g;
      // the scalar: the product over the set high bits
      double2 v = (j >= M && j < P.n && ((t >> (j - M)) & 1u)) ? g : make_double2(1.0, 0.0);
#pragma unroll
      for (int off = 16; off; off >>= 1)
        v = cmul(v, make_double2(__shfl_xor_sync(0xffffffffu, v.x, off), __shfl_xor_sync(0xffffffffu, v.y, off)));
      if (j == 0) scal = cmul(v, P.c);
    }
    __syncthreads();
    if (tid < 48) {
      const int which = tid >> 4, x = tid & 15;
      double2 v = which == 2 ? scal : make_double2(1.0, 0.0);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (((x >> k) & 1) && (which < 2 || k < KB)) v = cmul(v, f[which == 2 ? reg_bit(k) : CB + 4 * which + k]);
      (which == 0 ? tabA : which == 1 ? tabB : tabK)[x] = mk<R>((R)v.x, (R)v.y);
    }
    __syncthreads();
    const T p = cmul(tabA[tid & 15], tabB[tid >> 4]);
#pragma unroll
    for (int x = 0; x < NK; x += SV) {
      const float4 sv = *reinterpret_cast<const float4*>(&S[x / SV][tid][0]);
      const T* s = reinterpret_cast<const T*>(&sv);
#pragma unroll
      for (int i = 0; i < SV; ++i) a[x + i] = cmul(a[x + i], cmul(s[i], cmul(p, tabK[x + i])));
    }
#pragma unroll
    for (int k = 0; k < (NK >> CB); ++k) {
      if constexpr (CB == 1)
        reinterpret_cast<float4*>(at)[tid + k * NT] = make_float4(a[2 * k].x, a[2 * k].y, a[2 * k + 1].x, a[2 * k + 1].y);
      else
        at[tid + k * NT] = a[k];
    }
  }
}

// The tiled form of a diagonal, when it has one: every table entry of modulus 1
// (the factored form divides by them) and at least one whole tile.
template <typename R>
static bool plan_diag_tile(int n, const std::vector<Term>& terms, std::complex<double> scalar, DiagTileParams<R>& P) {
  constexpr int M = DiagTile<R>::M;
  if (n < M || n - M > kDiagHigh) return false;
  std::vector<std::complex<double>> u(n, 1.0), w((size_t)n * n, 1.0);
  for (const Term& t : terms) {
    for (const auto& v : t.tab)
      if (!(std::fabs(std::abs(v) - 1.0) < 1e-6)) return false;
    scalar *= t.tab[0];
    if (t.bits.size() == 1) {
      u[t.bits[0]] *= t.tab[1] / t.tab[0];
      continue;
    }
    const int a = t.bits[0], b = t.bits[1];  // table index = 2 b_a + b_b
    u[a] *= t.tab[2] / t.tab[0];
    u[b] *= t.tab[1] / t.tab[0];
    const auto v = t.tab[3] * t.tab[0] / (t.tab[1] * t.tab[2]);
    w[(size_t)a * n + b] *= v;
    w[(size_t)b * n + a] *= v;
  }
  auto d2 = [](std::complex<double> v) { return make_double2(v.real(), v.imag()); };
  std::memset(&P, 0, sizeof(P));
  P.n = n;
  P.n_tiles = 1u << (n - M);
  P.c = d2(scalar);
  for (int j = 0; j < n; ++j) P.u[j] = d2(u[j]);
  for (int a = 0; a < M; ++a)
    for (int b = 0; b < M; ++b) P.wl[a][b] = d2(w[(size_t)a * n + b]);
  for (int h = M; h < n; ++h)
    for (int j = 0; j < 32; ++j)
      P.wh[h - M][j] = (j < M || (h < j && j < n)) ? d2(w[(size_t)j * n + h]) : make_double2(1.0, 0.0);
  return true;
}

template <typename R>
static int launch_diag_tile(mq_state* h, const DiagTileParams<R>& P) {
  const uint32_t grid = std::min<uint32_t>(P.n_tiles, (uint32_t)h->num_sms * kDiagCtas);
  k_diag_tile<R><<<grid, 1 << kDiagLT, 0, h->stream>>>(reinterpret_cast<V2<R>*>(h->cur_buf()), P);
  MQ_LAUNCHED("k_diag_tile");
  h->launches += 1;
  h->sweeps += 1;
  return MQ_OK;
}

int launch_diag_terms(mq_state* h, int n_terms, const int32_t* kinds, const int32_t* wires, const double* params) {
  std::vector<Term> terms;
  std::complex<double> scalar;
  int rc = build_terms(h->n, n_terms, kinds, wires, params, terms, scalar);
  if (rc) return rc;
  if (terms.empty() && scalar == std::complex<double>(1.0, 0.0)) return MQ_OK;
  // The tiled form wherever it exists.  It measured faster than the window
  // tables for chains too (26 qubits: 177 against 219 us; complex128, 25
  // qubits: 176 against 201 us), at 18 qubits and more on the device alone
  // (6.2 against 9.6 us) and below that because the host plans no windows (12
  // qubits: 39 against 63 us a call, of which 5.5 against 3.6 us on the device).
  if (h->dtype == MQ_C64) {
    DiagTileParams<float> P;
    if (plan_diag_tile(h->n, terms, scalar, P)) return launch_diag_tile(h, P);
  } else {
    DiagTileParams<double> P;
    if (plan_diag_tile(h->n, terms, scalar, P)) return launch_diag_tile(h, P);
  }
  const int cap = h->dtype == MQ_C64 ? DiagCap<float>::v : DiagCap<double>::v;
  std::vector<PlannedLut> luts;
  for (int W = 10; W >= 1; --W) {
    luts = plan_luts(terms, W);
    size_t entries = 0;
    for (auto& L : luts) entries += lut_size(L);
    if ((int)luts.size() <= kMaxLuts && (int)entries <= cap) break;
    if (W == 1) break;  // fall through to multi-pass below
  }
  if (luts.empty()) {
    PlannedLut L;
    L.contig = true;
    L.vals = {1.0};
    luts.push_back(L);
  }
  realize(luts);
  for (auto& v : luts[0].vals) v *= scalar;
  // Split into passes that respect the parameter-block capacity.
  size_t i = 0;
  while (i < luts.size()) {
    std::vector<PlannedLut> pass;
    size_t entries = 0;
    while (i < luts.size() && (int)pass.size() < kMaxLuts && (int)(entries + luts[i].vals.size()) <= cap) {
      entries += luts[i].vals.size();
      pass.push_back(luts[i]);
      ++i;
    }
    if (pass.empty()) return fail(MQ_EUNSUPPORTED, "diagonal table exceeds capacity");
    rc = (h->dtype == MQ_C64) ? launch_diag_pass<float>(h, pass) : launch_diag_pass<double>(h, pass);
    if (rc) return rc;
  }
  return MQ_OK;
}

}  // namespace mq
