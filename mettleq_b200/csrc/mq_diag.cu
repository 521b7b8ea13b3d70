// Diagonal phase layers (b): RZ / U1 / Z / S / T, CZ / CPHASE / CRZ, ZZ and
// any mix of them, in ONE streaming pass.
//
// Replaces diag_pair_layer / diag_weighted_layer (shaders/diag.py:19-217),
// zz_chain_layer / zz_weighted_layer (shaders/zz.py:16-185) and the per-gate
// apply_diagonal passes of the CPU path (sim.py:94-138, device.py:1154-1211).
//
// The reference multiplies one unit phase per equal-angle group inside the
// kernel (zz.py:40-71).  Here a diagonal of unit-modulus terms is one angle per
// amplitude, a quadratic form of its index bits, summed up by tiles (k_diag_tile,
// below).  Small states, diagonals that are one small table and terms of other
// moduli take lookup tables (k_diag): the host factors the whole diagonal into
// at most eight, each indexed by a window of <= 10 index bits (or by a short list
// of scattered bits for far-apart pairs), every term's phase folded into exactly
// one in double precision.  The fused layers' epilogues use such tables too.
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
  int kind = 0;
  double th = 0;                       // the angle of kinds that have one
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
    tm.kind = kind;
    tm.th = th;
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
// bits: as an angle, the whole diagonal is
//   c + sum_j u_j b_j + sum_{i<j} w_ij b_i b_j,
// and for a tile of 2^M consecutive amplitudes (high bits H fixed) the pairs of
// low bits are the same in every tile (a thread keeps its 16 angles or 8 factors in
// shared memory), the pairs of high bits are one angle, and the mixed pairs leave
// one angle f_l = u_l + sum_{h in H} w_lh per low bit.  One warp adds up the f_l
// while the tile's loads are in flight.  An amplitude's angle is then the sum of
// three, whatever the graph: the thread's of the tile (eight bits), one of 16
// over the other bits, and its static one; complex64 takes one sine and cosine of
// the sum, complex128 (whose are long) multiplies three factors.
// Angles are fixed-point fractions of a turn in 64 bits: their sums are exact,
// whole turns drop out, and a factor is rounded once, where products of many
// factors were off by up to twice as much as the tables (complex128, chain of
// 17 qubits: 5.7e-16, the tables 3.2e-16, 1.5e-16 this way; complex64 6.7e-8,
// 5.0e-8, 4.2e-8).
// Bound by memory: 26 qubits, a chain and a random matching (38 bonds): 515 us
// with eight tables, 173 us this way in a replayed graph (164 us in a stream of
// calls, 6.5 TB/s); 12 qubits 3.8 and 3.7 us, 22 qubits 47 and 12 us.
template <typename R> struct DiagTile;
template <> struct DiagTile<float> { static constexpr int M = 12, CB = 1; };
template <> struct DiagTile<double> { static constexpr int M = 11, CB = 0; };
constexpr int kDiagLT = 8;  // 256 threads: index bits [CB, CB + 8)
// resident CTAs per SM; 26 qubits, complex64: 192 us with one, 173 with two, 179
// with three, 181 with four
constexpr int kDiagCtas = 2;
constexpr int kDiagHigh = 20;

using Turn = unsigned long long;  // 2^-64 of a turn

template <typename R>
struct DiagTileParams {
  static constexpr int M = DiagTile<R>::M;
  uint32_t n_tiles;
  int32_t n;
  Turn c;
  Turn u[32];
  Turn wl[M][M];            // w of low pairs (symmetric)
  Turn wh[kDiagHigh][32];   // wh[h - M][j]: w of (j, h) for j < h (else 0)
};

// e^{i angle}: quarter turns exactly, the rest (at most an eighth of a turn) by
// sincospi.
__device__ __forceinline__ double2 turn_cis(Turn a) {
  const unsigned q = (unsigned)((a + (Turn(1) << 61)) >> 62);
  const double x = (double)(long long)(a - ((Turn)q << 62)) * 0x1p-63;
  double s, c;
  sincospi(x, &s, &c);
  const double2 r = (q & 1u) ? make_double2(-s, c) : make_double2(c, s);
  return (q & 2u) ? make_double2(-r.x, -r.y) : r;
}

// The same for two 32-bit angles (an error of 7e-10): the Taylor series of sine
// and cosine on the rest, cut where the next term is below 2e-9, on the
// paired FP32 instructions.  sincospif instead took 3 % longer at 26 qubits.
__device__ __forceinline__ void turn_cis2(uint32_t a, uint32_t b, float2& x, float2& y) {
  const uint32_t qa = (a + (1u << 29)) >> 30, qb = (b + (1u << 29)) >> 30;
  const float2 r = make_float2((float)(int32_t)(a - (qa << 30)), (float)(int32_t)(b - (qb << 30)));
  auto both = [](float v) { return make_float2(v, v); };
  const float2 t = __fmul2_rn(r, both(1.4629180792671596e-9f));  // 2 pi / 2^32
  const float2 u = __fmul2_rn(t, t);
  float2 s = __ffma2_rn(u, both(1.f / 362880.f), both(-1.f / 5040.f));
  s = __ffma2_rn(s, u, both(1.f / 120.f));
  s = __ffma2_rn(s, u, both(-1.f / 6.f));
  s = __ffma2_rn(__fmul2_rn(t, u), s, t);
  float2 c = __ffma2_rn(u, both(-1.f / 3628800.f), both(1.f / 40320.f));
  c = __ffma2_rn(c, u, both(-1.f / 720.f));
  c = __ffma2_rn(c, u, both(1.f / 24.f));
  c = __ffma2_rn(c, u, both(-0.5f));
  c = __ffma2_rn(c, u, both(1.f));
  auto turned = [](uint32_t q, float cs, float sn) {
    const uint32_t sign = (q & 2u) << 30;
    const float re = (q & 1u) ? -sn : cs, im = (q & 1u) ? cs : sn;
    return make_float2(__uint_as_float(__float_as_uint(re) ^ sign), __uint_as_float(__float_as_uint(im) ^ sign));
  };
  x = turned(qa, c.x, s.x);
  y = turned(qb, c.y, s.y);
}
__device__ __forceinline__ uint32_t turn_high(Turn a) { return (uint32_t)((a + (Turn(1) << 31)) >> 32); }

template <typename R>
__global__ void __launch_bounds__(1 << kDiagLT, kDiagCtas) k_diag_tile(V2<R>* __restrict__ st,
                                                            const __grid_constant__ DiagTileParams<R> P) {
  using T = V2<R>;
  constexpr int M = DiagTile<R>::M, CB = DiagTile<R>::CB;
  constexpr bool C64 = sizeof(R) == 4;
  constexpr int NT = 1 << kDiagLT;
  constexpr int KB = M - kDiagLT;      // register bits: [0, CB) and [CB + 8, M)
  constexpr int NK = 1 << KB;
  __shared__ Turn wh[kDiagHigh][32];
  __shared__ Turn f[32], scal;
  __shared__ __align__(16) Turn ang[2][16];  // by four thread bits
  // by register bits: complex64 angles, complex128 factors
  __shared__ __align__(16) uint32_t angK[16];
  __shared__ double2 tabK[C64 ? 1 : 16];
  // a thread's static angles (four to 16 bytes) or factors
  __shared__ uint4 S[C64 ? NK / 4 : NK][NT];
  const int tid = threadIdx.x;
  const int nh = P.n - M;
  for (int j = tid; j < nh * 32; j += NT) wh[j >> 5][j & 31] = P.wh[j >> 5][j & 31];
  auto reg_bit = [](int k) { return k < CB ? k : kDiagLT + k; };
  // the static angles: pairs of low bits
  {
    Turn base = 0, cr[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) cr[k] = 0;
#pragma unroll 1
    for (int a = 0; a < kDiagLT; ++a) {
      const Turn on = (tid >> a) & 1 ? ~Turn(0) : 0;
      Turn with = 0;
#pragma unroll
      for (int b = 0; b < kDiagLT; ++b)
        if (b < a && ((tid >> b) & 1)) with += P.wl[CB + a][CB + b];
      base += with & on;
#pragma unroll
      for (int k = 0; k < KB; ++k) cr[k] += P.wl[CB + a][reg_bit(k)] & on;
    }
    uint32_t w[4];
#pragma unroll
    for (int x = 0; x < NK; ++x) {
      Turn v = base;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        if (!((x >> k) & 1)) continue;
        v += cr[k];
#pragma unroll
        for (int i = 0; i < k; ++i)
          if ((x >> i) & 1) v += P.wl[reg_bit(k)][reg_bit(i)];
      }
      if constexpr (C64) {
        w[x & 3] = turn_high(v);
        if ((x & 3) == 3) S[x / 4][tid] = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
        *reinterpret_cast<double2*>(&S[x][tid]) = turn_cis(v);
      }
    }
  }
  __syncthreads();
  for (uint32_t t = blockIdx.x; t < P.n_tiles; t += gridDim.x) {
    T* at = st + ((size_t)t << M);
    T a[NK];
#pragma unroll
    for (int k = 0; k < (NK >> CB); ++k) {
      if constexpr (C64) {
        const float4 v = reinterpret_cast<const float4*>(at)[tid + k * NT];
        a[2 * k] = mk<R>(v.x, v.y);
        a[2 * k + 1] = mk<R>(v.z, v.w);
      } else {
        a[k] = at[tid + k * NT];
      }
    }
    if (tid < 32) {
      const int j = tid;
      Turn g = j < P.n ? P.u[j] : 0;
      for (int h = 0; h < nh; ++h)
        if ((t >> h) & 1u) g += wh[h][j];
      f[j] = g;
      // the pairs of high bits and the set high bits' own angles
      Turn v = (j >= M && j < P.n && ((t >> (j - M)) & 1u)) ? g : 0;
#pragma unroll
      for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (j == 0) scal = v + P.c;
    }
    __syncthreads();
    if (tid < 48) {
      const int which = tid >> 4, x = tid & 15;
      Turn v = which == 2 ? scal : 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (((x >> k) & 1) && (which < 2 || k < KB)) v += f[which == 2 ? reg_bit(k) : CB + 4 * which + k];
      if (which < 2) ang[which][x] = v;
      else if constexpr (C64) angK[x] = turn_high(v);
      else tabK[x] = turn_cis(v);
    }
    __syncthreads();
    const Turn mine = ang[0][tid & 15] + ang[1][tid >> 4];
    if constexpr (C64) {
      const uint32_t p = turn_high(mine);
#pragma unroll
      for (int x = 0; x < NK; x += 4) {
        const uint4 s = S[x / 4][tid], k = *reinterpret_cast<const uint4*>(angK + x);
        T w[4];
        turn_cis2(p + k.x + s.x, p + k.y + s.y, w[0], w[1]);
        turn_cis2(p + k.z + s.z, p + k.w + s.w, w[2], w[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) a[x + i] = cmul(a[x + i], w[i]);
      }
    } else {
      const double2 p = turn_cis(mine);
#pragma unroll
      for (int x = 0; x < NK; ++x) {
        const double2 s = *reinterpret_cast<const double2*>(&S[x][tid]);
        a[x] = cmul(a[x], cmul(s, cmul(p, tabK[x])));
      }
    }
#pragma unroll
    for (int k = 0; k < (NK >> CB); ++k) {
      if constexpr (C64)
        reinterpret_cast<float4*>(at)[tid + k * NT] = make_float4(a[2 * k].x, a[2 * k].y, a[2 * k + 1].x, a[2 * k + 1].y);
      else
        at[tid + k * NT] = a[k];
    }
  }
}

// Angles to 2^-62 of a turn: of x turns, |x| <= 1/2; of a number of modulus 1.
static Turn to_turn(long double x) { return (Turn)std::llrint(x * 0x1p62L) << 2; }
constexpr long double kPerTurn = 0.159154943091895335768883763372514362L;  // 1 / (2 pi)
static Turn turn_of(std::complex<double> z) {
  return z == 1.0 ? 0 : to_turn(std::atan2((long double)z.imag(), (long double)z.real()) * kPerTurn);
}
// The angles of a term's table entries: from its own angle where it has one
// (an arctangent a term takes longer than the rest of the plan), and small
// enough for the product to keep 2^-62 of a turn.
static void term_turns(const Term& t, Turn (&a)[4]) {
  const bool has = t.kind != MQ_DIAG_1Q && t.kind != MQ_DIAG_2Q && std::fabs(t.th) <= 8.0;
  if (!has) {
    for (size_t i = 0; i < t.tab.size(); ++i) {
      size_t k = 0;  // equal and conjugate entries share one
      while (k < i && t.tab[k] != t.tab[i] && t.tab[k] != std::conj(t.tab[i])) ++k;
      a[i] = k == i ? turn_of(t.tab[i]) : t.tab[k] == t.tab[i] ? a[k] : 0 - a[k];
    }
    return;
  }
  const bool half = t.kind == MQ_DIAG_CRZ || t.kind == MQ_DIAG_RZ;
  long double x = (long double)(half ? t.th / 2 : t.th) * kPerTurn;
  const Turn w = t.tab[t.tab.size() - 1] == -1.0 ? Turn(1) << 63 : to_turn(x - std::rint(x));
  switch (t.kind) {
    case MQ_DIAG_ZZ: a[0] = a[3] = 0 - w; a[1] = a[2] = w; break;
    case MQ_DIAG_CPHASE: a[0] = a[1] = a[2] = 0; a[3] = w; break;
    case MQ_DIAG_CRZ: a[0] = a[1] = 0; a[2] = 0 - w; a[3] = w; break;
    case MQ_DIAG_RZ: a[0] = 0 - w; a[1] = w; break;
    default: a[0] = 0; a[1] = w; break;  // MQ_DIAG_PHASE
  }
}

// The tiled form of a diagonal, when it has one: every table entry of modulus 1
// to the rounding of its parts (complex64: to a hundredth of a result's), as
// an angle keeps no modulus, and at least one whole tile.
template <typename R>
static bool plan_diag_tile(int n, const std::vector<Term>& terms, std::complex<double> scalar, DiagTileParams<R>& P) {
  constexpr int M = DiagTile<R>::M;
  constexpr double off = sizeof(R) == 4 ? 1e-9 : 4.5e-16;
  if (n < M || n - M > kDiagHigh) return false;
  for (const Term& t : terms)
    for (const auto& v : t.tab)
      if (!(std::fabs(std::norm(v) - 1.0) <= off)) return false;
  if (!(std::fabs(std::norm(scalar) - 1.0) <= 16 * off)) return false;
  std::memset(&P, 0, sizeof(P));
  P.n = n;
  P.n_tiles = 1u << (n - M);
  P.c = turn_of(scalar);
  auto pair = [&](int h, int l, Turn w) {  // h > l
    if (h >= M) {
      P.wh[h - M][l] += w;
    } else {
      P.wl[h][l] += w;
      P.wl[l][h] += w;
    }
  };
  for (const Term& t : terms) {
    Turn a[4];
    term_turns(t, a);
    P.c += a[0];
    if (t.bits.size() == 1) {
      P.u[t.bits[0]] += a[1] - a[0];
      continue;
    }
    const int x = t.bits[0], y = t.bits[1];  // table index = 2 b_x + b_y
    P.u[x] += a[2] - a[0];
    P.u[y] += a[1] - a[0];
    pair(t.hi, t.lo, a[3] - a[1] - a[2] + a[0]);
  }
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

// Diagonals that are one small table stay with it: a look-up costs less than the
// tile's angles.  Measured, us on the device, table against tile (complex64):
// terms within six neighbouring bits, 14 qubits 1.7 / 3.8, 20 qubits 3.4 / 6.3,
// 22 qubits 7.4 / 12.1, 24 qubits 45.4 / 45.6, 26 qubits 174 / 173; up to four
// bits in pairs ten and more apart, 20 qubits 4.8 / 6.3, 22 qubits 13.6 / 12.1, 24
// qubits 56 / 46.  complex128: 20 qubits 5.8 and 6.3 / 9.7, 22 qubits 21.2 and 18.1 /
// 20.4, 24 qubits 97 / 90.  With more tables the tile is faster from 14 qubits on,
// and below as a call (12 qubits, chain: 53 against 62 us, of which 3.7 against
// 3.4 on the device: the host fills no tables).
static bool one_small_table(int n, int dtype, const std::vector<Term>& terms) {
  int lo = n, hi = -1;
  bool apart = true;
  uint32_t bits = 0;
  for (const Term& t : terms) {
    lo = std::min(lo, t.lo);
    hi = std::max(hi, t.hi);
    apart = apart && t.hi - t.lo >= 10;
    for (int b : t.bits) bits |= 1u << b;
  }
  if (hi - lo < 6) return dtype == MQ_C64 || n <= 23;
  return apart && __builtin_popcount(bits) <= 4 && n <= (dtype == MQ_C64 ? 21 : 23);
}

int launch_diag_terms(mq_state* h, int n_terms, const int32_t* kinds, const int32_t* wires, const double* params) {
  std::vector<Term> terms;
  std::complex<double> scalar;
  int rc = build_terms(h->n, n_terms, kinds, wires, params, terms, scalar);
  if (rc) return rc;
  if (terms.empty() && scalar == std::complex<double>(1.0, 0.0)) return MQ_OK;
  if (!one_small_table(h->n, h->dtype, terms)) {
    if (h->dtype == MQ_C64) {
      DiagTileParams<float> P;
      if (plan_diag_tile(h->n, terms, scalar, P)) return launch_diag_tile(h, P);
    } else {
      DiagTileParams<double> P;
      if (plan_diag_tile(h->n, terms, scalar, P)) return launch_diag_tile(h, P);
    }
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
