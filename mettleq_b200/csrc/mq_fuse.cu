// Gate-stream fusion on the host, for streams of ordinary gates (the Python
// front end hands over codes, wires and parameters as arrays and turns the
// segments returned here into layer dicts; fusion.py states the rules and
// handles every other stream).  Host code only: the per-gate work of a circuit
// call, which as interpreted code took longer than all of its kernels (20
// qubits, 20 layers, 1160 gates: 6.2 ms against 0.8 ms on the GPU).
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <exception>
#include <map>
#include <new>
#include <vector>

#include "mq_internal.cuh"

namespace mq {
namespace {

using C = std::complex<double>;

// the order of fusion.GATE_NAMES
enum Gate : int {
  G_H, G_I, G_X, G_Y, G_Z, G_S, G_SDG, G_T, G_TDG, G_SX, G_RX, G_RY, G_RZ, G_U1, G_U2, G_U3,
  G_CNOT, G_CH, G_CZ, G_CPHASE, G_CRX, G_CRY, G_CRZ, G_SWAP, G_ISWAP, G_XXPHASE, G_YYPHASE, G_ZZPHASE,
  G_TOFFOLI, G_FREDKIN, G_COUNT,
  // made here
  G_D2, G_QFTSTAGE
};
constexpr int kParams[G_COUNT] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 2, 3, 0, 0, 0, 1, 1, 1, 1, 0, 0, 1, 1, 1, 0, 0};
int arity(int g) { return g < G_CNOT ? 1 : g < G_TOFFOLI ? 2 : 3; }

struct Op {
  int code;
  int w[3];
  double p[3];
  int j = 0, m = 0, inverse = 0;  // G_QFTSTAGE: stage j of the wires [j, m)
};

enum Cat : int { K_SINGLE, K_DIAG, K_AFFINE, K_CONTROLLED, K_OTHER };
int category(const Op& o) {
  switch (o.code) {
    case G_CZ: case G_CPHASE: case G_CRZ: case G_ZZPHASE: case G_D2: return K_DIAG;
    case G_CNOT: case G_SWAP: return K_AFFINE;
    case G_CH: case G_CRX: case G_CRY: case G_TOFFOLI: return K_CONTROLLED;
    case G_QFTSTAGE: case G_XXPHASE: case G_YYPHASE: return K_OTHER + (o.code == G_QFTSTAGE ? 0 : o.code == G_XXPHASE ? 1 : 2);
    default: return K_SINGLE;
  }
}
constexpr int kCats = K_OTHER + 3;

struct M2 { C a, b, c, d; };
M2 mul(const M2& x, const M2& y) {
  return {x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}
const double kSq = 1.0 / std::sqrt(2.0);
M2 u3(double theta, double phi, double lam) {
  const double c = std::cos(theta / 2.0), s = std::sin(theta / 2.0);
  const double a = (phi + lam) / 2.0, b = (phi - lam) / 2.0;
  const double ca = std::cos(a), sa = std::sin(a), cb = std::cos(b), sb = std::sin(b);
  return {C(ca * c, -sa * c), C(-cb * s, sb * s), C(cb * s, sb * s), C(ca * c, sa * c)};
}
M2 matrix(int g, const double* p) {
  const C I(0, 1);
  switch (g) {
    case G_H: return {kSq, kSq, kSq, -kSq};
    case G_X: return {0, 1, 1, 0};
    case G_Y: return {0, -I, I, 0};
    case G_Z: return {1, 0, 0, -1};
    case G_S: return {1, 0, 0, I};
    case G_SDG: return {1, 0, 0, -I};
    case G_T: return {1, 0, 0, C(std::cos(M_PI / 4), std::sin(M_PI / 4))};
    case G_TDG: return {1, 0, 0, C(std::cos(M_PI / 4), -std::sin(M_PI / 4))};
    case G_SX: return {C(0.5, 0.5), C(0.5, -0.5), C(0.5, -0.5), C(0.5, 0.5)};
    case G_RX: case G_CRX: {
      const double c = std::cos(p[0] / 2.0), s = std::sin(p[0] / 2.0);
      return {c, C(0, -s), C(0, -s), c};
    }
    case G_RY: case G_CRY: {
      const double c = std::cos(p[0] / 2.0), s = std::sin(p[0] / 2.0);
      return {c, -s, s, c};
    }
    case G_RZ: {
      const double h = p[0] / 2.0;
      return {C(std::cos(h), -std::sin(h)), 0, 0, C(std::cos(h), std::sin(h))};
    }
    case G_U1: return {1, 0, 0, C(std::cos(p[0]), std::sin(p[0]))};
    case G_U2: return u3(M_PI / 2.0, p[0], p[1]);
    case G_U3: return u3(p[0], p[1], p[2]);
    case G_CH: return {kSq, kSq, kSq, -kSq};
    case G_TOFFOLI: return {0, 1, 1, 0};
    default: return {1, 0, 0, 1};
  }
}
bool near(const M2& m, const M2& r) {
  return std::abs(m.a - r.a) <= 1e-12 && std::abs(m.b - r.b) <= 1e-12 && std::abs(m.c - r.c) <= 1e-12 &&
         std::abs(m.d - r.d) <= 1e-12;
}

// fusion.decompose and fusion._mark_qft_stages
std::vector<Op> marked(const std::vector<Op>& in) {
  std::vector<Op> d;
  d.reserve(in.size() + 8);
  for (const Op& o : in) {
    if (o.code == G_ISWAP) {
      Op x = o;
      x.code = G_D2;
      d.push_back(x);
      x.code = G_SWAP;
      d.push_back(x);
    } else if (o.code == G_FREDKIN) {  // CNOT(b, a) TOFFOLI(c, a, b) CNOT(b, a)
      Op x = o;
      x.code = G_CNOT;
      x.w[0] = o.w[2];
      x.w[1] = o.w[1];
      d.push_back(x);
      Op t = o;
      t.code = G_TOFFOLI;
      d.push_back(t);
      d.push_back(x);
    } else {
      d.push_back(o);
    }
  }
  std::vector<Op> out;
  out.reserve(d.size());
  const size_t N = d.size();
  auto cp = [&](size_t i, int k, int j, double sign) {
    return i < N && d[i].code == G_CPHASE && d[i].w[0] == k && d[i].w[1] == j && k > j &&
           d[i].p[0] == sign * std::ldexp(M_PI, -(k - j));
  };
  for (size_t i = 0; i < N;) {
    Op st{};
    size_t next = 0;
    if (d[i].code == G_H) {
      const int j = d[i].w[0];
      int k = j + 1;
      size_t e = i + 1;
      while (cp(e, k, j, 1.0)) { ++k; ++e; }
      if (k > j + 1) {
        st.j = j; st.m = k; st.inverse = 0;
        next = e;
      }
    } else if (d[i].code == G_CPHASE && d[i].p[0] < 0) {
      const int k0 = d[i].w[0], j = d[i].w[1];
      int k = k0;
      size_t e = i;
      while (k > j && cp(e, k, j, -1.0)) { --k; ++e; }
      // k0 < j: no ladder, a bare H must follow at once (as fusion.py has it)
      if (k <= j && e < N && d[e].code == G_H && d[e].w[0] == j) {
        st.j = j; st.m = k0 + 1; st.inverse = 1;
        next = e + 1;
      }
    }
    if (next) {
      st.code = G_QFTSTAGE;
      out.push_back(st);
      i = next;
    } else {
      out.push_back(d[i++]);
    }
  }
  return out;
}

// fusion.dependency_schedule
std::vector<int> scheduled(const std::vector<Op>& ops, int n) {
  const int N = (int)ops.size();
  std::vector<int> order;
  order.reserve(N);
  std::vector<int> indeg(N, 0), last(n, -1), cat(N);
  std::vector<std::vector<int>> succ(N);
  std::vector<int> seen(N, -1);
  for (int i = 0; i < N; ++i) {
    cat[i] = category(ops[i]);
    const bool st = ops[i].code == G_QFTSTAGE;
    const int nw = st ? ops[i].m - ops[i].j : ops[i].code == G_D2 ? 2 : arity(ops[i].code);
    for (int k = 0; k < nw; ++k) {
      const int w = st ? ops[i].j + k : ops[i].w[k];
      const int p = last[w];
      if (p >= 0 && seen[p] != i) {
        seen[p] = i;
        ++indeg[i];
        succ[p].push_back(i);
      }
      last[w] = i;
    }
  }
  std::vector<int> ready[kCats], batch;
  for (int i = 0; i < N; ++i)
    if (!indeg[i]) ready[cat[i]].push_back(i);
  int current = -1;
  auto emit = [&](int c) {
    batch.swap(ready[c]);
    ready[c].clear();
    std::sort(batch.begin(), batch.end());
    for (int i : batch) {
      order.push_back(i);
      for (int s : succ[i])
        if (--indeg[s] == 0) ready[cat[s]].push_back(s);
    }
    batch.clear();
  };
  while ((int)order.size() < N) {
    if (current >= 0 && !ready[current].empty()) { emit(current); continue; }
    if (!ready[K_SINGLE].empty()) { emit(K_SINGLE); current = -1; continue; }
    int best = N;
    current = -1;
    for (int c = 0; c < kCats; ++c)
      for (int i : ready[c])
        if (i < best) { best = i; current = c; }
    if (current < 0) return {};  // cannot happen: the dependencies are acyclic
  }
  return order;
}

// Segment kinds of the output (fusion._decode)
enum Seg : int { S_QFT, S_U2, S_DIAG, S_XOR, S_PAIR, S_CU };

struct Out {
  std::vector<int32_t> i;
  std::vector<double> d;
  void put(std::initializer_list<int> v) { i.insert(i.end(), v.begin(), v.end()); }
  void put(const M2& m) {
    for (const C& v : {m.a, m.b, m.c, m.d}) {
      d.push_back(v.real());
      d.push_back(v.imag());
    }
  }
};

void term(Out& o, int kind, int a, int b, std::initializer_list<double> p) {
  o.put({kind, a, b});
  const size_t at = o.d.size();
  o.d.insert(o.d.end(), p.begin(), p.end());
  o.d.resize(at + 8, 0.0);
}
void diag_terms(Out& o, const Op& op) {
  switch (op.code) {
    case G_CZ: term(o, MQ_DIAG_CPHASE, op.w[0], op.w[1], {M_PI}); break;
    case G_CPHASE: term(o, MQ_DIAG_CPHASE, op.w[0], op.w[1], {op.p[0]}); break;
    case G_CRZ: term(o, MQ_DIAG_CRZ, op.w[0], op.w[1], {op.p[0]}); break;
    case G_ZZPHASE: term(o, MQ_DIAG_ZZ, op.w[0], op.w[1], {op.p[0]}); break;
    default: term(o, MQ_DIAG_2Q, op.w[0], op.w[1], {1, 0, 0, 1, 0, 1, 1, 0}); break;  // ISWAP's diag(1, i, i, 1)
  }
}

void window(Out& o, const std::vector<Op>& ops, const std::vector<int>& order, size_t i, size_t j, int n) {
  std::vector<M2> m(n, M2{1, 0, 0, 1});
  for (size_t k = i; k < j; ++k) {
    const Op& op = ops[order[k]];
    m[op.w[0]] = mul(matrix(op.code, op.p), m[op.w[0]]);
  }
  std::vector<int> active;
  bool diag = true, flip = true;
  for (int q = 0; q < n; ++q) {
    if (near(m[q], M2{1, 0, 0, 1})) continue;
    active.push_back(q);
    diag = diag && std::abs(m[q].b) <= 1e-15 && std::abs(m[q].c) <= 1e-15;
    flip = flip && near(m[q], M2{0, 1, 1, 0});
  }
  if (active.empty()) return;
  if (diag) {
    o.put({S_DIAG, (int)active.size()});
    for (int q : active) term(o, MQ_DIAG_1Q, q, -1, {m[q].a.real(), m[q].a.imag(), m[q].d.real(), m[q].d.imag()});
  } else if (flip) {
    uint32_t c = 0;
    for (int q : active) c ^= 1u << (n - 1 - q);
    o.put({S_XOR, (int)c});
    for (int k = 0; k < n; ++k) o.put({1 << (n - 1 - k)});
  } else {
    o.put({S_U2, (int)active.size()});
    for (int q : active) o.put({q});
    for (int q : active) o.put(m[q]);
  }
}

// fusion.affine_of
void affine(Out& o, const std::vector<Op>& ops, const std::vector<int>& order, size_t i, size_t j, int n) {
  std::vector<uint32_t> rows(n);
  for (int k = 0; k < n; ++k) rows[k] = 1u << (n - 1 - k);
  uint32_t c = 0;
  auto bit = [&](int q) { return 1u << (n - 1 - q); };
  for (size_t k = j; k-- > i;) {
    const Op& op = ops[order[k]];
    const int a = op.w[0], b = op.w[1];
    if (op.code == G_X) {
      c ^= bit(a);
    } else if (op.code == G_CNOT) {
      rows[b] ^= rows[a];
      if (c & bit(a)) c ^= bit(b);
    } else {
      std::swap(rows[a], rows[b]);
      if (((c & bit(a)) != 0) != ((c & bit(b)) != 0)) c ^= bit(a) | bit(b);
    }
  }
  o.put({S_XOR, (int)c});
  for (uint32_t r : rows) o.put({(int)r});
}

}  // namespace
}  // namespace mq

using namespace mq;

extern "C" {

int mq_fuse_stream(int n, int n_ops, const int32_t* codes, const int32_t* n_wires, const int32_t* wires,
                   const int32_t* n_params, const double* params, int32_t* ints, int64_t ints_cap, double* doubles,
                   int64_t doubles_cap, int64_t* used) {
  try {
    if (n < 1 || n > kMaxQubits || n_ops < 0) return fail(MQ_EINVAL, "bad stream size");
    if (n_ops > 0 && (!codes || !n_wires || !wires || !n_params)) return fail(MQ_EINVAL, "null stream arrays");
    if (!used || !ints || !doubles) return fail(MQ_EINVAL, "null output");
    std::vector<Op> in;
    in.reserve(n_ops);
    int64_t wi = 0, pi = 0;
    for (int i = 0; i < n_ops; ++i) {
      const int g = codes[i];
      if (g < 0 || g >= G_COUNT) return fail(MQ_EINVAL, "unknown gate code");
      if (n_wires[i] != arity(g)) return fail(MQ_EINVAL, "wrong wire count");
      if (n_params[i] < kParams[g]) return fail(MQ_EINVAL, "too few parameters");
      if (n_params[i] > 0 && !params) return fail(MQ_EINVAL, "null stream arrays");
      Op o{};
      o.code = g;
      for (int k = 0; k < arity(g); ++k) {
        o.w[k] = wires[wi + k];
        if (o.w[k] < 0 || o.w[k] >= n) return fail(MQ_EINVAL, "Qubit index out of range");
        for (int l = 0; l < k; ++l)
          if (o.w[l] == o.w[k]) return fail(MQ_EINVAL, "Control/target wires must be distinct");
      }
      // (infinities, NaN, and angles whose sum could be one: 1e300)
      for (int k = 0; k < n_params[i]; ++k)
        if (!(std::fabs(params[pi + k]) < 1e300)) return fail(MQ_EINVAL, "parameter is not finite");
      for (int k = 0; k < kParams[g]; ++k) o.p[k] = params[pi + k];
      wi += n_wires[i];
      pi += n_params[i];
      in.push_back(o);
    }
    const std::vector<Op> ops = marked(in);
    const std::vector<int> order = scheduled(ops, n);
    if (order.size() != ops.size()) return fail(MQ_EDEVICE, "operation dependency graph contains a cycle");
    Out out;
    const size_t N = order.size();
    auto at = [&](size_t k) -> const Op& { return ops[order[k]]; };
    auto is_single = [&](size_t k) { return category(at(k)) == K_SINGLE; };
    for (size_t i = 0; i < N;) {
      const Op& op = at(i);
      size_t j = i;
      const int cat = category(op);
      if (op.code == G_QFTSTAGE) {
        out.put({S_QFT, op.j, op.m, op.inverse});
        j = i + 1;
      } else if (cat == K_SINGLE) {
        while (j < N && is_single(j)) ++j;
        window(out, ops, order, i, j, n);
      } else if (cat == K_DIAG) {
        while (j < N && category(at(j)) == K_DIAG) ++j;
        out.put({S_DIAG, (int)(j - i)});
        for (size_t k = i; k < j; ++k) diag_terms(out, at(k));
      } else if (cat == K_AFFINE) {
        while (j < N && (category(at(j)) == K_AFFINE || at(j).code == G_X)) ++j;
        affine(out, ops, order, i, j, n);
      } else if (cat == K_CONTROLLED) {
        while (j < N && category(at(j)) == K_CONTROLLED) ++j;
        out.put({S_CU, (int)(j - i)});
        for (size_t k = i; k < j; ++k) {
          const Op& g = at(k);
          const int nc = arity(g.code) - 1;
          out.put({nc});
          for (int l = 0; l <= nc; ++l) out.put({g.w[l]});
          out.put(matrix(g.code, g.p));
        }
      } else {
        while (j < N && at(j).code == op.code) ++j;
        out.put({S_PAIR, op.code == G_YYPHASE ? 1 : 0, (int)(j - i)});
        for (size_t k = i; k < j; ++k) {
          out.put({at(k).w[0], at(k).w[1]});
          out.d.push_back(at(k).p[0]);
        }
      }
      i = j;
    }
    used[0] = (int64_t)out.i.size();
    used[1] = (int64_t)out.d.size();
    if (used[0] > ints_cap || used[1] > doubles_cap) return fail(MQ_EUNSUPPORTED, "output arrays too small");
    std::memcpy(ints, out.i.data(), out.i.size() * sizeof(int32_t));
    std::memcpy(doubles, out.d.data(), out.d.size() * sizeof(double));
    return MQ_OK;
  } catch (const std::bad_alloc&) {
    return fail(MQ_ENOMEM, "host allocation failed");
  } catch (const std::exception& ex) {
    return fail(MQ_EDEVICE, ex.what());
  } catch (...) {
    return fail(MQ_EDEVICE, "unknown C++ exception");
  }
}

}  // extern "C"
