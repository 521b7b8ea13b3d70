// Pauli expectations (e): <psi|P|psi> of a list of words.
//
// Replaces pauli_product_expectations, one functional copy of the state per word
// (_common.py:384-427).  Every sum has a fixed order, so results are
// bit-reproducible run to run.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "mq_pauli.cuh"

namespace mq {

// -------------------------------------------------------------- Pauli words
// <psi|P|psi> of a word with masks (x, z) is sum_i (-1)^{|i & z|} v_i,
// v_i = conj(a_{i^x}) a_i.  The pair (i, i^x) contributes
// (-1)^{|i & z|} (v_i + (-1)^{|x & z|} conj v_i): twice the real part of v_i,
// or twice i times its imaginary part, so each pair is read and multiplied
// once and one real sum per word is kept, in float64.  Three kernels share
// the words of a call (pauli_launch):
//   k_pauli_z     words without X or Y (x = 0), any number in one pass;
//   k_pauli_tile  words whose X and Y letters lie within four index bits of a
//                 tile window, up to kTileWords in one pass;
//   k_pauli       the rest, eight words of one x per pass over the state.
// A word's sum depends on its masks and the launch shape only, never on the
// other words of the call.
constexpr int kWords = 8;
constexpr int kGroups = 64;
struct PauliGroup {
  uint32_t x;
  uint16_t nw, imag;  // words; bit w: word w keeps the imaginary part
  uint32_t z[kWords];
};
struct PauliParams {
  uint32_t pairs;  // pairs (x != 0) or amplitudes (x = 0)
  uint32_t n_groups;
  PauliGroup g[kGroups];
};

// One group per block column (blockIdx.x % n_groups): the groups of a launch
// walk the state in step.  part[(group * kWords + word) * blocks + block].
// Bound by memory: 25 qubits, one word: 135 us reading both amplitudes of
// every pair twice, 39 us a group this way (15 groups of one launch).
template <typename R>
__global__ void __launch_bounds__(256) k_pauli(const V2<R>* __restrict__ st, const __grid_constant__ PauliParams P,
                                               double* __restrict__ part) {
  __shared__ double red[8][kWords];
  const uint32_t grp = blockIdx.x % P.n_groups, block = blockIdx.x / P.n_groups, blocks = gridDim.x / P.n_groups;
  const PauliGroup& G = P.g[grp];
  const uint32_t x = G.x;
  const int h = x ? 31 - __clz(x) : 0;
  const uint32_t low = (1u << h) - 1u;
  const int nw = G.nw;
  const uint32_t imag = G.imag;
  double acc[kWords];
#pragma unroll
  for (int w = 0; w < kWords; ++w) acc[w] = 0.0;
  const uint32_t stride = blocks * 256u;
  constexpr int U = 4;
  for (uint32_t u0 = block * 256u + threadIdx.x; u0 < P.pairs; u0 += U * stride) {
    V2<R> a[U], b[U];
    uint32_t id[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint64_t u = (uint64_t)u0 + (uint64_t)k * stride;
      id[k] = 0;
      a[k] = b[k] = mk<R>(0, 0);
      if (u < P.pairs) {
        // the pair's index with bit h clear; x = 0: every index, its own partner
        id[k] = x ? ((((uint32_t)u & ~low) << 1) | ((uint32_t)u & low)) : (uint32_t)u;
        a[k] = st[id[k]];
        b[k] = st[id[k] ^ x];
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const double ar = a[k].x, ai = a[k].y, br = b[k].x, bi = b[k].y;
      const double re = fma(br, ar, bi * ai);
      const double im = fma(br, ai, -(bi * ar));
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        if (w >= nw) break;
        const double v = (imag >> w) & 1u ? im : re;
        acc[w] += (__popc(id[k] & G.z[w]) & 1) ? -v : v;
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int w = 0; w < kWords; ++w) {
    if (w >= nw) break;
    double v = acc[w];
#pragma unroll
    for (int off = 16; off; off >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    if (lane == 0) red[warp][w] = v;
  }
  __syncthreads();
  if ((int)threadIdx.x < nw) {
    double v = 0.0;
    for (int k = 0; k < 8; ++k) v = __dadd_rn(v, red[k][threadIdx.x]);
    part[((size_t)grp * kWords + threadIdx.x) * blocks + block] = v;
  }
}

// Words without X or Y: sum_i (-1)^{|i & z|} p_i.  A tile of 2^12 consecutive
// probabilities is turned into its 4096 Walsh sums in three register steps of
// four bits; every word then takes one of them per tile, signed by the
// parity of the tile's high bits, so the cost does not grow with the number
// of words (one per thread and launch).  25 qubits, 24 ZZ words: three passes
// of 135 us before, one of 74 us now.
constexpr int kZBits = 12;
constexpr int kZThreads = 256;
struct PauliZParams {
  uint32_t n_tiles;
  int32_t nw;
  uint32_t z[kZThreads];
};
__device__ __forceinline__ void walsh16(double (&v)[16]) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      if (r & (1 << k)) continue;
      const double s = v[r] + v[r | (1 << k)], d = v[r] - v[r | (1 << k)];
      v[r] = s;
      v[r | (1 << k)] = d;
    }
}
// shared-memory place of entry i (16 banks of 8 bytes): bits 4-7 fold onto
// bits 0-3, so that the register steps over bits 1-4 and 5-8 spread over them
__device__ __forceinline__ uint32_t zslot(uint32_t i) { return i ^ ((i >> 4) & 15u) ^ ((i >> 8) & 15u); }

template <typename R>
__global__ void __launch_bounds__(kZThreads) k_pauli_z(const V2<R>* __restrict__ st,
                                                       const __grid_constant__ PauliZParams P,
                                                       double* __restrict__ part) {
  __shared__ double wal[1 << kZBits];
  const uint32_t tid = threadIdx.x;
  const uint32_t z = (int)tid < P.nw ? P.z[tid] : 0u;
  const uint32_t zl = zslot(z & ((1u << kZBits) - 1u)), zh = z >> kZBits;
  double acc = 0.0;
  for (uint32_t tile = blockIdx.x; tile < P.n_tiles; tile += gridDim.x) {
    const V2<R>* src = st + ((size_t)tile << kZBits);
    double v[16];  // bit 0 and bits 9-11 in registers
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t i = 2 * tid + 512 * k;
      if constexpr (sizeof(R) == 4) {
        const float4 q = *reinterpret_cast<const float4*>(src + i);
        v[2 * k] = amp2<R>(mk<R>(q.x, q.y));
        v[2 * k + 1] = amp2<R>(mk<R>(q.z, q.w));
      } else {
        v[2 * k] = amp2<R>(src[i]);
        v[2 * k + 1] = amp2<R>(src[i + 1]);
      }
    }
    walsh16(v);
    __syncthreads();  // the words of the previous tile have been read
#pragma unroll
    for (int r = 0; r < 16; ++r) wal[zslot((2 * tid) | (r & 1) | ((r >> 1) << 9))] = v[r];
    __syncthreads();
    // bits 1-4, then bits 5-8; the other eight bits are the thread's
#pragma unroll
    for (int step = 0; step < 2; ++step) {
      const int lo = step ? 5 : 1;
      const uint32_t low = (1u << lo) - 1u;
      const uint32_t i0 = ((tid & ~low) << 4) | (tid & low);
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = wal[zslot(i0 | ((uint32_t)r << lo))];
      walsh16(v);
#pragma unroll
      for (int r = 0; r < 16; ++r) wal[zslot(i0 | ((uint32_t)r << lo))] = v[r];
      __syncthreads();
    }
    const double t = wal[zl];
    acc += (__popc(tile & zh) & 1) ? -t : t;
  }
  if ((int)tid < P.nw) part[(size_t)tid * gridDim.x + blockIdx.x] = acc;
}

// res[idx[v]] = sum of part[v * blocks ..+ blocks): each thread a strided
// share in increasing order, then a fixed halving tree.
constexpr int kFinishThreads = 128;
struct PauliFinish {
  uint32_t blocks;
  uint16_t idx[kGroups * kWords];  // 0xffff: an unused slot
};
__global__ void __launch_bounds__(kFinishThreads) k_pauli_finish(const double* __restrict__ part,
                                                                 const __grid_constant__ PauliFinish F,
                                                                 double* __restrict__ res) {
  __shared__ double red[kFinishThreads];
  if (F.idx[blockIdx.x] == 0xffffu) return;
  const double* p = part + (size_t)blockIdx.x * F.blocks;
  double v = 0.0;
  for (uint32_t b = threadIdx.x; b < F.blocks; b += kFinishThreads) v = __dadd_rn(v, p[b]);
  red[threadIdx.x] = v;
  __syncthreads();
#pragma unroll
  for (int s = kFinishThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) red[threadIdx.x] = __dadd_rn(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) res[F.idx[blockIdx.x]] = red[0];
}

// The launch shape of a call's words: where each one goes.  The tile sweeps
// of an n-qubit state cover the index bits [0, M), then eight bits at a time
// over the low passengers that make a 128-byte run, each sweep overlapping the
// one below by a bit so that neighbouring bits always share a tile; a
// sweep's windows are the aligned nibbles of its tile and those shifted by two.
// A word goes to the first sweep, and there the first window, that holds its
// X mask.
struct PauliWindow {
  int sweep;
  std::vector<int> bits;  // four index bits, ascending
  uint32_t mask;
};
struct PauliSweep {
  std::vector<int> tile;  // M index bits, ascending
};
static void pauli_windows(int n, int M, std::vector<PauliSweep>& sweeps, std::vector<PauliWindow>& wins) {
  for (int lo = 0; lo < n; lo = sweeps.size() == 1 ? M - 1 : lo + 7) {
    if (!sweeps.empty() && lo + 1 >= n) break;  // only the shared bit is left
    PauliSweep s;
    if (sweeps.empty()) {
      for (int b = 0; b < M; ++b) s.tile.push_back(b);
    } else {
      for (int b = lo; b < std::min(lo + 8, n); ++b) s.tile.push_back(b);
      for (int b = 0; (int)s.tile.size() < M; ++b) s.tile.push_back(b);  // >= M - 8 passengers, all below lo
      std::sort(s.tile.begin(), s.tile.end());
    }
    sweeps.push_back(s);
    const int id = (int)sweeps.size() - 1;
    const int first = id == 0 ? 0 : (int)(std::find(s.tile.begin(), s.tile.end(), lo) - s.tile.begin());
    auto add = [&](int at) {
      at = std::min(at, M - 4);
      PauliWindow w;
      w.sweep = id;
      w.mask = 0;
      for (int k = 0; k < 4; ++k) {
        w.bits.push_back(s.tile[at + k]);
        w.mask |= 1u << s.tile[at + k];
      }
      wins.push_back(w);
    };
    for (int at = first; at < M; at += 4) add(at);
    for (int at = first + 2; at + 2 < M; at += 4) add(at);
    if (id > 0 && lo + 8 >= n) break;
  }
}

// Sums of every word into res[0 .. n_words) (device memory): twice nothing,
// the sum over pairs (x != 0) or amplitudes (x = 0) of the part the word
// keeps.  part: room for part_cap doubles, at least kWords * num_sms * 4.
static int pauli_launch(mq_state* h, int n_words, const uint64_t* xmask, const uint64_t* zmask, double* part,
                        size_t part_cap, double* res) {
  const int n = h->n;
  const bool c64 = h->dtype == MQ_C64;
  const int M = c64 ? PauliTile<float>::M : PauliTile<double>::M;
  auto odd = [](uint64_t v) { return (__builtin_popcountll(v) & 1) != 0; };
  auto finish = [&](uint32_t blocks, const std::vector<int>& idx) -> int {
    PauliFinish F;
    F.blocks = blocks;
    for (size_t v = 0; v < idx.size(); ++v) F.idx[v] = idx[v] < 0 ? 0xffffu : (uint16_t)idx[v];
    k_pauli_finish<<<(uint32_t)idx.size(), kFinishThreads, 0, h->stream>>>(part, F, res);
    MQ_LAUNCHED("k_pauli_finish");
    h->launches += 2;
    h->sweeps += 1;
    return MQ_OK;
  };
  std::vector<int> rest;
  std::vector<std::vector<int>> in_win;
  std::vector<PauliSweep> sweeps;
  std::vector<PauliWindow> wins;
  std::vector<int> zwords;
  // small states: one launch of the general kernel is all latency anyway
  if (n > kZBits) {
    pauli_windows(n, M, sweeps, wins);
    in_win.resize(wins.size());
  }
  for (int w = 0; w < n_words; ++w) {
    if (n > kZBits && xmask[w] == 0) {
      zwords.push_back(w);
      continue;
    }
    size_t k = 0;
    while (k < wins.size() && (xmask[w] & ~(uint64_t)wins[k].mask)) ++k;
    if (k < wins.size()) in_win[k].push_back(w);
    else rest.push_back(w);
  }
  // words without X or Y
  const uint32_t zgrid = (uint32_t)std::min<uint64_t>(h->dim() >> kZBits, (uint64_t)h->num_sms * 4);
  for (size_t i = 0; i < zwords.size();) {
    PauliZParams Z;
    std::memset(&Z, 0, sizeof(Z));
    Z.n_tiles = (uint32_t)(h->dim() >> kZBits);
    const size_t most = std::min<size_t>(kZThreads, part_cap / zgrid);
    std::vector<int> idx;
    for (; i < zwords.size() && idx.size() < most; ++i) {
      Z.z[idx.size()] = (uint32_t)zmask[zwords[i]];
      idx.push_back(zwords[i]);
    }
    Z.nw = (int32_t)idx.size();
    if (c64) k_pauli_z<float><<<zgrid, kZThreads, 0, h->stream>>>((const float2*)h->cur_buf(), Z, part);
    else k_pauli_z<double><<<zgrid, kZThreads, 0, h->stream>>>((const double2*)h->cur_buf(), Z, part);
    MQ_LAUNCHED("k_pauli_z");
    int rc = finish(zgrid, idx);
    if (rc) return rc;
  }
  // words of the tile windows, sweep by sweep
  for (size_t sw = 0; sw < sweeps.size(); ++sw) {
    std::vector<std::pair<int, int>> todo;  // (window, word)
    for (size_t k = 0; k < wins.size(); ++k)
      if (wins[k].sweep == (int)sw) {
        auto single = [&](int w) { return zmask[w] == 0 && (xmask[w] & (xmask[w] - 1)) == 0; };
        std::stable_partition(in_win[k].begin(), in_win[k].end(), single);
        for (int w : in_win[k]) todo.push_back({(int)k, w});
      }
    const uint32_t n_tiles = (uint32_t)(h->dim() >> M);
    const uint32_t grid = std::min<uint32_t>(n_tiles, (uint32_t)h->num_sms * 4);
    const size_t most = std::min<size_t>(kTileWords, part_cap / grid);
    for (size_t i = 0; i < todo.size();) {
      PauliTileParams P;
      std::memset(&P, 0, sizeof(P));
      P.n_tiles = n_tiles;
      for (int k = 0; k < M; ++k) P.tile_bit[k] = (uint8_t)sweeps[sw].tile[k];
      make_base_runs(P.runs, n, P.tile_bit, M);
      std::vector<int> idx;
      int open = -1;  // the window the launch's last entry belongs to
      for (; i < todo.size() && idx.size() < most; ++i) {
        const PauliWindow& W = wins[todo[i].first];
        if (todo[i].first != open) {
          if (P.n_win == kTileWins) break;
          open = todo[i].first;
          PauliWin& D = P.win[P.n_win++];
          std::memset(D.one, 0xff, sizeof(D.one));
          D.w0 = (uint16_t)idx.size();
          auto phys = [c64](uint32_t v) -> uint32_t { return c64 ? (v ^ ((v >> 3) & 0xEu)) : (v ^ ((v >> 3) & 7u)); };
          int j = 0, r = 0;
          for (int k = 0; k < M; ++k) {
            const uint32_t g = 1u << sweeps[sw].tile[k];
            if (W.mask & g) {
              D.s_reg[r++] = phys(1u << k);
            } else {
              D.s_grp[j] = phys(1u << k);
              D.g_grp[j++] = g;
            }
          }
        }
        const int w = todo[i].second;
        PauliTileWord& T = P.word[idx.size()];
        uint32_t zr = 0;
        for (int k = 0; k < 4; ++k) {
          if ((xmask[w] >> W.bits[k]) & 1u) T.x |= (uint8_t)(1 << k);
          if ((zmask[w] >> W.bits[k]) & 1u) zr |= 1u << k;
        }
        for (uint32_t r = 0; r < 16; ++r)
          if (odd(r & zr)) T.sgn |= (uint16_t)(1u << r);
        T.z = (uint32_t)zmask[w] & ~W.mask;
        T.imag = odd(xmask[w] & zmask[w]) ? 1 : 0;
        PauliWin& D = P.win[P.n_win - 1];
        if (zmask[w] == 0 && (T.x & (T.x - 1)) == 0 && D.one[__builtin_ctz(T.x)] == 0xff && D.w0 == idx.size()) {
          // single X letters come first in the window's list (a repeated one ends them)
          D.one[__builtin_ctz(T.x)] = (uint8_t)idx.size();
          D.w0 = (uint16_t)(idx.size() + 1);
        }
        idx.push_back(w);
        D.w1 = (uint16_t)idx.size();
        D.zs |= T.z;
      }
      P.n_words = (uint8_t)idx.size();
      int rc = launch_pauli_tile(h, P, grid, part);
      if (rc) return rc;
      rc = finish(grid, idx);
      if (rc) return rc;
    }
  }
  // the rest: groups of up to kWords words of one x
  std::vector<bool> done(rest.size(), false);
  std::vector<std::vector<int>> groups;
  for (size_t i = 0; i < rest.size(); ++i) {
    if (done[i]) continue;
    std::vector<int> g;
    for (size_t j = i; j < rest.size() && (int)g.size() < kWords; ++j)
      if (!done[j] && xmask[rest[j]] == xmask[rest[i]]) {
        g.push_back(rest[j]);
        done[j] = true;
      }
    groups.push_back(g);
  }
  std::stable_partition(groups.begin(), groups.end(), [&](const std::vector<int>& g) { return xmask[g[0]] == 0; });
  for (size_t i = 0; i < groups.size();) {
    PauliParams P;
    std::memset(&P, 0, sizeof(P));
    // x = 0 (small states only) sums amplitudes, the others pairs
    const bool diag = xmask[groups[i][0]] == 0;
    P.pairs = (uint32_t)(diag ? h->dim() : h->dim() >> 1);
    const uint32_t blocks = (uint32_t)std::min<uint64_t>(((uint64_t)P.pairs + 255) / 256, (uint64_t)h->num_sms * 4);
    const size_t most = std::min<size_t>(kGroups, part_cap / ((size_t)kWords * blocks));
    std::vector<int> idx;
    for (; i < groups.size() && P.n_groups < most && (xmask[groups[i][0]] == 0) == diag; ++i) {
      PauliGroup& G = P.g[P.n_groups++];
      G.x = (uint32_t)xmask[groups[i][0]];
      G.nw = (uint16_t)groups[i].size();
      for (int w = 0; w < kWords; ++w) {
        if (w >= G.nw) {
          idx.push_back(-1);
          continue;
        }
        const int id = groups[i][w];
        G.z[w] = (uint32_t)zmask[id];
        if (odd(xmask[id] & zmask[id])) G.imag |= (uint16_t)(1u << w);
        idx.push_back(id);
      }
    }
    if (c64) k_pauli<float><<<blocks * P.n_groups, 256, 0, h->stream>>>((const float2*)h->cur_buf(), P, part);
    else k_pauli<double><<<blocks * P.n_groups, 256, 0, h->stream>>>((const double2*)h->cur_buf(), P, part);
    MQ_LAUNCHED("k_pauli");
    int rc = finish(blocks, idx);
    if (rc) return rc;
  }
  return MQ_OK;
}

// A word's value from its sum: both members of a pair, then the factor i^ny.
static void pauli_value(uint64_t x, uint64_t z, int ny, double sum, double* out) {
  const double v = x ? 2.0 * sum : sum;
  const double none = v * 0.0 + 0.0;  // 0, or NaN where the sum is not finite
  const bool imag = (__builtin_popcountll(x & z) & 1) != 0;
  const double re = imag ? none : v, im = imag ? v : none;
  double fr = re, fi = im;
  switch ((ny % 4 + 4) % 4) {
    case 1: fr = -im; fi = re; break;
    case 2: fr = -re; fi = -im; break;
    case 3: fr = im; fi = -re; break;
    default: break;
  }
  out[0] = fr;
  out[1] = fi;
}

constexpr int kCallWords = 4096;  // words per pass over pauli_launch (bounds the result array)

int run_expval_pauli(mq_state* h, int n_words, const uint64_t* xmask, const uint64_t* zmask, const int32_t* ny,
                     double* out) {
  const uint64_t lim = h->dim() - 1;
  for (int w = 0; w < n_words; ++w)
    if ((xmask[w] & ~lim) || (zmask[w] & ~lim)) return fail(MQ_EINVAL, "Pauli mask outside the register");
  std::vector<double> host;
  for (int w0 = 0; w0 < n_words; w0 += kCallWords) {
    const int cnt = std::min(n_words - w0, kCallWords);
    // partial sums of one launch: at most one group of kWords slots per word,
    // over four blocks per SM
    const size_t cap = (size_t)std::min(cnt, kGroups) * kWords * (size_t)h->num_sms * 4;
    int rc = ensure_scratch(h, (cap + cnt) * sizeof(double));
    if (rc) return rc;
    double* res = (double*)h->scratch;
    rc = pauli_launch(h, cnt, xmask + w0, zmask + w0, res + cnt, cap, res);
    if (rc) return rc;
    host.resize(cnt);
    MQ_CUDA(cudaMemcpyAsync(host.data(), res, (size_t)cnt * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
    for (int w = 0; w < cnt; ++w)
      pauli_value(xmask[w0 + w], zmask[w0 + w], ny ? ny[w0 + w] : 0, host[w], out + 2 * (w0 + w));
  }
  return MQ_OK;
}

// ================================================ allocation-free expectations
// mq_expval_pauli_static computes the same values as mq_expval_pauli, but
// never allocates device memory.  mq_expval_pauli grows the handle's scratch
// buffer with cudaMalloc (and cudaFree) the first time it needs room for
// its per-block partial sums; cudaFree waits for the whole device.  Callers
// that run under a fixed device-memory budget (a serving loop that admits
// requests by their state footprint alone, or a host whose memory pool owns
// all free HBM) or that cannot stall other streams with that device-wide
// wait use this entry point instead.
//
// Its scratch is a file-scope device array of a fixed size: every GPU that
// loads the library holds these 131,200 bytes until the process exits.  The
// host reaches the array through the address that cudaGetSymbolAddress
// returns for the current device (the array's name in host code is only a
// host-side stand-in); the address is looked up once per device, on the
// first call made on that device, and kept for the life of the process.  A
// cudaDeviceReset (or any teardown of the device's primary context) makes
// the kept address stale: a process that resets a device must not call this
// entry point on it afterwards.
constexpr uint32_t kStaticBlocks = 1024;  // partial-sum blocks the array holds
static __device__ __align__(256) double2 g_pauli_static[kStaticBlocks * kWords + kWords];

constexpr int kStaticMaxDevices = 64;
static std::mutex g_static_mu;
static void* g_static_addr[kStaticMaxDevices] = {};

// Device address of g_pauli_static on `device`, which must be current.
static int pauli_static_scratch(int device, double2** out) {
  if (device < 0 || device >= kStaticMaxDevices) return fail(MQ_EUNSUPPORTED, "device ordinal beyond 63");
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_addr[device]) {
    void* p = nullptr;
    MQ_CUDA(cudaGetSymbolAddress(&p, g_pauli_static));
    g_static_addr[device] = p;
  }
  *out = reinterpret_cast<double2*>(g_static_addr[device]);
  return MQ_OK;
}

int run_expval_pauli_static(mq_state* h, int n_words, const uint64_t* xmask, const uint64_t* zmask,
                            const int32_t* ny, double* out) {
  const uint64_t lim = h->dim() - 1;
  for (int w = 0; w < n_words; ++w)
    if ((xmask[w] & ~lim) || (zmask[w] & ~lim)) return fail(MQ_EINVAL, "Pauli mask outside the register");
  // the launch shapes are those of run_expval_pauli (the result bits depend
  // on them): up to four blocks per SM
  const uint32_t grid = (uint32_t)h->num_sms * 4;
  if (grid > kStaticBlocks)
    return fail(MQ_EUNSUPPORTED, "mq_expval_pauli_static: this GPU needs " + std::to_string(grid) +
                                     " partial-sum blocks; the static scratch holds 1024 (GPUs of up to 256 SMs)");
  double2* scratch = nullptr;
  int rc = pauli_static_scratch(h->device, &scratch);
  if (rc) return rc;
  double* partials = reinterpret_cast<double*>(scratch);
  const size_t cap = (size_t)kStaticBlocks * kWords * 2;
  double* res = partials + cap;
  // Every slot read below is written earlier in the same call (each kernel
  // writes the slots of all its words, k_pauli_finish one result per word),
  // so whatever an earlier call left in the array is never read and nothing
  // has to be cleared.
  for (int w0 = 0; w0 < n_words; w0 += kWords) {
    const int cnt = std::min(n_words - w0, kWords);
    rc = pauli_launch(h, cnt, xmask + w0, zmask + w0, partials, cap, res);
    if (rc) return rc;
    double host[kWords];
    MQ_CUDA(cudaMemcpyAsync(host, res, (size_t)cnt * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
    for (int w = 0; w < cnt; ++w)
      pauli_value(xmask[w0 + w], zmask[w0 + w], ny ? ny[w0 + w] : 0, host[w], out + 2 * (w0 + w));
  }
  return MQ_OK;
}

}  // namespace mq
