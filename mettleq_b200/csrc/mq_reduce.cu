// Probabilities, seeded sampling and Pauli expectations (e).
//
// Replaces the reference's MLX library calls on this path:
//   probabilities_array: |a|^2, transpose, sum           (sim.py:322-343)
//   sample_array: log(max(p,1e-30)) + mx.random.categorical (sim.py:383-419)
//   pauli_product_expectations: one functional copy per word (_common.py:384-427)
//
// Every reduction has a fixed order so results are bit-reproducible run to
// run and can be restated exactly on the CPU:
//   * p_i = re^2 + im^2 in float64 with explicitly rounded operations;
//   * block sums: 32 lanes add entries lane, lane+32, ... sequentially, then
//     an XOR butterfly over the lanes;
//   * longer sums are sequential over <= 1024 partial sums, in two levels.
// Sampling uses Philox4x32-10 (counter = shot + stream_offset, key = seed),
// u = 53 random bits / 2^53, target t = u * total, a binary search over block
// offsets and a sequential running sum inside the chosen block.
#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "mq_internal.cuh"

namespace mq {

constexpr uint32_t kBlock = 1024;
constexpr uint32_t kSuper = 1024;

template <typename R>
__device__ __forceinline__ double amp2(V2<R> a) {
  const double re = (double)a.x, im = (double)a.y;
  return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
}

template <typename R> struct StateSrc {
  const V2<R>* st;
  __device__ __forceinline__ double operator()(uint32_t i) const { return amp2<R>(st[i]); }
};
struct VecSrc {
  const double* q;
  __device__ __forceinline__ double operator()(uint32_t i) const { return q[i]; }
};

// -------------------------------------------------------------- full |a|^2
template <typename R, typename O>
__global__ void k_amp2_out(const V2<R>* __restrict__ st, O* __restrict__ out, uint32_t dim) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += stride) out[i] = (O)amp2<R>(st[i]);
}

// -------------------------------------------------------------- block sums
template <typename Src>
__global__ void k_block_sums(Src src, uint32_t bs, uint32_t nb, double* __restrict__ S) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= nb) return;
  const uint32_t base = warp * bs;
  double acc = 0.0;
  for (uint32_t j = lane; j < bs; j += 32) acc = __dadd_rn(acc, src(base + j));
#pragma unroll
  for (int off = 16; off; off >>= 1) acc = __dadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, off));
  if (lane == 0) S[warp] = acc;
}

// Marginal chunk sums in bucket-major order.  Entry j of that order is the
// amplitude at XOR of img[t] over j's set bits (the selected and the remaining
// index bits permuted); a chunk is cs consecutive entries, lane l summing
// entries l, l + 32, ....  Where index bits 0-3 (128 bytes of complex64) hold
// selected qubits, the entries of one chunk are strided and the bytes between
// them belong to the S-bit sibling chunks that differ in those qubits only: a
// warp sums all 2^S of them together, so each line it touches is used whole.
// Chunks of fewer than 32 entries share a warp (lane bits above the chunk's
// are chunk bits).  27 qubits, 9 selected: 304 us with one warp per chunk and
// table look-ups for every address, 168 us this way (6.4 TB/s).
struct ChunkParams {
  uint8_t nb, cb;    // bits of j, bits of a chunk (cs = 2^cb)
  uint8_t spos[4];   // j bit positions (all >= max(cb, 5)) of the sibling qubits, ascending
  uint32_t img[32];  // index bit (as a mask) of every j bit
};

template <typename R, int S>
__global__ void __launch_bounds__(256) k_chunk_sums(const V2<R>* __restrict__ st, const __grid_constant__ ChunkParams P,
                                                    double* __restrict__ D) {
  constexpr int NS = 1 << S;
  __shared__ uint32_t step[32];
  const int lane = threadIdx.x & 31;
  // index offsets of j bits 5-9 (a chunk's successive 32-entry rows)
  const int rb = P.cb > 5 ? P.cb - 5 : 0;
  if (threadIdx.x < 32) {
    uint32_t g = 0;
    for (int t = 0; t < rb; ++t)
      if ((threadIdx.x >> t) & 1u) g |= P.img[5 + t];
    step[threadIdx.x] = g;
  }
  __syncthreads();
  uint32_t g_lane = 0;
#pragma unroll
  for (int t = 0; t < 5; ++t)
    if (t < P.nb && ((lane >> t) & 1)) g_lane |= P.img[t];
  uint32_t g_sib[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    g_sib[s] = 0;
#pragma unroll
    for (int t = 0; t < S; ++t)
      if ((s >> t) & 1) g_sib[s] |= P.img[P.spos[t]];
  }
  const int wb = max((int)P.cb, 5);  // j bits a warp covers
  const bool lane_on = P.nb >= 5 || (lane >> P.nb) == 0;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t n_units = P.nb > wb + S ? 1u << (P.nb - wb - S) : 1u;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n_units; w += warps) {
    // j of the warp's first entry: w's bits around the sibling positions
    uint32_t j0 = w << wb;
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const uint32_t low = (1u << P.spos[t]) - 1u;
      j0 = ((j0 & ~low) << 1) | (j0 & low);
    }
    const uint32_t base =
        __reduce_or_sync(0xffffffffu, (lane < P.nb && ((j0 >> lane) & 1u)) ? P.img[lane] : 0u) | g_lane;
    double acc[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) acc[s] = 0.0;
    if (lane_on) {
      constexpr int U = NS >= 8 ? 1 : 8 / NS;  // rows in flight
      const int rows = 1 << rb;
      int i = 0;
      for (; i + U <= rows; i += U) {
        V2<R> v[U][NS];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int s = 0; s < NS; ++s) v[u][s] = st[base | step[i + u] | g_sib[s]];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int s = 0; s < NS; ++s) acc[s] = __dadd_rn(acc[s], amp2<R>(v[u][s]));
      }
      for (; i < rows; ++i)
#pragma unroll
        for (int s = 0; s < NS; ++s) acc[s] = __dadd_rn(acc[s], amp2<R>(st[base | step[i] | g_sib[s]]));
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
#pragma unroll
      for (int off = 16; off; off >>= 1)
        if ((off >> P.cb) == 0) acc[s] = __dadd_rn(acc[s], __shfl_xor_sync(0xffffffffu, acc[s], off));
      uint32_t js = j0 | (uint32_t)lane;
#pragma unroll
      for (int t = 0; t < S; ++t)
        if ((s >> t) & 1) js |= 1u << P.spos[t];
      if (lane_on && (P.cb >= 5 ? lane == 0 : (lane & ((1 << P.cb) - 1)) == 0)) D[js >> P.cb] = acc[s];
    }
  }
}

// Sequential sums of consecutive runs: out[t] = sum of in[t*len .. t*len+cnt)
// with cnt = min(len, total - t*len) restricted to the run's own group.  The
// long runs take a warp each, which stages kSuper entries in shared memory
// and adds them in order (every lane alike, from broadcast reads); runs of at
// most 16 entries (two lines) a thread each.  512 runs of 256 entries: 22 us
// by one thread per run, 4.8 us by warps; 65536 runs of two (27 qubits, 16
// selected): a call of 282 us by warps, 260 by threads.
constexpr int kSeqWarps = 4;
__global__ void __launch_bounds__(32 * kSeqWarps) k_seq_sums_warp(const double* __restrict__ in, uint32_t group_len,
                                                                  uint32_t run_len, uint32_t runs_per_group,
                                                                  uint32_t n_runs, double* __restrict__ out) {
  __shared__ __align__(16) double stage[kSeqWarps][kSuper];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t t = blockIdx.x * kSeqWarps + warp;
  if (t >= n_runs) return;
  const uint32_t g = t / runs_per_group, r = t % runs_per_group;
  const uint32_t start = g * group_len + r * run_len;
  const uint32_t end = min(start + run_len, (g + 1) * group_len);
  double* v = stage[warp];
  double acc = 0.0;
  for (uint32_t at = start; at < end; at += kSuper) {
    const uint32_t cnt = min(end - at, kSuper);
    __syncwarp();
    for (uint32_t i = lane; i < cnt; i += 32) v[i] = in[at + i];
    __syncwarp();
    uint32_t i = 0;
    for (; i + 8 <= cnt; i += 8) {
      double q[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) q[k] = v[i + k];
#pragma unroll
      for (int k = 0; k < 8; ++k) acc = __dadd_rn(acc, q[k]);
    }
    for (; i < cnt; ++i) acc = __dadd_rn(acc, v[i]);
  }
  if (lane == 0) out[t] = acc;
}

__global__ void k_seq_sums(const double* __restrict__ in, uint32_t group_len, uint32_t run_len,
                           uint32_t runs_per_group, uint32_t n_runs, double* __restrict__ out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_runs) return;
  const uint32_t g = t / runs_per_group, r = t % runs_per_group;
  const uint32_t start = g * group_len + r * run_len;
  const uint32_t end = min(start + run_len, (g + 1) * group_len);
  double acc = 0.0;
  for (uint32_t i = start; i < end; ++i) acc = __dadd_rn(acc, in[i]);
  out[t] = acc;
}

// The running sums below are sequential by definition (each addition rounds
// on the one before it), so their length is bound by the latency of a double
// addition.  What can be taken off that chain is the memory access: one CTA
// per run stages its values in shared memory with coalesced loads, one thread
// adds them from there, and the CTA writes the results back coalesced.
// Measured at 28 qubits (256 runs of 1024): 188 us with one thread per run
// reading and writing device memory itself, 8.8 us this way.
constexpr int kPrefixThreads = 256;

// v[0..cnt) -> its exclusive running sums, in place; returns the total.
// Eight values are read ahead of the eight additions that use them.
__device__ __forceinline__ double exclusive_sums(double* v, uint32_t cnt) {
  double e = 0.0;
  uint32_t i = 0;
  for (; i + 8 <= cnt; i += 8) {
    double q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = v[i + k];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[i + k] = e;
      e = __dadd_rn(e, q[k]);
    }
  }
  for (; i < cnt; ++i) {
    const double s = v[i];
    v[i] = e;
    e = __dadd_rn(e, s);
  }
  return e;
}

// Exclusive running sums inside super-blocks of kSuper blocks (one CTA each).
__global__ void __launch_bounds__(kPrefixThreads) k_local_prefix(const double* __restrict__ S, uint32_t nb,
                                                                 double* __restrict__ L, double* __restrict__ T,
                                                                 int32_t* __restrict__ LP) {
  __shared__ __align__(16) double v[kSuper];
  __shared__ int32_t last;
  const uint32_t start = blockIdx.x * kSuper;
  const uint32_t cnt = min(nb - start, kSuper);
  if (threadIdx.x == 0) last = -1;
  __syncthreads();
  int32_t mine = -1;
  for (uint32_t i = threadIdx.x; i < cnt; i += kPrefixThreads) {
    const double s = S[start + i];
    v[i] = s;
    if (s > 0.0) mine = (int32_t)(start + i);
  }
  if (mine >= 0) atomicMax(&last, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    T[blockIdx.x] = exclusive_sums(v, cnt);
    LP[blockIdx.x] = last;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < cnt; i += kPrefixThreads) L[start + i] = v[i];
}

struct SampleMeta {
  double total;
  int32_t last_block;
  int32_t pad;
};

// Exclusive running sum over the super-blocks (at most 2^31 / 2^20 = 2048 of
// them), by one CTA.
constexpr uint32_t kMaxSupers = 2048;
__global__ void __launch_bounds__(kPrefixThreads) k_super_prefix(const double* __restrict__ T,
                                                                 const int32_t* __restrict__ LP, uint32_t ng,
                                                                 double* __restrict__ E, SampleMeta* __restrict__ meta) {
  __shared__ double v[kMaxSupers];
  __shared__ int32_t last;
  if (threadIdx.x == 0) last = -1;
  __syncthreads();
  int32_t mine = -1;
  for (uint32_t g = threadIdx.x; g < ng; g += kPrefixThreads) {
    v[g] = T[g];
    mine = max(mine, LP[g]);
  }
  if (mine >= 0) atomicMax(&last, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    meta->total = exclusive_sums(v, ng);
    meta->last_block = last;
  }
  __syncthreads();
  for (uint32_t g = threadIdx.x; g < ng; g += kPrefixThreads) E[g] = v[g];
}

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    if (r) { k.x += W0; k.y += W1; }
    const uint32_t lo0 = M0 * c.x, hi0 = __umulhi(M0, c.x);
    const uint32_t lo1 = M1 * c.z, hi1 = __umulhi(M1, c.z);
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
  }
  return c;
}

// The target of shot s on the scale of the total.
__device__ __forceinline__ double shot_target(int64_t s, uint64_t seed, uint64_t offset, double total) {
  const uint64_t ctr = (uint64_t)s + offset;
  const uint4 x = philox4x32_10(make_uint4((uint32_t)ctr, (uint32_t)(ctr >> 32), 0u, 0u),
                                make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  const uint64_t bits = ((((uint64_t)x.y) << 32) | x.x) >> 11;
  const double u = (double)bits * 0x1p-53;
  return __dmul_rn(u, total);
}

// One thread per shot: a binary search for the block, then its entries one
// by one.  Bound by the latency of 1024 dependent reads and additions, about
// 120 us whatever the number of shots, until they fill the GPU.  The better
// one from kThreadShots shots: 20 qubits, a call of 16000 shots 232 us (170 with
// a warp per shot), of 32000 262 (262), of 128000 572 (831); at 2 to 8 qubits
// the two are equal near 16000.
constexpr int64_t kThreadShots = 24576;
template <typename Src>
__global__ void k_draw_threads(Src src, uint32_t bs, uint32_t nb, const double* __restrict__ L,
                               const double* __restrict__ E, const SampleMeta* __restrict__ meta, uint64_t seed,
                               uint64_t offset, int64_t shots, int64_t* __restrict__ out) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= shots) return;
  const double t = shot_target(s, seed, offset, meta->total);
  uint32_t lo = 0, hi = nb - 1;
  while (lo < hi) {
    const uint32_t mid = (lo + hi + 1) >> 1;
    const double c = __dadd_rn(E[mid / kSuper], L[mid]);
    if (c <= t) lo = mid; else hi = mid - 1;
  }
  uint32_t b = lo;
  if ((int32_t)b > meta->last_block) b = (uint32_t)max(meta->last_block, 0);
  double r = __dadd_rn(E[b / kSuper], L[b]);
  const uint32_t base = b * bs;
  int64_t found = -1;
  for (uint32_t i = 0; i < bs; ++i) {
    r = __dadd_rn(r, src(base + i));
    if (r > t) { found = i; break; }
  }
  if (found < 0) {
    for (int64_t i = (int64_t)bs - 1; i >= 0; --i)
      if (src(base + (uint32_t)i) > 0.0) { found = i; break; }
    if (found < 0) found = 0;
  }
  out[s] = (int64_t)base + found;
}

// One warp per shot.  The block is found by a 32-way search over the
// (non-decreasing) block offsets; its entries are staged in shared memory
// with coalesced loads and summed in order by every lane alike (a broadcast
// read each), so the chain costs the latency of a double addition per entry
// instead of a dependent 8-byte gather: 1000 shots of 28 qubits took 200 us
// with one thread per shot, 22 us this way.
constexpr int kDrawWarps = 4;
template <typename Src>
__global__ void __launch_bounds__(32 * kDrawWarps)
k_draw(Src src, uint32_t bs, uint32_t nb, const double* __restrict__ L, const double* __restrict__ E,
       const SampleMeta* __restrict__ meta, uint64_t seed, uint64_t offset, int64_t shots, int64_t* __restrict__ out) {
  __shared__ __align__(16) double stage[kDrawWarps][kBlock];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* p = stage[warp];
  const int64_t s = (int64_t)blockIdx.x * kDrawWarps + warp;
  if (s >= shots) return;
  const double t = shot_target(s, seed, offset, meta->total);
  // the last block whose offset is <= t (block 0 if none is)
  uint32_t lo = 0, hi = nb - 1;
  while (lo < hi) {
    const uint32_t span = hi - lo;
    auto probe = [&](int i) -> uint32_t { return lo + (uint32_t)(((uint64_t)span * (uint32_t)(i + 1) + 31) >> 5); };
    const uint32_t m = probe(lane);
    const double c = __dadd_rn(E[m / kSuper], L[m]);
    const int below = __popc(__ballot_sync(0xffffffffu, c <= t));
    const uint32_t l0 = below ? probe(below - 1) : lo;
    hi = below < 32 ? probe(below) - 1 : hi;
    lo = l0;
  }
  uint32_t b = lo;
  if ((int32_t)b > meta->last_block) b = (uint32_t)max(meta->last_block, 0);
  const uint32_t base = b * bs;
  int32_t last = -1;
  for (uint32_t i = lane; i < bs; i += 32) {
    const double v = src(base + i);
    p[i] = v;
    if (v > 0.0) last = (int32_t)i;
  }
  __syncwarp();
  double r = __dadd_rn(E[b / kSuper], L[b]);
  int32_t found = -1;
  uint32_t i = 0;
  // the running sum never falls, so a group of eight holds the first entry
  // above t when its last partial sum is above t
  for (; i + 8 <= bs && found < 0; i += 8) {
    double q[8];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const double2 w = *reinterpret_cast<const double2*>(p + i + k);
      q[k] = w.x;
      q[k + 1] = w.y;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = r = __dadd_rn(r, q[k]);
    if (r > t) {
#pragma unroll
      for (int k = 7; k >= 0; --k)
        if (q[k] > t) found = (int32_t)i + k;
    }
  }
  for (; i < bs && found < 0; ++i) {
    r = __dadd_rn(r, p[i]);
    if (r > t) found = (int32_t)i;
  }
  if (found < 0) found = max(__reduce_max_sync(0xffffffffu, last), 0);
  if (lane == 0) out[s] = (int64_t)base + found;
}

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

// Words whose X and Y letters lie within a window of four tile bits.  A tile
// (2^12 complex64 or 2^11 complex128 amplitudes: 32 KB) is loaded once; for
// every window in use each thread takes groups of 16 amplitudes that differ
// in the window's bits to registers, in float64, and sums the eight pairs of
// every word there (two products per pair).  Sums per word and thread stay in
// shared memory.  Bound by the float64 work (16 products per 16 amplitudes
// and word) and the float32 -> float64 conversions of every window; 25
// qubits, 25 X words: 25 passes of 135 us before, three of 79 us on average now
// (117 with every word through the switch).
constexpr int kTileWords = 24;
constexpr int kTileWins = 6;
constexpr int kPauliLT = 7;
constexpr int kPauliSmem = 32768 + kTileWords * (1 << kPauliLT) * 8;
template <typename R> struct PauliTile;
template <> struct PauliTile<float> { static constexpr int M = 12; };
template <> struct PauliTile<double> { static constexpr int M = 11; };
struct PauliWin {
  uint32_t s_reg[4], s_grp[8], g_grp[8];
  uint16_t w0, w1;  // words [w0, w1) of the window
  uint32_t zs;      // Z letters of its words outside it (0: signs need no index)
  uint8_t one[4];   // word X on the window's bit k alone, no Z letters; 0xff: none
};
struct PauliTileWord {
  uint32_t z;         // Z mask outside the window (index bits)
  uint16_t sgn;       // bit r: register pattern r carries the sign -1
  uint8_t x, imag;    // X mask over the window's four bits; the imaginary part is kept
};
struct PauliTileParams {
  uint32_t n_tiles;
  uint8_t n_win, n_words, pad[2];
  uint8_t tile_bit[16];
  BaseRuns runs;
  PauliWin win[kTileWins];
  PauliTileWord word[kTileWords];
};

// Four running sums: their additions' latency, not their rate, would bound two.
template <int X, bool IMAG, bool SIGNED>
__device__ __forceinline__ double pair_sum(const double (&ar)[16], const double (&ai)[16], uint32_t sgn) {
  // the zeros are opaque, so that the compiler does not compute one case's
  // products for another (hoisted out of the switch over X they spill)
  double s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) asm volatile("mov.f64 %0, 0d0000000000000000;" : "=d"(s[k]));
  if constexpr (SIGNED) asm volatile("" : "+r"(sgn));
  int n = 0;
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    if ((r ^ X) < r) continue;
    double xr = ar[r], xi = ai[r];
    if constexpr (SIGNED) {
      const int flip = (int)((sgn << (31 - r)) & 0x80000000u);
      xr = __hiloint2double(__double2hiint(xr) ^ flip, __double2loint(xr));
      xi = __hiloint2double(__double2hiint(xi) ^ flip, __double2loint(xi));
    }
    const int j = n++ & 1;
    s[j] = fma(ar[r ^ X], IMAG ? xi : xr, s[j]);  // Re or Im of conj(b) a
    s[2 + j] = fma(ai[r ^ X], IMAG ? xr : xi, s[2 + j]);
  }
  return IMAG ? (s[0] + s[1]) - (s[2] + s[3]) : (s[0] + s[1]) + (s[2] + s[3]);
}
template <int X>
__device__ __forceinline__ double pair_sum(const double (&ar)[16], const double (&ai)[16], uint32_t sgn, bool imag) {
  if (imag) return pair_sum<X, true, true>(ar, ai, sgn);
  return sgn ? pair_sum<X, false, true>(ar, ai, sgn) : pair_sum<X, false, false>(ar, ai, sgn);
}

template <typename R>
__global__ void __launch_bounds__(1 << kPauliLT, 4) k_pauli_tile(const V2<R>* __restrict__ st,
                                                              const __grid_constant__ PauliTileParams P,
                                                              double* __restrict__ part) {
  using T = V2<R>;
  constexpr int M = PauliTile<R>::M;
  constexpr int NT = 1 << kPauliLT;
  constexpr int CB = sizeof(T) == 8 ? 1 : 0;  // log2 amplitudes per 16-byte chunk
  constexpr int CPT = (1 << (M - CB)) / NT;
  constexpr int GPT = (1 << (M - 4)) / NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* tile = reinterpret_cast<T*>(smem_raw);
  double* acc = reinterpret_cast<double*>(smem_raw + (sizeof(T) << M));  // [word][thread]
  const uint32_t tid = threadIdx.x;
  for (int w = 0; w < P.n_words; ++w) acc[w * NT + tid] = 0.0;
  uint32_t g_t = 0;
#pragma unroll
  for (int b = 0; b < kPauliLT; ++b)
    if ((tid >> b) & 1u) g_t |= 1u << P.tile_bit[CB + b];
  const uint32_t s_t = tid ^ ((tid >> 3) & 7u);
  for (uint32_t t = blockIdx.x; t < P.n_tiles; t += gridDim.x) {
    const uint32_t base = deposit_runs(t, P.runs);
    __syncthreads();  // the previous tile has been read
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      uint32_t g = base | g_t;
#pragma unroll
      for (int b = 0; b < M - CB - kPauliLT; ++b)
        if ((k >> b) & 1) g |= 1u << P.tile_bit[CB + kPauliLT + b];
      const uint32_t kk = (uint32_t)(k * NT);
      cp_async<16>(smem_u32(tile) + 16u * (s_t ^ (kk ^ ((kk >> 3) & 7u))), st + g);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    for (int win = 0; win < P.n_win; ++win) {
      const PauliWin& W = P.win[win];
#pragma unroll 1
      for (int g = 0; g < GPT; ++g) {
        const uint32_t q = tid + (uint32_t)(g * NT);
        uint32_t sq = 0, gq = base;
#pragma unroll
        for (int j = 0; j < M - 4; ++j)
          if ((q >> j) & 1u) sq ^= W.s_grp[j];
        if (W.zs)
#pragma unroll
          for (int j = 0; j < M - 4; ++j)
            if ((q >> j) & 1u) gq |= W.g_grp[j];
        double ar[16], ai[16];
        if (CB == 1 && W.s_reg[0] == 1u) {  // the pair (r, r+1) is one 16-byte chunk
#pragma unroll
          for (int r = 0; r < 16; r += 2) {
            uint32_t o = sq;
#pragma unroll
            for (int k = 1; k < 4; ++k)
              if (r & (1 << k)) o ^= W.s_reg[k];
            const float4 v = *reinterpret_cast<const float4*>(tile + o);
            ar[r] = v.x;
            ai[r] = v.y;
            ar[r + 1] = v.z;
            ai[r + 1] = v.w;
          }
        } else {
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            uint32_t o = sq;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (r & (1 << k)) o ^= W.s_reg[k];
            const T v = tile[o];
            ar[r] = v.x;
            ai[r] = v.y;
          }
        }
        // converted once here, not again for every word
#pragma unroll
        for (int r = 0; r < 16; ++r) asm volatile("" : "+d"(ar[r]), "+d"(ai[r]));
        // single X letters (a transverse field) without the switch below
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t w = W.one[k];
          if (w == 0xffu) continue;
          double s[4];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = ((j >> k) << (k + 1)) | (j & ((1 << k) - 1)), r1 = r | (1 << k);
            if (j < 2) {
              s[j] = ar[r] * ar[r1];
              s[2 + j] = ai[r] * ai[r1];
            } else {
              s[j & 1] = fma(ar[r], ar[r1], s[j & 1]);
              s[2 + (j & 1)] = fma(ai[r], ai[r1], s[2 + (j & 1)]);
            }
          }
          acc[w * NT + tid] += (s[0] + s[1]) + (s[2] + s[3]);
        }
        for (int w = W.w0; w < W.w1; ++w) {
          const PauliTileWord& D = P.word[w];
          double s;
          switch (D.x) {
#define MQ_PAULI_CASE(X) case X: s = pair_sum<X>(ar, ai, D.sgn, D.imag); break;
            MQ_PAULI_CASE(1) MQ_PAULI_CASE(2) MQ_PAULI_CASE(3) MQ_PAULI_CASE(4) MQ_PAULI_CASE(5) MQ_PAULI_CASE(6)
            MQ_PAULI_CASE(7) MQ_PAULI_CASE(8) MQ_PAULI_CASE(9) MQ_PAULI_CASE(10) MQ_PAULI_CASE(11)
            MQ_PAULI_CASE(12) MQ_PAULI_CASE(13) MQ_PAULI_CASE(14)
            default: s = pair_sum<15>(ar, ai, D.sgn, D.imag); break;
#undef MQ_PAULI_CASE
          }
          acc[w * NT + tid] += (__popc(gq & D.z) & 1) ? -s : s;
        }
      }
    }
  }
  // the words' sums over the block: a fixed halving tree
  for (int s = NT / 2; s > 0; s >>= 1) {
    __syncthreads();
    for (int j = (int)tid; j < P.n_words * s; j += NT) {
      const int w = j / s, i = j % s;
      acc[w * NT + i] = __dadd_rn(acc[w * NT + i], acc[w * NT + i + s]);
    }
  }
  __syncthreads();
  if ((int)tid < P.n_words) part[(size_t)tid * gridDim.x + blockIdx.x] = acc[tid * NT];
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

// ================================================================ host side
static uint32_t grid_for(uint64_t threads, int bs) { return (uint32_t)std::max<uint64_t>(1, (threads + bs - 1) / bs); }

template <int S>
static void launch_chunks(mq_state* h, const ChunkParams& P, double* D) {
  const int wb = std::max<int>(P.cb, 5);
  const uint64_t units = P.nb > wb + S ? uint64_t(1) << (P.nb - wb - S) : 1;
  const uint32_t grid = (uint32_t)std::min<uint64_t>((units + 7) / 8, (uint64_t)h->num_sms * 8);
  if (h->dtype == MQ_C64) k_chunk_sums<float, S><<<grid, 256, 0, h->stream>>>((const float2*)h->cur_buf(), P, D);
  else k_chunk_sums<double, S><<<grid, 256, 0, h->stream>>>((const double2*)h->cur_buf(), P, D);
}

static int launch_seq(mq_state* h, const double* in, uint32_t group_len, uint32_t run_len, uint32_t runs_per_group,
                      uint32_t n_runs, double* out) {
  if (std::min(run_len, group_len) > 16)  // a run ends with its group
    k_seq_sums_warp<<<grid_for(n_runs, kSeqWarps), 32 * kSeqWarps, 0, h->stream>>>(in, group_len, run_len,
                                                                                   runs_per_group, n_runs, out);
  else
    k_seq_sums<<<grid_for(n_runs, 128), 128, 0, h->stream>>>(in, group_len, run_len, runs_per_group, n_runs, out);
  MQ_LAUNCHED("k_seq_sums");
  h->launches += 1;
  return MQ_OK;
}

// Deterministic marginal over `wires` (k < n or permuted order) into device
// memory: *q = the 2^k values, somewhere in work[0 .. 2 nc + 2^k).
static int marginal_device(mq_state* h, const int32_t* wires, int k, double* work, double** q) {
  const int n = h->n;
  ChunkParams P;
  std::memset(&P, 0, sizeof(P));
  std::vector<bool> sel(n, false);
  for (int t = 0; t < k; ++t) sel[n - 1 - wires[t]] = true;
  int t = 0;
  for (int b = 0; b < n; ++b)
    if (!sel[b]) P.img[t++] = 1u << b;  // remaining bits ascending = low j bits
  for (int s = k - 1; s >= 0; --s) P.img[t++] = 1u << (n - 1 - wires[s]);  // first wire = MSB of bucket
  const uint64_t bucket_len = uint64_t(1) << (n - k);
  const uint32_t cs = (uint32_t)std::min<uint64_t>(kBlock, bucket_len);
  const uint32_t nc = (uint32_t)((uint64_t(1) << n) / cs);
  const uint32_t ncb = (uint32_t)(bucket_len / cs);      // chunks per bucket
  const uint32_t nsb = (ncb + kSuper - 1) / kSuper;       // super-chunks per bucket
  const uint32_t nbk = 1u << k;
  P.nb = (uint8_t)n;
  while ((1u << P.cb) < cs) ++P.cb;
  // siblings: selected qubits on index bits 0-3, outside the bits of a warp
  int S = 0;
  for (int j = std::max<int>(P.cb, 5); j < n && S < 4; ++j)
    if (j >= n - k && P.img[j] < 16u) P.spos[S++] = (uint8_t)j;
  double* D = work;
  double* Pp = work + nc;
  double* out = Pp + nc;
  switch (S) {
    case 0: launch_chunks<0>(h, P, D); break;
    case 1: launch_chunks<1>(h, P, D); break;
    case 2: launch_chunks<2>(h, P, D); break;
    case 3: launch_chunks<3>(h, P, D); break;
    default: launch_chunks<4>(h, P, D); break;
  }
  MQ_LAUNCHED("k_chunk_sums");
  h->launches += 1;
  h->sweeps += 1;
  // a level of one entry per run is the entry itself (0 + x = x)
  int rc = MQ_OK;
  if (ncb > 1) {
    rc = launch_seq(h, D, ncb, kSuper, nsb, nbk * nsb, Pp);
    D = Pp;
  }
  if (!rc && nsb > 1) {
    rc = launch_seq(h, D, nsb, nsb, 1, nbk, out);
    D = out;
  }
  *q = D;
  return rc;
}

static bool natural_order(int n, const int32_t* wires, int k) {
  if (!wires || k < 0) return true;
  if (k != n) return false;
  for (int i = 0; i < n; ++i)
    if (wires[i] != i) return false;
  return true;
}

static int check_wires(int n, const int32_t* wires, int k) {
  if (!wires || k < 0) return MQ_OK;
  if (k > n) return fail(MQ_EINVAL, "more wires than qubits");
  std::vector<bool> seen(n, false);
  for (int i = 0; i < k; ++i) {
    if (wires[i] < 0 || wires[i] >= n) return fail(MQ_EINVAL, "Qubit index out of range");
    if (seen[wires[i]]) return fail(MQ_EINVAL, "Duplicate qubit indices");
    seen[wires[i]] = true;
  }
  return MQ_OK;
}

// |a|^2 of every amplitude, natural order, into out (device memory of the
// handle's device), asynchronously on the handle's stream.
int run_probabilities_device(mq_state* h, int out_dtype, void* out) {
  const uint32_t dim = (uint32_t)h->dim();
  const uint32_t grid = (uint32_t)std::min<uint64_t>((dim + 255) / 256, (uint64_t)h->num_sms * 16);
  if (h->dtype == MQ_C64) {
    if (out_dtype == 0) k_amp2_out<float, float><<<grid, 256, 0, h->stream>>>((const float2*)h->cur_buf(), (float*)out, dim);
    else k_amp2_out<float, double><<<grid, 256, 0, h->stream>>>((const float2*)h->cur_buf(), (double*)out, dim);
  } else {
    if (out_dtype == 0) k_amp2_out<double, float><<<grid, 256, 0, h->stream>>>((const double2*)h->cur_buf(), (float*)out, dim);
    else k_amp2_out<double, double><<<grid, 256, 0, h->stream>>>((const double2*)h->cur_buf(), (double*)out, dim);
  }
  MQ_LAUNCHED("k_amp2_out");
  h->launches += 1;
  h->sweeps += 1;
  return MQ_OK;
}

int run_probabilities(mq_state* h, const int32_t* wires, int k, int out_dtype, void* out) {
  int rc = check_wires(h->n, wires, k);
  if (rc) return rc;
  const int n = h->n;
  if (natural_order(n, wires, k)) {
    rc = ensure_alt(h);
    if (rc) return rc;
    const uint32_t dim = (uint32_t)h->dim();
    void* stage = h->buf[1 - h->cur];
    const uint32_t grid = (uint32_t)std::min<uint64_t>((dim + 255) / 256, (uint64_t)h->num_sms * 16);
    if (h->dtype == MQ_C64) {
      if (out_dtype == 0) k_amp2_out<float, float><<<grid, 256, 0, h->stream>>>((const float2*)h->cur_buf(), (float*)stage, dim);
      else k_amp2_out<float, double><<<grid, 256, 0, h->stream>>>((const float2*)h->cur_buf(), (double*)stage, dim);
    } else {
      if (out_dtype == 0) k_amp2_out<double, float><<<grid, 256, 0, h->stream>>>((const double2*)h->cur_buf(), (float*)stage, dim);
      else k_amp2_out<double, double><<<grid, 256, 0, h->stream>>>((const double2*)h->cur_buf(), (double*)stage, dim);
    }
    MQ_LAUNCHED("k_amp2_out");
    h->launches += 1;
    h->sweeps += 1;
    MQ_CUDA(cudaMemcpyAsync(out, stage, (size_t)dim * (out_dtype == 0 ? 4 : 8), cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
    return MQ_OK;
  }
  const uint64_t nc = (uint64_t(1) << n) / std::min<uint64_t>(kBlock, uint64_t(1) << (n - k));
  const size_t nbk = size_t(1) << k;
  const size_t need = (nc + nc + nbk) * 8 + 256;
  rc = ensure_scratch(h, need);
  if (rc) return rc;
  double* q = nullptr;
  rc = marginal_device(h, wires, k, (double*)h->scratch, &q);
  if (rc) return rc;
  if (out_dtype == 1) {
    MQ_CUDA(cudaMemcpyAsync(out, q, nbk * 8, cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
  } else {
    std::vector<double> tmp(nbk);
    MQ_CUDA(cudaMemcpyAsync(tmp.data(), q, nbk * 8, cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
    for (size_t i = 0; i < nbk; ++i) ((float*)out)[i] = (float)tmp[i];
  }
  return MQ_OK;
}

// Up to this many shots the call waits for the GPU once, and the shots pass
// through host memory of its own; above, copying them twice takes longer than
// the second wait.
constexpr int64_t kStagedShots = 8192;

template <typename Src>
static int sample_from(mq_state* h, Src src, uint32_t m, uint64_t seed, uint64_t offset, int64_t shots,
                       int64_t* out, double* work) {
  const uint32_t bs = std::min<uint32_t>(kBlock, m);
  const uint32_t nb = m / bs;
  const uint32_t ng = (nb + kSuper - 1) / kSuper;
  double* S = work;
  double* L = S + nb;
  double* T = L + nb;
  double* E = T + ng;
  int32_t* LP = (int32_t*)(E + ng);
  SampleMeta* meta = (SampleMeta*)(((uintptr_t)(LP + ng) + 15) & ~(uintptr_t)15);
  int64_t* dout = (int64_t*)(meta + 1);
  k_block_sums<Src><<<grid_for((uint64_t)nb * 32, 256), 256, 0, h->stream>>>(src, bs, nb, S);
  MQ_LAUNCHED("k_block_sums");
  k_local_prefix<<<ng, kPrefixThreads, 0, h->stream>>>(S, nb, L, T, LP);
  MQ_LAUNCHED("k_local_prefix");
  k_super_prefix<<<1, kPrefixThreads, 0, h->stream>>>(T, LP, ng, E, meta);
  MQ_LAUNCHED("k_super_prefix");
  SampleMeta hm;
  auto total = [&]() -> int {  // a state without probability is refused before any shot is handed out
    if (!(hm.total > 0.0)) return fail(MQ_EINVAL, "Simulator returned a zero-probability state");
    return MQ_OK;
  };
  if (shots <= kStagedShots) {
    // the total and the shots, which follow it, come back in one copy
    if (shots > 0) {
      k_draw<Src><<<grid_for((uint64_t)shots, kDrawWarps), 32 * kDrawWarps, 0, h->stream>>>(
          src, bs, nb, L, E, meta, seed, offset, shots, dout);
      MQ_LAUNCHED("k_draw");
    }
    const size_t bytes = sizeof(SampleMeta) + (size_t)shots * 8;
    std::unique_ptr<char[]> host(new char[bytes]);
    MQ_CUDA(cudaMemcpyAsync(host.get(), meta, bytes, cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
    std::memcpy(&hm, host.get(), sizeof(hm));
    int rc = total();
    if (rc) return rc;
    if (shots > 0) std::memcpy(out, host.get() + sizeof(SampleMeta), (size_t)shots * 8);
  } else {
    MQ_CUDA(cudaMemcpyAsync(&hm, meta, sizeof(hm), cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
    int rc = total();
    if (rc) return rc;
    if (shots < kThreadShots)
      k_draw<Src><<<grid_for((uint64_t)shots, kDrawWarps), 32 * kDrawWarps, 0, h->stream>>>(
          src, bs, nb, L, E, meta, seed, offset, shots, dout);
    else
      k_draw_threads<Src><<<grid_for((uint64_t)shots, 128), 128, 0, h->stream>>>(src, bs, nb, L, E, meta, seed, offset,
                                                                                 shots, dout);
    MQ_LAUNCHED("k_draw");
    MQ_CUDA(cudaMemcpyAsync(out, dout, (size_t)shots * 8, cudaMemcpyDeviceToHost, h->stream));
    MQ_CUDA(cudaStreamSynchronize(h->stream));
  }
  h->launches += 4;
  h->sweeps += 1;
  return MQ_OK;
}

static size_t sample_work_bytes(uint32_t m, int64_t shots) {
  const uint32_t bs = std::min<uint32_t>(kBlock, m);
  const uint32_t nb = m / bs;
  const uint32_t ng = (nb + kSuper - 1) / kSuper;
  return (size_t)(2 * nb + 2 * ng) * 8 + (size_t)ng * 4 + 64 + (size_t)std::max<int64_t>(shots, 1) * 8 + 64;
}

int run_sample(mq_state* h, const int32_t* wires, int k, uint64_t seed, uint64_t offset, int64_t shots, int64_t* out) {
  int rc = check_wires(h->n, wires, k);
  if (rc) return rc;
  if (shots < 0) return fail(MQ_EINVAL, "shots must be non-negative");
  const int n = h->n;
  if (natural_order(n, wires, k)) {
    const uint32_t m = (uint32_t)h->dim();
    rc = ensure_scratch(h, sample_work_bytes(m, shots));
    if (rc) return rc;
    if (h->dtype == MQ_C64) return sample_from(h, StateSrc<float>{(const float2*)h->cur_buf()}, m, seed, offset, shots, out, (double*)h->scratch);
    return sample_from(h, StateSrc<double>{(const double2*)h->cur_buf()}, m, seed, offset, shots, out, (double*)h->scratch);
  }
  if (k == 0) {
    for (int64_t s = 0; s < shots; ++s) out[s] = 0;
    return MQ_OK;
  }
  const uint64_t nc = (uint64_t(1) << n) / std::min<uint64_t>(kBlock, uint64_t(1) << (n - k));
  const size_t nbk = size_t(1) << k;
  const size_t marg = (nc + nc + nbk) * 8 + 256;
  rc = ensure_scratch(h, marg + sample_work_bytes((uint32_t)nbk, shots) + 64);
  if (rc) return rc;
  double* q = nullptr;
  rc = marginal_device(h, wires, k, (double*)h->scratch, &q);
  if (rc) return rc;
  double* swork = (double*)((((uintptr_t)h->scratch + marg) + 63) & ~(uintptr_t)63);
  return sample_from(h, VecSrc{q}, (uint32_t)nbk, seed, offset, shots, out, swork);
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
      const size_t smem = (h->amp_bytes() << M) + sizeof(double) * idx.size() * (1u << kPauliLT);
      if (c64) {
        MQ_CUDA(cudaFuncSetAttribute(k_pauli_tile<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPauliSmem));
        k_pauli_tile<float><<<grid, 1 << kPauliLT, smem, h->stream>>>((const float2*)h->cur_buf(), P, part);
      } else {
        MQ_CUDA(cudaFuncSetAttribute(k_pauli_tile<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPauliSmem));
        k_pauli_tile<double><<<grid, 1 << kPauliLT, smem, h->stream>>>((const double2*)h->cur_buf(), P, part);
      }
      MQ_LAUNCHED("k_pauli_tile");
      int rc = finish(grid, idx);
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
