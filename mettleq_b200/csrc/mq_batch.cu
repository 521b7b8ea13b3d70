// Batched circuits (the batching direction): many independent circuits of
// uneven width in one CUDA-graph launch.
//
// The reference runs a batch as a Python loop, one circuit and one launch
// sequence at a time (integrations/qiskit.py:505-514).  Here a batch of
// layered circuits (per layer: a 2x2 on every qubit, optionally followed by
// the CNOT ladder 0->1->...->n-1) is planned once and captured as one graph:
//
//   * circuits of at most kSmallMax qubits run whole inside shared memory:
//     k_batch_small is a persistent kernel whose CTAs take circuits from an
//     atomic counter, start from |0...0>, apply every layer in place (the
//     ladder is a gather between two shared buffers) and write the
//     probabilities and <Z_0>; nothing but the outputs touches HBM;
//   * larger circuits run in groups of one width (k_group_sweep), one launch
//     per layer and sweep for the whole group, on parallel lanes (one stream
//     each, the lanes are parallel branches of the graph).  With a tile plan of
//     mq_batch_set_tiles they run one by one through the general tile sweeps.
//
// Gate matrices live in device memory (read by the kernels when they run),
// so one captured graph serves every later parameter set: a run is one
// host-to-device copy of the matrices and one graph launch.
#include <algorithm>
#include <cstring>
#include <exception>
#include <map>
#include <new>
#include <numeric>
#include <vector>

#include "mq_internal.cuh"

namespace mq {

constexpr int kSmallMax = 13;  // 2 x 2^13 complex64 = 128 KiB of shared memory

struct SmallCircuit {
  uint32_t n, depth, ladder, index;
  uint64_t mats_off;   // doubles: depth * n * 8, layer-major, qubit-major
  uint64_t probs_off;  // floats
};

__device__ __forceinline__ uint32_t bslot(uint32_t i) { return i ^ ((i >> 3) & 0xEu); }

// u0 x0 + u1 x1 on the paired FP32 instructions, the entries given as
// (u.x, u.x, -u.y, u.y).  Both components take the rounding steps of
//   fma(u0.x, x0.x, fma(-u0.y, x0.y, fma(u1.x, x1.x, -u1.y x1.y)))
//   fma(u0.x, x0.y, fma(u0.y, x0.x, fma(u1.x, x1.y, u1.y x1.x))).
__device__ __forceinline__ float2 cmac2p(float4 u0, float2 x0, float4 u1, float2 x1) {
  const float2 s0 = make_float2(x0.y, x0.x), s1 = make_float2(x1.y, x1.x);
  return __ffma2_rn(x0, make_float2(u0.x, u0.y),
                    __ffma2_rn(s0, make_float2(u0.z, u0.w),
                               __ffma2_rn(x1, make_float2(u1.x, u1.y), __fmul2_rn(s1, make_float2(u1.z, u1.w)))));
}

template <int NT>
__global__ void __launch_bounds__(NT) k_batch_small(const SmallCircuit* __restrict__ circ, uint32_t n_circ,
                                                    const double* __restrict__ mats, float* __restrict__ probs,
                                                    double* __restrict__ z0, uint32_t* __restrict__ next,
                                                    uint32_t half) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ float4 um[kSmallMax][4];  // an entry u as (u.x, u.x, -u.y, u.y)
  __shared__ uint32_t cid;
  __shared__ double zred[NT / 32];
  const int tid = threadIdx.x;
  for (;;) {
    __syncthreads();
    if (tid == 0) cid = atomicAdd(next, 1u);
    __syncthreads();
    const uint32_t c = cid;
    if (c >= n_circ) break;
    const SmallCircuit C = circ[c];
    const int n = (int)C.n;
    const uint32_t E = 1u << n;
    float2* a = sm;
    float2* b = sm + half;
    for (uint32_t i = tid; i < E; i += NT) a[bslot(i)] = make_float2(i == 0 ? 1.f : 0.f, 0.f);
    for (uint32_t l = 0; l < C.depth; ++l) {
      __syncthreads();
      for (int j = tid; j < n * 4; j += NT) {
        const double* m = mats + C.mats_off + ((size_t)l * n * 4 + j) * 2;
        const float x = (float)m[0], y = (float)m[1];
        um[j >> 2][j & 3] = make_float4(x, x, -y, y);
      }
      __syncthreads();
      // 2x2 on every qubit, four index bits per register pass; the last pass
      // is shifted down to [n-4, n) and skips the bits already done
      for (int g0 = 0; g0 < n; g0 += 4) {
        const int lo = n >= 4 ? min(g0, n - 4) : 0;
        const int nb = n >= 4 ? 4 : n;
        const uint32_t groups = E >> nb;
        for (uint32_t gi = tid; gi < groups; gi += NT) {
          const uint32_t base = ((gi >> lo) << (lo + nb)) | (gi & ((1u << lo) - 1u));
          float2 v[16];
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (r < (1 << nb)) v[r] = a[bslot(base | ((uint32_t)r << lo))];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int bit = lo + k;
            if (k >= nb || bit < g0) continue;
            const int q = n - 1 - bit;
            const float4 u[4] = {um[q][0], um[q][1], um[q][2], um[q][3]};
#pragma unroll
            for (int r = 0; r < 16; ++r) {
              if ((r & (1 << k)) || r >= (1 << nb)) continue;
              const float2 x0 = v[r], x1 = v[r | (1 << k)];
              v[r] = cmac2p(u[0], x0, u[1], x1);
              v[r | (1 << k)] = cmac2p(u[2], x0, u[3], x1);
            }
          }
#pragma unroll
          for (int r = 0; r < 16; ++r)
            if (r < (1 << nb)) a[bslot(base | ((uint32_t)r << lo))] = v[r];
        }
        __syncthreads();
      }
      if (C.ladder) {
        // CNOT(0,1), ..., CNOT(n-2,n-1): out[y] = in[y ^ (y >> 1)]
        for (uint32_t y = tid; y < E; y += NT) b[bslot(y)] = a[bslot(y ^ (y >> 1))];
        __syncthreads();
        float2* t = a;
        a = b;
        b = t;
      }
    }
    double zacc = 0.0;
    for (uint32_t i = tid; i < E; i += NT) {
      const float2 v = a[bslot(i)];
      const double p = (double)v.x * v.x + (double)v.y * v.y;
      probs[C.probs_off + i] = (float)p;
      zacc += ((i >> (n - 1)) & 1u) ? -p : p;
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) zacc += __shfl_xor_sync(0xffffffffu, zacc, off);
    if ((tid & 31) == 0) zred[tid >> 5] = zacc;
    __syncthreads();
    if (tid == 0) {
      double z = 0.0;
      for (int w = 0; w < NT / 32; ++w) z += zred[w];
      z0[C.index] = z;
    }
  }
}

// ------------------------------------------------- groups of larger circuits
// Circuits of one width (and ladder choice) run together, sorted by depth:
// their states lie one after the other, and a layer of all circuits that are
// still that deep is one launch per sweep.  A sweep of one 14- to 20-qubit
// circuit fills a fraction of the GPU for about 10 us, and a graph of one such
// node per circuit, layer and sweep is bound by its nodes: 256 circuits of 10
// to 20 qubits, 9.0 ms with 3400 sweeps of single circuits, 4.3 ms this way (20
// qubits, 32 circuits: 5.2 -> 3.2 ms; 14 and 15 qubits, 100 circuits: 1.54 -> 0.42).
// What bounds a sweep now is the complex 2x2 arithmetic and its latency (24 warps
// an SM).  The gates of an amplitude are applied in the order and with the
// rounding of the single circuits' sweeps (fill_order): the states are the same
// bits.
struct GroupCirc {
  uint64_t mats_off;   // doubles: the circuit's matrices, layer-major
  uint64_t probs_off;  // floats
  uint32_t index, depth;
};

struct GroupSweep {
  const float2* src;
  float2* dst;
  const GroupCirc* circ;
  const double* mats;
  uint32_t layer;
  uint32_t n_tiles;    // circuits << (n - 12)
  uint8_t n, start, cnt;  // target bits [start, start + cnt)
  uint8_t ladder;      // low sweep: CNOT ladder at the write-back
};

// Tile-local index of register pattern r of the thread's group, register bits
// [4P, 4P + 4).
template <int P>
__device__ __forceinline__ uint32_t nib_index(uint32_t tid, uint32_t r) {
  if constexpr (P == 0) return (tid << 4) | r;
  else if constexpr (P == 1) return (tid & 15u) | (r << 4) | ((tid >> 4) << 8);
  else return tid | (r << 8);
}

constexpr int kSweepThreads = 256;
// 80 registers a thread; 256 circuits of 10 to 20 qubits: 4.25 ms a run, 4.47
// with 2 CTAs (the two tile buffers leave no room for 4)
constexpr int kSweepCtas = 3;

constexpr size_t kSweepSmem = 2 * 4096 * sizeof(float2);

// One phase: 16 amplitudes differing in tile bits [4P, 4P + 4), the gates of
// the first `cnt` of these bits in ascending order.  (Scalar FP32 instructions
// instead of cmac2p: 5.19 against 4.98 ms a batch run.)
template <int P>
__device__ __forceinline__ void group_gates(const float2* tile, uint32_t tid, int cnt, const float4 (*um)[4], float2 (&a)[16]) {
  if constexpr (P == 0) {
#pragma unroll
    for (int r = 0; r < 16; r += 2) {
      const float4 v = *reinterpret_cast<const float4*>(tile + bslot(nib_index<P>(tid, r)));
      a[r] = make_float2(v.x, v.y);
      a[r + 1] = make_float2(v.z, v.w);
    }
  } else {
#pragma unroll
    for (int r = 0; r < 16; ++r) a[r] = tile[bslot(nib_index<P>(tid, r))];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= cnt) break;
    const float4 u[4] = {um[k][0], um[k][1], um[k][2], um[k][3]};
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      if (r & (1 << k)) continue;
      const float2 x0 = a[r], x1 = a[r | (1 << k)];
      a[r] = cmac2p(u[0], x0, u[1], x1);
      a[r | (1 << k)] = cmac2p(u[2], x0, u[3], x1);
    }
  }
}
template <int P>
__device__ __forceinline__ void group_phase(float2* tile, uint32_t tid, int cnt, const float4 (*um)[4]) {
  float2 a[16];
  group_gates<P>(tile, tid, cnt, um, a);
  if constexpr (P == 0) {
#pragma unroll
    for (int r = 0; r < 16; r += 2)
      *reinterpret_cast<float4*>(tile + bslot(nib_index<P>(tid, r))) =
          make_float4(a[r].x, a[r].y, a[r + 1].x, a[r + 1].y);
  } else {
#pragma unroll
    for (int r = 0; r < 16; ++r) tile[bslot(nib_index<P>(tid, r))] = a[r];
  }
}

// A sweep of one layer over a group: tiles of 2^12 amplitudes, register phases
// on the tile's nibbles, from the top target bits down.  LOW: the tile is the
// index bits [0, 12), targets [0, cnt), the ladder out[y] = in[y ^ (y >> 1)] at
// the write-back (an output tile reads one input tile).  Else cnt <= 8 high
// targets in tile bits [4, 4 + cnt) over the passengers 0-3; the tile's
// remaining bits are the index bits from 4 up, so a run is 2^(12 - cnt)
// amplitudes.  In place unless the ladder permutes.  The next tile and its
// matrices are loaded while this one is worked on: 24 warps an SM did not cover
// the wait (4.69 -> 4.56 ms a batch run).
template <bool LOW>
__global__ void __launch_bounds__(kSweepThreads, kSweepCtas) k_group_sweep(const __grid_constant__ GroupSweep P) {
  extern __shared__ __align__(16) float2 tiles[];  // two buffers of 4096
  __shared__ float4 um[2][12][4];                  // by buffer, tile bit
  __shared__ double2 raw[48];                      // the next tile's matrices as they are in memory
  uint32_t tid = threadIdx.x;
  const int n = P.n, cnt = P.cnt, pas = 12 - cnt;
  // consecutive chunks of a tile are consecutive in memory: chunk order over
  // (passengers, targets), tile-local order (passengers 0-3, targets, other
  // passengers)
  auto local_of = [&](uint32_t i) -> uint32_t {
    if constexpr (LOW) return i;
    const uint32_t low = i & 15u, mid = (i >> 4) & ((1u << (pas - 4)) - 1u), tg = i >> pas;
    return low | (tg << 4) | (mid << (4 + cnt));
  };
  auto offset_of = [&](uint32_t i) -> uint32_t {
    if constexpr (LOW) return i;
    else return (i & ((1u << pas) - 1u)) | ((i >> pas) << P.start);
  };
  // high sweeps: offset of a tile-local index (bits 4 and up)
  auto place = [&](uint32_t l) -> uint32_t {
    return (((l >> 4) & ((1u << cnt) - 1u)) << P.start) | ((l >> (4 + cnt)) << 4);
  };
  auto base_of = [&](uint32_t h) -> uint32_t {  // of the input tile
    if constexpr (LOW) {
      return (P.ladder ? h ^ (h >> 1) : h) << 12;
    } else {
      const int run = P.start - pas;  // free bits between the passengers and the targets
      return ((h & ((1u << run) - 1u)) << pas) | ((h >> run) << (P.start + cnt));
    }
  };
  auto load = [&](uint32_t t, float2* tile) {
    const float2* src = P.src + ((size_t)(t >> (n - 12)) << n) + base_of(t & ((1u << (n - 12)) - 1u));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t i = 2 * tid + 512 * k;
      cp_async<16>(smem_u32(tile + bslot(local_of(i))), src + offset_of(i));
    }
    if ((int)tid < 4 * cnt) {
      const double* m = P.mats + P.circ[t >> (n - 12)].mats_off + ((size_t)P.layer * n + (n - 1 - (P.start + (tid >> 2)))) * 8;
      cp_async<16>(smem_u32(raw + tid), m + 2 * (tid & 3u));
    }
    cp_async_commit();
  };
  auto arrive = [&](int buf) {  // a thread converts the entry it has loaded itself
    cp_async_wait<0>();
    if ((int)tid < 4 * cnt) {
      const float x = (float)raw[tid].x, y = (float)raw[tid].y;
      um[buf][(LOW ? 0 : 4) + (tid >> 2)][tid & 3u] = make_float4(x, x, -y, y);
    }
  };
  int buf = 0;
  if (blockIdx.x < P.n_tiles) {
    load(blockIdx.x, tiles);
    arrive(0);
  }
  for (uint32_t t = blockIdx.x; t < P.n_tiles; t += gridDim.x, buf ^= 1) {
    // keeps the per-chunk addresses from being held (spilled) across tiles
    asm volatile("" : "+r"(tid));
    float2* tile = tiles + 4096 * buf;
    __syncthreads();  // the tile and its matrices are here, the previous tile has left
    const uint32_t next = t + gridDim.x;
    if (next < P.n_tiles) load(next, tiles + 4096 * (buf ^ 1));
    asm volatile("" : "+r"(tid));
    if constexpr (LOW) {
      if (cnt > 8) {
        group_phase<2>(tile, tid, cnt - 8, &um[buf][8]);
        __syncthreads();
      }
      if (cnt > 4) {
        group_phase<1>(tile, tid, min(cnt - 4, 4), &um[buf][4]);
        __syncwarp();
      }
      group_phase<0>(tile, tid, min(cnt, 4), &um[buf][0]);
    } else {
      if (cnt > 4) {
        group_phase<2>(tile, tid, cnt - 4, &um[buf][8]);
        __syncthreads();
      }
      // the last phase's 16 amplitudes go straight to memory: 16 lanes are the
      // passengers 0-3, so every run is a whole line (4.56 -> 4.42 ms a batch run)
      float2 a[16];
      group_gates<1>(tile, tid, min(cnt, 4), &um[buf][4], a);
      asm volatile("" : "+r"(tid));
      const uint32_t rest = (tid >> 4) << 8;  // tile bits 8-11
      float2* out = P.dst + ((size_t)(t >> (n - 12)) << n) + base_of(t & ((1u << (n - 12)) - 1u)) + place(rest) + (tid & 15u);
      uint32_t step[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) step[k] = place(16u << k);
#pragma unroll
      for (int r = 0; r < 16; ++r)
        out[((r & 1) ? step[0] : 0u) + ((r & 2) ? step[1] : 0u) + ((r & 4) ? step[2] : 0u) + ((r & 8) ? step[3] : 0u)] = a[r];
    }
    if constexpr (LOW) {
      // phases 1 and 0 and the ladder keep tile bits 9-11 apart (the ladder
      // maps each value to one), so a warp reads only what it wrote: two
      // block barriers less, 4.42 -> 4.32 ms a batch run
      __syncwarp();
      asm volatile("" : "+r"(tid));
      const uint32_t h = t & ((1u << (n - 12)) - 1u);
      uint32_t block = tid >> 5;
      if (P.ladder) {
        block ^= (h & 1u) << 2;
        block ^= block >> 1;
        block ^= block >> 2;
      }
      float2* out = P.dst + ((size_t)(t >> (n - 12)) << n) + (h << 12);
      const uint32_t cl = (h & 1u) << 11;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t i = (block << 9) + 2 * (tid & 31u) + 64 * k;
        uint32_t l = i;
        if (P.ladder) l = i ^ (i >> 1) ^ cl;
        const float4 v = *reinterpret_cast<const float4*>(tile + bslot(l & ~1u));
        *reinterpret_cast<float4*>(out + i) = (l & 1u) ? make_float4(v.z, v.w, v.x, v.y) : v;
      }
    }
    if (next < P.n_tiles) arrive(buf ^ 1);
  }
}

// The state after the first layer, written once instead of a cleared state and
// a layer of sweeps on it: from |0...0> every amplitude is the product of one
// entry of each qubit's first column, multiplied up in the order of the
// sweeps' gates (then the ladder).  Circuits without layers stay |0...0>.
struct GroupFirst {
  float2* dst;
  const GroupCirc* circ;
  const double* mats;
  uint32_t n_tiles;
  uint8_t n, ladder;
  uint8_t order[32];  // index bits in gate order; the last four are 0, 1, 2, 3
};
__global__ void __launch_bounds__(kSweepThreads) k_group_first(const __grid_constant__ GroupFirst P) {
  __shared__ float2 col[32][2];  // by gate order
  const uint32_t tid = threadIdx.x;
  const int n = P.n;
  // a gate on amplitudes (v, 0): the rounding of cmac2p with x1 = 0
  auto times = [](float2 u, float2 v) { return make_float2(fmaf(u.x, v.x, -u.y * v.y), fmaf(u.x, v.y, u.y * v.x)); };
  uint32_t have = 0xffffffffu;
  for (uint32_t t = blockIdx.x; t < P.n_tiles; t += gridDim.x) {
    const uint32_t cid = t >> (n - 12);
    const uint32_t h = t & ((1u << (n - 12)) - 1u);
    const uint32_t depth = P.circ[cid].depth;
    if (cid != have) {
      have = cid;
      __syncthreads();
      if ((int)tid < 2 * n) {
        const int j = tid >> 1, e = tid & 1;
        float2 v = make_float2(e ? 0.f : 1.f, 0.f);
        if (depth) {
          const double* m = P.mats + P.circ[cid].mats_off + (size_t)(n - 1 - P.order[j]) * 8 + 4 * e;
          v = make_float2((float)m[0], (float)m[1]);
        }
        col[j][e] = v;
      }
      __syncthreads();
    }
    const bool lad = P.ladder && depth;
    float2* out = P.dst + ((size_t)cid << n);
    // 16 amplitudes of the product, consecutive before the ladder: the ladder
    // maps them to 16 of one 16-aligned run of outputs
    const uint32_t x0 = ((lad ? h ^ (h >> 1) : h) << 12) | (tid << 4);
    // (the low 12 bits are enumerated over all threads, so the tile's set of
    // inputs is the set its outputs read)
    float2 v[16];
    v[0] = make_float2(1.f, 0.f);
    for (int j = 0; j < n - 4; ++j) v[0] = times(col[j][(x0 >> P.order[j]) & 1u], v[0]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 c0 = col[n - 4 + k][0], c1 = col[n - 4 + k][1];
#pragma unroll
      for (int r = 0; r < (1 << k); ++r) {
        v[r | (1 << k)] = times(c1, v[r]);
        v[r] = times(c0, v[r]);
      }
    }
    // output index of input x: y ^ (y >> 1) = x, the prefix XOR from the top;
    // the low 12 bits start from the parity of the bits above
    uint32_t y0 = x0 & 4095u;
    if (lad) {
      y0 ^= y0 >> 1;
      y0 ^= y0 >> 2;
      y0 ^= y0 >> 4;
      y0 ^= y0 >> 8;
      y0 &= 4095u;
      if (h & 1u) y0 ^= 4095u;  // y's bit 12 is h's bit 0
    }
    const uint32_t at = (h << 12) | (y0 & ~15u);
    const uint32_t top = (y0 & 16u) ? 15u : 0u;  // y's bit 4 flips the prefix of the low four
#pragma unroll
    for (int r = 0; r < 16; r += 2) {
      // outputs (e, e + 1) of the run, e even, read inputs g(e), g(e) ^ 1
      const int g = r ^ (r >> 1);
      if (lad) {
        const uint32_t e = (uint32_t)r ^ top;  // output offset whose input pattern is g(r), or its partner
        const float2 p = v[g & 15], q = v[(g ^ 1) & 15];
        // e and e ^ 1 are one pair; e is odd when top is set
        *reinterpret_cast<float4*>(out + at + (e & ~1u)) =
            (e & 1u) ? make_float4(q.x, q.y, p.x, p.y) : make_float4(p.x, p.y, q.x, q.y);
      } else {
        *reinterpret_cast<float4*>(out + at + r) = make_float4(v[r].x, v[r].y, v[r + 1].x, v[r + 1].y);
      }
    }
  }
}

// Probabilities and per-block partial sums of <Z_0> of a group: `blocks`
// blocks per circuit; a circuit's state is in the buffer its number of
// permuted layers left it in.
struct GroupProbs {
  const float2* buf[2];
  const GroupCirc* circ;
  float* probs;
  double* zpart;
  uint32_t blocks;
  uint8_t n, ladder;
};
__global__ void __launch_bounds__(256) k_group_probs(const __grid_constant__ GroupProbs P) {
  __shared__ double red[8];
  const uint32_t cid = blockIdx.x / P.blocks, block = blockIdx.x % P.blocks;
  const GroupCirc C = P.circ[cid];
  const float2* st = P.buf[(P.ladder && C.depth > 1) ? ((C.depth - 1) & 1u) : 0u] + ((size_t)cid << P.n);
  float* probs = P.probs + C.probs_off;
  const uint32_t pairs = 1u << (P.n - 1);
  double acc = 0.0;
  for (uint32_t i = block * 256u + threadIdx.x; i < pairs; i += P.blocks * 256u) {
    const float4 v = reinterpret_cast<const float4*>(st)[i];
    const double p0 = (double)v.x * v.x + (double)v.y * v.y, p1 = (double)v.z * v.z + (double)v.w * v.w;
    probs[2 * i] = (float)p0;
    probs[2 * i + 1] = (float)p1;
    acc += ((i >> (P.n - 2)) & 1u) ? -(p0 + p1) : p0 + p1;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double z = 0.0;
    for (int w = 0; w < 8; ++w) z += red[w];
    P.zpart[blockIdx.x] = z;
  }
}
// <Z_0> of the group's circuits from their blocks' sums, a warp each
__global__ void k_group_z(const double* __restrict__ zpart, uint32_t blocks, const GroupCirc* __restrict__ circ,
                          uint32_t count, double* __restrict__ z0) {
  const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= count) return;
  const uint32_t lane = threadIdx.x & 31;
  double z = 0.0;
  for (uint32_t b = lane; b < blocks; b += 32) z += zpart[(size_t)c * blocks + b];
#pragma unroll
  for (int off = 16; off; off >>= 1) z += __shfl_xor_sync(0xffffffffu, z, off);
  if (lane == 0) z0[circ[c].index] = z;
}

// probabilities of a full state and per-block partial sums of <Z_0>
__global__ void __launch_bounds__(256) k_probs_z(const float2* __restrict__ st, uint32_t dim, int n,
                                                 float* __restrict__ probs, double* __restrict__ zpart) {
  __shared__ double red[8];
  double acc = 0.0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += stride) {
    const float2 v = st[i];
    const double p = (double)v.x * v.x + (double)v.y * v.y;
    probs[i] = (float)p;
    acc += ((i >> (n - 1)) & 1u) ? -p : p;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double z = 0.0;
    for (int w = 0; w < 8; ++w) z += red[w];
    zpart[blockIdx.x] = z;
  }
}

__global__ void k_zsum(const double* __restrict__ zpart, uint32_t nb, double* __restrict__ out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double z = 0.0;
  for (uint32_t b = 0; b < nb; ++b) z += zpart[b];
  *out = z;
}

__global__ void k_basis0(float2* st) {
  if (threadIdx.x == 0 && blockIdx.x == 0) st[0] = make_float2(1.f, 0.f);
}

}  // namespace mq

using namespace mq;

struct mq_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int n_circ = 0;
  std::vector<int32_t> n, depth;
  std::vector<uint8_t> ladder;
  std::vector<uint64_t> mats_off, probs_off;
  uint64_t mats_total = 0, probs_total = 0;
  double* d_mats = nullptr;
  // small circuits
  std::vector<int> small;
  SmallCircuit* d_small = nullptr;
  uint32_t* d_next = nullptr;
  int small_threads = 256;
  // large circuits
  std::vector<int> large;
  int lanes = 1;
  std::vector<std::vector<int>> lane_work;  // single circuits (single_work)
  // groups of circuits of one width and ladder choice, deepest first
  struct Group {
    int n = 0;
    bool ladder = false;
    std::vector<int> circ;
    uint32_t first = 0;  // their GroupCirc entries start here
  };
  std::vector<Group> groups;
  std::vector<std::vector<int>> lane_groups;
  std::vector<size_t> lane_amps;  // amplitudes of a lane's largest group
  std::vector<float2*> lane_buf[2];
  GroupCirc* d_group = nullptr;
  std::vector<cudaStream_t> lane_stream;
  std::vector<cudaEvent_t> lane_event;
  cudaEvent_t fork_event = nullptr;
  std::vector<std::map<int, mq_state*>> lane_state;
  double* d_zpart = nullptr;
  uint32_t zblocks = 0;   // most blocks of one circuit
  size_t zslots = 0;      // partial sums of a lane
  int num_sms = 148;
  // sweep plan of the large circuits (mq_batch_set_tiles; 0 / -1 = defaults)
  int tile_max = 0, tile_pas = -1, tile_min = 0;
  cudaGraphExec_t exec = nullptr;
  float* graph_probs = nullptr;
  double* graph_z0 = nullptr;
};

namespace mq {

static void state_free(mq_state* h) {
  if (h->buf[0]) cudaFree(h->buf[0]);
  if (h->buf[1]) cudaFree(h->buf[1]);
  if (h->scratch) cudaFree(h->scratch);
  delete h;
}

static void batch_free(mq_batch* b) {
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  for (auto& m : b->lane_state)
    for (auto& kv : m) state_free(kv.second);
  for (auto s : b->lane_stream) cudaStreamDestroy(s);
  for (auto e : b->lane_event) cudaEventDestroy(e);
  if (b->fork_event) cudaEventDestroy(b->fork_event);
  if (b->d_mats) cudaFree(b->d_mats);
  if (b->d_small) cudaFree(b->d_small);
  if (b->d_next) cudaFree(b->d_next);
  if (b->d_zpart) cudaFree(b->d_zpart);
  for (auto& v : b->lane_buf)
    for (float2* p : v)
      if (p) cudaFree(p);
  if (b->d_group) cudaFree(b->d_group);
  if (b->own_stream && b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

// A lane's workspace state for n qubits (both buffers allocated up front:
// nothing may allocate while the graph is being captured).
static int make_lane_state(mq_batch* b, int lane, int n) {
  auto* h = new mq_state();
  h->n = n;
  h->dtype = MQ_C64;
  h->device = b->device;
  h->num_sms = b->num_sms;
  h->device_sms = b->num_sms;
  h->stream = b->lane_stream[lane];
  h->tile_max = b->tile_max;
  h->tile_pas = b->tile_pas;
  h->tile_min = b->tile_min;
  h->state_bytes = (size_t(1) << n) * 8;
  cudaError_t e = cudaMalloc(&h->buf[0], h->state_bytes);
  if (e == cudaSuccess) e = cudaMalloc(&h->buf[1], h->state_bytes);
  if (e != cudaSuccess) {
    state_free(h);
    return cuda_fail(e, "cudaMalloc(batch lane state)");
  }
  b->lane_state[lane][n] = h;
  return MQ_OK;
}

template <int NT>
static int launch_small(mq_batch* b, float* probs, double* z0, bool configure) {
  if (configure) {  // the limit is the kernel's, not the batch's: always the largest
    MQ_CUDA(cudaFuncSetAttribute(k_batch_small<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(2 * sizeof(float2) << kSmallMax)));
    return MQ_OK;
  }
  // two buffers of the widest circuit: a batch of up to 12 qubits has two and
  // more CTAs on an SM (200 circuits of 6 to 12 qubits: 85 -> 78 us, with cmac2p)
  int widest = 1;
  for (int c : b->small) widest = std::max(widest, (int)b->n[c]);
  const uint32_t half = 1u << widest;
  const size_t smem = 2 * sizeof(float2) * (size_t)half;
  int bps = 0;
  MQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_batch_small<NT>, NT, smem));
  const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(b->small.size(), (uint64_t)b->num_sms * std::max(1, bps)));
  k_batch_small<NT><<<grid, NT, smem, b->stream>>>(b->d_small, (uint32_t)b->small.size(), b->d_mats, probs, z0, b->d_next,
                                             half);
  MQ_LAUNCHED("k_batch_small");
  return MQ_OK;
}

static int small_dispatch(mq_batch* b, float* probs, double* z0, bool configure) {
  switch (b->small_threads) {
    case 128: return launch_small<128>(b, probs, z0, configure);
    case 512: return launch_small<512>(b, probs, z0, configure);
    default: return launch_small<256>(b, probs, z0, configure);
  }
}

// The large circuits of a lane one by one through the general sweeps, with the
// tile plan of mq_batch_set_tiles.
static int record_lane_single(mq_batch* b, int l, float* probs, double* z0) {
  uint32_t cols[32];
  cudaStream_t s = b->lane_stream[l];
  double* zpart = b->d_zpart + (size_t)l * b->zslots;
  for (int c : b->lane_work[l]) {
    const int n = b->n[c];
    mq_state* h = b->lane_state[l].at(n);
    h->cur = 0;
    MQ_CUDA(cudaMemsetAsync(h->buf[0], 0, h->state_bytes, s));
    k_basis0<<<1, 32, 0, s>>>(reinterpret_cast<float2*>(h->buf[0]));
    MQ_LAUNCHED("k_basis0");
    // CNOT ladder: columns A e_j of out[y] = in[A y], A e_j = e_j + e_{j-1}
    for (int j = 0; j < n; ++j) cols[j] = (1u << j) | (j ? (1u << (j - 1)) : 0u);
    for (int d = 0; d < b->depth[c]; ++d) {
      const double* md = b->d_mats + b->mats_off[c] + (size_t)d * n * 8;
      int rc = launch_layer(h, nullptr, nullptr, 0, nullptr, nullptr, nullptr, b->ladder[c] ? cols : nullptr, 0, md);
      if (rc) return rc;
    }
    const uint32_t dim = 1u << n;
    const uint32_t grid = std::min<uint32_t>(b->zblocks, std::max<uint32_t>(1, dim / 256));
    k_probs_z<<<grid, 256, 0, s>>>(reinterpret_cast<const float2*>(h->cur_buf()), dim, n, probs + b->probs_off[c], zpart);
    MQ_LAUNCHED("k_probs_z");
    k_zsum<<<1, 32, 0, s>>>(zpart, grid, z0 + c);
    MQ_LAUNCHED("k_zsum");
  }
  return MQ_OK;
}

// <Z_0> blocks of one circuit of a group: 16 pairs of amplitudes a thread,
// at most zblocks.
static uint32_t group_blocks(const mq_batch* b, int n) {
  return (uint32_t)std::min<uint64_t>(b->zblocks, std::max<uint64_t>(1, (uint64_t(1) << n) / 8192));
}

// Target bits (start, count) of a layer's sweeps on n qubits, the low sweep
// first in the list and last in the layer: the split of the general sweeps
// with 12-bit tiles and four passengers (mq_tile.cu split_bits).
static std::vector<std::pair<int, int>> group_split(int n) {
  const int n_hi = (n - 12 + 7) / 8;
  const int low = std::max(n - n_hi * 8, std::min(12, (n + n_hi) / (n_hi + 1)));
  std::vector<std::pair<int, int>> out = {{0, low}};
  int start = low;
  for (int i = 0; i < n_hi; ++i) {
    const int cnt = (n - low) / n_hi + (i < (n - low) % n_hi ? 1 : 0);
    out.push_back({start, cnt});
    start += cnt;
  }
  return out;
}
// The index bits in the order their gates are applied to an amplitude: the
// high sweeps, then the low one; in a sweep the remainder of its bits over
// four from the top, then nibbles downwards, each ascending.
static void fill_order(const std::vector<std::pair<int, int>>& split, uint8_t* order) {
  int k = 0;
  for (size_t i = 1; i <= split.size(); ++i) {
    const auto [start, cnt] = split[i % split.size()];
    for (int at = start + cnt; at > start;) {
      const int len = (at - start) % 4 ? (at - start) % 4 : 4;
      at -= len;
      for (int b = 0; b < len; ++b) order[k++] = (uint8_t)(at + b);
    }
  }
}

static int record_lane_groups(mq_batch* b, int l, float* probs, double* z0) {
  cudaStream_t s = b->lane_stream[l];
  double* zpart = b->d_zpart + (size_t)l * b->zslots;
  float2* buf[2] = {b->lane_buf[0][l], b->lane_buf[1][l]};
  for (int gi : b->lane_groups[l]) {
    const mq_batch::Group& G = b->groups[gi];
    const int n = G.n;
    const uint32_t count = (uint32_t)G.circ.size();
    auto grid = [&](uint32_t tiles) { return std::min<uint32_t>(tiles, (uint32_t)b->num_sms * kSweepCtas); };
    const auto split = group_split(n);
    GroupFirst F;
    std::memset(&F, 0, sizeof(F));
    F.dst = buf[0];
    F.circ = b->d_group + G.first;
    F.mats = b->d_mats;
    F.n_tiles = count << (n - 12);
    F.n = (uint8_t)n;
    F.ladder = G.ladder;
    fill_order(split, F.order);
    k_group_first<<<grid(F.n_tiles), kSweepThreads, 0, s>>>(F);
    MQ_LAUNCHED("k_group_first");
    int cur = 0;
    for (int d = 1; d < b->depth[G.circ[0]]; ++d) {
      uint32_t live = 0;
      while (live < count && b->depth[G.circ[live]] > d) ++live;
      GroupSweep P;
      std::memset(&P, 0, sizeof(P));
      P.circ = b->d_group + G.first;
      P.mats = b->d_mats;
      P.layer = (uint32_t)d;
      P.n_tiles = live << (n - 12);
      P.n = (uint8_t)n;
      P.ladder = G.ladder;
      P.src = P.dst = buf[cur];
      for (size_t g = 1; g < split.size(); ++g) {
        P.start = (uint8_t)split[g].first;
        P.cnt = (uint8_t)split[g].second;
        k_group_sweep<false><<<grid(P.n_tiles), kSweepThreads, kSweepSmem, s>>>(P);
        MQ_LAUNCHED("k_group_sweep");
      }
      if (G.ladder) cur ^= 1;
      P.dst = buf[cur];
      P.start = 0;
      P.cnt = (uint8_t)split[0].second;
      k_group_sweep<true><<<grid(P.n_tiles), kSweepThreads, kSweepSmem, s>>>(P);
      MQ_LAUNCHED("k_group_sweep");
    }
    GroupProbs Q;
    Q.buf[0] = buf[0];
    Q.buf[1] = buf[1];
    Q.circ = b->d_group + G.first;
    Q.probs = probs;
    Q.zpart = zpart;
    Q.blocks = group_blocks(b, n);
    Q.n = (uint8_t)n;
    Q.ladder = G.ladder;
    k_group_probs<<<count * Q.blocks, 256, 0, s>>>(Q);
    MQ_LAUNCHED("k_group_probs");
    k_group_z<<<(count + 3) / 4, 128, 0, s>>>(zpart, Q.blocks, Q.circ, count, z0);
    MQ_LAUNCHED("k_group_z");
  }
  return MQ_OK;
}

// A tile plan other than the default: every large circuit runs on its own.
static bool custom_tiles(int tile_max, int tile_pas, int tile_min) {
  return tile_max != 0 || tile_pas >= 0 || tile_min != 0;
}
static bool single_circuits(const mq_batch* b) { return custom_tiles(b->tile_max, b->tile_pas, b->tile_min); }

// Record the whole batch on b->stream (being captured).
static int record_batch(mq_batch* b, float* probs, double* z0) {
  const bool single = single_circuits(b);
  if (!b->large.empty()) {
    MQ_CUDA(cudaEventRecord(b->fork_event, b->stream));
    for (int l = 0; l < b->lanes; ++l) MQ_CUDA(cudaStreamWaitEvent(b->lane_stream[l], b->fork_event, 0));
  }
  if (!b->small.empty()) {
    MQ_CUDA(cudaMemsetAsync(b->d_next, 0, sizeof(uint32_t), b->stream));
    int rc = small_dispatch(b, probs, z0, false);
    if (rc) return rc;
  }
  if (b->large.empty()) return MQ_OK;
  for (int l = 0; l < b->lanes; ++l) {
    int rc = single ? MQ_OK : record_lane_groups(b, l, probs, z0);
    if (!rc) rc = record_lane_single(b, l, probs, z0);
    if (rc) return rc;
    MQ_CUDA(cudaEventRecord(b->lane_event[l], b->lane_stream[l]));
    MQ_CUDA(cudaStreamWaitEvent(b->stream, b->lane_event[l], 0));
  }
  return MQ_OK;
}

// Most amplitudes of a group (32 MB; a wider circuit is a group of its own).
// 256 circuits of 10 to 20 qubits on 16 lanes: 4.36 ms a run with 2^20, 4.33 with
// 2^21, 4.25 with 2^22, 4.23 with 2^23 (twice the memory).
constexpr size_t kGroupAmps = size_t(1) << 22;

// The large circuits that run one by one, all of them with a tile plan set by
// mq_batch_set_tiles, else those of 24 qubits and more, where the general
// sweeps with TMA tiles are as fast (24 qubits, 6 circuits: 12.5 ms both; 23
// qubits, 8 circuits: 8.6 against 8.2 ms in groups), by lane (longest
// processing time first).
constexpr int kGroupMaxQubits = 23;
using LaneWork = std::vector<std::vector<int>>;
static LaneWork single_work(const mq_batch* b, bool all) {
  LaneWork work(b->lanes);
  std::vector<int> order;
  for (int c : b->large)
    if (all || b->n[c] > kGroupMaxQubits) order.push_back(c);
  auto load = [&](int c) { return (uint64_t)std::max(1, b->depth[c]) << b->n[c]; };
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return load(x) > load(y); });
  std::vector<uint64_t> sum(b->lanes, 0);
  for (int c : order) {
    const int l = (int)(std::min_element(sum.begin(), sum.end()) - sum.begin());
    work[l].push_back(c);
    sum[l] += load(c);
  }
  return work;
}

// The device memory of a plan (its single circuits' states and, for the
// default tiles, the groups' buffers): what is missing is allocated, what is
// there stays.
static int acquire(mq_batch* b, const LaneWork& work, bool groups) {
  for (int i = 0; i < 2 && groups; ++i)
    for (int l = 0; l < b->lanes; ++l) {
      if (b->lane_buf[i][l] || !b->lane_amps[l]) continue;
      const cudaError_t e = cudaMalloc(&b->lane_buf[i][l], b->lane_amps[l] * sizeof(float2));
      if (e != cudaSuccess) {
        b->lane_buf[i][l] = nullptr;
        return cuda_fail(e, "cudaMalloc(batch group buffers)");
      }
    }
  for (int l = 0; l < b->lanes; ++l)
    for (int c : work[l])
      if (!b->lane_state[l].count(b->n[c])) {
        int rc = make_lane_state(b, l, b->n[c]);
        if (rc) return rc;
      }
  return MQ_OK;
}
// Gives back what a plan does not use (nothing runs before the first capture).
static void release_other(mq_batch* b, const LaneWork& work, bool groups) {
  for (int l = 0; l < b->lanes; ++l) {
    auto& m = b->lane_state[l];
    for (auto it = m.begin(); it != m.end();) {
      const bool used = std::any_of(work[l].begin(), work[l].end(), [&](int c) { return b->n[c] == it->first; });
      if (used) {
        ++it;
      } else {
        state_free(it->second);
        it = m.erase(it);
      }
    }
  }
  for (int i = 0; i < 2 && !groups; ++i)
    for (float2*& p : b->lane_buf[i]) {
      if (p) cudaFree(p);
      p = nullptr;
    }
}
// Changes the tile plan as a whole or not at all: when the memory of the new
// plan is not to be had, also not in place of the old plan's, the old plan is
// in force again (mq_batch_run asks for its memory once more).
static int change_plan(mq_batch* b, int tile_max, int tile_pas, int tile_min) {
  const bool all = custom_tiles(tile_max, tile_pas, tile_min), had_all = single_circuits(b);
  LaneWork work = single_work(b, all);
  int rc = acquire(b, work, !all);
  if (rc == MQ_ENOMEM) {
    release_other(b, work, !all);
    rc = acquire(b, work, !all);
  }
  if (rc) {
    const std::string why = mq_last_error();
    release_other(b, b->lane_work, !had_all);
    acquire(b, b->lane_work, !had_all);
    return fail(rc, why);
  }
  release_other(b, work, !all);
  b->lane_work = std::move(work);
  b->tile_max = tile_max;
  b->tile_pas = tile_pas;
  b->tile_min = tile_min;
  for (auto& m : b->lane_state)
    for (auto& kv : m) {
      kv.second->tile_max = tile_max;
      kv.second->tile_pas = tile_pas;
      kv.second->tile_min = tile_min;
    }
  return MQ_OK;
}

// Groups of the large circuits, their lanes (longest processing time first)
// and their table (their buffers: acquire).
static cudaError_t plan_groups(mq_batch* b) {
  std::map<std::pair<int, int>, std::vector<int>> by;  // (n, ladder)
  for (int c : b->large)
    if (b->n[c] <= kGroupMaxQubits) by[{b->n[c], b->ladder[c]}].push_back(c);
  std::vector<GroupCirc> table;
  for (auto& [key, list] : by) {
    std::stable_sort(list.begin(), list.end(), [&](int x, int y) { return b->depth[x] > b->depth[y]; });
    const size_t most = std::max<size_t>(1, kGroupAmps >> key.first);
    // groups of equal size, each with the whole range of depths
    const size_t ng = (list.size() + most - 1) / most;
    for (size_t g = 0; g < ng; ++g) {
      mq_batch::Group G;
      G.n = key.first;
      G.ladder = key.second != 0;
      G.first = (uint32_t)table.size();
      for (size_t i = g; i < list.size(); i += ng) {
        const int c = list[i];
        G.circ.push_back(c);
        table.push_back({b->mats_off[c], b->probs_off[c], (uint32_t)c, (uint32_t)b->depth[c]});
      }
      b->groups.push_back(std::move(G));
    }
  }
  auto load = [&](const mq_batch::Group& G) {
    uint64_t v = 0;
    for (int c : G.circ) v += (uint64_t)std::max(1, b->depth[c]) << G.n;
    return v;
  };
  b->lane_groups.resize(b->lanes);
  std::vector<int> order(b->groups.size());
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return load(b->groups[x]) > load(b->groups[y]); });
  std::vector<uint64_t> sum(b->lanes, 0);
  b->lane_amps.assign(b->lanes, 0);
  for (int g : order) {
    const int l = (int)(std::min_element(sum.begin(), sum.end()) - sum.begin());
    b->lane_groups[l].push_back(g);
    sum[l] += load(b->groups[g]);
    b->lane_amps[l] = std::max(b->lane_amps[l], b->groups[g].circ.size() << b->groups[g].n);
    b->zslots = std::max<size_t>(b->zslots, b->groups[g].circ.size() * group_blocks(b, b->groups[g].n));
  }
  cudaError_t e = cudaSuccess;
  for (auto& v : b->lane_buf) v.assign(b->lanes, nullptr);
  if (!table.empty()) e = cudaMalloc(&b->d_group, table.size() * sizeof(GroupCirc));
  if (e == cudaSuccess && !table.empty())
    e = cudaMemcpy(b->d_group, table.data(), table.size() * sizeof(GroupCirc), cudaMemcpyHostToDevice);
  return e;
}

}  // namespace mq

#define MQ_TRY_BEGIN try {
#define MQ_TRY_END                                                      \
  }                                                                     \
  catch (const std::bad_alloc&) { return fail(MQ_ENOMEM, "host allocation failed"); } \
  catch (const std::exception& ex) { return fail(MQ_EDEVICE, ex.what()); } \
  catch (...) { return fail(MQ_EDEVICE, "unknown C++ exception"); }

extern "C" {

int mq_batch_create(int device, void* stream, int n_circuits, const int32_t* n_qubits, const int32_t* depth,
                    const uint8_t* ladder, int lanes, int small_threads, mq_batch** out) {
  MQ_TRY_BEGIN
  if (!out) return fail(MQ_EINVAL, "null output handle");
  *out = nullptr;
  if (n_circuits < 0 || (n_circuits > 0 && (!n_qubits || !depth))) return fail(MQ_EINVAL, "invalid circuit arrays");
  if (lanes < 1 || lanes > 64) return fail(MQ_EINVAL, "lanes must be in [1, 64]");
  if (small_threads != 128 && small_threads != 256 && small_threads != 512)
    return fail(MQ_EINVAL, "small_threads must be 128, 256 or 512");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return fail(MQ_EDEVICE, "no CUDA device is available");
  }
  if (device < 0 || device >= ndev) return fail(MQ_EINVAL, "device index out of range");
  for (int c = 0; c < n_circuits; ++c) {
    if (n_qubits[c] < 1 || n_qubits[c] > 30) return fail(MQ_EINVAL, "batched circuits take 1 to 30 qubits");
    if (depth[c] < 0) return fail(MQ_EINVAL, "negative depth");
  }
  DeviceGuard g(device);
  auto* b = new mq_batch();
  b->device = device;
  b->n_circ = n_circuits;
  b->lanes = lanes;
  b->small_threads = small_threads;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && sms > 0) b->num_sms = sms;
  if (stream) {
    b->stream = (cudaStream_t)stream;
  } else {
    cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) { delete b; return cuda_fail(e, "cudaStreamCreate"); }
    b->own_stream = true;
  }
  b->n.assign(n_qubits, n_qubits + n_circuits);
  b->depth.assign(depth, depth + n_circuits);
  b->ladder.assign(n_circuits, 1);
  if (ladder) b->ladder.assign(ladder, ladder + n_circuits);
  for (int c = 0; c < n_circuits; ++c) {
    b->mats_off.push_back(b->mats_total);
    b->probs_off.push_back(b->probs_total);
    b->mats_total += (uint64_t)b->depth[c] * b->n[c] * 8;
    b->probs_total += uint64_t(1) << b->n[c];
    (b->n[c] <= kSmallMax ? b->small : b->large).push_back(c);
  }
  auto bail = [&](cudaError_t e, const char* where) {
    const int rc = cuda_fail(e, where);
    batch_free(b);
    return rc;
  };
  cudaError_t e = cudaMalloc(&b->d_mats, std::max<uint64_t>(8, b->mats_total * sizeof(double)));
  if (e != cudaSuccess) return bail(e, "cudaMalloc(batch matrices)");
  if (!b->small.empty()) {
    std::vector<SmallCircuit> sc;
    // largest circuits first: the atomic counter hands them out early
    std::vector<int> order = b->small;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
      return ((uint64_t)b->depth[x] << b->n[x]) > ((uint64_t)b->depth[y] << b->n[y]);
    });
    for (int c : order)
      sc.push_back({(uint32_t)b->n[c], (uint32_t)b->depth[c], (uint32_t)b->ladder[c], (uint32_t)c, b->mats_off[c],
                    b->probs_off[c]});
    e = cudaMalloc(&b->d_small, sc.size() * sizeof(SmallCircuit));
    if (e == cudaSuccess) e = cudaMalloc(&b->d_next, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemcpy(b->d_small, sc.data(), sc.size() * sizeof(SmallCircuit), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return bail(e, "batch small-circuit setup");
    int rc = small_dispatch(b, nullptr, nullptr, true);
    if (rc) { batch_free(b); return rc; }
  }
  if (!b->large.empty()) {
    e = cudaFuncSetAttribute(k_group_sweep<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepSmem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_group_sweep<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSweepSmem);
    if (e != cudaSuccess) return bail(e, "batch sweep setup");
    b->zblocks = (uint32_t)b->num_sms * 4;
    b->lanes = std::min<int>(lanes, (int)b->large.size());
    e = plan_groups(b);
    if (e != cudaSuccess) return bail(e, "batch group setup");
    for (int l = 0; l < b->lanes; ++l) {
      cudaStream_t s;
      cudaEvent_t ev;
      e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
      if (e != cudaSuccess) return bail(e, "cudaStreamCreate(lane)");
      b->lane_stream.push_back(s);
      e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
      if (e != cudaSuccess) return bail(e, "cudaEventCreate(lane)");
      b->lane_event.push_back(ev);
    }
    e = cudaEventCreateWithFlags(&b->fork_event, cudaEventDisableTiming);
    if (e != cudaSuccess) return bail(e, "cudaEventCreate(fork)");
    b->lane_state.resize(b->lanes);
    b->lane_work = single_work(b, false);
    int rc = acquire(b, b->lane_work, true);
    if (rc) { batch_free(b); return rc; }
    b->zslots = std::max<size_t>(b->zslots, b->zblocks);
    e = cudaMalloc(&b->d_zpart, (size_t)b->lanes * b->zslots * sizeof(double));
    if (e != cudaSuccess) return bail(e, "cudaMalloc(batch partials)");
  }
  *out = b;
  return MQ_OK;
  MQ_TRY_END
}

int mq_batch_info(const mq_batch* b, uint64_t* mats_count, uint64_t* probs_count, int* n_small, int* n_large) {
  if (!b) return fail(MQ_EINVAL, "null batch handle");
  if (mats_count) *mats_count = b->mats_total;
  if (probs_count) *probs_count = b->probs_total;
  if (n_small) *n_small = (int)b->small.size();
  if (n_large) *n_large = (int)b->large.size();
  return MQ_OK;
}

int mq_batch_set_tiles(mq_batch* b, int tile_max, int passengers, int tile_min) {
  if (!b) return fail(MQ_EINVAL, "null batch handle");
  if (b->exec) return fail(MQ_EINVAL, "the tile plan is fixed once the batch has run (its graph is captured)");
  if (tile_max != 0 && (tile_max < 6 || tile_max > 12)) return fail(MQ_EINVAL, "tile_max must be 0 or in [6, 12]");
  if (passengers < -1 || passengers > 5) return fail(MQ_EINVAL, "passengers must be -1 or in [0, 5]");
  if (tile_min < 0 || tile_min > 12) return fail(MQ_EINVAL, "tile_min must be 0 or in [1, 12]");
  if (tile_max && passengers >= tile_max) return fail(MQ_EINVAL, "passengers must leave room for targets in a tile");
  if (b->large.empty()) {  // no sweeps: the plan is only noted
    b->tile_max = tile_max;
    b->tile_pas = passengers;
    b->tile_min = tile_min;
    return MQ_OK;
  }
  MQ_TRY_BEGIN
  DeviceGuard g(b->device);
  return change_plan(b, tile_max, passengers, tile_min);
  MQ_TRY_END
}

int mq_batch_run(mq_batch* b, const double* mats, float* probs_dev, double* z0_dev) {
  MQ_TRY_BEGIN
  if (!b) return fail(MQ_EINVAL, "null batch handle");
  if (b->n_circ == 0) return MQ_OK;
  if ((b->mats_total && !mats) || !probs_dev || !z0_dev) return fail(MQ_EINVAL, "null batch arrays");
  DeviceGuard g(b->device);
  if (b->mats_total)
    MQ_CUDA(cudaMemcpyAsync(b->d_mats, mats, b->mats_total * sizeof(double), cudaMemcpyHostToDevice, b->stream));
  if (!b->exec || b->graph_probs != probs_dev || b->graph_z0 != z0_dev) {
    if (b->exec) {
      cudaGraphExecDestroy(b->exec);
      b->exec = nullptr;
    }
    if (!b->large.empty()) {  // all there, unless a refused plan could not be undone
      int rc = acquire(b, b->lane_work, !single_circuits(b));
      if (rc) return rc;
    }
    MQ_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    int rc = record_batch(b, probs_dev, z0_dev);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
    if (rc) {
      if (graph) cudaGraphDestroy(graph);
      return rc;
    }
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture(batch)");
    e = cudaGraphInstantiate(&b->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate(batch)");
    b->graph_probs = probs_dev;
    b->graph_z0 = z0_dev;
  }
  MQ_CUDA(cudaGraphLaunch(b->exec, b->stream));
  return MQ_OK;
  MQ_TRY_END
}

int mq_batch_sync(mq_batch* b) {
  if (!b) return fail(MQ_EINVAL, "null batch handle");
  DeviceGuard g(b->device);
  MQ_CUDA(cudaStreamSynchronize(b->stream));
  return MQ_OK;
}

int mq_batch_destroy(mq_batch* b) {
  if (!b) return MQ_OK;
  DeviceGuard g(b->device);
  cudaStreamSynchronize(b->stream);
  batch_free(b);
  return MQ_OK;
}

}  // extern "C"
