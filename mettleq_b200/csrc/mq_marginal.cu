// Marginals (e): the probabilities of some qubits, summed in a fixed order
// (probabilities_array's transpose and sum, sim.py:322-343): chunks of at most
// 1024 entries by 32 lanes and an XOR butterfly, then sequential runs.  A file
// of its own, since a process loads a file's kernels as a whole on the first
// use of one.
#include <algorithm>
#include <cstring>
#include <vector>

#include "mq_marginal.cuh"

namespace mq {

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

// ================================================================ host side
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

int marginal_device(mq_state* h, const int32_t* wires, int k, double* work, double** q) {
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
  int rc = MQ_OK;
  // a level of one entry per run is the entry itself (0 + x = x)
  if (!rc && ncb > 1) {
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

}  // namespace mq
