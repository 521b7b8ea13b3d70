// Probabilities and seeded sampling (e).
//
// Replaces the reference's MLX library calls on this path:
//   probabilities_array: |a|^2, transpose, sum           (sim.py:322-343)
//   sample_array: log(max(p,1e-30)) + mx.random.categorical (sim.py:383-419)
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
#include <vector>

#include "mq_marginal.cuh"

namespace mq {

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

// ================================================================ host side
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
  SampleMeta hm = {};
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

}  // namespace mq
