// Pauli words within a window of four tile bits: the kernel, in a file of its own
// (a process loads a file's kernels as a whole on the first use of one, and
// this one is by far the longest).
#include "mq_pauli.cuh"

namespace mq {

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

int launch_pauli_tile(mq_state* h, const PauliTileParams& P, uint32_t grid, double* part) {
  const size_t smem = 32768 + sizeof(double) * P.n_words * (1u << kPauliLT);
  if (h->dtype == MQ_C64) {
    MQ_CUDA(cudaFuncSetAttribute(k_pauli_tile<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPauliSmem));
    k_pauli_tile<float><<<grid, 1 << kPauliLT, smem, h->stream>>>((const float2*)h->cur_buf(), P, part);
  } else {
    MQ_CUDA(cudaFuncSetAttribute(k_pauli_tile<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPauliSmem));
    k_pauli_tile<double><<<grid, 1 << kPauliLT, smem, h->stream>>>((const double2*)h->cur_buf(), P, part);
  }
  MQ_LAUNCHED("k_pauli_tile");
  return MQ_OK;
}

}  // namespace mq
