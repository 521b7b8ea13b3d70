// The window sweeps of Pauli words (mq_pauli_tile.cu), launched by mq_pauli.cu.
#pragma once

#include "mq_internal.cuh"

namespace mq {

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

// One sweep's words: the sums of each block to part[word * grid + block].
int launch_pauli_tile(mq_state* h, const PauliTileParams& P, uint32_t grid, double* part);

}  // namespace mq
