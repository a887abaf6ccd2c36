// What the host side (qmv_rows.cu) and the kernel (qmv_rows.cuh, one translation unit per field width) of the row-owning decode
// product share.
#pragma once

#include "kernels.h"

namespace b200q {
namespace rows {

constexpr int kConsumers = 16;    // warps that multiply; one K slice each
// Runs: tiles of 8 columns at most, token rows that they take.  (Four tiles would hold 64 registers of x: 8 rows through [14336, 4096]
// at 6 bits, groups of 32, 47 us where the register-path kernel takes 27.)
constexpr int kRunTiles = 2;
__host__ __device__ constexpr int run_rows(int group) { return 8 * kRunTiles * group / 128; }
// Runs: chunks of 128 k per warp and phase, 16 registers of x each per tile.  More would save phases, but registers of x beyond
// 32 push the loop's addresses out to memory (one row through [28672, 8192], 6 bits in groups of 32: 46 us with four chunks, 40
// with two; units, 4 bits, [14336, 4096]: 13.8 us with 64 registers, 10.3 with 32, and less code to fetch before the first product).
__host__ __device__ constexpr int run_chunks(int tiles) { return tiles == 1 ? 2 : 1; }

__host__ __device__ constexpr int cmin(int a, int b) { return a < b ? a : b; }
__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }

// Compile-time shape of one (bits, group size, token tiles) instantiation of the units form.  A "unit" is 16 packed
// bytes of one row (what one ldmatrix row holds); lane t of a quad owns word t of every unit.
// WIDE (2 bits, up to 8 tokens, K from 4224 to 8192): 64 registers of x, so that a phase is all of K and a row 2 KB: in phases of 4096
// the 16 copies of 1 KB that a stage takes cost the loader more than HBM takes for them (rule and figures: lay_out).
template <int BITS, int G, int MT, bool WIDE = false>
struct UnitsCfg {
  static_assert(BITS == 2 || BITS == 4 || BITS == 8, "field widths of this form");
  static constexpr int GB = G * BITS / 8;                  // packed bytes of one group of one row
  static_assert(GB >= 16, "a group must fill at least one 16-byte unit");
  static constexpr int UG = GB / 16;                       // units per group
  static constexpr int KW = 32 / BITS;                     // k values per 32-bit word
  static constexpr int NP = KW / 2;                        // registers of pairs that a word unpacks to
  static constexpr int UW = cmax(2 * UG, cmin(cmin((MT == 1 && !WIDE ? 32 : 64) / (MT * NP), 8 * UG), 16));   // units per warp and phase
  static constexpr int NGW = UW / UG;                      // groups per warp and phase
  static_assert(NGW >= 2 && NGW <= 8 && NGW % 2 == 0, "groups are processed in pairs, eight at most feed one bias MMA");
};

// What a launch works on.  Plain: one matrix.  Grouped: the matrices of the experts that have rows.  Gated: the same
// with two matrices per expert, y = silu(gate) * up; their stages alternate, so both results of a row group meet in
// the reducer warp and neither product goes through memory.
enum class Work { Plain, Grouped, Gated };

// Buffers of partial sums of the stages being reduced; floats between two tokens' 16 rows in them (20: stores free of bank
// conflicts; grouped launches always have room for 8 tokens and spare it).
__host__ __device__ constexpr int partial_bufs(Work w) { return w == Work::Gated ? 4 : 2; }
__host__ __device__ constexpr int tok_pitch(Work w) { return w == Work::Plain ? 20 : 16; }

struct RowsParams {
  const uint16_t* x;   // 16-bit elements of either type
  uint16_t* y[kMaxPeers];
  int n_out;
  long long ld, col0;
  PeerSignal sig;       // completion signal towards the ranks that receive y (n == 0: none)
  const uint32_t* wq[2];
  const uint16_t* scales[2];
  const uint16_t* biases[2];
  int M, N, K;
  int blk_each, blk_more;    // plain: 8-row blocks per thread block; the first blk_more have one more
  int row_bytes, groups;     // of a packed row
  // K in phases of phase_items groups (units form) or chunks of 128 k (runs), cnt of them per consumer warp
  int nph, phase_items, cnt, items, n_active;
  int phase_groups;
  uint32_t phase_bytes;
  int ng;                    // runs: groups per chunk
  int s_piece, s_bytes;      // bytes per copy of scales; per row and phase, with the zeros that fill up the last warp's share
  int nst;                   // ring stages
  // a stage: eight pairs of rows, the second phase_bytes after the first; then eight pairs of scales (shalf), eight of biases
  uint32_t pitch, spitch, shalf, slot_bytes, off_scales;
  uint32_t off_slots, off_run, off_pbuf, pbuf_bytes, pwarp_bytes;
  uint32_t* status;     // may be null
  int early;            // weights, scales and biases may be read before the previous kernel ended
  // grouped (gather_qmm) launches only: device-side table of tiles of up to 8 expert-sorted rows
  const int4* tiles;       // expert, first row, rows
  const int* n_tiles;
  const int* src_slot;     // per sorted pair: which x it multiplies (null: x is in sorted order)
  const int* dst_slot;     // per sorted pair: which y it writes (null: y is in sorted order)
  int per_slot;            // rows per pair
  int rgs;                 // 16-row groups per matrix
};

struct RowsPlan {
  bool ok, runs, f16, wide;
  int shape;           // units: group size; runs: column tiles (1 or 2)
  int mt, grid;
  Work work;
  size_t smem;
  RowsParams prm;
};

template <int BITS>
int launch_rows(const RowsPlan& pl, cudaStream_t st);   // qmv_rows_<BITS>.cu

}  // namespace rows
}  // namespace b200q
