// Host side of the row-owning decode product (qmv_rows.cuh): which problems it takes, how K and the shared memory are laid out.
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "qmv_rows.h"

namespace b200q {
namespace rows {

constexpr size_t kSmemLimit = 227 * 1024;

bool pdl_on() {
  static const bool on = [] {
    const char* e = getenv("B200Q_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

// Groups (units form) that a warp's registers hold.
int units_groups(int bits, int group, int mt, bool wide) {
  if (wide) return group == 64 ? UnitsCfg<2, 64, 1, true>::NGW : UnitsCfg<2, 128, 1, true>::NGW;
#define B200Q_UNITS_CASE(BITS_, G_) \
  if (bits == BITS_ && group == G_) return mt == 2 ? UnitsCfg<BITS_, G_, 2>::NGW : UnitsCfg<BITS_, G_, 1>::NGW;
  B200Q_UNITS_CASE(2, 64) B200Q_UNITS_CASE(2, 128)
  B200Q_UNITS_CASE(4, 32) B200Q_UNITS_CASE(4, 64) B200Q_UNITS_CASE(4, 128)
  B200Q_UNITS_CASE(8, 32) B200Q_UNITS_CASE(8, 64) B200Q_UNITS_CASE(8, 128)
#undef B200Q_UNITS_CASE
  return 0;
}

// Everything that does not depend on pointers.  `tokens`: rows of x per tile; max_rg: row groups of a matrix that a block may
// have (times two when gated); stages: row groups that it has in all, at most.
constexpr int64_t kWideRows = 16384;
bool lay_out(RowsPlan& pl, int64_t rows, int tokens, int64_t K, int group, int bits, int64_t max_rg, int64_t stages) {
  RowsParams& p = pl.prm;
  if (K < 128 || K % 128 != 0 || K > (1 << 24)) return false;   // (rows of whole 16 bytes, whole groups)
  p.K = (int)K;
  p.row_bytes = (int)(K * bits / 8);
  p.groups = (int)(K / group);
  pl.runs = runs_form(bits, group);
  int most, item_bytes, item_groups;
  if (pl.runs) {
    p.ng = 128 / group;
    const int tiles = (tokens * p.ng + 7) / 8;
    if (tiles > kRunTiles) return false;
    pl.shape = tiles;
    most = run_chunks(pl.shape);
    p.items = (int)(K / 128);
    item_bytes = 16 * bits;
    item_groups = p.ng;
  } else {
    pl.shape = group;
    // Us with two phases and with one (1, 4, 8 rows): groups of 128, [28672, 8192] 27.2, 27.3, 27.6 / 23.1, 24.1, 24.8; [4096, 8192] 7.4,
    // 7.6, 8.1 / 6.8, 7.4, 8.0.  Groups of 64, [28672, 8192] 28.3, 28.4, 28.9 / 24.4, 25.8, 26.4; [4096, 8192] 7.4, 7.5, 8.2 / 7.3, 8.1,
    // 8.8, and with rows of scales off 16-byte boundaries [14336, 8064] 23.1 to 23.8 / 25.5 to 27.4: only many aligned rows pay for the
    // longer start.
    pl.wide = bits == 2 && pl.mt == 1 && pl.work == Work::Plain && K > 4096 && K <= 8192 &&
              (group == 128 || (rows >= kWideRows && K % 512 == 0));
    most = units_groups(bits, group, pl.mt, pl.wide);
    if (most == 0) return false;
    p.ng = 1;
    p.items = p.groups;
    item_bytes = group * bits / 8;
    item_groups = 1;
  }
  // As many items per warp as leave room for three stages, or two large ones; with long rows fewer, in more phases.
  for (; most >= 1; --most) {
    // phases as equal as whole shares of the warps allow, a share in each of them the same
    p.nph = (p.items + kConsumers * most - 1) / (kConsumers * most);
    p.phase_items = (p.items + p.nph - 1) / p.nph;
    p.cnt = (p.phase_items + kConsumers - 1) / kConsumers;
    if (!pl.runs)   // (pairs of groups, whose scales are one word)
      while (p.cnt < 2 || (p.cnt & (p.cnt - 1)) != 0) ++p.cnt;
    if (p.nph > 1) {   // (rows of scales from 16-byte boundaries in every phase where the first has them)
      p.phase_items = kConsumers * p.cnt;
      p.nph = (p.items + p.phase_items - 1) / p.phase_items;
    }
    p.n_active = (p.phase_items + p.cnt - 1) / p.cnt;
    p.phase_bytes = (uint32_t)p.phase_items * item_bytes;
    p.phase_groups = p.phase_items * item_groups;
    // pairs that eight lanes read at once without bank conflicts: an odd multiple of 16 bytes; of 32 where they read 8 bytes each
    const uint32_t step = pl.runs && bits % 2 == 0 ? 32 : 16;
    p.pitch = (2 * p.phase_bytes + step - 1) / step * step;
    if ((p.pitch / step) % 2 == 0) p.pitch += step;
    p.s_bytes = 2 * p.n_active * p.cnt * item_groups;
    p.shalf = ((uint32_t)p.s_bytes + 15) / 16 * 16;
    p.spitch = 2 * p.shalf + 16;
    p.off_scales = 8 * p.pitch;
    p.slot_bytes = (p.off_scales + 16 * p.spitch + 127) / 128 * 128;
    size_t off = 1024;   // barriers, abort flag
    p.off_run = (uint32_t)off;
    if (p.nph > 1) off += (size_t)max_rg * pl.mt * 512;
    p.off_pbuf = (uint32_t)off;
    p.pwarp_bytes = (uint32_t)tokens * tok_pitch(pl.work) * 4;
    p.pbuf_bytes = p.n_active * p.pwarp_bytes;
    off += (size_t)partial_bufs(pl.work) * p.pbuf_bytes;
    off = (off + 127) / 128 * 128;
    p.off_slots = (uint32_t)off;
    int64_t nst = off < kSmemLimit ? (int64_t)((kSmemLimit - off) / p.slot_bytes) : 0;
    if (nst < 3 && !(nst == 2 && (most == 1 || p.slot_bytes > 48 * 1024))) continue;
    if (nst > 16) nst = 16;
    if (nst > stages * p.nph) nst = stages * p.nph;
    p.nst = (int)(nst < 1 ? 1 : nst);
    pl.smem = off + (size_t)p.nst * p.slot_bytes;
    return true;
  }
  return false;
}

// The widest copy that every row's scales and biases of every phase are aligned to.
void align_scales(RowsParams& p, int nw) {
  uintptr_t al = (uintptr_t)p.groups * 2 | (p.nph > 1 ? (uintptr_t)p.phase_groups * 2 : 0);
  for (int i = 0; i < nw; ++i) al |= reinterpret_cast<uintptr_t>(p.scales[i]) | reinterpret_cast<uintptr_t>(p.biases[i]);
  p.s_piece = (al & 15) == 0 ? 16 : ((al & 7) == 0 ? 8 : ((al & 3) == 0 ? 4 : 2));
}

RowsPlan make_plan(const QmmArgs& a) {
  RowsPlan pl{};
  if ((a.dtype != B200Q_BF16 && !(a.dtype == B200Q_F16 && a.peers.n == 0)) || !a.transpose || a.w_batched || a.batch != 1) return pl;
  if (a.M < 1 || a.M > 16 || a.N < 1 || a.K < 1 || a.N > (1ll << 30)) return pl;
  pl.work = Work::Plain;
  pl.f16 = a.dtype == B200Q_F16;
  pl.mt = a.M > 8 ? 2 : 1;
  const int nblk8 = (int)((a.N + 7) / 8);
  pl.grid = cmin(nblk8, sm_count());
  const int max_rg = ((nblk8 + pl.grid - 1) / pl.grid + 1) / 2;
  if (!lay_out(pl, a.N, (int)a.M, a.K, a.group, a.bits, max_rg, max_rg)) return pl;
  RowsParams& p = pl.prm;
  p.blk_each = nblk8 / pl.grid;
  p.blk_more = nblk8 % pl.grid;
  p.x = (const uint16_t*)a.x;
  p.wq[0] = a.wq;
  p.scales[0] = (const uint16_t*)a.scales;
  p.biases[0] = (const uint16_t*)a.biases;
  align_scales(p, 1);
  if (a.peers.n > 0) {
    p.n_out = a.peers.n; p.ld = a.peers.ld; p.col0 = a.peers.col0;
    for (int q = 0; q < a.peers.n; ++q) p.y[q] = (uint16_t*)a.peers.y[q];
    p.sig = a.peers.sig;
  } else {
    p.n_out = 1; p.ld = a.N; p.col0 = 0; p.y[0] = (uint16_t*)a.y;
  }
  p.M = (int)a.M; p.N = (int)a.N;
  pl.ok = true;
  return pl;
}

RowsPlan make_group_plan(const RowsGroup& a) {
  RowsPlan pl{};
  if (a.N < 1 || a.K < 1) return pl;
  const int nw = a.wq[1] ? 2 : 1;
  for (int i = 0; i < nw; ++i) {
    if (reinterpret_cast<uintptr_t>(a.wq[i]) & 15) return pl;
    if ((reinterpret_cast<uintptr_t>(a.scales[i]) | reinterpret_cast<uintptr_t>(a.biases[i])) & 1) return pl;
  }
  const int64_t rgs = (a.N + 15) / 16, units = a.max_tiles * rgs;
  if (units > (1ll << 30)) return pl;
  pl.work = nw == 2 ? Work::Gated : Work::Grouped;
  pl.mt = 1;
  pl.grid = (int)(units < sm_count() ? units : sm_count());
  const int64_t most = (units + pl.grid - 1) / pl.grid;
  const int tile = rows_tile(a.bits, a.group);
  if (!lay_out(pl, a.N, tile, a.K, a.group, a.bits, (most < rgs ? most : rgs) * nw, most * nw)) return pl;
  RowsParams& p = pl.prm;
  p.x = (const uint16_t*)a.x;
  for (int i = 0; i < nw; ++i) {
    p.wq[i] = a.wq[i];
    p.scales[i] = (const uint16_t*)a.scales[i];
    p.biases[i] = (const uint16_t*)a.biases[i];
  }
  align_scales(p, nw);
  p.n_out = 1; p.ld = a.N; p.col0 = 0; p.y[0] = (uint16_t*)a.y;
  p.M = tile; p.N = (int)a.N;
  p.tiles = static_cast<const int4*>(a.tiles);
  p.n_tiles = a.n_tiles;
  p.src_slot = a.src_slot; p.dst_slot = a.dst_slot;
  p.per_slot = (int)a.per_slot;
  p.rgs = (int)rgs;
  p.status = a.status;
  pl.ok = true;
  return pl;
}

int launch_plan(const RowsPlan& pl, int bits, cudaStream_t st) {
  int rc = B200Q_ERR_UNSUPPORTED;
  B200Q_DISPATCH_BITS(bits, BITS, { rc = launch_rows<BITS>(pl, st); });
  return rc;
}

// 17 to 32 rows: two passes; the second finds the matrix in L2 when it fits.  Sharded output (peer buffers, completion signal)
// stays single-pass.
constexpr int kPassRows = 16;
int passes(const QmmArgs& a) { return (int)((a.M + kPassRows - 1) / kPassRows); }
QmmArgs pass_args(const QmmArgs& a, int i) {
  QmmArgs h = a;
  const int64_t row0 = (int64_t)i * kPassRows, rows = a.M - row0;
  h.M = rows < kPassRows ? rows : kPassRows;
  h.x = static_cast<const char*>(a.x) + (size_t)row0 * a.K * 2;
  h.y = static_cast<char*>(a.y) + (size_t)row0 * a.N * 2;
  return h;
}

}  // namespace rows

// Process-wide promise that packed weights, scales and biases are not written by the
// operation that precedes a matmul on its stream (set by b200q_set_weights_constant or
// B200Q_WEIGHTS_CONSTANT=1).  Only then may the decode kernel request them before the
// previous kernel has finished (programmatic dependent launch).
static int g_weights_constant = -1;
bool weights_constant() {
  if (g_weights_constant < 0) {
    const char* e = getenv("B200Q_WEIGHTS_CONSTANT");
    g_weights_constant = (e && e[0] == '1') ? 1 : 0;
  }
  return g_weights_constant == 1;
}
void set_weights_constant(int on) { g_weights_constant = on ? 1 : 0; }

// Rows of x:
//   units form   up to 16; 17 to 32 with K in whole turns of the 16 warps: two passes
//   runs form    up to 16 in groups of 128, 8 of 64, 4 of 32: what two column tiles take
bool qmv_rows_supported(const QmmArgs& a) {
  using namespace rows;
  if (a.M < 1 || a.M > 32 || a.K < 1 || a.group < 1) return false;
  if ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.wq)) & 15) return false;
  if ((reinterpret_cast<uintptr_t>(a.scales) | reinterpret_cast<uintptr_t>(a.biases)) & 1) return false;
  if (runs_form(a.bits, a.group) && a.M > run_rows(a.group)) return false;
  if (a.M > 16 && a.K % (kConsumers * a.group) != 0) return false;
  const int n = passes(a);
  if (n == 1) return make_plan(a).ok;
  if (a.peers.n > 0) return false;
  return make_plan(pass_args(a, 0)).ok && make_plan(pass_args(a, n - 1)).ok;
}

int qmv_rows(const QmmArgs& a, cudaStream_t st) {
  using namespace rows;
  const int n = passes(a);
  for (int i = 0; i < n; ++i) {
    RowsPlan pl = make_plan(n == 1 ? a : pass_args(a, i));
    if (!pl.ok) return fail(B200Q_ERR_UNSUPPORTED, "[quantized_matmul] qmv_rows: unsupported problem");
    pl.prm.early = weights_constant() ? 1 : 0;
    if (a.ws && a.ws_bytes >= kStatusBytes)
      pl.prm.status = reinterpret_cast<uint32_t*>(static_cast<char*>(a.ws) + a.ws_bytes - kStatusBytes);
    if (int rc = launch_plan(pl, a.bits, st)) return rc;
  }
  return B200Q_OK;
}

int rows_tile(int bits, int group) { return runs_form(bits, group) ? rows::cmin(8, rows::run_rows(group)) : 8; }

bool qmv_rows_grouped_supported(const RowsGroup& a) { return rows::make_group_plan(a).ok; }

int qmv_rows_grouped(const RowsGroup& a, cudaStream_t st) {
  const rows::RowsPlan pl = rows::make_group_plan(a);
  if (!pl.ok) return fail(B200Q_ERR_UNSUPPORTED, "[gather_qmm] qmv_rows: unsupported problem");
  return rows::launch_plan(pl, a.bits, st);
}

}  // namespace b200q
