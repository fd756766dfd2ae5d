// tsm_tile.cu -- how the any-layout tensor-core kernels (tsm_tile.cuh) are
// launched: each operand's way into shared memory, the chunk and the grid.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>

#include "tsm_errors.h"
#include "tsm_registry.cuh"
#include "tsm_tile.h"
#include "tsm_tmap.h"

namespace tsm {
namespace {

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Rows whose dense width-w copies are whole multiples of 16 bytes.
int64_t whole_rows(int64_t n, int64_t row_bytes) {
  int64_t unit = 16;
  while (unit > 1 && row_bytes % 2 == 0) {
    row_bytes /= 2;
    unit /= 2;
  }
  return n - n % unit;
}

// Shared pitch (elements) of a tensor-box or row-gathered operand: FP64 the
// next 4 mod 8 (conflict-free fragment loads; columns past the pitch read on
// into the next row, which only reaches entries of C that are not written);
// FP32 the next multiple of 4, not of 32 (2-way conflicts at worst: one FP32
// fragment load is half the bytes).
template <typename T>
int padded_pitch(int w) {
  if (sizeof(T) == 8) return w <= 4 ? 4 : (w + 3) / 8 * 8 + 4;
  const int p = (w + 3) / 4 * 4;
  return p % 32 == 0 ? p + 4 : p;
}

template <typename T>
TileOperand<T> operand(const T* base, int64_t n, int w, int64_t s_row, int64_t s_col, bool bulk_ok) {
  TileOperand<T> x{};
  x.base = base;
  x.s_row = s_row;
  x.s_col = s_col;
  x.w = x.cols = w;
  const int64_t row_bytes = s_row * int64_t(sizeof(T));
  const bool rows = s_col == 1 && s_row >= w && n <= static_cast<int64_t>(INT_MAX) - 4096;
  if (s_col == 1 && s_row == w && aligned16(base) && bulk_ok && w % (sizeof(T) == 8 ? 8 : 16) != 0) {
    x.load = kTileBulk;
  } else if (rows && aligned16(base) && row_bytes % 16 == 0) {
    x.load = kTileTma;
  } else if (rows && n >= 64) {
    x.load = kTilePhases;
  } else {
    x.load = s_row < s_col ? kTileCols : kTileRows;
  }
  return x;
}

// The shared layout of an operand whose load is settled: pitch, and how a
// k-step's address moves, with (phased) or without an operand in phases.
template <typename T>
void lay_out(TileOperand<T>& x, bool phased, int64_t ld) {
  constexpr int E = 16 / int(sizeof(T));  // elements per 16 bytes
  if (phased && x.load == kTileTma) x.load = kTilePhases;
  if (x.load == kTileBulk)
    x.pitch = x.w;
  else if (x.load == kTileTma)
    x.pitch = padded_pitch<T>(x.w);
  else if (x.load == kTilePhases)
    x.pitch = padded_pitch<T>(x.w + E - 1);
  else  // gathered: an odd pitch spreads rows written by neighbouring lanes, or read 4 apart, over the banks
    x.pitch = phased || x.load == kTileCols ? x.w | 1 : padded_pitch<T>(x.w);
  if (x.load == kTilePhases) {
    const int64_t first = static_cast<int64_t>(reinterpret_cast<uintptr_t>(x.base) / sizeof(T));
    for (int q = 0; q < 4; ++q) x.shift[q] = static_cast<unsigned char>((first + q * ld) % E);
  }
}

template <typename T>
void set_steps(TileOperand<T>& x, bool phased, int rs) {
  const int P = x.pitch;
  if (x.load == kTilePhases) {
    x.phase_bytes = (rs / 4 * P * int(sizeof(T)) + 127) / 128 * 128;
    x.q_step = x.phase_bytes / int(sizeof(T));
    x.j_step = 4 * P;
    x.t_step = P;
  } else {
    x.q_step = phased ? P : 4 * P;
    x.j_step = 16 * P;
    x.t_step = phased ? 4 * P : P;
  }
}

template <typename T>
bool encode(TileArgs<T>& a, int o) {
  const TileOperand<T>& x = a.x[o];
  const auto type = sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  if (x.load == kTileTma)
    return encode_rowmajor_map(&a.t[o][0], type, sizeof(T), x.base, a.p.n, x.w, x.s_row, x.pitch, a.rs / a.boxes,
                               CU_TENSOR_MAP_SWIZZLE_NONE, &last_error());
  if (x.load != kTilePhases) return true;
  for (int q = 0; q < 4; ++q)  // n >= 64: every phase has rows
    if (!encode_rowmajor_map(&a.t[o][q], type, sizeof(T), x.base + q * x.s_row - x.shift[q], (a.p.n - q + 3) / 4,
                             x.w + x.shift[q], 4 * x.s_row, x.pitch, a.rs / 4, CU_TENSOR_MAP_SWIZZLE_NONE,
                             &last_error()))
      return false;
  return true;
}

}  // namespace

namespace {

struct Joint {
  int width = 0;  // columns from the first of A's and B's to the last; 0: load them apart
  int a_first = 0, b_first = 0;
};

// Row-major operands that are column blocks of one matrix, at most two columns apart.
Joint joint_columns(const void* A, int m, int64_t lda, const void* B, int k, int64_t ldb, size_t esize) {
  Joint j;
  const intptr_t bytes = reinterpret_cast<intptr_t>(B) - reinterpret_cast<intptr_t>(A);
  const intptr_t most = intptr_t(esize) * 66;
  if (lda != ldb || bytes % intptr_t(esize) != 0 || bytes < -most || bytes > most) return j;
  const int64_t apart = bytes / intptr_t(esize);
  const int64_t a0 = apart < 0 ? -apart : 0, b0 = apart < 0 ? 0 : apart;
  const int64_t width = std::max(a0 + m, b0 + k);
  if (width > lda || width > m + k + 2) return j;
  j.width = static_cast<int>(width);
  j.a_first = static_cast<int>(a0);
  j.b_first = static_cast<int>(b0);
  return j;
}

}  // namespace

bool tile_joint(const void* A, int m, int64_t lda, const void* B, int k, int64_t ldb, size_t esize, bool* phases) {
  const Joint j = joint_columns(A, m, lda, B, k, ldb, esize);
  const bool aligned = aligned16(j.a_first == 0 ? A : B);
  *phases = !(aligned && (lda == j.width || lda * int64_t(esize) % 16 == 0));
  return j.width > 0;
}

template <typename T>
tsm_status launch_tile(const Variant* v, int sms, cudaStream_t stream, PlainArgs<T> p, int64_t a_row, int64_t a_col,
                       int64_t b_row, int64_t b_col, int64_t max_ctas) {
  TileArgs<T> a{};
  a.swap = (p.m <= v->wa && p.k <= v->wb) ? 0 : 1;
  if (p.m == 1) a_col = 1;  // a stride along an extent of one is never used
  if (p.k == 1) b_col = 1;
  if (p.n <= 1) {  // nor a row stride, which may be more than a tensor map holds
    a_row = p.m * a_col;
    b_row = p.k * b_col;
  }
  p.symmetric = p.A == p.B && p.m == p.k && a_row == b_row && a_col == b_col;
  const bool row_major = a_col == 1 && b_col == 1;
  const Joint j = row_major ? joint_columns(p.A, p.m, a_row, p.B, p.k, b_row, sizeof(T)) : Joint{};
  a.joint = j.width > 0;
  // Rows a bulk copy leaves are read by the reduction's epilogue, row-major.
  const int64_t bulk_n = a.joint ? whole_rows(p.n, j.width * int64_t(sizeof(T)))
                                 : std::min(whole_rows(p.n, p.m * int64_t(sizeof(T))),
                                            whole_rows(p.n, p.k * int64_t(sizeof(T))));
  const bool bulk_ok = row_major || bulk_n == p.n;
  TileOperand<T> xa, xb;
  if (a.joint) {
    xa = xb = operand<T>(j.a_first == 0 ? p.A : p.B, p.n, j.width, a_row, 1, bulk_ok);
    xa.cols = p.m;
    xb.cols = p.k;
  } else {
    xa = operand<T>(p.A, p.n, p.m, a_row, a_col, bulk_ok);
    xb = operand<T>(p.B, p.n, p.k, b_row, b_col, bulk_ok);
  }
  a.x[0] = a.swap ? xb : xa;
  a.x[1] = a.swap ? xa : xb;
  const int nops = a.joint ? 1 : 2;
  const bool phased = a.x[0].load == kTilePhases || a.x[1].load == kTilePhases;
  for (int o = 0; o < 2; ++o) lay_out(a.x[o], phased, a.x[o].s_row);
  const bool bulk = xa.load == kTileBulk || xb.load == kTileBulk;
  p.rows_main = bulk ? bulk_n : p.n;
  p.lda = a_row;
  p.ldb = b_row;

  // Chunk: as many rows as three stages hold, at most 1024; fewer where the
  // rows would not fill the grid evenly, but no less than 16 KB of them (64 to
  // 256): a CTA costs its share of the cross-CTA sum.
  const int unit = phased ? 16 : 8;
  const int elems = a.x[0].pitch + (nops == 2 ? a.x[1].pitch : 0);
  const int pad = kTilePad * int(sizeof(T)) + 128 + 4 * 128;  // reads past the end, rounding of offset and phases
  const int budget = int(kTileData) / kTileStages / 128 * 128 - nops * pad;
  const int most = std::min(1024, budget / (elems * int(sizeof(T)))) / unit * unit;
  const int64_t grid_max = max_ctas > 0 ? std::min<int64_t>(sms, max_ctas) : sms;
  const int least = std::min(most, std::max(64, std::min(256, 16384 / (elems * int(sizeof(T))) / unit * unit)));
  const int64_t waves = std::max<int64_t>(1, (p.rows_main + grid_max * most - 1) / (grid_max * most));
  const int64_t even = (p.rows_main + grid_max * waves - 1) / (grid_max * waves);
  a.rs = static_cast<int>(std::min<int64_t>(most, std::max<int64_t>(least, (even + unit - 1) / unit * unit)));
  a.boxes = 1;
  if (!phased) {
    a.boxes = (a.rs + 255) / 256;
    a.rs = a.rs / (8 * a.boxes) * (8 * a.boxes);  // equal boxes of whole 8-row groups
  }
  a.row_q = phased ? 1 : 4;
  a.row_t = phased ? 4 : 1;
  int offset = 0;
  for (int o = 0; o < nops; ++o) {
    set_steps(a.x[o], phased, a.rs);
    a.x[o].offset = offset;
    const int data = a.x[o].load == kTilePhases ? 4 * a.x[o].phase_bytes : a.rs * a.x[o].pitch * int(sizeof(T));
    offset += (data + kTilePad * int(sizeof(T)) + 127) / 128 * 128;
  }
  if (a.joint) {
    set_steps(a.x[1], phased, a.rs);
    a.x[1].offset = 0;
    a.x[0].first = a.swap ? j.b_first : j.a_first;
    a.x[1].first = a.swap ? j.a_first : j.b_first;
  }
  a.stage_bytes = offset;
  p.num_chunks = (p.rows_main + a.rs - 1) / a.rs;
  a.p = p;
  if (p.n > 0)
    for (int o = 0; o < nops; ++o)
      if (!encode(a, o)) return TSM_ERROR_CUDA;
  const int64_t grid = std::max<int64_t>(1, std::min(p.num_chunks, grid_max));
  void* args[] = {&a};
  const cudaError_t e = cudaLaunchKernel(v->kernel, dim3(static_cast<unsigned>(grid)), dim3(v->threads), args, v->smem,
                                         stream);
  if (e != cudaSuccess) {
    last_error() = std::string("cudaLaunchKernel(tile): ") + cudaGetErrorString(e);
    return TSM_ERROR_CUDA;
  }
  return TSM_SUCCESS;
}

template tsm_status launch_tile<double>(const Variant*, int, cudaStream_t, PlainArgs<double>, int64_t, int64_t,
                                        int64_t, int64_t, int64_t);
template tsm_status launch_tile<float>(const Variant*, int, cudaStream_t, PlainArgs<float>, int64_t, int64_t, int64_t,
                                       int64_t, int64_t);

}  // namespace tsm
