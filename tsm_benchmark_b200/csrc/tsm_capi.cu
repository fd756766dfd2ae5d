// tsm_capi.cu -- the C ABI (include/tsm.h): argument checks, variant choice,
// grid sizing and launches for the plain FP64 path.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/tsm.h"
#include "tsm_errors.h"
#include "tsm_registry.cuh"
#include "tsm_tile.h"
#include "tsm_tmap.h"

namespace tsm {
namespace {
thread_local std::string g_last_cuda_error;
}  // namespace

std::string& last_error() { return g_last_cuda_error; }

namespace {

tsm_status cuda_fail(cudaError_t e, const char* what) {
  char buf[256];
  std::snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
  g_last_cuda_error = buf;
  return TSM_ERROR_CUDA;
}

// Workspace layout: [counter u32][error u32][group counters u32 x 62][partials].
constexpr size_t kWsHeader = 256;
constexpr int kMaxCtasPerSm = 4;

struct DeviceState {
  int sms = 0;
  std::vector<signed char> attr_done;  // per variant: smem attribute set / failed
  std::vector<int> occupancy;          // per variant: CTAs per SM (0 = unknown)
};

std::mutex g_mu;
std::unordered_map<int, DeviceState> g_devices;

const std::vector<const Variant*>& variants() {
  static const std::vector<const Variant*> all = [] {
    std::vector<const Variant*> v;
    for (int p = 0; p < kVariantPartCount; ++p)
      for (int i = 0; i < kVariantParts[p].count; ++i) v.push_back(&kVariantParts[p].rows[i]);
    return v;
  }();
  return all;
}

tsm_status current_device(int* dev, DeviceState** st) {
  cudaError_t e = cudaGetDevice(dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  std::lock_guard<std::mutex> lk(g_mu);
  DeviceState& s = g_devices[*dev];
  if (s.sms == 0) {
    e = cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, *dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute");
    s.attr_done.assign(variants().size(), 0);
    s.occupancy.assign(variants().size(), 0);
  }
  *st = &s;
  return TSM_SUCCESS;
}

// Sets the dynamic shared-memory limit of a variant once per device and
// caches how many of its CTAs fit on one SM.
tsm_status prepare_variant(DeviceState* st, int idx) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (st->attr_done[idx] == 1) return TSM_SUCCESS;
  if (st->attr_done[idx] == -1) return TSM_ERROR_UNSUPPORTED;
  const Variant* v = variants()[idx];
  cudaError_t e = cudaFuncSetAttribute(v->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(v->smem));
  if (e != cudaSuccess) {
    st->attr_done[idx] = -1;
    return cuda_fail(e, "cudaFuncSetAttribute");
  }
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, v->kernel, v->threads, v->smem);
  if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
  if (occ < 1) {
    st->attr_done[idx] = -1;
    return TSM_ERROR_UNSUPPORTED;
  }
  st->occupancy[idx] = std::min(occ, kMaxCtasPerSm);
  st->attr_done[idx] = 1;
  return TSM_SUCCESS;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// C = A^T A: B is the same matrix as A (same data, pitch and width).
bool is_gram(int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb) {
  return A == B && lda == ldb && m == k;
}

bool applicable(const Variant* v, int dtype, int64_t n, int m, int k, const void* A, int64_t lda, const void* B,
                int64_t ldb) {
  if (v->dtype != dtype) return false;
  if (v->gram && !is_gram(m, k, A, lda, B, ldb)) return false;
  if (v->kind == kKindTile) return (m <= v->wa && k <= v->wb) || (m <= v->wb && k <= v->wa);
  if (v->exact ? (m != v->wa || k != v->wb) : (m > v->wa || k > v->wb)) return false;
  if (v->kind == kKindBulk) {
    if (lda != m || ldb != k) return false;
    if (!aligned16(A) || !aligned16(B)) return false;
  }
  if (v->kind == kKindDmma) {
    // Tensor maps: 16-byte aligned bases and row pitches, 32-bit row
    // coordinates.
    if ((lda * 8) % 16 != 0 || (ldb * 8) % 16 != 0) return false;
    if (!aligned16(A) || !aligned16(B)) return false;
    if (n > static_cast<int64_t>(INT_MAX) - v->rows) return false;
  }
  return true;
}

// Tensor map of a row-major FP64 operand (rows x width, pitch ld elements)
// with boxes of 16 columns x `box_rows` rows and the 128-byte swizzle the
// DMMA kernels read with.
tsm_status encode_operand_map(CUtensorMap* map, const double* base, int64_t rows, int width, int64_t ld,
                              int box_rows) {
  if (!encode_rowmajor_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, base, rows, width, ld, 16, box_rows,
                           CU_TENSOR_MAP_SWIZZLE_128B, &g_last_cuda_error))
    return TSM_ERROR_CUDA;
  return TSM_SUCCESS;
}

// Generated: preferred variant per (m, k, n) from the tuning table.
}  // namespace

extern const char* const kTunedDefaults[];  // "m k nmin name", null-terminated
extern const int kTunedDefaultCount;
extern const char* const kTunedGram[];  // "w nmin name": Gram variants, null-terminated
extern const int kTunedGramCount;

namespace {

int find_variant(const char* name) {
  const auto& vs = variants();
  for (size_t i = 0; i < vs.size(); ++i)
    if (std::strcmp(vs[i]->name, name) == 0) return static_cast<int>(i);
  return -1;
}

// The tuning tables, read once (every call used to scan their text and look
// the names up: 15 us of a 25 us call): per width pair the entries by rising
// nmin, table order for equal ones.
struct TunedEntry {
  long long nmin;
  int variant;
};
struct TunedTables {
  std::vector<TunedEntry> plain[65][65];
  std::vector<TunedEntry> gram[65];
};

const TunedTables& tuned() {
  static const TunedTables* tables = [] {
    auto* t = new TunedTables;
    auto add = [](std::vector<TunedEntry>& v, long long nmin, int variant) {
      const auto at = std::upper_bound(v.begin(), v.end(), nmin,
                                       [](long long a, const TunedEntry& e) { return a < e.nmin; });
      v.insert(at, TunedEntry{nmin, variant});
    };
    for (int i = 0; i < kTunedDefaultCount; ++i) {
      int m = 0, k = 0;
      long long nmin = 0;
      char name[96] = {0};
      if (std::sscanf(kTunedDefaults[i], "%d %d %lld %95s", &m, &k, &nmin, name) != 4) continue;
      const int idx = find_variant(name);
      if (idx >= 0 && m >= 1 && m <= 64 && k >= 1 && k <= 64) add(t->plain[m][k], nmin, idx);
    }
    for (int i = 0; i < kTunedGramCount; ++i) {
      int w = 0;
      long long nmin = 0;
      char name[96] = {0};
      if (std::sscanf(kTunedGram[i], "%d %lld %95s", &w, &nmin, name) != 3) continue;
      const int idx = find_variant(name);
      if (idx >= 0 && w >= 1 && w <= 64 && variants()[idx]->gram) add(t->gram[w], nmin, idx);
    }
    return t;
  }();
  return *tables;
}

bool pitched_prefers_tile(bool f64, int64_t n, int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb);

// The entry with the largest nmin <= n, if it holds for the operands, or -1.  The
// table was timed on dense, aligned operands.  Others keep its choice among the
// tensor-box kernels, which load any 16-byte pitch as they load dense rows, and
// a tile kernel where the rule for pitched rows agrees; the bulk kernels do not
// take them, and an entry for fewer rows, or a kernel that was the best on
// dense rows, says nothing about theirs (narrow slices of 8 x 4 at 3 x 10^6 rows
// took the tile kernel that had won on 4096 dense ones: 123 us, direct 71).
int tuned_variant(const std::vector<TunedEntry>& entries, int dtype, int64_t n, int m, int k, const void* A,
                  int64_t lda, const void* B, int64_t ldb, bool tiles = true) {
  const bool dense = lda == m && ldb == k && aligned16(A) && aligned16(B);
  for (auto e = entries.rbegin(); e != entries.rend(); ++e) {
    const Variant* v = variants()[e->variant];
    if (e->nmin > n || (!tiles && v->kind == kKindTile)) continue;
    if (!applicable(v, dtype, n, m, k, A, lda, B, ldb)) return -1;
    const bool holds = dense || v->kind == kKindDmma ||
                       (v->kind == kKindTile && pitched_prefers_tile(dtype == kF64, n, m, k, A, lda, B, ldb));
    return holds ? e->variant : -1;
  }
  return -1;
}

int first_in_table(int dtype, int64_t n, int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb) {
  const auto& vs = variants();
  for (size_t i = 0; i < vs.size(); ++i)
    if (vs[i]->kind != kKindTile && applicable(vs[i], dtype, n, m, k, A, lda, B, ldb)) return static_cast<int>(i);
  return -1;
}

// The tile variant (tsm_tile.cuh) with the least capacities for m x k.
int tile_variant(int dtype, int m, int k) {
  static const std::vector<int> index = [] {
    std::vector<int> v(2 * 8 * 8, -1);
    const auto& vs = variants();
    for (size_t i = 0; i < vs.size(); ++i)
      if (vs[i]->kind == kKindTile)
        v[(vs[i]->dtype * 8 + vs[i]->wa / 8 - 1) * 8 + vs[i]->wb / 8 - 1] = static_cast<int>(i);
    return v;
  }();
  return index[(dtype * 8 + (std::max(m, k) - 1) / 8) * 8 + (std::min(m, k) - 1) / 8];
}

// The SIMT kernels are compiled for powers of two: the columns one works on for w.
int padded_width(int w) {
  int p = 1;
  while (p < w) p *= 2;
  return p;
}

// Whether an m x k product that has no tuned entry runs on the tile kernel
// rather than on `v`, the first variant in the table that takes it.
//
// FP32 squares compiled exactly stay, but for few rows of wide ones, where
// their long chunks leave SMs idle: SIMT -> tile, us, 16 x 16 at n = 1000 9.2 ->
// 5.8, at 2^18 15.4 -> 13.5, at 2^20 28.3 -> 30.7; 32 x 32 at 2^16 19.9 -> 17.1;
// 64 x 64 at 2^16 49.6 -> 41.9, at 2^20 254 -> 293; 8 x 8 at 2^18 9.5 -> 11.0.
//
// The rest run on SIMT register tiles of a larger capacity, over bulk copies of
// contiguous rows or over direct loads.
//
// Contiguous rows.  The SIMT capacity kernels pad to powers of two, load one
// element at a time and meet bank conflicts at even widths; they keep up with
// HBM only on narrow rows, where the tile kernel's 4-row steps bound it.
// B200, 400 MB of operands, SIMT -> tile, us: FP64 1 x 1 60 -> 152, 3 x 3
// 63 -> 66, 8 x 1 62 -> 64, 3 x 5 67 -> 62, 5 x 5 82 -> 64, 13 x 13 87 -> 64,
// 24 x 24 179 -> 64, 37 x 37 463 -> 85, 63 x 63 352 -> 139 (FP64-bound).
// Below 64 MB launch and cross-CTA sum decide: 3 x 7 at n = 200001 9.4 -> 10.7,
// 5 x 8 at 1000 5.2 -> 5.8, 13 x 13 at 1000 7.7 -> 5.4, 64 x 5 8.6 -> 6.0.
// FP32, 300 MB.  The tile kernel widens to FP64, and the FP64 pipe bounds it on
// narrow rows: 4 x 4 50 -> 77, 12 x 4 52 -> 62, 63 x 3 51 -> 56.  The SIMT kernels fall
// behind where a thread holds 8 columns of either side (from 5 on: 5 x 5 79 -> 69, 6
// x 20 87 -> 60, 13 x 8 61 -> 54), where rows of a multiple of 32 bytes put their
// lanes on the same banks (16 x 3 70 -> 57, 40 x 2 78 -> 56, but 17 x 3 70 -> 72), and
// where a quarter of a side padded to 64 is padding (36 x 3 74 -> 58, 48 x 3 the
// last).  Padded to 32 the two are within 15 % (17 x 3 70 -> 72, 31 x 3 51 -> 57) and the
// FP64 sums decide: 25 x 3 at 2^22 rows is 9e-9 off in one, 1.3e-7 in FP32.
//
// Strided or unaligned rows: pitched_prefers_tile.
bool prefers_tile(const Variant* v, int64_t n, int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb) {
  const int lo = std::min(m, k), hi = std::max(m, k);
  const bool f64 = v->dtype == kF64;
  if (v->exact) return !f64 && v->kind == kKindBulk && lo >= 16 && n * (m + k) <= int64_t(1) << 23;
  if (v->kind == kKindBulk && !is_gram(m, k, A, lda, B, ldb))
    return f64 ? m * k >= 100 || m + k >= 18 || (m + k >= 10 && n * (m + k) >= int64_t(1) << 23)
               : lo >= 5 || (hi >= 16 && hi % 8 == 0) || (lo >= 3 && hi > 16 && hi <= 48);
  return pitched_prefers_tile(f64, n, m, k, A, lda, B, ldb);
}

// The same for strided or unaligned rows (and A^T A, whose rows are loaded once).
// The direct kernels issue a load per element and lane and pad widths to powers
// of two; tensor boxes cost by the row, so narrow slices that are loaded apart
// stay direct: SIMT -> tile, us at 300 MB, 16-byte pitches, 8 x 8 91 -> 94, 4 x
// 16 83 -> 86, 8 x 16 87 -> 81, 7 x 20 116 -> 73; odd pitches or unaligned bases,
// 13 x 8 80 -> 92, 16 x 4 63 -> 78, 8 x 16 74 -> 55..67, 7 x 20 110 -> 71, 13 x 13
// 174 -> 84, 1 x 64 75 -> 50.  Within L2 the direct kernels' loads wait on its
// latency: at 6 MB 8 x 4 10.4 -> 8.6, 16 x 4 10.0 -> 8.3, 8 x 8 FP32 10.3 -> 8.2.  At
// 0.5 MB launch and sum decide: 1 x 64 4.8 -> 5.4, 8 x 16 5.7 -> 6.2.
// Neighbouring slices come as one: FP64 4 x 8 54 -> 50, 8 x 8 75 -> 50, 40 x 20
// 720 -> 68; FP32 8 x 3 74 -> 76, 5 x 5 118 -> 82, 40 x 1 81 -> 74.  In phases (an
// odd pitch that the columns do not fill) they take four boxes for one: 4 x 4 58
// -> 75, 8 x 4 57 -> 93, 8 x 8 59 -> 56; within L2 the boxes keep up (60 MB 4 x 4
// 1.2 times slower, 20 MB as fast, 6 MB 9.9 -> 8.3).  FP32 4 x 8 63 -> 80 stays, with
// its sums in FP64.  A^T A of 5 and 6 columns, boxes of 12 half filled: 300 MB 171
// -> 228 and 145 -> 191, 60 MB as fast or faster.  On a
// thousand rows narrow ones cost the same or less direct: 3 x 5 4.8 -> 5.1, FP32 5
// x 8 4.8 -> 5.7; 13 x 13 7.0 -> 5.5.
bool pitched_prefers_tile(bool f64, int64_t n, int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb) {
  const int lo = std::min(m, k), hi = std::max(m, k);
  const int64_t e = f64 ? 8 : 4;
  const int simt_work = padded_width(m) * padded_width(k);  // products a row
  const bool small = m * k < 100 && n < (1 << 14);
  if (is_gram(m, k, A, lda, B, ldb))  // one load for both operands
    return m >= 5 && !small && (!f64 || m > 6 || n * m * e < int64_t(128) << 20);
  bool phases = false;
  if (tile_joint(A, m, lda, B, k, ldb, static_cast<size_t>(e), &phases)) {
    if (f64 && phases && simt_work < 64 && n * (m + k) * e >= int64_t(32) << 20) return false;
    return !small && (f64 ? m + k >= 8 : (lo >= 3 && m * k >= 25) || hi >= 40);
  }
  const int64_t elems = n * (m + k);
  if (f64 && simt_work < 256 && elems < (1 << 17)) return false;
  if (simt_work >= 32 && elems >= (1 << 18) && elems * e < (16 << 20)) return true;
  const bool maps = aligned16(A) && aligned16(B) && lda * e % 16 == 0 && ldb * e % 16 == 0;
  return m * k >= (maps ? 64 : 128) || m + k >= 28;
}

int default_variant(int dtype, int64_t n, int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb,
                    bool tiles = true) {
  const auto& vs = variants();
  // 0. C = A^T A: a Gram variant (A streamed once): the tuned one, else the
  //    first in table order.
  if (is_gram(m, k, A, lda, B, ldb)) {
    const int best = tuned_variant(tuned().gram[m], dtype, n, m, k, A, lda, B, ldb);
    if (best >= 0) return best;
    for (size_t i = 0; i < vs.size(); ++i)
      if (vs[i]->gram && applicable(vs[i], dtype, n, m, k, A, lda, B, ldb)) return static_cast<int>(i);
  }
  // 1. The tuning table.
  const int best = tuned_variant(tuned().plain[m][k], dtype, n, m, k, A, lda, B, ldb, tiles);
  if (best >= 0) return best;
  // 2. Table order: the generator lists exact variants first, then capacity
  //    bulk variants from the smallest capacity up, then direct ones; the tile
  //    kernel in place of a capacity one where it is faster.
  const int idx = first_in_table(dtype, n, m, k, A, lda, B, ldb);
  if (tiles && idx >= 0 && prefers_tile(vs[idx], n, m, k, A, lda, B, ldb)) return tile_variant(dtype, m, k);
  return idx;
}

// Rows the bulk kernels stream: every copy of rows * width elements must be a
// multiple of 16 bytes, so up to three final rows may be left to the epilogue.
int64_t bulk_rows(int64_t n, int m, int k, size_t esize) {
  auto need = [esize](int w) {
    const size_t bytes = static_cast<size_t>(w) * esize;
    size_t g = 16;
    size_t b = bytes;
    while (b) {
      const size_t t = g % b;
      g = b;
      b = t;
    }
    return static_cast<int64_t>(16 / g);
  };
  const int64_t ra = need(m), rb = need(k);
  const int64_t r0 = ra > rb ? ra : rb;  // both are powers of two
  return n - n % r0;
}

tsm_status check_args(int64_t n, int m, int k, const void* A, int64_t lda, const void* B, int64_t ldb,
                      const void* C, int64_t ldc) {
  if (n < 0 || m < 1 || k < 1 || m > 64 || k > 64) return TSM_ERROR_INVALID_VALUE;
  if (lda < m || ldb < k || ldc < k) return TSM_ERROR_INVALID_VALUE;
  if (C == nullptr) return TSM_ERROR_INVALID_VALUE;
  if (n > 0 && (A == nullptr || B == nullptr)) return TSM_ERROR_INVALID_VALUE;
  return TSM_SUCCESS;
}

size_t workspace_bytes_for(int sms, int m, int k) {
  return kWsHeader + static_cast<size_t>(sms) * kMaxCtasPerSm * m * k * sizeof(double);
}

// Rows the main loop streams, chunk count and grid for variant v (p.n, p.m,
// p.k set).  Bulk: 16-byte copies leave up to three final rows of an
// odd-width operand to the reduction epilogue.  DMMA: the tensor maps
// zero-fill past row n, so every row is streamed.
template <typename T>
int64_t plan_grid(const Variant* v, const DeviceState* st, int idx, PlainArgs<T>& p) {
  const int64_t max_grid = static_cast<int64_t>(st->sms) * st->occupancy[idx];
  if (v->kind == kKindBulk || v->kind == kKindDmma) {
    p.rows_main = v->kind == kKindBulk ? bulk_rows(p.n, p.m, p.k, sizeof(T)) : p.n;
    p.num_chunks = (p.rows_main + v->rows - 1) / v->rows;
    return std::max<int64_t>(1, std::min<int64_t>(p.num_chunks, max_grid));
  }
  p.rows_main = p.n;
  p.num_chunks = 0;
  const int tiles = (v->wa / v->ta) * (v->wb / v->tb);
  const int64_t row_groups = v->threads / tiles;
  return std::max<int64_t>(1, std::min<int64_t>((p.n + row_groups - 1) / row_groups, max_grid));
}

template <typename T>
void set_workspace(PlainArgs<T>& p, void* ws) {
  unsigned char* base = static_cast<unsigned char*>(ws);
  p.counter = reinterpret_cast<unsigned*>(base);
  p.error = reinterpret_cast<unsigned*>(base) + 1;
  p.partials = reinterpret_cast<double*>(base + kWsHeader);
}

template <typename T>
tsm_status launch_variant(const Variant* v, const PlainArgs<T>& p, int64_t grid, cudaStream_t stream) {
  cudaError_t e;
  if (v->kind == kKindDmma) {
    if constexpr (sizeof(T) == 8) {
      DmmaArgs d{};
      d.p = p;
      d.p.symmetric = is_gram(p.m, p.k, p.A, p.lda, p.B, p.ldb) ? 1 : 0;
      if (p.n > 0) {  // n = 0: no chunks, the maps are never read
        const int box_rows = dmma_box_rows(v->rows);
        tsm_status s = encode_operand_map(&d.ta, p.A, p.n, p.m, p.lda, box_rows);
        if (s == TSM_SUCCESS && !v->gram) s = encode_operand_map(&d.tb, p.B, p.n, p.k, p.ldb, box_rows);
        if (s != TSM_SUCCESS) return s;
      }
      void* args[] = {&d};
      e = cudaLaunchKernel(v->kernel, dim3(static_cast<unsigned>(grid)), dim3(v->threads), args, v->smem, stream);
    } else {
      return TSM_ERROR_UNSUPPORTED;
    }
  } else {
    PlainArgs<T> q = p;
    q.symmetric = is_gram(p.m, p.k, p.A, p.lda, p.B, p.ldb) ? 1 : 0;  // C = A^T A: written exactly symmetric
    void* args[] = {&q};
    e = cudaLaunchKernel(v->kernel, dim3(static_cast<unsigned>(grid)), dim3(v->threads), args, v->smem, stream);
  }
  if (e != cudaSuccess) return cuda_fail(e, "cudaLaunchKernel");
  return TSM_SUCCESS;
}

template <typename T>
tsm_status launch_plain(cudaStream_t stream, int64_t n, int m, int k, const T* A, int64_t lda, const T* B,
                        int64_t ldb, T* C, int64_t ldc, int accumulate, void* ws, size_t ws_bytes, int variant,
                        int64_t max_ctas = 0) {
  constexpr int dtype = DTypeOf<T>::value;
  tsm_status s = check_args(n, m, k, A, lda, B, ldb, C, ldc);
  if (s != TSM_SUCCESS) return s;
  int dev = 0;
  DeviceState* st = nullptr;
  if ((s = current_device(&dev, &st)) != TSM_SUCCESS) return s;
  if (ws == nullptr || ws_bytes < workspace_bytes_for(st->sms, m, k) || !aligned16(ws))
    return TSM_ERROR_WORKSPACE;

  const auto& vs = variants();
  int idx = variant;
  if (idx < 0) {
    idx = default_variant(dtype, n, m, k, A, lda, B, ldb);
    if (idx < 0) return TSM_ERROR_UNSUPPORTED;
  } else if (idx >= static_cast<int>(vs.size()) || !applicable(vs[idx], dtype, n, m, k, A, lda, B, ldb)) {
    return TSM_ERROR_UNSUPPORTED;
  }
  if ((s = prepare_variant(st, idx)) != TSM_SUCCESS) return s;
  const Variant* v = vs[idx];

  PlainArgs<T> p{};
  p.A = A;
  p.B = B;
  p.C = C;
  p.n = n;
  p.m = m;
  p.k = k;
  p.lda = lda;
  p.ldb = ldb;
  p.ldc = ldc;
  p.accumulate = accumulate ? 1 : 0;
  set_workspace(p, ws);

  if (v->kind == kKindTile) return launch_tile<T>(v, st->sms, stream, p, lda, 1, ldb, 1, max_ctas);
  int64_t grid = plan_grid(v, st, idx, p);
  if (max_ctas > 0) grid = std::min(grid, max_ctas);  // every kernel deals its rows over any grid >= 1
  return launch_variant(v, p, grid, stream);
}

}  // namespace

tsm_status run_tile_f64(cudaStream_t stream, int64_t n, int m, int k, const double* A, int64_t a_row, int64_t a_col,
                        const double* B, int64_t b_row, int64_t b_col, double* C, int64_t ldc, int accumulate,
                        void* ws, size_t ws_bytes) {
  int dev = 0;
  DeviceState* st = nullptr;
  tsm_status s = current_device(&dev, &st);
  if (s != TSM_SUCCESS) return s;
  if (ws == nullptr || ws_bytes < workspace_bytes_for(st->sms, m, k) || !aligned16(ws)) return TSM_ERROR_WORKSPACE;
  const int idx = tile_variant(kF64, m, k);
  if (idx < 0) return TSM_ERROR_UNSUPPORTED;
  if ((s = prepare_variant(st, idx)) != TSM_SUCCESS) return s;
  PlainArgs<double> p{};
  p.A = A;
  p.B = B;
  p.C = C;
  p.n = n;
  p.m = m;
  p.k = k;
  p.ldc = ldc;
  p.accumulate = accumulate ? 1 : 0;
  set_workspace(p, ws);
  return launch_tile<double>(variants()[idx], st->sms, stream, p, a_row, a_col, b_row, b_col, 0);
}

namespace {

// ------------------------------------------------------- timeout self-test
// One thread waits on an mbarrier that nothing ever arrives on, through the
// same bounded wait every pipeline uses, then records the timeout in the
// workspace's error word -- the failure path of the kernels, exercised on
// purpose (a wait that runs out; no fault, no trap).
__global__ void selftest_wait_kernel(unsigned* error, uint64_t limit_ns) {
  __shared__ uint64_t bar;
  __shared__ int abort;
  if (threadIdx.x == 0) {
    dev::mbar_init(&bar, 1);
    abort = 0;
    dev::fence_mbar_init();
    if (!dev::mbar_wait_for(&bar, 0, &abort, limit_ns)) atomicOr(error, dev::kErrTimeout);
  }
}

// ----------------------------------------------------------------- fills
__global__ void fill_uniform_kernel(double* x, int64_t count, uint64_t seed, uint64_t stream_id) {
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += step) {
    uint64_t z = seed + ((stream_id << 40) + static_cast<uint64_t>(i) + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const double u = static_cast<double>(z >> 11) * 0x1.0p-53;
    x[i] = 2.0 * u - 1.0;
  }
}

}  // namespace
}  // namespace tsm

using namespace tsm;

extern "C" {

int tsm_version(void) { return 100; }

const char* tsm_status_string(tsm_status s) {
  switch (s) {
    case TSM_SUCCESS: return "success";
    case TSM_ERROR_INVALID_VALUE: return "invalid value (shape, pointer or leading dimension)";
    case TSM_ERROR_WORKSPACE: return "workspace missing, unaligned or too small";
    case TSM_ERROR_CUDA: return "CUDA runtime error";
    case TSM_ERROR_UNSUPPORTED: return "no compiled variant supports this request";
    case TSM_ERROR_DEVICE_TIMEOUT: return "a kernel gave up a bounded wait";
  }
  return "unknown status";
}

const char* tsm_last_cuda_error(void) { return g_last_cuda_error.c_str(); }

size_t tsm_gemm_tn_workspace_size(int64_t n, int m, int k) {
  (void)n;
  if (m < 1 || k < 1 || m > 64 || k > 64) return 0;
  int dev = 0;
  DeviceState* st = nullptr;
  if (current_device(&dev, &st) != TSM_SUCCESS) return 0;
  return workspace_bytes_for(st->sms, m, k);
}

tsm_status tsm_gemm_tn_f64(tsm_stream_t stream, int64_t n, int m, int k, const double* A, int64_t lda,
                           const double* B, int64_t ldb, double* C, int64_t ldc, int accumulate, void* workspace,
                           size_t workspace_bytes) {
  return launch_plain<double>(static_cast<cudaStream_t>(stream), n, m, k, A, lda, B, ldb, C, ldc, accumulate,
                              workspace, workspace_bytes, -1);
}

tsm_status tsm_gram_f64(tsm_stream_t stream, int64_t n, int m, const double* A, int64_t lda, double* C, int64_t ldc,
                        int accumulate, void* workspace, size_t workspace_bytes) {
  return launch_plain<double>(static_cast<cudaStream_t>(stream), n, m, m, A, lda, A, lda, C, ldc, accumulate,
                              workspace, workspace_bytes, -1);
}

tsm_status tsm_gemm_tn_f64_variant(tsm_stream_t stream, int64_t n, int m, int k, const double* A, int64_t lda,
                                   const double* B, int64_t ldb, double* C, int64_t ldc, int accumulate,
                                   void* workspace, size_t workspace_bytes, int variant) {
  return launch_plain<double>(static_cast<cudaStream_t>(stream), n, m, k, A, lda, B, ldb, C, ldc, accumulate,
                              workspace, workspace_bytes, variant);
}

tsm_status tsm_gemm_tn_f64_launch(tsm_stream_t stream, int64_t n, int m, int k, const double* A, int64_t lda,
                                  const double* B, int64_t ldb, double* C, int64_t ldc, int accumulate,
                                  void* workspace, size_t workspace_bytes, int variant, int64_t max_ctas) {
  return launch_plain<double>(static_cast<cudaStream_t>(stream), n, m, k, A, lda, B, ldb, C, ldc, accumulate,
                              workspace, workspace_bytes, variant, max_ctas);
}

tsm_status tsm_gemm_tn_f32(tsm_stream_t stream, int64_t n, int m, int k, const float* A, int64_t lda,
                           const float* B, int64_t ldb, float* C, int64_t ldc, int accumulate, void* workspace,
                           size_t workspace_bytes) {
  return launch_plain<float>(static_cast<cudaStream_t>(stream), n, m, k, A, lda, B, ldb, C, ldc, accumulate,
                             workspace, workspace_bytes, -1);
}

tsm_status tsm_gemm_tn_f32_variant(tsm_stream_t stream, int64_t n, int m, int k, const float* A, int64_t lda,
                                   const float* B, int64_t ldb, float* C, int64_t ldc, int accumulate,
                                   void* workspace, size_t workspace_bytes, int variant) {
  return launch_plain<float>(static_cast<cudaStream_t>(stream), n, m, k, A, lda, B, ldb, C, ldc, accumulate,
                             workspace, workspace_bytes, variant);
}

int tsm_gemm_tn_default_variant(int dtype, int64_t n, int m, int k, const void* A, int64_t lda, const void* B,
                                int64_t ldb) {
  if (dtype != kF64 && dtype != kF32) return -1;
  if (check_args(n, m, k, A, lda, B, ldb, A ? A : B, k) != TSM_SUCCESS) return -1;
  return default_variant(dtype, n, m, k, A, lda, B, ldb);
}

int tsm_variant_count(void) { return static_cast<int>(variants().size()); }

tsm_status tsm_variant_get_info(int index, tsm_variant_info* info) {
  if (index < 0 || index >= tsm_variant_count() || info == nullptr) return TSM_ERROR_INVALID_VALUE;
  const Variant* v = variants()[index];
  std::memset(info, 0, sizeof(*info));
  std::strncpy(info->name, v->name, sizeof(info->name) - 1);
  info->kind = v->kind;
  info->dtype = v->dtype;
  info->wa = v->wa;
  info->wb = v->wb;
  info->ta = v->ta;
  info->tb = v->tb;
  info->exact = v->exact;
  info->threads = v->threads;
  info->stages = v->stages;
  info->rows = v->rows;
  info->unroll = v->unroll;
  info->smem_bytes = v->smem;
  info->gram = v->gram;
  return TSM_SUCCESS;
}

tsm_status tsm_selftest_wait_timeout(tsm_stream_t stream, void* workspace, size_t workspace_bytes,
                                     unsigned limit_us) {
  if (workspace == nullptr || workspace_bytes < kWsHeader || !aligned16(workspace)) return TSM_ERROR_WORKSPACE;
  if (limit_us == 0 || limit_us > 2000000u) return TSM_ERROR_INVALID_VALUE;
  unsigned* error = reinterpret_cast<unsigned*>(workspace) + 1;
  selftest_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(error, uint64_t(limit_us) * 1000u);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "selftest_wait_kernel");
  return TSM_SUCCESS;
}

tsm_status tsm_workspace_check(tsm_stream_t stream, void* workspace, unsigned* bits) {
  if (workspace == nullptr) return TSM_ERROR_WORKSPACE;
  unsigned host = 0;
  unsigned* err = static_cast<unsigned*>(workspace) + 1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(&host, err, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(unsigned), s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "tsm_workspace_check");
  if (bits) *bits = host;
  return host ? TSM_ERROR_DEVICE_TIMEOUT : TSM_SUCCESS;
}

tsm_status tsm_fill_uniform_f64(tsm_stream_t stream, double* x, int64_t count, uint64_t seed, uint64_t stream_id) {
  if (count < 0 || (count > 0 && x == nullptr)) return TSM_ERROR_INVALID_VALUE;
  if (count == 0) return TSM_SUCCESS;
  int dev = 0;
  DeviceState* st = nullptr;
  tsm_status s = current_device(&dev, &st);
  if (s != TSM_SUCCESS) return s;
  const int64_t blocks = std::min<int64_t>((count + 255) / 256, static_cast<int64_t>(st->sms) * 16);
  fill_uniform_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, count, seed,
                                                                                                    stream_id);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fill_uniform_kernel");
  return TSM_SUCCESS;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free entry point: tsm_gemm_tn_f64_noalloc.
//
// Some callers cannot hand the library a workspace.  A plugin loaded into a
// host program that owns every device allocation (its own pool, no
// cudaMalloc from plug-ins), or a latency-bound loop where a cudaMalloc --
// which may synchronise the whole device -- is not allowed after start-up,
// can still call this.  The scratch the kernels need (a launch counter, an
// error word and one m x k partial per CTA) lives in the file-scope array
// below instead, which every GPU that loads this library holds until the
// process exits.
//
// Limits and sharing:
//   * kStaticScratchBytes (4 MiB) bounds a call: 256 B of header plus
//     (CTAs launched) * m * k * 8 B of partials.  A request that would need
//     more returns TSM_ERROR_WORKSPACE and runs nothing.
//   * All calls on a device share the one array and it keeps whatever the
//     last call left.  The launch counters must start at zero, so each call
//     zeroes them (stream-ordered) before its launch.  Calls that overlap on
//     the GPU (different streams, other threads) race on the array and give
//     wrong results: serialise them.
//   * The first call on each device looks the array's device address up
//     (cudaGetSymbolAddress, with that device current); make that first call
//     before any stream capture.  Like every per-device state of the
//     library, that address does not survive cudaDeviceReset: do not reset a
//     device while the library is in use on it.
//   * A kernel that gives up a bounded wait sets a bit in the array's error
//     word; tsm_noalloc_check reads and clears it.
// ---------------------------------------------------------------------------
namespace tsm {
namespace {
constexpr size_t kStaticScratchBytes = size_t(4) << 20;
constexpr int kStaticScratchDevices = 64;
}  // namespace
}  // namespace tsm

static __device__ __align__(256) unsigned char tsm_static_scratch[tsm::kStaticScratchBytes];

namespace tsm {
namespace {

std::mutex g_static_mu;
void* g_static_ptr[kStaticScratchDevices] = {};

// Device address of tsm_static_scratch on device `dev` (current), looked up
// once per device.  In host code the array's name is only a host-side
// stand-in, never a device address.
tsm_status static_scratch(int dev, void** out) {
  if (dev < 0 || dev >= kStaticScratchDevices) return TSM_ERROR_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (g_static_ptr[dev] == nullptr) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, tsm_static_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(tsm_static_scratch)");
    g_static_ptr[dev] = p;
  }
  *out = g_static_ptr[dev];
  return TSM_SUCCESS;
}

}  // namespace
}  // namespace tsm

extern "C" tsm_status tsm_gemm_tn_f64_noalloc(tsm_stream_t stream, int64_t n, int m, int k, const double* A,
                                              int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc,
                                              int accumulate) {
  using namespace tsm;
  tsm_status s = check_args(n, m, k, A, lda, B, ldb, C, ldc);
  if (s != TSM_SUCCESS) return s;
  int dev = 0;
  DeviceState* st = nullptr;
  if ((s = current_device(&dev, &st)) != TSM_SUCCESS) return s;
  void* scratch = nullptr;
  if ((s = static_scratch(dev, &scratch)) != TSM_SUCCESS) return s;

  PlainArgs<double> p{};
  p.A = A;
  p.B = B;
  p.C = C;
  p.n = n;
  p.m = m;
  p.k = k;
  p.lda = lda;
  p.ldb = ldb;
  p.ldc = ldc;
  p.accumulate = accumulate ? 1 : 0;
  // What the array holds is decided by the grid of the SIMT or exact variant;
  // the tile kernel, where it takes that one's place, runs on a grid that fits.
  int idx = default_variant(kF64, n, m, k, A, lda, B, ldb, false);
  if (idx < 0) return TSM_ERROR_UNSUPPORTED;
  if ((s = prepare_variant(st, idx)) != TSM_SUCCESS) return s;
  const int64_t grid = plan_grid(variants()[idx], st, idx, p);
  const size_t per_cta = static_cast<size_t>(m) * k * sizeof(double);
  if (kWsHeader + static_cast<size_t>(grid) * per_cta > kStaticScratchBytes) return TSM_ERROR_WORKSPACE;
  const int tile = default_variant(kF64, n, m, k, A, lda, B, ldb);
  if (variants()[tile]->kind == kKindTile) {
    idx = tile;
    if ((s = prepare_variant(st, idx)) != TSM_SUCCESS) return s;
  }
  const Variant* v = variants()[idx];
  set_workspace(p, scratch);

  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(p.counter, 0, sizeof(unsigned), cs);
  if (e == cudaSuccess) e = cudaMemsetAsync(p.counter + 2, 0, kWsHeader - 2 * sizeof(unsigned), cs);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(static scratch counters)");
  if (v->kind == kKindTile)
    return launch_tile<double>(v, st->sms, cs, p, lda, 1, ldb, 1,
                               static_cast<int64_t>((kStaticScratchBytes - kWsHeader) / per_cta));
  return launch_variant(v, p, grid, cs);
}

// Reads and clears the error word of the static scratch: the counterpart of
// tsm_workspace_check for tsm_gemm_tn_f64_noalloc, whose kernels record a
// bounded wait that ran out there instead of in a caller's workspace.  The
// word is sticky across calls until read.  Allocates nothing.
extern "C" tsm_status tsm_noalloc_check(tsm_stream_t stream, unsigned* bits) {
  using namespace tsm;
  int dev = 0;
  DeviceState* st = nullptr;
  tsm_status s = current_device(&dev, &st);
  if (s != TSM_SUCCESS) return s;
  void* scratch = nullptr;
  if ((s = static_scratch(dev, &scratch)) != TSM_SUCCESS) return s;
  return tsm_workspace_check(stream, scratch, bits);
}
