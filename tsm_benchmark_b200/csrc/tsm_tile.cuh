// tsm_tile.cuh -- C (m x k) = A^T B for ANY widths up to 64, any element
// strides and any alignment, FP64 or FP32 storage, on the FP64 tensor cores
// (mma.sync m8n8k4 .f64).  The kernels of tsm_dmma.cuh take widths that are
// multiples of 16, those of tsm_plain.cuh are fastest on the widths they were
// compiled for; this one takes the rest: widths like 24, 37 or 13, column
// slices, odd pitches, operands of different layouts.
//
// Tiles.  Columns are padded to 8 x 8 tiles of C only in the arithmetic: TA x
// TB tiles for widths up to 8 TA and 8 TB.  A column beyond the width holds
// whatever lies in shared memory there and only ever reaches entries of C
// that are not written, so nothing is masked in the row loop (rows are, in
// the one partial chunk at the end).
//
// Loads.  Every operand has its own way into shared memory, picked on the
// host (tsm_tile.cu), so that one kernel serves every pair of layouts:
//   * kTileBulk   -- contiguous rows: one 1-D bulk copy per chunk, shared
//                    pitch = width;
//   * kTileTma    -- 16-byte row pitch and base: 2-D tensor boxes of `pitch`
//                    columns, the ones past the width zero-filled by the TMA
//                    unit;
//   * kTilePhases -- row-major with any pitch and base, which one tensor map
//                    cannot describe: rows q, q + 4, q + 8, ... (phase q of
//                    4) have a pitch of 4 ld elements, always a multiple of
//                    16 bytes, so each phase gets a map of its own, based at
//                    the 16-byte boundary at or before its first row
//                    (shift[q] elements before it), and a part of the stage;
//   * kTileRows / kTileCols -- anything else: the producer warps copy element
//                    by element with cp.async, lanes along the operand's
//                    shorter stride (columns or rows).
// Operands that are (nearly) neighbouring column blocks of one row-major
// matrix -- a basis and the vectors after it, or B = A -- are loaded as one,
// columns from the first of the two to the last: whole rows where the blocks
// fill them, and half the tensor-box rows, which bound narrow slices.
//
// Row order.  A k-step's four rows (one per lane tq) may be any four, the same
// in both operands: rows 4 ks + tq, or, where an operand comes in phases, the
// rows q + 16 j + 4 tq of phase q = ks mod 4, j = ks / 4.  Each operand's
// address is linear in (q, j, tq) either way.
//
// Bank conflicts.  With FP64 the 16 lanes of a half-warp read 4 rows x 4
// columns and hit 16 different bank pairs when rows are 4 mod 8 elements
// apart, the pitch of the padded loads (in phases: consecutive rows of one
// phase; the other operand's rows are then 4 pitches apart and its pitch odd).
// A 1-D copy has no choice of pitch: odd widths cost 2-way conflicts, which
// stay below the HBM time of their rows.
//
// Warps.  8 consumer warps = R regions of MT x NT tiles x S row slots; 4
// producer warps (one issues the TMA copies, all four gather).
//
// Reduction, waits and errors as in tsm_plain.cuh.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "tsm_device.cuh"
#include "tsm_plain.cuh"

namespace tsm {

enum TileLoad : int { kTileBulk = 0, kTileTma = 1, kTilePhases = 2, kTileRows = 3, kTileCols = 4 };

constexpr int kTileStages = 3;
constexpr int kTileConsumers = 8, kTileProducers = 4;
constexpr int kTileThreads = 32 * (kTileConsumers + kTileProducers);
constexpr size_t kTileData = 224 * 1024;  // ring, then the reduction sheets
constexpr size_t kTileSmem = 128 + kTileData + 2 * kTileStages * sizeof(uint64_t) + 16;
// Elements past a chunk's last row that its padded columns may reach.
constexpr int kTilePad = 72;  // up to 63 columns and a phase's shift of 3

template <typename T>
struct TileOperand {
  const T* base;
  int64_t s_row, s_col;  // element strides
  int w;                 // columns loaded
  int cols;              // columns of the operand
  int pitch;             // elements between rows in shared memory
  int load;              // TileLoad
  int offset;            // bytes from the stage's start to where it is loaded
  int first;             // column of the load that is the operand's first
  int q_step, j_step, t_step;  // elements between k-steps of one j, between j, between lanes tq
  int phase_bytes;       // kTilePhases: bytes between the phases' parts of the stage
  unsigned char shift[4];  // kTilePhases: elements in front of a phase's rows
};

template <typename T>
struct TileArgs {
  PlainArgs<T> p;       // num_chunks = ceil(rows_main / rs)
  TileOperand<T> x[2];  // the operand with TA tiles, then the one with TB
  int rs;               // rows per chunk, a multiple of 8 (of 16 in phases)
  int boxes;            // kTileTma: tensor boxes per chunk (rs / boxes rows each)
  int stage_bytes;
  int swap;             // 1: x[0] is B and x[1] is A
  int joint;            // 1: x[1]'s columns lie in what x[0] loads
  int row_q, row_t;     // row of a k-step's lane: q * row_q + 16 j + tq * row_t
  CUtensorMap t[2][4];  // kTileTma: t[o][0], {w columns, n rows}; kTilePhases: t[o][q]
};

// How TA x TB tiles are split over the warps: RA x RB regions of MT x NT tiles
// (the last ones padded), at most 25 tiles (50 accumulators a lane); the fewest
// DMMAs first, then the fewest shared loads.
struct TileRegion {
  int ra, rb, mt, nt;
};
__host__ __device__ constexpr TileRegion tile_region(int ta, int tb) {
  TileRegion best{0, 0, 0, 0};
  int best_cost = 1 << 30;
  for (int ra = 1; ra <= 8; ra *= 2)
    for (int rb = 1; ra * rb <= 8; rb *= 2) {
      const int mt = (ta + ra - 1) / ra, nt = (tb + rb - 1) / rb;
      if (mt * nt > 25) continue;
      const int cost = ra * rb * (100 * mt * nt + mt + nt);
      if (cost < best_cost) {
        best_cost = cost;
        best = TileRegion{ra, rb, mt, nt};
      }
    }
  return best;
}

template <int TA, int TB>
struct TileKernel {
  static_assert(TA >= TB && TB >= 1 && TA <= 8, "wider operand first, up to 64 columns");
  static constexpr TileRegion G = tile_region(TA, TB);
  static constexpr int RA = G.ra, RB = G.rb, MT = G.mt, NT = G.nt;
  static constexpr int R = RA * RB;
  static constexpr int S = kTileConsumers / R;  // row slots
  // Few tiles: several k-steps' loads in flight, and two sets of accumulators, or
  // a warp's DMMAs would wait for its loads and for one another.
  static constexpr int V = MT * NT <= 2 ? 4 : (MT * NT <= 8 ? 2 : 1);
  static constexpr int U = MT * NT <= 4 ? 2 : 1;
  static_assert(size_t(S) * 8 * TA * 8 * TB * sizeof(double) <= kTileData, "reduction sheets fit");
};

namespace detail {

// Element-by-element copy of a chunk's `rows` rows by the producer warps (pt:
// producer thread), lanes along the rows (kTileCols) or the columns.  What
// bounds it is the copies a producer warp can issue (3.0 TB/s with both
// operands gathered); whole columns to a warp, with fewer address steps but
// uneven shares, ran 127 -> 151 us at 400 MB of 13 x 13.
template <typename T>
__device__ __forceinline__ void tile_gather(const TileOperand<T>& x, unsigned char* dst, int64_t r0, int rows, int pt) {
  const bool cols = x.load == kTileCols;
  const T* src = x.base + r0 * x.s_row;
  const int ext = cols ? rows : x.w;  // the extent lanes run along
  const int64_t si = cols ? x.s_row : x.s_col, so = cols ? x.s_col : x.s_row;
  const int di = cols ? x.pitch : 1, dn = cols ? 1 : x.pitch;
  const int total = x.w * rows;
  constexpr int NP = 32 * kTileProducers;
  int in = pt % ext, out = pt / ext;
  const int step_in = NP % ext, step_out = NP / ext;
  const uint32_t d = dev::smem_u32(dst);
#pragma unroll 4
  for (int q = pt; q < total; q += NP) {
    dev::cp_async<sizeof(T)>(d + static_cast<uint32_t>((in * di + out * dn) * int(sizeof(T))), src + in * si + out * so);
    in += step_in;
    out += step_out;
    if (in >= ext) {
      in -= ext;
      ++out;
    }
  }
}

}  // namespace detail

template <typename T, int TA, int TB>
__global__ void __launch_bounds__(kTileThreads, 1) tsm_tn_tile_kernel(const __grid_constant__ TileArgs<T> args) {
  using K = TileKernel<TA, TB>;
  constexpr int CW = kTileConsumers, STAGES = kTileStages;
  const PlainArgs<T>& p = args.p;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128u - (dev::smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kTileData);
  uint64_t* empty = full + STAGES;
  volatile int* abort = reinterpret_cast<volatile int*>(empty + STAGES);
  unsigned* s_is_last = reinterpret_cast<unsigned*>(empty + STAGES) + 1;

  const int t = threadIdx.x;
  const int warp = t >> 5, lane = t & 31;
  const int nops = args.joint ? 1 : 2;
  bool gathers = args.x[0].load >= kTileRows;
  if (nops == 2) gathers = gathers || args.x[1].load >= kTileRows;
  if (t == 0) {
    for (int s = 0; s < STAGES; ++s) {
      dev::mbar_init(&full[s], gathers ? 1 + 32 * kTileProducers : 1);
      dev::mbar_init(&empty[s], CW);
    }
    *abort = 0;
    dev::fence_mbar_init();
  }
  if (warp == CW && lane == 0 && blockIdx.x < p.num_chunks) {
    if (args.x[0].load == kTileTma) dev::prefetch_tensormap(&args.t[0][0]);
    if (nops == 2 && args.x[1].load == kTileTma) dev::prefetch_tensormap(&args.t[1][0]);
  }
  __syncthreads();

  const int64_t G = gridDim.x;
  const int rs = args.rs;
  const int region = warp % K::R, slot0 = warp / K::R;
  const int ra = region % K::RA, rb = region / K::RA;
  const int g = lane >> 2, tq = lane & 3;
  double acc[K::U][K::MT][K::NT][2];
#pragma unroll
  for (int u = 0; u < K::U; ++u)
#pragma unroll
    for (int i = 0; i < K::MT; ++i)
#pragma unroll
      for (int j = 0; j < K::NT; ++j) acc[u][i][j][0] = acc[u][i][j][1] = 0.0;

  if (warp >= CW) {
    // ---------------- producers: one thread issues the TMA copies, all gather.
    if (warp == CW || gathers) {
      const int pt = t - CW * 32;
      int64_t issued = 0;
      const uint64_t policy = dev::policy_evict_first();
      for (int64_t c = blockIdx.x; c < p.num_chunks; c += G, ++issued) {
        const int s = static_cast<int>(issued % STAGES);
        const int64_t round = issued / STAGES;
        bool ok = true;
        if (lane == 0 && round > 0) ok = dev::mbar_wait(&empty[s], static_cast<uint32_t>((round - 1) & 1), abort);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        __syncwarp();
        if (!ok) {
          if (lane == 0) {
            *abort = 1;
            atomicOr(p.error, dev::kErrTimeout);
          }
          break;
        }
        unsigned char* stage = smem + s * args.stage_bytes;
        const int64_t r0 = c * rs;
        const int rows = static_cast<int>(p.rows_main - r0 < rs ? p.rows_main - r0 : rs);
        if (pt == 0) {
          uint32_t tx = 0;
          for (int o = 0; o < nops; ++o) {
            const TileOperand<T>& x = args.x[o];
            if (x.load == kTileBulk) tx += static_cast<uint32_t>(rows * x.w * int(sizeof(T)));
            if (x.load == kTileTma || x.load == kTilePhases)
              tx += static_cast<uint32_t>(rs * x.pitch * int(sizeof(T)));
          }
          dev::mbar_arrive_expect_tx(&full[s], tx);
          for (int o = 0; o < nops; ++o) {
            const TileOperand<T>& x = args.x[o];
            if (x.load == kTileBulk)
              dev::bulk_g2s_evict_first(stage + x.offset, x.base + r0 * x.w,
                                        static_cast<uint32_t>(rows * x.w * int(sizeof(T))), &full[s], policy);
            if (x.load == kTileTma) {
              const int box = rs / args.boxes;
              for (int q = 0; q < args.boxes; ++q)
                dev::tma_load_2d(stage + x.offset + q * box * x.pitch * int(sizeof(T)), &args.t[o][0], 0,
                                 static_cast<int>(r0) + q * box, &full[s], policy);
            }
            if (x.load == kTilePhases)
              for (int q = 0; q < 4; ++q)
                dev::tma_load_2d(stage + x.offset + q * x.phase_bytes, &args.t[o][q], 0, static_cast<int>(r0 / 4),
                                 &full[s], policy);
          }
        }
        if (gathers) {
          __syncwarp();
          for (int o = 0; o < nops; ++o)
            if (args.x[o].load >= kTileRows) detail::tile_gather(args.x[o], stage + args.x[o].offset, r0, rows, pt);
          dev::cp_async_mbar_arrive(&full[s]);
        }
      }
      dev::cp_async_wait_all();
    }
  } else {
    // ---------------- consumers: k-steps (4 rows) of this warp's slot.
    const TileOperand<T>& xa = args.x[0];
    const TileOperand<T>& xb = args.x[1];
    const int qa = xa.q_step, ja = xa.j_step, qb = xb.q_step, jb = xb.j_step;
    const int base_a = 8 * K::MT * ra + g + tq * xa.t_step, base_b = 8 * K::NT * rb + g + tq * xb.t_step;
    const int ksteps = rs / 4;
    int64_t it = 0;
    bool ok = true;  // false: a wait ran out, the remaining chunks are gone through without any
    for (int64_t c = blockIdx.x; c < p.num_chunks; c += G, ++it) {
      const int s = static_cast<int>(it % STAGES);
      if (ok && !dev::mbar_wait(&full[s], static_cast<uint32_t>((it / STAGES) & 1), abort)) {
        ok = false;  // no lane leaves the loop: its MMAs and barriers take the whole warp
        *abort = 1;
        atomicOr(p.error, dev::kErrTimeout);
      }
      const unsigned char* stage = smem + s * args.stage_bytes;
      const T* sa = reinterpret_cast<const T*>(stage + xa.offset) + xa.first + base_a;
      const T* sb = reinterpret_cast<const T*>(stage + xb.offset) + xb.first + base_b;
      const int64_t left = p.rows_main - c * rs;
      // The slots take turns at the chunk's first k-step: chunks need not hold whole rounds of slots.
      const int slot = (slot0 + static_cast<int>(it)) % K::S;
      auto at_a = [&](int ks) { return sa + ((ks & 3) * qa + xa.shift[ks & 3] + (ks >> 2) * ja); };
      auto at_b = [&](int ks) { return sb + ((ks & 3) * qb + xb.shift[ks & 3] + (ks >> 2) * jb); };
      auto mma = [&](double (&d)[K::MT][K::NT][2], const double (&a)[K::MT], const double (&b)[K::NT]) {
#pragma unroll
        for (int i = 0; i < K::MT; ++i)
#pragma unroll
          for (int j = 0; j < K::NT; ++j) dev::dmma_m8n8k4(d[i][j][0], d[i][j][1], a[i], b[j]);
      };
      if (left >= rs) {
        const T* pa = at_a(slot);
        const T* pb = at_b(slot);
        int ks = slot;
#pragma unroll 1
        for (; ks + (K::V - 1) * K::S < ksteps; ks += K::V * K::S) {
          double a[K::V][K::MT], b[K::V][K::NT];
#pragma unroll
          for (int v = 0; v < K::V; ++v) {
            // q is the same for all of a slot's k-steps when S is a multiple of 4
            const T* ya = K::S % 4 == 0 ? pa + v * (K::S / 4) * ja : at_a(ks + v * K::S);
            const T* yb = K::S % 4 == 0 ? pb + v * (K::S / 4) * jb : at_b(ks + v * K::S);
#pragma unroll
            for (int i = 0; i < K::MT; ++i) a[v][i] = static_cast<double>(ya[8 * i]);
#pragma unroll
            for (int j = 0; j < K::NT; ++j) b[v][j] = static_cast<double>(yb[8 * j]);
          }
          pa += K::V * (K::S / 4) * ja;
          pb += K::V * (K::S / 4) * jb;
#pragma unroll
          for (int v = 0; v < K::V; ++v) mma(acc[v % K::U], a[v], b[v]);
        }
        if constexpr (K::V > 1) {
#pragma unroll 1
          for (; ks < ksteps; ks += K::S) {
            const T* ya = at_a(ks);
            const T* yb = at_b(ks);
            double a[K::MT], b[K::NT];
#pragma unroll
            for (int i = 0; i < K::MT; ++i) a[i] = static_cast<double>(ya[8 * i]);
#pragma unroll
            for (int j = 0; j < K::NT; ++j) b[j] = static_cast<double>(yb[8 * j]);
            mma(acc[0], a, b);
          }
        }
      } else {
        // The last chunk: rows past the end contribute zeros.  They are read (the
        // stage holds them) and replaced with a select: no lane may branch
        // around a load here, or the warp could reach the warp-wide MMAs in
        // two parts, which never end.
        const int rows = static_cast<int>(left);
#pragma unroll 1
        for (int ks = slot; ks < ksteps; ks += K::S) {
          const int row0 = (ks & 3) * args.row_q + 16 * (ks >> 2);
          if (row0 >= rows) continue;
          const bool in = row0 + tq * args.row_t < rows;
          const T* ya = at_a(ks);
          const T* yb = at_b(ks);
          double a[K::MT], b[K::NT];
#pragma unroll
          for (int i = 0; i < K::MT; ++i) {
            const double v = static_cast<double>(ya[8 * i]);
            a[i] = in ? v : 0.0;
          }
#pragma unroll
          for (int j = 0; j < K::NT; ++j) {
            const double v = static_cast<double>(yb[8 * j]);
            b[j] = in ? v : 0.0;
          }
          __syncwarp();
          mma(acc[0], a, b);
        }
      }
      __syncwarp();
      if (lane == 0) dev::mbar_arrive(&empty[s]);
    }
  }

  __syncthreads();
  if (*abort && warp == CW && lane == 0) {
    // Let every copy this CTA issued land before the ring is reused (bounded).
    int64_t issued = 0;
    for (int64_t c = blockIdx.x; c < p.num_chunks; c += G) ++issued;
    volatile int no_abort = 0;
    for (int64_t q = issued > STAGES ? issued - STAGES : 0; q < issued; ++q)
      if (!dev::mbar_wait(&full[q % STAGES], static_cast<uint32_t>((q / STAGES) & 1), &no_abort)) break;
  }
  __syncthreads();

  // Each warp's tiles -> its slot's m x k sheet: D[g][2 tq + e] of tile (i, j)
  // is column 8 (ra MT + i) + g of x[0] times column 8 (rb NT + j) + 2 tq + e of x[1].
  const int mk = p.m * p.k;
  double* red = reinterpret_cast<double*>(smem);
  if (warp < CW) {
    const int w0 = args.x[0].cols, w1 = args.x[1].cols;
    const int s0 = args.swap ? 1 : p.k, s1 = args.swap ? p.k : 1;
    double* sheet = red + slot0 * mk;
#pragma unroll
    for (int i = 0; i < K::MT; ++i) {
      const int c0 = 8 * (ra * K::MT + i) + g;
#pragma unroll
      for (int j = 0; j < K::NT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c1 = 8 * (rb * K::NT + j) + 2 * tq + e;
          double v = acc[0][i][j][e];
          if constexpr (K::U == 2) v += acc[1][i][j][e];
          if (c0 < w0 && c1 < w1) sheet[c0 * s0 + c1 * s1] = v;
        }
    }
  }
  __syncthreads();
  detail::finish_partials<64 * TA * TB>(p, red, K::S, t, kTileThreads, s_is_last);
}

}  // namespace tsm
