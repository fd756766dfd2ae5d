// tsm_tsmm_tile.cuh -- Y (n x q) = X (n x p) W (p x q), or Y += X W, for any
// p, q <= 64 on the FP64 tensor cores; X and Y dense and 16-byte aligned.  The
// kernels of tsm_tsmm_dmma.cuh are compiled for powers of two: other widths
// were padded to the next one, took a guarded path with a load per element,
// and stored Y element by element.  Here
//   * X's rows (and, for Y += X W, Y's old rows) stream through a ring of
//     1-D bulk copies, as they lie: pitch p (q);
//   * W's fragments lie in shared memory in lane order, zero-padded, as
//     doubles: a conflict-free 8-byte load each, shared by four row groups;
//   * a warp takes units of 32 rows x 16 columns (8 where one 8-column tile is
//     left), round-robin over the chunks' units, so widths need not divide the
//     warps;
//   * results go to the stage's Y rows in shared memory (added to the old ones
//     there), and a storing warp writes the chunk's rows with ONE bulk copy:
//     whole 128-byte lines whatever q is.
// The sum over p runs in the order of tsm_tsmm_dmma.cuh (k-step 2 kb + e:
// columns 8 kb + 2 t + e).  Up to 7 columns on either side lanes take whole
// rows instead (tsmm_rows).
//
// 16 consumer warps, four a scheduler: with 8 the chain of a unit (loads,
// dependent MMAs, stores) left the tensor pipe idle (13 x 13 FP64, 400 MB: 110
// us; 79 with 16; 67 with the unit's loops specialised for even and odd widths).
//
// A bulk copy of X brings bank conflicts with it (rows p apart: 2-way for odd
// p, 4-way for p = 16, 48): at most 4 shared-memory cycles per DMMA issued, the
// DMMA's own cost.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "tsm_device.cuh"
#include "tsm_tsmm.cuh"
#include "tsm_tsmm_dmma.cuh"  // load_pair

namespace tsm {

constexpr int kTsmmTileStages = 4;
constexpr int kTsmmTileCW = 16;                                // consumer warps
constexpr int kTsmmTileThreads = 32 * (kTsmmTileCW + 2);      // + the loading and the storing warp
constexpr size_t kTsmmTileData = 224 * 1024;                  // W fragments, then the ring
constexpr size_t kTsmmTileSmem = 128 + kTsmmTileData + 3 * kTsmmTileStages * sizeof(uint64_t) + 16;

template <typename T>
struct TsmmTileArgs {
  TsmmArgs<T> a;       // split: chunks of prob[0]
  int rs;              // rows per chunk, a multiple of 32
  int w_offset[2];     // bytes from the start of shared memory to a problem's W fragments
  int ring;            // ... to the ring
  int y_offset[2];     // bytes from a stage's start to its Y rows
  int stage_bytes;
};

// k-steps of 4 of p columns (pairs of them beyond p = 4) and 8-column tiles of q.
__host__ __device__ constexpr int tsmm_ksteps(int p) { return p <= 4 ? 1 : 2 * ((p + 7) / 8); }
__host__ __device__ constexpr int tsmm_tiles(int q) { return (q + 7) / 8; }
// Rows to lanes instead of tiles: an 8 x 8 MMA tile is mostly padding there,
// and a row's p q multiplications cost less than its bytes.  B200, 400 MB read
// and written, backward, MMA units -> rows to lanes, us: FP64 1 x 1 210 -> 71,
// 3 x 3 87 -> 66, 7 x 7 71 -> 65; FP32 2 x 4 156 -> 86, 3 x 3 155 -> 77, 7 x 7
// 103 -> 92.  At 8 columns the rows' stride meets bank conflicts: 5 x 8 FP64 69
// -> 91.
__host__ __device__ constexpr bool tsmm_narrow(int p, int q) { return p <= 7 && q <= 7; }

namespace detail {

__device__ __forceinline__ void put_pair(double* y, double v0, double v1) {
  *reinterpret_cast<double2*>(y) = make_double2(v0, v1);
}
__device__ __forceinline__ void put_pair(float* y, double v0, double v1) {
  *reinterpret_cast<float2*>(y) = make_float2(static_cast<float>(v0), static_cast<float>(v1));
}

// One unit: RG groups of 8 rows from row0 on x NTG tiles from tile j0.  BETA:
// Y += (the old rows lie at y); XP, YP: p, q even (pairs are aligned).
template <int RG, int NTG, bool BETA, bool XP, bool YP, typename T>
__device__ __forceinline__ void tsmm_unit(const T* x, T* y, const double* wf, int p, int q, int ksteps, int nt, int row0,
                                          int j0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double* w = wf + j0 * 32 + lane;
  const T* xr = x + (row0 + g) * p;
  const int p8 = 8 * p, q8 = 8 * q;
  double d[RG][NTG][2];
#pragma unroll
  for (int i = 0; i < RG; ++i)
#pragma unroll
    for (int j = 0; j < NTG; ++j) d[i][j][0] = d[i][j][1] = 0.0;
  // Columns at or past p read a valid one and are replaced by zeros with a
  // select: no lane may branch around a load here, or the warp could reach the
  // warp-wide MMAs in two parts, which never end.
  if (ksteps == 1) {  // p <= 4: column t
    const int col = min(t, p - 1);
    double a[RG];
#pragma unroll
    for (int i = 0; i < RG; ++i) {
      const double v = static_cast<double>(xr[i * p8 + col]);
      a[i] = t < p ? v : 0.0;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < RG; ++i)
#pragma unroll
      for (int j = 0; j < NTG; ++j) dev::dmma_m8n8k4(d[i][j][0], d[i][j][1], a[i], w[32 * j]);
  } else {
    auto step = [&](const double (&a)[RG][2]) {  // two k-steps
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        double b[NTG];
#pragma unroll
        for (int j = 0; j < NTG; ++j) b[j] = w[(e * nt + j) * 32];
#pragma unroll
        for (int j = 0; j < NTG; ++j)
#pragma unroll
          for (int i = 0; i < RG; ++i) dev::dmma_m8n8k4(d[i][j][0], d[i][j][1], a[i][e], b[j]);
      }
      w += 64 * nt;
    };
    const T* xk = xr + 2 * t;
    const int whole = p >> 3;
#pragma unroll 2
    for (int kb = 0; kb < whole; ++kb, xk += 8) {
      double a[RG][2];
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        if constexpr (XP) {
          load_pair(xk + i * p8, a[i][0], a[i][1]);
        } else {
          a[i][0] = static_cast<double>(xk[i * p8]);
          a[i][1] = static_cast<double>(xk[i * p8 + 1]);
        }
      }
      step(a);
    }
    if (p & 7) {  // past p: the next row's values, not zeros
      const int kappa = 8 * whole + 2 * t, c0 = min(kappa, p - 1), c1 = min(kappa + 1, p - 1);
      double a[RG][2];
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        const double v0 = static_cast<double>(xr[i * p8 + c0]), v1 = static_cast<double>(xr[i * p8 + c1]);
        a[i][0] = kappa < p ? v0 : 0.0;
        a[i][1] = kappa + 1 < p ? v1 : 0.0;
      }
      __syncwarp();
      step(a);
    }
  }
  // D[g][2t + {0,1}] of tile j -> Y[row][8 (j0 + j) + 2 t + {0,1}]
  __syncwarp();
  T* yr = y + (row0 + g) * q + 8 * j0 + 2 * t;
#pragma unroll
  for (int j = 0; j < NTG; ++j) {
    const int left = q - 8 * (j0 + j) - 2 * t;  // columns of Y from this lane's first on
    if constexpr (YP) {
      if (left > 0) {
#pragma unroll
        for (int i = 0; i < RG; ++i) {
          T* dst = yr + i * q8 + 8 * j;
          if constexpr (BETA) {
            double o0, o1;
            load_pair(dst, o0, o1);
            put_pair(dst, d[i][j][0] + o0, d[i][j][1] + o1);
          } else {
            put_pair(dst, d[i][j][0], d[i][j][1]);
          }
        }
      }
    } else {
      if (left > 0) {
#pragma unroll
        for (int i = 0; i < RG; ++i) {
          T* dst = yr + i * q8 + 8 * j;
          dst[0] = static_cast<T>(BETA ? d[i][j][0] + static_cast<double>(dst[0]) : d[i][j][0]);
        }
      }
      if (left > 1) {
#pragma unroll
        for (int i = 0; i < RG; ++i) {
          T* dst = yr + i * q8 + 8 * j + 1;
          dst[0] = static_cast<T>(BETA ? d[i][j][1] + static_cast<double>(dst[0]) : d[i][j][1]);
        }
      }
    }
  }
}

// Narrow problems: a lane takes a row, its P values in registers and W (p x q
// doubles, row-major) broadcast from shared memory.  A unit is 32 rows.
template <int P, bool BETA, typename T>
__device__ __forceinline__ int tsmm_rows(const T* x, T* y, const double* w, int q, int rows, int u, int lane) {
  const int units = (rows + 31) / 32;
#pragma unroll 1
  for (; u < units; u += kTsmmTileCW) {
    const T* xr = x + (32 * u + lane) * P;
    T* yr = y + (32 * u + lane) * q;
    double v[P];
    if constexpr (P % 2 == 0) {
#pragma unroll
      for (int a = 0; a < P; a += 2) load_pair(xr + a, v[a], v[a + 1]);
    } else {
#pragma unroll
      for (int a = 0; a < P; ++a) v[a] = static_cast<double>(xr[a]);
    }
#pragma unroll 4
    for (int o = 0; o < q; ++o) {
      double s = v[0] * w[o];
#pragma unroll
      for (int a = 1; a < P; ++a) s = fma(v[a], w[a * q + o], s);
      yr[o] = static_cast<T>(BETA ? s + static_cast<double>(yr[o]) : s);
    }
  }
  return u - units;
}

template <bool BETA, typename T>
__device__ __forceinline__ int tsmm_rows(const T* x, T* y, const double* w, int p, int q, int rows, int u, int lane) {
  switch (p) {
    case 1: return tsmm_rows<1, BETA>(x, y, w, q, rows, u, lane);
    case 2: return tsmm_rows<2, BETA>(x, y, w, q, rows, u, lane);
    case 3: return tsmm_rows<3, BETA>(x, y, w, q, rows, u, lane);
    case 4: return tsmm_rows<4, BETA>(x, y, w, q, rows, u, lane);
    case 5: return tsmm_rows<5, BETA>(x, y, w, q, rows, u, lane);
    case 6: return tsmm_rows<6, BETA>(x, y, w, q, rows, u, lane);
    default: return tsmm_rows<7, BETA>(x, y, w, q, rows, u, lane);
  }
}

// This warp's units of a chunk, from unit `u` on; returns the first one past the chunk.
template <int RG, bool BETA, bool XP, bool YP, typename T>
__device__ __forceinline__ int tsmm_units(const T* x, T* y, const double* wf, int p, int q, int rows, int u, int lane) {
  const int ks = tsmm_ksteps(p), nt = tsmm_tiles(q), groups = (nt + 1) / 2;
  const int units = (rows + 8 * RG - 1) / (8 * RG) * groups;
  int rb = u / groups, cg = u - rb * groups;
#pragma unroll 1
  for (; u < units; u += kTsmmTileCW) {
    if (2 * cg + 1 < nt)
      tsmm_unit<RG, 2, BETA, XP, YP>(x, y, wf, p, q, ks, nt, 8 * RG * rb, 2 * cg, lane);
    else
      tsmm_unit<RG, 1, BETA, XP, YP>(x, y, wf, p, q, ks, nt, 8 * RG * rb, 2 * cg, lane);
    cg += kTsmmTileCW;
    while (cg >= groups) {
      cg -= groups;
      ++rb;
    }
  }
  return u - units;
}

template <bool BETA, bool XP, bool YP, typename T>
__device__ __forceinline__ int tsmm_units(const T* x, T* y, const double* wf, int p, int q, int rows, int u, int lane) {
  return p + q <= 64 ? tsmm_units<4, BETA, XP, YP>(x, y, wf, p, q, rows, u, lane)
                     : tsmm_units<2, BETA, XP, YP>(x, y, wf, p, q, rows, u, lane);
}

}  // namespace detail

template <typename T>
__global__ void __launch_bounds__(kTsmmTileThreads, 1) tsm_tsmm_tile_kernel(const __grid_constant__ TsmmTileArgs<T> args) {
  constexpr int CW = kTsmmTileCW, STAGES = kTsmmTileStages;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128u - (dev::smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kTsmmTileData);  // rows have landed
  uint64_t* done = full + STAGES;                                      // results are in the stage's Y rows
  uint64_t* empty = done + STAGES;                                     // ... and have been read by the store
  volatile int* abort = reinterpret_cast<volatile int*>(empty + STAGES);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int64_t G = gridDim.x, total = args.a.total_chunks;
  unsigned char* ring = smem + args.ring;
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      dev::mbar_init(&full[s], 1);
      dev::mbar_init(&done[s], CW);
      dev::mbar_init(&empty[s], 1);
    }
    *abort = 0;
    dev::fence_mbar_init();
  }
  __syncthreads();

  if (warp == CW) {
    // ---------------- loading warp: X rows, and Y's old rows where they count.
    if (lane == 0) {
      int64_t issued = 0;
      const uint64_t policy = dev::policy_evict_first();
      for (int64_t c = blockIdx.x; c < total; c += G, ++issued) {
        const int s = static_cast<int>(issued % STAGES);
        const int64_t round = issued / STAGES;
        if (round > 0 && !dev::mbar_wait(&empty[s], static_cast<uint32_t>((round - 1) & 1), abort)) {
          *abort = 1;
          atomicOr(args.a.error, dev::kErrTimeout);
          break;
        }
        int pi;
        int64_t r0;
        detail::tsmm_chunk(args.a, c, args.rs, pi, r0);
        const TsmmProblem<T>& pr = args.a.prob[pi];
        const int64_t rows = pr.rows_main - r0 < args.rs ? pr.rows_main - r0 : args.rs;
        const uint32_t xb = static_cast<uint32_t>(rows * pr.p * int64_t(sizeof(T)));
        const uint32_t yb = pr.beta ? static_cast<uint32_t>(rows * pr.q * int64_t(sizeof(T))) : 0u;
        unsigned char* stage = ring + s * args.stage_bytes;
        dev::mbar_arrive_expect_tx(&full[s], xb + yb);
        dev::bulk_g2s_evict_first(stage, pr.X + r0 * pr.p, xb, &full[s], policy);
        if (yb) dev::bulk_g2s_evict_first(stage + args.y_offset[pi], pr.Y + r0 * pr.q, yb, &full[s], policy);
      }
    }
  } else if (warp == CW + 1) {
    // ---------------- storing warp: a finished chunk's Y rows, one bulk copy.
    if (lane == 0) {
      const uint64_t policy = dev::policy_evict_first();
      int64_t it = 0;
      for (int64_t c = blockIdx.x; c < total; c += G, ++it) {
        const int s = static_cast<int>(it % STAGES);
        if (!dev::mbar_wait(&done[s], static_cast<uint32_t>((it / STAGES) & 1), abort)) {
          *abort = 1;
          atomicOr(args.a.error, dev::kErrTimeout);
          break;
        }
        int pi;
        int64_t r0;
        detail::tsmm_chunk(args.a, c, args.rs, pi, r0);
        const TsmmProblem<T>& pr = args.a.prob[pi];
        const int64_t rows = pr.rows_main - r0 < args.rs ? pr.rows_main - r0 : args.rs;
        dev::bulk_s2g(pr.Y + r0 * pr.q, ring + s * args.stage_bytes + args.y_offset[pi],
                      static_cast<uint32_t>(rows * pr.q * int64_t(sizeof(T))), policy);
        dev::bulk_commit();
        dev::bulk_wait_read<0>();  // the stage is free once the store has read it
        dev::mbar_arrive(&empty[s]);
      }
      dev::bulk_wait_all();
    }
  } else {
    // ---------------- consumer warps
    const int g = lane >> 2, t = lane & 3;
    // W's fragments, all of both problems: lane (g, t) of k-step s, tile j
    // holds W[kappa(s, t)][8 j + g], zero past p or q.
    for (int pi = 0; pi < args.a.nprob; ++pi) {
      const TsmmProblem<T>& pr = args.a.prob[pi];
      double* wf = reinterpret_cast<double*>(smem + args.w_offset[pi]);
      if (tsmm_narrow(pr.p, pr.q)) {
        for (int f = tid; f < pr.p * pr.q; f += CW * 32) {
          const int a = f / pr.q, o = f - a * pr.q;
          const double w = static_cast<double>(pr.W[a * pr.w_row + o * pr.w_col]);
          wf[f] = pr.negate ? -w : w;
        }
        continue;
      }
      const int ks = tsmm_ksteps(pr.p), nt = tsmm_tiles(pr.q);
      for (int f = warp; f < ks * nt; f += CW) {
        const int s = f / nt, j = f - s * nt;
        const int kappa = ks > 1 ? 8 * (s >> 1) + 2 * t + (s & 1) : t, o = 8 * j + g;
        double w = 0.0;
        if (kappa < pr.p && o < pr.q)
          w = static_cast<double>(pr.W[static_cast<int64_t>(kappa) * pr.w_row + static_cast<int64_t>(o) * pr.w_col]);
        wf[f * 32 + lane] = pr.negate ? -w : w;
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(CW * 32) : "memory");

    int64_t it = 0;
    bool ok = true;  // false: a wait ran out, the remaining chunks are gone through without any
    int turn = warp;  // this warp's first unit of the chunk: units go round the warps across chunks
    for (int64_t c = blockIdx.x; c < total; c += G, ++it) {
      const int s = static_cast<int>(it % STAGES);
      int pi;
      int64_t r0;
      detail::tsmm_chunk(args.a, c, args.rs, pi, r0);
      const TsmmProblem<T>& pr = args.a.prob[pi];
      const int64_t left = pr.rows_main - r0;
      const int rows = static_cast<int>(left < args.rs ? left : args.rs);
      const int p = pr.p, q = pr.q;
      const unsigned char* stage = ring + s * args.stage_bytes;
      const T* x = reinterpret_cast<const T*>(stage);
      T* y = reinterpret_cast<T*>(const_cast<unsigned char*>(stage) + args.y_offset[pi]);
      const double* wf = reinterpret_cast<const double*>(smem + args.w_offset[pi]);
      if (ok && !dev::mbar_wait(&full[s], static_cast<uint32_t>((it / STAGES) & 1), abort)) {
        ok = false;  // no lane leaves the loop: its MMAs and barriers take the whole warp
        *abort = 1;
        atomicOr(args.a.error, dev::kErrTimeout);
      }
      if (tsmm_narrow(p, q)) {
        turn = pr.beta ? detail::tsmm_rows<true>(x, y, wf, p, q, rows, turn, lane)
                       : detail::tsmm_rows<false>(x, y, wf, p, q, rows, turn, lane);
      } else
      switch ((pr.beta ? 4 : 0) | (p & 1 ? 0 : 2) | (q & 1 ? 0 : 1)) {
        case 0: turn = detail::tsmm_units<false, false, false>(x, y, wf, p, q, rows, turn, lane); break;
        case 1: turn = detail::tsmm_units<false, false, true>(x, y, wf, p, q, rows, turn, lane); break;
        case 2: turn = detail::tsmm_units<false, true, false>(x, y, wf, p, q, rows, turn, lane); break;
        case 3: turn = detail::tsmm_units<false, true, true>(x, y, wf, p, q, rows, turn, lane); break;
        case 4: turn = detail::tsmm_units<true, false, false>(x, y, wf, p, q, rows, turn, lane); break;
        case 5: turn = detail::tsmm_units<true, false, true>(x, y, wf, p, q, rows, turn, lane); break;
        case 6: turn = detail::tsmm_units<true, true, false>(x, y, wf, p, q, rows, turn, lane); break;
        default: turn = detail::tsmm_units<true, true, true>(x, y, wf, p, q, rows, turn, lane); break;
      }
      dev::fence_proxy_async_smem();  // the store reads what was written here
      __syncwarp();
      if (lane == 0) dev::mbar_arrive(&done[s]);
    }
    // Rows the ring did not stream (fewer than 16 bytes' worth per problem):
    // CTA 0 computes them from global memory, one output per thread.
    if (blockIdx.x == 0) {
      for (int pi = 0; pi < args.a.nprob; ++pi) {
        const TsmmProblem<T>& pr = args.a.prob[pi];
        const int64_t tail = pr.n - pr.rows_main;
        for (int64_t e = tid; e < tail * pr.q; e += CW * 32) {
          const int64_t r = pr.rows_main + e / pr.q;
          const int o = static_cast<int>(e % pr.q);
          double v = 0.0;
          for (int a = 0; a < pr.p; ++a)
            v = fma(static_cast<double>(pr.X[r * pr.ldx + a]),
                    static_cast<double>(pr.W[static_cast<int64_t>(a) * pr.w_row + static_cast<int64_t>(o) * pr.w_col]),
                    v);
          if (pr.negate) v = -v;
          detail::store_y(pr, r, o, static_cast<T>(v));
        }
      }
    }
  }

  __syncthreads();
  if (*abort && warp == CW && lane == 0) {
    // Let every load this CTA issued land before it exits (bounded).
    int64_t issued = 0;
    for (int64_t c = blockIdx.x; c < total; c += G) ++issued;
    volatile int no_abort = 0;
    for (int64_t q = issued > STAGES ? issued - STAGES : 0; q < issued; ++q)
      if (!dev::mbar_wait(&full[q % STAGES], static_cast<uint32_t>((q / STAGES) & 1), &no_abort)) break;
  }
}

}  // namespace tsm
