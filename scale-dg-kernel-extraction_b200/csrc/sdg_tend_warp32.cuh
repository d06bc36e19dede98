// Mixed-form RK-stage kernel at Nq = 8: one warp per element, each lane
// contracting whole lines from registers.
//
// The element's q, u, v, w arrive in shared memory through a tensor map with
// the 128-byte swizzle: 16-byte word c of 128-byte row r sits at word
// c ^ (r & 7).  In that layout three readings of the same data are all free of
// bank conflicts, and the warp makes each where it needs it:
//
//   x-lines (j,k), 16-byte words along i: lane L takes (L & 7, L >> 3) and
//           (L & 7, 4 + (L >> 3)), packed in the two halves of float2;
//   y-lines (i,k), 8-byte words: lane (c, k) = (L & 3, L >> 2) takes the
//           neighbouring lines i = 2c, 2c + 1;
//   z-lines (i,j), 8-byte words: lane (c, j) takes the columns i = 2c, 2c + 1,
//           in which the node is finally updated and stored.
//
// So the volume fluxes are formed where they are contracted, and the lane that
// holds a line holds both of its ends: it evaluates the two face fluxes there.
// Through shared memory pass only the line sums (x to y to z, over the
// element's own w, which is in registers by then), the x fluxes (to the y-lines,
// over two inner words of the x-line's u) and the lift of the four x/y faces
// (y to z, over v).  No block barrier, no face or flux buffers.  The packed FP32
// instructions (__ffma2_rn) advance the two lines of a lane together.  Every
// node's operations and their order are those of tend_kernel.
//
// Tiles, ring, producer warp, in-tile neighbours and bounded waits are those
// of tend_warp_kernel.
//
// Measured (32^3 elements, us per launch of RK stage 1 / 2 / 3): 90 / 83 / 89
// against 99 / 97 / 101 for the block kernel it replaced, i.e. 4.5 / 5.7 / 6.1
// TB/s of the 24 / 28 / 32 algorithmic bytes per node, where a copy reaches
// 6.5.  Instructions per element 1900 -> 1050, L1 data pipe 74 -> 48 % busy.
// Stage 1 also converts its FP64 state in all three readings.  Eleven warps of
// 168 registers measured better than fourteen of 128 (8 KB an element: the
// slots would hold them), which spill.
//
// It takes the batch and meshes of more than 64 elements an SM; smaller ones stay with
// tend_pipe_kernel (warp32_few).
#pragma once

#include <cuda.h>

#include "sdg_in_tile.h"
#include "sdg_tend_warp.cuh"

namespace sdg {

// The forms that run this kernel.
template <int NQ, typename TC, bool EXACT>
constexpr bool kWarp32Kernel = NQ == 8 && sizeof(TC) == 4 && !EXACT;

// Tensor maps of one stage's inputs q, u, v, w (encode_field_map).
struct alignas(64) FieldMaps {
  CUtensorMap m[4];
};
static_assert(sizeof(FieldMaps) == kFieldMapsBytes, "FieldMaps");

template <typename TQ>
struct Warp32Plan {
  static constexpr int NP = 512;
  static constexpr size_t QB = NP * sizeof(TQ);
  static constexpr size_t VB = NP * sizeof(float);
  static constexpr size_t ELEM = QB + 3 * VB;     // 8 KB, 10 KB with FP64 q
  static constexpr int ELEMS = kWarpElems32;  // per tile at most
  static constexpr int WARPS = ELEMS;         // consumer warps
  static constexpr int NSTAGE = 2;
  static constexpr int THREADS = 32 * (WARPS + 1);
  static constexpr size_t SLOT = ELEMS * ELEM;
  // The swizzle acts on address bits: slots start at 1024-byte boundaries.
  static constexpr size_t OFF_C = NSTAGE * SLOT + 16 * NSTAGE;
  static constexpr size_t BYTES = OFF_C + 4 * 128 + 1024;  // contexts as in WarpPlan
};
static_assert(Warp32Plan<float>::BYTES <= kPipeMaxSmem &&
                  Warp32Plan<double>::BYTES <= kPipeMaxSmem,
              "warp kernel: shared memory");

// Tiled copy of the map's box at row `row` (no multicast); dst 128-byte
// aligned, the innermost coordinate is 0.
__device__ __forceinline__ void tma_rows_g2s(void* dst, const CUtensorMap* map, int row,
                                             uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(row), "r"(smem_u32(bar))
      : "memory");
}

// Before a block's first use of a tensor map that the host copied to global
// memory: what the copy wrote is what its tensor copies read.
__device__ __forceinline__ void tensormap_acquire(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}

// Word index of node (i,j,k) in a swizzled element of floats or doubles.
template <typename T>
__device__ __forceinline__ int swz(int i, int j, int k) {
  if constexpr (sizeof(T) == 4) {
    const int row = 2 * k + (j >> 2);
    return 32 * row + 4 * (((2 * (j & 3) + (i >> 2)) ^ row) & 7) + (i & 3);
  } else {
    const int row = 4 * k + (j >> 1);
    return 16 * row + 2 * (((4 * (j & 1) + (i >> 1)) ^ row) & 7) + (i & 1);
  }
}

// A value of a lane's two lines, packed.
struct Lines {
  using V = float2;
  static __device__ __forceinline__ V make(float a, float b) { return make_float2(a, b); }
  static __device__ __forceinline__ float lo(V a) { return a.x; }
  static __device__ __forceinline__ float hi(V a) { return a.y; }
  static __device__ __forceinline__ V dup(float a) { return make_float2(a, a); }
  static __device__ __forceinline__ V mul(V a, V b) { return __fmul2_rn(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
  static __device__ __forceinline__ V neg(V a) { return make_float2(-a.x, -a.y); }
  static __device__ __forceinline__ V abs(V a) { return make_float2(fabsf(a.x), fabsf(a.y)); }
  // a*b - c*d, three roundings: scalar, because the compiler fuses a packed
  // product into a packed sum.
  static __device__ __forceinline__ V sub_products(V a, V b, V c, V d) {
    return make_float2(__fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(c.x, d.x)),
                       __fsub_rn(__fmul_rn(a.y, b.y), __fmul_rn(c.y, d.y)));
  }
  // Neighbouring nodes of the lane's two lines, and back.
  static __device__ __forceinline__ V ld(const float* p) {
    return *reinterpret_cast<const float2*>(p);
  }
  static __device__ __forceinline__ void st(float* p, V a) { *reinterpret_cast<float2*>(p) = a; }
};
__device__ __forceinline__ float ld_early(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_early_state(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

template <typename TQ, typename TO, bool BATCH>
__global__ void __launch_bounds__(Warp32Plan<TQ>::THREADS, 1)
    tend_warp32_kernel(const __grid_constant__ TendArgs<TQ, float, TO, float> A,
                       const __grid_constant__ DMat<8, float> D,
                       const __grid_constant__ FieldMaps M) {
  using P = Warp32Plan<TQ>;
  using Ctx = TileCtx<TQ, float, TO, float>;
  using L = Lines;
  using V = typename L::V;
  constexpr int NP = P::NP;
  constexpr int NS = P::NSTAGE;
  constexpr unsigned kAll = 0xffffffffu;
  pdl_trigger();
  extern __shared__ unsigned char smem_any[];
  unsigned char* smem = smem_any + ((1024 - (smem_u32(smem_any) & 1023)) & 1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + NS * P::SLOT);
  uint64_t* empty = full + NS;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int es = warp;  // element of the tile
  const int tw = A.tile_elems;  // elements per tile (single instance)
  const int ntiles = BATCH ? A.ntiles : (A.nelem + tw - 1) / tw;
  auto context = [&](int tile) {
    Ctx t = tile_ctx<1, BATCH>(A, tile, ntiles);
    if constexpr (!BATCH) {
      t.e0 = A.elem0 + tile * tw;
      t.n = min(tw, A.nelem - tile * tw);
    }
    return t;
  };
  if (threadIdx.x == 0) {
    for (int k = 0; k < NS; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], P::WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  // Contexts of the block's tiles, as in tend_warp_kernel (batched launches).
  static_assert(sizeof(Ctx) <= 128, "context ring");
  auto ctx_at = [&](int it) -> Ctx* {
    return reinterpret_cast<Ctx*>(smem + P::OFF_C + 128 * (it & 3));
  };
  // Copies of tile `tile` into slot `slot`: the velocities (parts & 1), then q
  // (parts & 2) with q0 into L2, where the epilogue's loads find it (without:
  // stage 2 85.6 instead of 78.1 us at 32^3).
  int acquired = -1;  // instance whose maps this block last acquired
  auto copy = [&](int it, int tile, int slot, int parts) {
    const Ctx t = context(tile);
    const CUtensorMap* maps = M.m;
    if constexpr (BATCH) {
      const int inst = A.tiles[tile].inst;
      maps = static_cast<const CUtensorMap*>(A.insts[inst].maps);
      if (parts & 1) {
        *ctx_at(it) = t;
        if (tile + gridDim.x < ntiles) *ctx_at(it + 1) = context(tile + gridDim.x);
        // The tables are rewritten in place when members come and go.
        if (inst != acquired)
#pragma unroll
          for (int f = 0; f < 4; ++f) tensormap_acquire(maps + f);
        acquired = inst;
      }
    }
    unsigned char* dst = smem + slot * P::SLOT;
    constexpr int RQ = static_cast<int>(P::QB / 128), RV = static_cast<int>(P::VB / 128);
    if (parts & 1) {
      mbar_arrive_expect_tx(&full[slot], static_cast<uint32_t>(t.n * P::ELEM));
      for (int s = 0; s < t.n; ++s)
#pragma unroll
        for (int f = 1; f < 4; ++f)
          tma_rows_g2s(dst + s * P::ELEM + P::QB + (f - 1) * P::VB, maps + f, (t.e0 + s) * RV,
                       &full[slot]);
    }
    if (!(parts & 2)) return;
    for (int s = 0; s < t.n; ++s)
      tma_rows_g2s(dst + s * P::ELEM, maps, (t.e0 + s) * RQ, &full[slot]);
    if (A.rk_a != 0.0)
      bulk_prefetch_l2(t.q0 + static_cast<size_t>(t.e0) * NP,
                       static_cast<uint32_t>(t.n * NP * sizeof(double)));
  };
  if (warp == P::WARPS) {
    // Producer, as in tend_warp_kernel.
    int ahead = 0;
    for (; A.chained && lane == 0 && ahead < NS; ++ahead) {
      const int tile = blockIdx.x + ahead * gridDim.x;
      if (tile >= ntiles || tile + 1 == A.inject_skip) break;
      copy(ahead, tile, ahead, 1);
    }
    if (A.chained) pdl_wait();
    for (int it = 0; lane == 0; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      if (tile >= ntiles) break;
      const int slot = it % NS;
      if (it >= NS && !mbar_wait_bounded(&empty[slot], ((it / NS) - 1) & 1, A.wait_spins)) {
        atomicExch(A.status, kStatusWaitTimeout);
        break;
      }
      if (tile + 1 == A.inject_skip) continue;  // test hook: leave the slot empty
      copy(it, tile, slot, it < ahead ? 2 : 3);
    }
    return;
  }

  // This lane's lines: x (xj, xk), (xj, xk + 4); y (yi, yk), (yi + 1, yk); z (yi, zj),
  // (yi + 1, zj).
  const int xj = lane & 7, xk = lane >> 3;
  const int yi = 2 * (lane & 3);
  const int yk = lane >> 2;
  const int zj = yk;
  // Lift factors of the faces +x and -x at this lane's i.
  const V lx2 = L::make(D.lx[8 + yi], D.lx[9 + yi]);
  const V lx4 = L::make(D.lx[yi], D.lx[1 + yi]);

  // Face-neighbour row and metric factors, one word per lane, a tile ahead.
  auto load_row = [&](const Ctx& t, int* row, float* met) {
    const long e = t.e0 + min(es, t.n - 1);
    if (lane < 6) *row = ldro(t.pbase + 6 * e + lane);
    if (lane < 9) *met = ldro(lane < 3 ? t.escale + 3 * e + lane : t.fscale + 6 * e + lane - 3);
  };
  // Plus-side values at the two ends of each line (0: low, 1: high).  An x
  // neighbour in the tile is read from shared memory later (in_x: its element
  // of the tile, else -1).
  V xq[2], xu[2], yq[2], yv[2], zq[2], zw[2];
  int in_x[2] = {-1, -1};
  // Two values at p and p + d: of a velocity, of the state.
  auto early = [&](const float* p, int d) {
    const float a = ld_early(p);
    return L::make(a, ld_early(p + d));
  };
  auto early_state = [&](const TQ* p, int d) {
    const float a = static_cast<float>(ld_early_state(p));
    return L::make(a, static_cast<float>(ld_early_state(p + d)));
  };
  auto gather = [&](const Ctx& t, int row) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      // x: faces -x (3), +x (1); node (7 or 0, j, k) of the neighbour.
      const int p = __shfl_sync(kAll, row, s == 0 ? 3 : 1);
      const int d = node_in_tile(p, t.e0, t.n, NP);
      in_x[s] = d >= 0 ? d / NP : -1;
      if (in_x[s] < 0) {
        const long n = p >= 0 ? static_cast<long>(p) + (s == 0 ? 7 : 0) + 8 * xj + 64 * xk
                              : static_cast<long>(-1 - p) + xj + 8 * xk;
        xq[s] = early_state(t.q + n, p >= 0 ? 256 : 32);
        xu[s] = early(t.u + n, p >= 0 ? 256 : 32);
      }
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      // y: faces -y (0), +y (2); nodes (i; 7 or 0; k).  A halo face may start
      // at an odd node, so these are single words.
      const int p = __shfl_sync(kAll, row, s == 0 ? 0 : 2);
      const long n = p >= 0 ? static_cast<long>(p) + (s == 0 ? 56 : 0) + 64 * yk + yi
                            : static_cast<long>(-1 - p) + 8 * yk + yi;
      yq[s] = early_state(t.q + n, 1);
      yv[s] = early(t.v + n, 1);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      // z: faces -z (4), +z (5); nodes (i; j; 7 or 0).
      const int p = __shfl_sync(kAll, row, 4 + s);
      const long n = (p >= 0 ? static_cast<long>(p) + (s == 0 ? 448 : 0)
                             : static_cast<long>(-1 - p)) + 2 * lane;
      zq[s] = early_state(t.q + n, 1);
      zw[s] = early(t.w + n, 1);
    }
  };
  // Upwind flux of upwind_flux (sdg_tend.cuh), rounded alike: sg = -1, 1 and
  // the halving are exact, so they move freely; hs = fscale / 2.
  auto flux = [](V qM, V vM, V qp, V vp, bool low, float hs) {
    const V t = L::sub_products(qp, vp, qM, vM);
    const V h = L::mul(L::abs(L::add(vp, vM)), L::add(qp, L::neg(qM)));
    return L::mul(L::dup(hs), L::fma(L::dup(-0.5f), h, low ? L::neg(t) : t));
  };
  // Node (i,j,k) of q as float, of both lines.
  auto ld_q = [](const TQ* p) {
    if constexpr (sizeof(TQ) == 4) {
      return L::ld(reinterpret_cast<const float*>(p));
    } else {
      const double2 v = *reinterpret_cast<const double2*>(p);
      return L::make(static_cast<float>(v.x), static_cast<float>(v.y));
    }
  };

  // Context of the block's tile it (batched: once its copies are there).
  auto of_tile = [&](int it, int tile) {
    if constexpr (BATCH) return *ctx_at(it);
    else return context(tile);
  };

  float met = 0.0f;
  if (blockIdx.x < ntiles) {
    int row = 0;
    const Ctx t = context(blockIdx.x);
    load_row(t, &row, &met);
    if (A.chained) pdl_wait();
    gather(t, row);
  }

  for (int it = 0;; ++it) {
    const int tile = blockIdx.x + it * gridDim.x;
    if (tile >= ntiles) break;
    const bool more = tile + gridDim.x < ntiles;
    const int slot = it % NS;
    if constexpr (BATCH) {  // the contexts come with the copies
      const uint32_t parity = (it / NS) & 1;
      const bool ok = mbar_wait_bounded(&full[slot], parity, A.wait_spins);
      if (__all_sync(kAll, ok) == 0) {
        // Wait for the copies still in flight (bounded) and leave.
        if (lane == 0) {
          atomicExch(A.status, kStatusWaitTimeout);
          if (more) mbar_wait_bounded(&full[(it + 1) % NS], ((it + 1) / NS) & 1, A.wait_spins);
          mbar_wait_bounded(&full[slot], parity, A.wait_spins);
        }
        return;
      }
    }
    const Ctx C = of_tile(it, tile);
    const Ctx N = more ? of_tile(it + 1, tile + gridDim.x) : C;
    const bool active = es < C.n;  // idle warps of a short tile keep pace
    const long base = static_cast<long>(C.e0 + (active ? es : 0)) * NP + 2 * lane;
    unsigned char* st = smem + slot * P::SLOT;
    unsigned char* sb = st + es * P::ELEM;
    const TQ* sq = reinterpret_cast<const TQ*>(sb);
    float* su = reinterpret_cast<float*>(sb + P::QB);
    float* sv = reinterpret_cast<float*>(sb + P::QB + P::VB);
    float* sw = reinterpret_cast<float*>(sb + P::QB + 2 * P::VB);

    int row_n = 0;
    float met_n = 0.0f;
    load_row(N, &row_n, &met_n);
    const float e1 = __shfl_sync(kAll, met, 0), e2 = __shfl_sync(kAll, met, 1),
                e3 = __shfl_sync(kAll, met, 2);
    float hs[6];  // fscale / 2 of the faces
#pragma unroll
    for (int f = 0; f < 6; ++f) hs[f] = 0.5f * __shfl_sync(kAll, met, 3 + f);

    if constexpr (!BATCH) {
      const uint32_t parity = (it / NS) & 1;
      const bool ok = mbar_wait_bounded(&full[slot], parity, A.wait_spins);
      if (__all_sync(kAll, ok) == 0) {
        // Wait for the copies still in flight (bounded) and leave.
        if (lane == 0) {
          atomicExch(A.status, kStatusWaitTimeout);
          if (more) mbar_wait_bounded(&full[(it + 1) % NS], ((it + 1) / NS) & 1, A.wait_spins);
          mbar_wait_bounded(&full[slot], parity, A.wait_spins);
        }
        return;
      }
    }

    // ---- Columns: q and the z-flux; w's place then takes the line sums -------
    V fz[8], wl, wh, ql, qh;
    double2 qd[sizeof(TQ) == 8 ? 8 : 1];
    V qf[sizeof(TQ) == 8 ? 1 : 8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      V q2;
      const TQ* pq = sq + swz<TQ>(yi, zj, k);
      if constexpr (sizeof(TQ) == 8) {
        qd[k] = *reinterpret_cast<const double2*>(pq);
        q2 = L::make(static_cast<float>(qd[k].x), static_cast<float>(qd[k].y));
      } else {
        q2 = qf[k] = ld_q(pq);
      }
      const V w2 = L::ld(sw + swz<float>(yi, zj, k));
      if (k == 0) { ql = q2; wl = w2; }
      if (k == 7) { qh = q2; wh = w2; }
      fz[k] = L::mul(q2, w2);
    }
    __syncwarp();

    // ---- x-lines -------------------------------------------------------------
    {
      V F[8], q0e, q7e, u0e, u7e;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        V q[4], u[4];
        if constexpr (sizeof(TQ) == 8) {
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const double2 x = *reinterpret_cast<const double2*>(sq + swz<TQ>(4 * h + 2 * m, xj, xk));
            const double2 y =
                *reinterpret_cast<const double2*>(sq + swz<TQ>(4 * h + 2 * m, xj, xk + 4));
            q[2 * m] = L::make(static_cast<float>(x.x), static_cast<float>(y.x));
            q[2 * m + 1] = L::make(static_cast<float>(x.y), static_cast<float>(y.y));
          }
        } else {
          const float4 x = *reinterpret_cast<const float4*>(sq + swz<TQ>(4 * h, xj, xk));
          const float4 y =
              *reinterpret_cast<const float4*>(sq + swz<TQ>(4 * h, xj, xk + 4));
          q[0] = L::make(x.x, y.x); q[1] = L::make(x.y, y.y);
          q[2] = L::make(x.z, y.z); q[3] = L::make(x.w, y.w);
        }
        const float4 ua = *reinterpret_cast<const float4*>(su + swz<float>(4 * h, xj, xk));
        const float4 ub =
            *reinterpret_cast<const float4*>(su + swz<float>(4 * h, xj, xk + 4));
        u[0] = L::make(ua.x, ub.x); u[1] = L::make(ua.y, ub.y);
        u[2] = L::make(ua.z, ub.z); u[3] = L::make(ua.w, ub.w);
#pragma unroll
        for (int m = 0; m < 4; ++m) F[4 * h + m] = L::mul(q[m], u[m]);
        if (h == 0) { q0e = q[0]; u0e = u[0]; }
        else { q7e = q[3]; u7e = u[3]; }
      }
      V r[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        r[i] = L::mul(L::dup(D.d[8 * i]), F[0]);
#pragma unroll
        for (int l = 1; l < 8; ++l) r[i] = L::fma(L::dup(D.d[8 * i + l]), F[l], r[i]);
      }
#pragma unroll
      for (int s = 0; s < 2; ++s)
        if (in_x[s] >= 0) {
          const unsigned char* nb = st + in_x[s] * P::ELEM;
          const TQ* nq = reinterpret_cast<const TQ*>(nb);
          const float* nu = reinterpret_cast<const float*>(nb + P::QB);
          const int i = s == 0 ? 7 : 0;
          xq[s] = L::make(static_cast<float>(nq[swz<TQ>(i, xj, xk)]),
                          static_cast<float>(nq[swz<TQ>(i, xj, xk + 4)]));
          xu[s] = L::make(nu[swz<float>(i, xj, xk)], nu[swz<float>(i, xj, xk + 4)]);
        }
      // (f2, f4) of this line over nodes 2, 3 of its u: a neighbour reads only
      // the ends.
      const V f4 = flux(q0e, u0e, xq[0], xu[0], true, hs[3]);
      const V f2 = flux(q7e, u7e, xq[1], xu[1], false, hs[1]);
      *reinterpret_cast<float2*>(su + swz<float>(2, xj, xk)) = make_float2(L::lo(f2), L::lo(f4));
      *reinterpret_cast<float2*>(su + swz<float>(2, xj, xk + 4)) =
          make_float2(L::hi(f2), L::hi(f4));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        *reinterpret_cast<float4*>(sw + swz<float>(4 * h, xj, xk)) = make_float4(
            L::lo(r[4 * h]), L::lo(r[4 * h + 1]), L::lo(r[4 * h + 2]), L::lo(r[4 * h + 3]));
        *reinterpret_cast<float4*>(sw + swz<float>(4 * h, xj, xk + 4)) = make_float4(
            L::hi(r[4 * h]), L::hi(r[4 * h + 1]), L::hi(r[4 * h + 2]), L::hi(r[4 * h + 3]));
      }
    }
    // q0 (in L2 since the tile's copies were issued).
    constexpr bool kQ0 = sizeof(TQ) == 4;  // stages 2 and 3
    double2 q0[kQ0 ? 8 : 1];
    if constexpr (kQ0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) q0[k] = ld_early_stream2(C.q0 + base + 64 * k);
    }
    __syncwarp();

    // ---- y-lines ---------------------------------------------------------------
    {
      V F[8], q0e, q7e, v0e, v7e;
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        const V q2 = ld_q(sq + swz<TQ>(yi, l, yk));
        const V v2 = L::ld(sv + swz<float>(yi, l, yk));
        F[l] = L::mul(q2, v2);
        if (l == 0) { q0e = q2; v0e = v2; }
        if (l == 7) { q7e = q2; v7e = v2; }
      }
      const V f1 = flux(q0e, v0e, yq[0], yv[0], true, hs[0]);
      const V f3 = flux(q7e, v7e, yq[1], yv[1], false, hs[2]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float* o = sw + swz<float>(yi, j, yk);
        V y = L::mul(L::dup(D.d[8 * j]), F[0]);
#pragma unroll
        for (int l = 1; l < 8; ++l) y = L::fma(L::dup(D.d[8 * j + l]), F[l], y);
        L::st(o, L::fma(L::dup(e2), y, L::mul(L::dup(e1), L::ld(o))));
        // Lift of the faces -y, +x, +y, -x, in that order.
        const float2 f24 = *reinterpret_cast<const float2*>(su + swz<float>(2, j, yk));
        V lf = L::mul(L::dup(D.ly[j]), f1);
        lf = L::fma(lx2, L::dup(f24.x), lf);
        lf = L::fma(L::dup(D.ly[8 + j]), f3, lf);
        lf = L::fma(lx4, L::dup(f24.y), lf);
        L::st(sv + swz<float>(yi, j, yk), lf);
      }
    }
    __syncwarp();

    // ---- z-lines ---------------------------------------------------------------
    const V f5 = flux(ql, wl, zq[0], zw[0], true, hs[4]);
    const V f6 = flux(qh, wh, zq[1], zw[1], false, hs[5]);
    V acc[8], lf[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      acc[k] = L::ld(sw + swz<float>(yi, zj, k));
      lf[k] = L::ld(sv + swz<float>(yi, zj, k));
    }
    // This warp is done with the slot: the next copies may overwrite it.  (With
    // q read again for the update and the slot freed after it: 91 / 88 / 96 us
    // per stage at 32^3.)
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[slot]);
    if (more) gather(N, row_n);
    met = met_n;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      V dz = L::mul(fz[0], L::dup(D.d[8 * k]));
#pragma unroll
      for (int l = 1; l < 8; ++l) dz = L::fma(fz[l], L::dup(D.d[8 * k + l]), dz);
      lf[k] = L::fma(L::dup(D.lz[k]), f5, lf[k]);
      lf[k] = L::fma(L::dup(D.lz[8 + k]), f6, lf[k]);
      acc[k] = L::add(L::fma(L::dup(e3), dz, acc[k]), lf[k]);  // -dqdt
    }
    if (!active) continue;
    // ---- RK update in FP64 (main.f90:70-71), store ------------------------------
    using AD = Ar<double, false>;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double q2[2], r[2];
      if constexpr (sizeof(TQ) == 8) {
        q2[0] = qd[k].x;
        q2[1] = qd[k].y;
      } else {
        q2[0] = static_cast<double>(L::lo(qf[k]));
        q2[1] = static_cast<double>(L::hi(qf[k]));
      }
      const float a[2] = {-L::lo(acc[k]), -L::hi(acc[k])};
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        r[m] = AD::mul(A.rk_b, AD::mad(C.dt, static_cast<double>(a[m]), q2[m]));
        if constexpr (kQ0) r[m] = AD::mad(A.rk_a, m == 0 ? q0[k].x : q0[k].y, r[m]);
      }
      TO* o = C.out + base + 64 * k;
      if constexpr (sizeof(TO) == 8)
        *reinterpret_cast<double2*>(o) = make_double2(r[0], r[1]);
      else
        *reinterpret_cast<float2*>(o) =
            make_float2(static_cast<float>(r[0]), static_cast<float>(r[1]));
    }
  }
}

}  // namespace sdg
