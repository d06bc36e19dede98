// Fast FP64 tendency / RK-stage kernel at Nq = 8: one warp per element, every
// contraction and the lift in one fragment layout of the FP64 tensor cores.
//
// A k-plane of an element is an 8x8 (j, i) block.  Lane L = 4g + c of the warp
// holds nodes (i = 2c, 2c+1; j = g) of each of the eight planes: 16-byte
// words, consecutive over the lanes, which is the C-fragment layout of mma.sync
// m8n8k4 (rows j, columns i).  So
//
//   x   C(j,i) = sum_l Fx(l,j) D(i,l)   A = Fx, formed from q and u at l = c and
//                                       c + 4 of row g, B = D
//   y   C(j,i) = sum_l D(j,l) Fy(i,l)   A = D, B = Fy, whose fragments the warp
//                                       transposes through shared memory
//   x/y lift   C(j,i) = l1(j) f1(i) + f2(j) l2(i) + l3(j) f3(i) + f4(j) l4(i)
//                                       one k-step: A = (l1,f2,l3,f4)(j),
//                                       B = (f1,l2,f3,l4)(i)
//   z   each lane holds whole columns: eight FMAs per node from registers,
//       and the two z-lift terms
//
// meet in the lane that updates and stores the node.  In the lift step lane (g, c)
// needs exactly one face flux per plane, that of face node (g, k) of face c in
// (-y, +x, +y, -x), and computes it itself: no flux goes through shared memory, and
// no phase needs more than one warp, so there is no block barrier.
//
// The tensor core adds its four products one after another in ascending l, each
// with one rounding (checked against FMA chains), so every node's operations and
// their order are those of tend_kernel, and so are the bits.  (With l = 2c + s in
// step s the A fragments of x come from registers, and with dt, the stage
// coefficient and the metric factors folded into D, w and the flux scale the sums
// need no scaling: meshes of 1,000 to 8,000 elements took 3 to 10 % less, 32^3 the
// same, but each folded operand is a rounding more: 2.37e-16 instead of 2.13e-16
// against 64 bits after five steps.)
//
// A tile is up to seven consecutive elements, one per warp; an eighth warp
// keeps a ring of two tiles (q, u, v, w: 16 KB an element) filled by bulk
// copies, full/empty mbarriers between it and the seven, one block per SM.  A
// slot is refilled, two tiles ahead, once every warp has its sums.
// The Fy transposition reuses the element's own w, which is in registers by
// then; q, u and v stay as copied, so a face neighbour in the same tile is
// read from shared memory.  The other plus-side values come from global memory
// (L2), loaded a tile ahead.  Every bounded wait and the status word work as
// in tend_pipe_kernel.
//
// Measured (32^3 elements): 123 / 134 / 133 us per single launch of RK stage 1 / 2 /
// 3 and 375 us a chained step, against 153 / 160 / 160 and 469 for the block kernel
// it replaced (two warps per element, line buffers and fluxes in shared memory); the
// step is 6.1 TB/s of the 40 / 48 / 48 algorithmic bytes per node, where a copy
// reaches 6.56.  Shared-memory pipe 75 -> 38 % busy; seven warps per SM, about 1,100
// instructions per element.  Tried on the way: seven independent warps with a ring
// each and all face values from L2, 153 / 183 / 183 (the -x/+x faces are 8-byte words
// 64 bytes apart, each a 32-byte sector); without any neighbour's values 111 / 130.
//
// H warps per element (1, 2 or 4): the latency form for meshes too small to
// give every warp of the GPU an element.  Warp h of an element takes planes
// [8h/H, 8(h+1)/H); the columns of q*w meet in shared memory for the
// z-derivative.  Each node goes through the same operations, so the results
// do not depend on H.
#pragma once

#include "sdg_tend_pipe.cuh"

namespace sdg {

// The forms that run the warp-per-element kernel.
template <int NQ, typename TC, bool EXACT>
constexpr bool kWarpKernel = NQ == 8 && sizeof(TC) == 8 && !EXACT;

// Loads that stay where they are written (asm volatile), so that the values
// are on their way while the warp works; the compiler otherwise sinks them
// towards their use.  The state is not constant over the kernel (ld_state).
__device__ __forceinline__ double ld_early(const double* p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_early_state(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_early2(const double* p) {
  double2 v;
  asm volatile("ld.global.nc.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double2 ld_early_state2(const double* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
// q0 is read once, and in stage 3 it is the array the kernel writes.
__device__ __forceinline__ double2 ld_early_stream2(const double* p) {
  double2 v;
  asm volatile("ld.global.cs.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}

template <int H, int E>
struct WarpPlan {
  static constexpr int NQ = 8;
  static constexpr int NP = 512;
  static constexpr int ELEMS = E;               // per tile at most
  static constexpr int WARPS = ELEMS * H;       // consumer warps
  static constexpr int NSTAGE = 2;
  static constexpr int THREADS = 32 * (WARPS + 1);
  static constexpr size_t FIELD = ELEMS * NP * sizeof(double);  // one field of a slot
  static constexpr size_t SLOT = 4 * FIELD;
  // Fy transposition and q*w columns, where w is not reused (H > 1).
  static constexpr size_t EXCH = H > 1 ? 2 * FIELD : 0;
  static constexpr size_t OFF_C = NSTAGE * SLOT + EXCH + 16 * NSTAGE;
  static constexpr size_t BYTES = OFF_C + 4 * 128;  // four batched tiles' contexts
};
static_assert(WarpPlan<1, kWarpElems>::BYTES <= kPipeMaxSmem &&
                  WarpPlan<2, 4>::BYTES <= kPipeMaxSmem, "warp kernel: shared memory");

// Barriers of the `threads` threads of some warps: a plain one, and one that
// also gives each of them whether all came with `ok`.
__device__ __forceinline__ void bar_sync_warps(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ bool bar_and_warps(int id, int threads, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "bar.red.and.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"(static_cast<uint32_t>(ok))
      : "memory");
  return r != 0;
}

// VEC: the arrays are 16-byte aligned (bulk copies and 16-byte accesses);
// otherwise the warp fills its slot with plain loads and stores word by word.
template <bool STAGE, bool BATCH, bool VEC, int H, int E>
__global__ void __launch_bounds__((WarpPlan<H, E>::THREADS), 1)
    tend_warp_kernel(const __grid_constant__ TendArgs<double, double, double, double> A,
                     const __grid_constant__ DMat<8, double> D) {
  using P = WarpPlan<H, E>;
  static_assert(H == 1 || VEC, "plain loads: one warp per element");
  constexpr int KP = 8 / H;   // planes of a warp
  using Ctx = TileCtx<double, double, double, double>;
  constexpr int NP = P::NP;
  constexpr size_t EB = NP * sizeof(double);  // bytes of an element's field
  constexpr int NS = VEC ? P::NSTAGE : 1;
  constexpr unsigned kAll = 0xffffffffu;
  using AR = Ar<double, false>;
  pdl_trigger();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw + P::NSTAGE * P::SLOT + P::EXCH);
  uint64_t* empty = full + P::NSTAGE;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;
  const int es = warp / H;                  // element of the tile
  const int k0 = H == 1 ? 0 : (warp - es * H) * KP;  // first plane of this warp
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

  if constexpr (VEC) {
    if (threadIdx.x == 0) {
      for (int k = 0; k < NS; ++k) {
        mbar_init(&full[k], 1);
        mbar_init(&empty[k], P::WARPS);
      }
      fence_barrier_init();
    }
    __syncthreads();
  }
  // Contexts of the block's tiles it and it + 1 (index it & 3): written before
  // the copies of tile it are announced, so whoever has waited for those reads
  // both here instead of through the tile and instance tables (batched p = 7
  // stage, 9,900 elements: 62 -> 47 us).
  Ctx* ring = reinterpret_cast<Ctx*>(smem_raw + P::OFF_C);
  static_assert(sizeof(Ctx) <= 128, "context ring");
  auto ctx_at = [&](int it) -> Ctx& {
    return *reinterpret_cast<Ctx*>(reinterpret_cast<unsigned char*>(ring) + 128 * (it & 3));
  };
  // Copies of the block's tile it into its slot: the velocities (parts & 1),
  // then q with the prefetch of q0 (parts & 2).
  auto copy = [&](int it, int parts) {
    const int tile = blockIdx.x + it * gridDim.x, slot = it % NS;
    const Ctx t = context(tile);
    if constexpr (BATCH) {
      if (parts & 1) {
        ctx_at(it) = t;
        if (tile + gridDim.x < ntiles) ctx_at(it + 1) = context(tile + gridDim.x);
      }
    }
    const size_t off = static_cast<size_t>(t.e0) * EB;
    const uint32_t bytes = static_cast<uint32_t>(t.n * EB);
    unsigned char* dst = smem_raw + slot * P::SLOT;
    const void* src[4] = {t.q, t.u, t.v, t.w};
    if (parts & 1) {
      mbar_arrive_expect_tx(&full[slot], 4 * bytes);
#pragma unroll
      for (int k = 1; k < 4; ++k)
        bulk_g2s(dst + k * P::FIELD, static_cast<const unsigned char*>(src[k]) + off, bytes,
                 &full[slot]);
    }
    if (!(parts & 2)) return;
    bulk_g2s(dst, static_cast<const unsigned char*>(src[0]) + off, bytes, &full[slot]);
    if (STAGE && A.rk_a != 0.0)
      bulk_prefetch_l2(reinterpret_cast<const unsigned char*>(t.q0) + off, bytes);
  };
  if (warp == P::WARPS) {
    // Producer: fills slot it % NS with this block's tile it once the seven
    // warps are done with tile it - NS.
    // The first tiles' velocities go before the wait for the previous stage.
    int ahead = 0;
    for (; VEC && A.chained && lane == 0 && ahead < NS; ++ahead) {
      const int tile = blockIdx.x + ahead * gridDim.x;
      if (tile >= ntiles || tile + 1 == A.inject_skip) break;
      copy(ahead, 1);
    }
    if (A.chained) pdl_wait();
    for (int it = 0; VEC && lane == 0; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      if (tile >= ntiles) break;
      const int slot = it % NS;
      if (it >= NS && !mbar_wait_bounded(&empty[slot], ((it / NS) - 1) & 1, A.wait_spins)) {
        atomicExch(A.status, kStatusWaitTimeout);
        break;  // the consumers wait for what is in flight
      }
      if (tile + 1 == A.inject_skip) continue;  // test hook: leave the slot empty
      copy(it, it < ahead ? 2 : 3);
    }
    return;
  }

  // Face of this lane: c = 0, 1, 2, 3: -y, +x, +y, -x, the order of the lift's
  // sum, face node (g, k); minus- and plus-side node of plane k = 0.
  const int face = c;
  const int moff = c == 0 ? g : (c == 1 ? 8 * g + 7 : (c == 2 ? g + 56 : 8 * g));
  const int poff = c == 0 ? g + 56 : (c == 1 ? 8 * g : (c == 2 ? g : 8 * g + 7));
  const bool yface = (c & 1) == 0;
  const double sgn = (c == 0 || c == 3) ? -1.0 : 1.0;
  // Lift factor l_f of this lane's face at normal index g (faces -y, +y along
  // j; -x, +x along i).
  const double lf = ldro(A.lift + NP * face + ((face & 1) ? g : 8 * g));
  // D fragments: D(g, c) and D(g, c + 4), B of the x and A of the y products.
  const double d0 = D.d[8 * g + c], d1 = D.d[8 * g + c + 4];
  // x fragments: nodes i = c, c + 4 of row j = g.  The lanes of every other pair
  // of rows read them in the other order, which keeps the loads free of bank
  // conflicts.
  const bool swap = (g & 2) != 0;
  const int xa = 8 * g + (swap ? c + 4 : c), xb = 8 * g + (swap ? c : c + 4);

  // Face-neighbour row (lanes 0-5) and metric factors (lanes 0-2 escale, 3-8
  // fscale) of a tile, one word per lane, shared out by shuffles: loaded a
  // tile ahead, so that nothing waits for them.
  auto load_row = [&](const Ctx& t, int* row, double* met) {
    const long e = t.e0 + min(es, t.n - 1);
    if (lane < 6) *row = ldro(t.pbase + 6 * e + lane);
    if (lane < 9) *met = ldro(lane < 3 ? t.escale + 3 * e + lane : t.fscale + 6 * e + lane - 3);
  };
  // Plus-side values of this lane's x or y face nodes (g, k): from a
  // neighbour in the tile later, from shared memory (inside: its first node
  // within the tile), else loaded here.
  double qP[KP], vP[KP];
  double2 qZ[2], wZ[2];
  int inside = -1;
  auto gather = [&](const Ctx& t, int row) {
    const int pf = __shfl_sync(kAll, row, face);
    const long d = static_cast<long>(pf) - static_cast<long>(t.e0) * NP;
    inside = (VEC && pf >= 0 && d >= 0 && d < t.n * NP) ? static_cast<int>(d) : -1;
    if (inside >= 0) return;
    // Neighbour element: plane stride 64; halo: contiguous face nodes.
    const int ks = pf >= 0 ? 64 : 8;
    const long n0 = pf >= 0 ? static_cast<long>(pf) + poff : static_cast<long>(-1 - pf) + g;
    const double* pq = t.q + n0 + k0 * ks;
    const double* pv = (yface ? t.v : t.u) + n0 + k0 * ks;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      qP[k] = ld_early_state(pq + k * ks);
      vP[k] = ld_early(pv + k * ks);
    }
  };
  // Plus-side values of the z faces at this lane's two columns.
  auto gather_z = [&](const Ctx& t, int row) {
#pragma unroll
    for (int z = 0; z < 2; ++z) {
      const int pz = __shfl_sync(kAll, row, 4 + z);
      const long n0 = (pz >= 0 ? static_cast<long>(pz) + (z == 0 ? 448 : 0)
                               : static_cast<long>(-1 - pz)) + 2 * lane;
      // A halo face may start at an odd node.
      if (VEC && (n0 & 1) == 0) {
        qZ[z] = ld_early_state2(t.q + n0);
        wZ[z] = ld_early2(t.w + n0);
      } else {
        qZ[z] = make_double2(ld_state(t.q + n0), ld_state(t.q + n0 + 1));
        wZ[z] = make_double2(ldro(t.w + n0), ldro(t.w + n0 + 1));
      }
    }
  };
  // upwind_flux (sdg_tend.cuh), rounded alike: the sign factors out of the
  // products exactly; hs = fscale / 2.
  auto flux = [](double qM, double vM, double qp, double vp, double sg, double hs) {
    const double t = AR::sub(AR::mul(qp, vp), AR::mul(qM, vM));
    const double alpha = AR::mul(0.5, fabs(AR::add(vp, vM)));
    return AR::mul(hs, fma(sg, t, -AR::mul(alpha, AR::sub(qp, qM))));
  };

  // Waits for the slot of the block's tile it (bounded); false: leave.
  auto wait_full = [&](int it) -> bool {
    const int slot = it % NS;
    const uint32_t parity = (it / NS) & 1;
    const bool ok = mbar_wait_bounded(&full[slot], parity, A.wait_spins);
    // The warps that share an element leave together, or none does.
    if (H == 1 ? __all_sync(kAll, ok) != 0 : bar_and_warps(1 + es, 32 * H, ok)) return true;
    // Wait for the copies still in flight (bounded) first.
    if (lane == 0) {
      atomicExch(A.status, kStatusWaitTimeout);
      if (blockIdx.x + (it + 1) * gridDim.x < ntiles)
        mbar_wait_bounded(&full[(it + 1) % NS], ((it + 1) / NS) & 1, A.wait_spins);
      mbar_wait_bounded(&full[slot], parity, A.wait_spins);
    }
    return false;
  };

  double met = 0.0;
  if (blockIdx.x < ntiles) {
    int row = 0;
    const Ctx t = context(blockIdx.x);
    load_row(t, &row, &met);
    if (A.chained) pdl_wait();
    gather(t, row);
    gather_z(t, row);
  }

  for (int it = 0;; ++it) {
    const int tile = blockIdx.x + it * gridDim.x;
    if (tile >= ntiles) break;
    const bool more = tile + gridDim.x < ntiles;
    const int slot = it % NS;
    Ctx C, N;
    if constexpr (BATCH) {
      if (!wait_full(it)) return;
      C = ctx_at(it);
      N = ctx_at(more ? it + 1 : it);
    } else {
      C = context(tile);
      N = context(more ? tile + gridDim.x : tile);
    }
    const bool active = es < C.n;  // idle warps of a short tile keep pace
    const long base = static_cast<long>(C.e0 + (active ? es : 0)) * NP + 64 * k0 + 2 * lane;
    unsigned char* sb = smem_raw + slot * P::SLOT;
    double* tq = reinterpret_cast<double*>(sb);  // the tile's fields
    double* tu = reinterpret_cast<double*>(sb + P::FIELD);
    double* tv = reinterpret_cast<double*>(sb + 2 * P::FIELD);
    double* sq = tq + es * NP;                   // this element's
    double* su = tu + es * NP;
    double* sv = tv + es * NP;
    double* sw = reinterpret_cast<double*>(sb + 3 * P::FIELD) + es * NP;
    // Fy transposition and q*w columns.
    double* sy = H == 1 ? sw : reinterpret_cast<double*>(smem_raw + NS * P::SLOT) + es * NP;
    double* sz = sy + P::FIELD / sizeof(double);

    // ---- q0 (in L2 since the tile's copies were issued) and the next row ---
    double2 q0[KP];
    const bool use_q0 = STAGE && A.rk_a != 0.0;
    if (use_q0) {
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        const double* p = C.q0 + base + 64 * k;
        if constexpr (VEC) q0[k] = ld_early_stream2(p);
        else q0[k] = make_double2(p[0], p[1]);
      }
    }
    int row_n = 0;
    double met_n = 0.0;
    load_row(N, &row_n, &met_n);

    const double e1 = __shfl_sync(kAll, met, 0);
    const double e2 = __shfl_sync(kAll, met, 1);
    const double e3 = __shfl_sync(kAll, met, 2);
    const double hsf = AR::mul(0.5, __shfl_sync(kAll, met, 3 + face));
    const double hsz0 = AR::mul(0.5, __shfl_sync(kAll, met, 7));
    const double hsz1 = AR::mul(0.5, __shfl_sync(kAll, met, 8));

    // ---- The element's q, u, v, w ------------------------------------------
    if constexpr (VEC) {
      if constexpr (!BATCH) {
        if (!wait_full(it)) return;
      }
    } else {
      __syncwarp();
      for (int n = 0; n < NP; n += 32) {
        sq[lane + n] = C.q[base - lane + n];
        su[lane + n] = C.u[base - lane + n];
        sv[lane + n] = C.v[base - lane + n];
        sw[lane + n] = C.w[base - lane + n];
      }
      __syncwarp();
    }

    // q: this warp's planes; fz: the whole columns of q*w.
    double fz[16], q[2 * KP];
    double ql[2], qh[2], wl[2], wh[2];
    // ---- Fluxes of the z columns, Fy to its transposition buffer ------------
    constexpr int KG = KP < 4 ? KP : 4;
#pragma unroll
    for (int h = 0; h < KP / KG; ++h) {
      double fy[2 * KG];
#pragma unroll
      for (int kk = 0; kk < KG; ++kk) {
        const int k = KG * h + kk, n = 64 * (k0 + k) + 2 * lane;
        const double2 q2 = *reinterpret_cast<const double2*>(sq + n);
        const double2 v2 = *reinterpret_cast<const double2*>(sv + n);
        const double2 w2 = *reinterpret_cast<const double2*>(sw + n);
        q[2 * k] = q2.x;
        q[2 * k + 1] = q2.y;
        if (H == 1 && k == 0) { wl[0] = w2.x; wl[1] = w2.y; }
        if (H == 1 && k == 7) { wh[0] = w2.x; wh[1] = w2.y; }
        const double z0 = AR::mul(q2.x, w2.x), z1 = AR::mul(q2.y, w2.y);
        if constexpr (H == 1) {
          fz[2 * k] = z0;
          fz[2 * k + 1] = z1;
        } else {
          *reinterpret_cast<double2*>(sz + n) = make_double2(z0, z1);
        }
        fy[2 * kk] = AR::mul(q2.x, v2.x);
        fy[2 * kk + 1] = AR::mul(q2.y, v2.y);
      }
      __syncwarp();  // every lane has read its w of these planes
      // F_y(i,j) of plane k at 64k + 8j + 2((i>>1) ^ (j&2)) + (i&1): the pair
      // stores and the fragment loads below are free of bank conflicts.
#pragma unroll
      for (int kk = 0; kk < KG; ++kk)
        *reinterpret_cast<double2*>(sy + 64 * (k0 + KG * h + kk) + 8 * g + 2 * (c ^ (g & 2))) =
            make_double2(fy[2 * kk], fy[2 * kk + 1]);
    }
    if constexpr (H == 1) {
      __syncwarp();
      ql[0] = q[0]; ql[1] = q[1];
      qh[0] = q[2 * KP - 2]; qh[1] = q[2 * KP - 1];
    } else {
      const double2 a0 = *reinterpret_cast<const double2*>(sq + 2 * lane);
      const double2 a1 = *reinterpret_cast<const double2*>(sw + 2 * lane);
      const double2 a2 = *reinterpret_cast<const double2*>(sq + 448 + 2 * lane);
      const double2 a3 = *reinterpret_cast<const double2*>(sw + 448 + 2 * lane);
      ql[0] = a0.x; ql[1] = a0.y;
      wl[0] = a1.x; wl[1] = a1.y;
      qh[0] = a2.x; qh[1] = a2.y;
      wh[0] = a3.x; wh[1] = a3.y;
      bar_sync_warps(1 + es, 32 * H);  // the columns of q*w are complete
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        const double2 z = *reinterpret_cast<const double2*>(sz + 64 * l + 2 * lane);
        fz[2 * l] = z.x;
        fz[2 * l + 1] = z.y;
      }
    }

    // ---- z-derivative and z fluxes -------------------------------------------
    // D(k,l) and the z-lift factors: constant-bank operands where the plane is
    // known at compile time (H = 1), uniform loads otherwise.
    double dz[2 * KP];
#pragma unroll
    for (int k = 0; k < 2 * KP; ++k) {
      dz[k] = AR::mul(fz[k & 1], D.d[8 * (k0 + (k >> 1))]);
#pragma unroll
      for (int l = 1; l < 8; ++l)
        dz[k] = AR::mad(fz[2 * l + (k & 1)], D.d[8 * (k0 + (k >> 1)) + l], dz[k]);
    }
    const double f5[2] = {flux(ql[0], wl[0], qZ[0].x, wZ[0].x, -1.0, hsz0),
                          flux(ql[1], wl[1], qZ[0].y, wZ[0].y, -1.0, hsz0)};
    const double f6[2] = {flux(qh[0], wh[0], qZ[1].x, wZ[1].x, 1.0, hsz1),
                          flux(qh[1], wh[1], qZ[1].y, wZ[1].y, 1.0, hsz1)};

    // ---- x and y products, lift, RK update and store, plane by plane ---------
    const double* sf = yface ? sv : su;
    if (inside >= 0) {
      const double* nq = tq + inside + poff + 64 * k0;
      const double* nf = (yface ? tv : tu) + inside + poff + 64 * k0;
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        qP[k] = nq[64 * k];
        vP[k] = nf[64 * k];
      }
    }
    const int yb = 8 * c + 2 * ((g >> 1) ^ (c & 2)) + (g & 1);
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int n = 64 * (k0 + k);
      const double ga = AR::mul(sq[n + xa], su[n + xa]), gb = AR::mul(sq[n + xb], su[n + xb]);
      double x0, x1, y0, y1, l0, l1;
      dmma_m8n8k4(x0, x1, swap ? gb : ga, d0, 0.0, 0.0);
      dmma_m8n8k4(x0, x1, swap ? ga : gb, d1, x0, x1);
      dmma_tile8(d0, d1, sy[n + yb], sy[n + yb + 32], &y0, &y1);
      const double f = flux(sq[n + moff], sf[n + moff], qP[k], vP[k], sgn, hsf);
      dmma_m8n8k4(l0, l1, yface ? lf : f, yface ? f : lf, 0.0, 0.0);
      const double xs[2] = {x0, x1}, ys[2] = {y0, y1}, ls[2] = {l0, l1};
      // The results take dz's place: no branch parts the planes here.
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double lt = AR::mad(D.lz[8 + k0 + k], f6[m], AR::mad(D.lz[k0 + k], f5[m], ls[m]));
        double acc = AR::mad(e2, ys[m], AR::mul(e1, xs[m]));
        acc = AR::mad(e3, dz[2 * k + m], acc);
        double r = -AR::add(acc, lt);
        // q = rk_a*q0 + rk_b*(q + dt*dqdt), main.f90:70-71.
        if constexpr (STAGE) r = AR::mul(A.rk_b, AR::mad(C.dt, r, q[2 * k + m]));
        dz[2 * k + m] = r;
      }
    }
    // This warp is done with the slot: the next copies may overwrite it.
    fence_proxy_async_smem();
    __syncwarp();
    if (VEC && lane == 0) mbar_arrive(&empty[slot]);
    // The next element's plus-side values: on their way through the first half
    // of the next iteration.
    if (more) {
      gather(N, row_n);
      gather_z(N, row_n);
    }
    met = met_n;

    if (use_q0) {
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        dz[2 * k] = AR::mad(A.rk_a, q0[k].x, dz[2 * k]);
        dz[2 * k + 1] = AR::mad(A.rk_a, q0[k].y, dz[2 * k + 1]);
      }
    }
    if (!active) continue;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      double* o = C.out + base + 64 * k;
      if constexpr (VEC) {
        *reinterpret_cast<double2*>(o) = make_double2(dz[2 * k], dz[2 * k + 1]);
      } else {
        o[0] = dz[2 * k];
        o[1] = dz[2 * k + 1];
      }
    }
  }
}

}  // namespace sdg
