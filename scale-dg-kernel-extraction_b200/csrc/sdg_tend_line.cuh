// Line form of the persistent fused kernel: each thread contracts whole lines
// read straight from the copied fields.
//
// tend_pipe_kernel reads every field by columns, writes the volume fluxes into
// line buffers, reads them by lines, writes the results back and collects
// everything by columns; minus sides and fluxes of the faces pass through
// buffers too: about 25 words per node through shared memory.  Here thread
// (a, b) of an element takes in turn
//
//   x-line (j,k) = (a,b): reads q and u along i, contracts, stores the sums in
//           S; it holds both ends of the line, so it evaluates the -x and +x
//           fluxes of face node (a,b) and leaves them for the y-lines;
//   y-line (i,k) = (a,b): reads q and v along j, contracts, adds to S; it
//           evaluates the -y and +y fluxes and forms the lift of the four x/y
//           faces at its nodes, over its own line of v;
//   column (i,j) = (a,b): reads q and w along k, contracts, evaluates the z
//           fluxes, adds S and the lift, updates and stores the node:
//
// about 18 words, two barriers a tile, no face buffers.  Every node's
// operations and their order are those of tend_kernel, in all forms (exact ones
// included), so the results are the other kernels' bits.
//
// A tile is E consecutive elements of one thread per line and element.  A
// producer warp keeps q of two tiles and u, v, w of one in shared memory (bulk
// copies, one mbarrier per field): u is free for the next tile after the
// x-lines, the others once every warp holds its columns.  A face neighbour in x
// that lies in the tile is read from shared memory; the other plus-side values
// are loaded a tile ahead (L2).  Waits are bounded as in tend_pipe_kernel; the
// two barriers carry the verdict, so that a block leaves as one.
#pragma once

#include "sdg_in_tile.h"
#include "sdg_tend_warp.cuh"

namespace sdg {

// Elements per tile and blocks per SM, as measured: shared memory holds 4 to 6
// elements of 9 or 10 nodes a side and one of 14 to 16 (FP64); more blocks
// compute while others wait at a barrier, larger tiles read more neighbours
// from shared memory.  Sum of the three RK stages at ~16 M DOF in us, (E, blocks):
// Nq = 10 (2,2) 525, (4,1) 563 and (1,3) 578; 11 (1,3) 557, (3,1) 584; 12 (2,1)
// 536, (1,2) 634; 13 (2,1) 516, (1,2) 642; 2 (32,4) 794, (64,3) 852, (64,4)
// 1039; FP32 2 (48,4) 527, (32,6) 542, (128,2) 577.  One tile table serves the
// three stages of the mixed form.
template <int NQ, typename TC>
struct LineTile {
  static constexpr bool F64 = sizeof(TC) == 8;
  static constexpr int E = NQ == 2 ? (F64 ? 32 : 48)
                           : (NQ == 10 || NQ == 12 || NQ == 13) ? 2 : 1;
  static constexpr int BLOCKS = NQ == 2 ? 4 : NQ == 11 ? 3 : NQ <= 10 ? 2 : 1;
};

// Where the automatic variant takes this kernel.  Measured against it (sum of
// the three RK stages at ~16 M DOF in us, this kernel / the one before):
//   fast FP64   p = 1 794 / 1099, p = 9 525 / 598, p = 10 557 / 621, p = 11 536 /
//               754, p = 12 516 / 635, p = 13 679 / 856, p = 14 754 / 1021, p = 15
//               797 / 932; slower at p = 2-6 (p = 3 761 / 551: many short lines a
//               thread, two waits each), p = 8 about equal
//   exact       p = 11 752 / 1178, p = 12 709 / 967, p = 13 861 / 1137; slower at
//               p = 10 (909 / 776), 14, 15; p = 1, 8, 9 gain 3-15 % on large
//               meshes and lose as much or more on small ones
//   mixed       p = 1 527 / 801; slower elsewhere (p = 15 531 / 419), where the
//               block kernels pack the x and y lines of a thread
template <int NQ, typename TC, bool EXACT>
constexpr bool kLineAuto =
    EXACT ? NQ >= 12 && NQ <= 14 : NQ == 2 || (sizeof(TC) == 8 && NQ >= 10);

// Whether a launch of n elements of one instance stays with the kernels before
// this one (`part`: some of a mesh's elements; `chained`: a programmatic dependent
// launch, whose barrier set-up and first copies hide behind the stage before).
// us per launch at 148 SMs, this kernel / the one before, on boxes near a cube:
//   p = 1        tiles of a few elements, four threads each, with their own set-up
//                and seven copies.  FP64 chained 1728 elements 2.75 / 2.60, 2548 2.76
//                / 2.77, 4096 2.83 / 3.51; single stages 4624 3.61 / 3.23, 5000 3.69
//                / 3.91; tendency 4624 3.39 / 3.08, 5508 3.44 / 3.74.  Mixed chained
//                4096 2.84 / 2.40, 4624 2.82 / 2.79, 5508 2.83 / 3.42; single stages
//                9240 3.76 / 3.47, 10000 3.88 / 3.93.
//   p = 9, 11, 12  single stages, whose first tile nothing hides: p = 9 64 elements
//                5.22 / 5.02, 294 6.45 / 6.28, 343 and more faster; p = 11 64 6.08 /
//                5.94, p = 12 80 7.29 / 6.75, 140 and more equal or faster.  Chained
//                ones are faster from the start (p = 9 64 4.78 / 5.05).  A part of a
//                host-buffer call follows another part's launch that it does not
//                read: five steps of 9^3 at p = 9 443 / 481 us.
//   p = 10       single stages and parts 64 6.33 / 5.43, 252 equal; chained 64 equal,
//                80 5.94 / 5.41, 144 7.03 / 5.64 (blocks of the next stage share the
//                SM), 180 to 294 equal, 343 7.83 / 10.09.  And where the second round
//                of three blocks an SM is a third full while that of two is full: 576
//                13.16 / 12.27; 448 10.84 / 11.88, 648 13.49 / 14.96.
//   p = 15       one block an SM against two: 64 10.77 / 10.54, 216 19.76 / 15.45, 512
//                40.05 / 36.82, 592 equal.
//   exact        the lift table's loads one by one: p = 11 64 7.60 / 7.29 (single 8.25 /
//                7.29), 144 7.69 / 7.85; p = 12 single 64 9.48 / 9.20.
template <int NQ, typename TC, bool EXACT, bool STAGE>
inline bool line_few(long n, long sms, bool chained, bool part) {
  constexpr bool F64 = sizeof(TC) == 8;
  const bool single = STAGE && !chained && !part;
  long per = 0;  // elements per SM
  if (EXACT) per = 2;
  else if (NQ == 16) per = 4;
  else if (NQ == 2) per = chained ? (F64 ? 17 : 30) : F64 ? 32 : 64;
  else if (NQ == 11) per = STAGE ? 2 : 0;
  else if (NQ == 10) per = single ? 2 : 0;
  else if (NQ == 12 || NQ == 13) per = single ? 1 : 0;
  return n <= per * sms || (NQ == 11 && !EXACT && STAGE && 2 * n > 7 * sms && n <= 4 * sms);
}
// The orders and forms at which it may.
template <int NQ, bool EXACT>
constexpr bool kLineFew = EXACT || NQ == 2 || (NQ >= 10 && NQ <= 13) || NQ == 16;

template <int NQ, typename TQ, typename TV, typename TC>
struct LinePlan {
  using LT = LineTile<NQ, TC>;
  static constexpr int E = LT::E;
  static constexpr int NQ2 = NQ * NQ;
  static constexpr int NP = NQ2 * NQ;
  static constexpr int LINES = E * NQ2;
  static constexpr int WARPS = (LINES + 31) / 32;  // consumer warps
  static constexpr int CTHREADS = 32 * WARPS;
  static constexpr int THREADS = CTHREADS + 32;
  static constexpr bool LATE = sizeof(TC) == 8 && NQ >= 9;
  // The x-line's sums go to S as they are formed (p = 14 in all 885 -> 754 us;
  // at Nq = 14 they go together: 679, not 900).
  static constexpr bool STORE_EACH = NQ != 14;
  static constexpr size_t r16(size_t x) { return (x + 15) & ~size_t(15); }
  // Fields are copied with their range widened to 16-byte boundaries.
  static constexpr size_t QB = r16(sizeof(TQ) * E * NP + 32);
  static constexpr size_t VB = r16(sizeof(TV) * E * NP + 32);
  static constexpr size_t EB = r16(sizeof(TC) * 3 * E + 32);  // escale rows
  static constexpr size_t FB = r16(sizeof(TC) * 6 * E + 32);  // fscale rows
  static constexpr size_t PB = r16(sizeof(int) * 6 * E + 32);  // neighbour rows
  static constexpr size_t CB = 128;                            // TileCtx
  // Two of: q, rows, context.
  static constexpr size_t OFF_E = QB;
  static constexpr size_t OFF_F = OFF_E + EB;
  static constexpr size_t OFF_P = OFF_F + FB;
  static constexpr size_t OFF_C = OFF_P + PB;
  static constexpr size_t SLOT = OFF_C + CB;
  static constexpr size_t OFF_U = 2 * SLOT;
  static constexpr size_t OFF_V = OFF_U + VB;
  static constexpr size_t OFF_W = OFF_V + VB;
  static constexpr size_t OFF_S = OFF_W + VB;                      // line sums
  static constexpr size_t OFF_X = OFF_S + r16(sizeof(TC) * E * NP);  // x fluxes
  static constexpr size_t OFF_B = OFF_X + r16(2 * sizeof(TC) * LINES);
  static constexpr size_t BYTES = OFF_B + 8 * 8;
};

// Line of NQ values at p, by the widest words its alignment gives (fields and
// sums start at 16-byte boundaries where NQ is even).
template <int NQ, typename T>
struct LineIO {
  static constexpr int BYTES = NQ * static_cast<int>(sizeof(T));
  static constexpr int W = (NQ % 2 != 0) ? 1 : (BYTES % 16 == 0 ? 16 : 8) / static_cast<int>(sizeof(T));
  static __device__ __forceinline__ void load(const T* p, T (&v)[NQ]) {
    if constexpr (W == 1) {
#pragma unroll
      for (int l = 0; l < NQ; ++l) v[l] = p[l];
    } else if constexpr (W * sizeof(T) == 16 && sizeof(T) == 4) {
#pragma unroll
      for (int l = 0; l < NQ; l += 4) {
        const float4 x = *reinterpret_cast<const float4*>(p + l);
        v[l] = x.x; v[l + 1] = x.y; v[l + 2] = x.z; v[l + 3] = x.w;
      }
    } else {
      using V2 = typename Pair2<T>::type;
#pragma unroll
      for (int l = 0; l < NQ; l += 2) {
        const V2 x = *reinterpret_cast<const V2*>(p + l);
        v[l] = x.x; v[l + 1] = x.y;
      }
    }
  }
  static __device__ __forceinline__ void store(T* p, const T (&v)[NQ]) {
    if constexpr (W == 1) {
#pragma unroll
      for (int l = 0; l < NQ; ++l) p[l] = v[l];
    } else if constexpr (W * sizeof(T) == 16 && sizeof(T) == 4) {
#pragma unroll
      for (int l = 0; l < NQ; l += 4)
        *reinterpret_cast<float4*>(p + l) = make_float4(v[l], v[l + 1], v[l + 2], v[l + 3]);
    } else {
      using V2 = typename Pair2<T>::type;
#pragma unroll
      for (int l = 0; l < NQ; l += 2) *reinterpret_cast<V2*>(p + l) = V2{v[l], v[l + 1]};
    }
  }
};

template <int NQ, typename TQ, typename TV, typename TO, typename TC, bool EXACT, int ORDER,
          bool STAGE, bool BATCH>
__global__ void __launch_bounds__((LinePlan<NQ, TQ, TV, TC>::THREADS),
                                  (LineTile<NQ, TC>::BLOCKS))
    tend_line_kernel(const __grid_constant__ TendArgs<TQ, TV, TO, TC> A,
                     const __grid_constant__ DMat<NQ, TC> D) {
  using P = LinePlan<NQ, TQ, TV, TC>;
  using AR = Ar<TC, EXACT>;
  using Ctx = TileCtx<TQ, TV, TO, TC>;
  using V2 = typename Pair2<TC>::type;
  static_assert(sizeof(TV) == sizeof(TC), "the lift goes over v");
  static_assert(sizeof(Ctx) <= P::CB, "TileCtx fits its slot area");
  constexpr int NQ2 = P::NQ2;
  constexpr int NP = P::NP;
  extern __shared__ __align__(128) unsigned char smem[];
  TC* S = reinterpret_cast<TC*>(smem + P::OFF_S);
  V2* X = reinterpret_cast<V2*>(smem + P::OFF_X);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P::OFF_B);
  uint64_t *fq = bars, *fu = bars + 2, *fv = bars + 3, *fw = bars + 4;  // filled
  uint64_t *eu = bars + 5, *done = bars + 6;  // u free; q, v, w and S free
  const int tw = A.tile_elems;  // elements per tile (single instance), at most E
  const int ntiles = BATCH ? A.ntiles : (A.nelem + tw - 1) / tw;
  const unsigned spins = A.wait_spins;

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int k = 0; k < 5; ++k) mbar_init(&bars[k], 1);
    mbar_init(eu, 1);
    mbar_init(done, P::WARPS);
    fence_barrier_init();
  }
  __syncthreads();

  if (threadIdx.x >= P::CTHREADS) {
    // ---- Producer -----------------------------------------------------------
    if (threadIdx.x != P::CTHREADS) return;
    // One field of tile context c to `dst`.
    auto copy = [&](const void* src, size_t per, const Ctx& c, unsigned char* dst,
                    uint64_t* bar, bool expect) {
      size_t lo;
      uint32_t by, sh;
      tile_range(c.e0, c.n, per, &lo, &by, &sh);
      if (expect) mbar_arrive_expect_tx(bar, by);
      bulk_g2s(dst, static_cast<const unsigned char*>(src) + lo, by, bar);
    };
    auto bytes_of = [&](size_t per, const Ctx& c) {
      size_t lo;
      uint32_t by, sh;
      tile_range(c.e0, c.n, per, &lo, &by, &sh);
      return by;
    };
    // Rows, context and the promise of q; then q itself, with q0 into L2.
    auto rows = [&](const Ctx& c, int slot) {
      unsigned char* d = smem + slot * P::SLOT;
      *reinterpret_cast<Ctx*>(d + P::OFF_C) = c;
      mbar_arrive_expect_tx(&fq[slot], bytes_of(sizeof(TQ) * NP, c) + bytes_of(sizeof(TC) * 3, c) +
                                           bytes_of(sizeof(TC) * 6, c) + bytes_of(24, c));
      copy(c.escale, sizeof(TC) * 3, c, d + P::OFF_E, &fq[slot], false);
      copy(c.fscale, sizeof(TC) * 6, c, d + P::OFF_F, &fq[slot], false);
      copy(c.pbase, 24, c, d + P::OFF_P, &fq[slot], false);
    };
    auto state = [&](const Ctx& c, int slot) {
      copy(c.q, sizeof(TQ) * NP, c, smem + slot * P::SLOT, &fq[slot], false);
      if (STAGE && A.rk_a != 0.0) {
        size_t lo;
        uint32_t by, sh;
        tile_range(c.e0, c.n, sizeof(double) * NP, &lo, &by, &sh);
        bulk_prefetch_l2(reinterpret_cast<const unsigned char*>(c.q0) + lo, by);
      }
    };
    for (int it = 0;; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      if (tile >= ntiles) break;
      const bool skip = tile + 1 == A.inject_skip;  // test hook: no copies
      Ctx c = tile_ctx<1, BATCH>(A, tile, ntiles);
      if constexpr (!BATCH) {
        c.e0 = A.elem0 + tile * tw;
        c.n = min(tw, A.nelem - tile * tw);
      }
      const int slot = it & 1;
      // The slot is free: the iteration before waited for `done` of tile it - 2.
      // (A second wait for that phase could find the barrier two phases on,
      // where its parity reads as not yet complete.)
      bool ok = true;
      // Velocities before the wait for the previous stage.
      const bool q_last = it == 0 && A.chained;
      if (!skip) {
        rows(c, slot);
        if (!q_last) state(c, slot);
        if (it == 0) {
          copy(c.u, sizeof(TV) * NP, c, smem + P::OFF_U, fu, true);
          copy(c.v, sizeof(TV) * NP, c, smem + P::OFF_V, fv, true);
          copy(c.w, sizeof(TV) * NP, c, smem + P::OFF_W, fw, true);
        }
      }
      if (q_last) {
        pdl_wait();
        if (!skip) state(c, slot);
      }
      if (it > 0) {
        ok = ok && mbar_wait_bounded(eu, (it - 1) & 1, spins);
        if (ok && !skip) copy(c.u, sizeof(TV) * NP, c, smem + P::OFF_U, fu, true);
        ok = ok && mbar_wait_bounded(done, (it - 1) & 1, spins);
        if (ok && !skip) {
          copy(c.v, sizeof(TV) * NP, c, smem + P::OFF_V, fv, true);
          copy(c.w, sizeof(TV) * NP, c, smem + P::OFF_W, fw, true);
        }
      }
      if (!ok) {
        atomicExch(A.status, kStatusWaitTimeout);
        break;
      }
    }
    return;
  }

  // ---- Consumers --------------------------------------------------------------
  const int t = threadIdx.x;
  const bool mine = t < P::LINES;  // the last warp's rest keeps pace
  const int s = mine ? t / NQ2 : 0;
  const int n = mine ? t - s * NQ2 : 0;
  const int a = n % NQ;
  const int b = n / NQ;

  // Plus-side values at face node n of faces -y, +x, +y, -x, -z, +z.
  TC qP[6], vP[6];
  int in_x[2] = {-1, -1};  // +x, -x: first node of the neighbour in the tile
  auto gather = [&](int slot) {
    const unsigned char* d = smem + slot * P::SLOT;
    Ctx c;
    if constexpr (BATCH) c = *reinterpret_cast<const Ctx*>(d + P::OFF_C);
    else {
      const Ctx& m = *reinterpret_cast<const Ctx*>(d + P::OFF_C);
      c.e0 = m.e0;
      c.n = m.n;
      c.q = A.q;
      c.u = A.u;
      c.v = A.v;
      c.w = A.w;
    }
    if (!mine || s >= c.n) return;
    const int* row = reinterpret_cast<const int*>(d + P::OFF_P + tile_shift(c.e0, 24)) + 6 * s;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int pb = row[f];
      if (f == 1 || f == 3) {
        in_x[f == 3] = node_in_tile(pb, c.e0, c.n, NP);
        if (in_x[f == 3] >= 0) continue;
      }
      const long idx = pb >= 0 ? static_cast<long>(pb) + opp_offset<NQ>(f, a, b)
                               : static_cast<long>(-1 - pb) + n;
      qP[f] = static_cast<TC>(ld_state(c.q + idx));
      vP[f] = static_cast<TC>((f == 1 || f == 3) ? ldro(c.u + idx)
                                                 : (f >= 4 ? ldro(c.w + idx) : ldro(c.v + idx)));
    }
  };

  if (A.chained) pdl_wait();
  if (blockIdx.x < ntiles) {
    if (!mbar_wait_bounded(&fq[0], 0, spins)) atomicExch(A.status, kStatusWaitTimeout);
    else gather(0);
  }

  for (int it = 0;; ++it) {
    const int tile = blockIdx.x + it * gridDim.x;
    if (tile >= ntiles) break;
    const bool more = tile + gridDim.x < ntiles;
    const int slot = it & 1;
    unsigned char* d = smem + slot * P::SLOT;

    bool ok = mbar_wait_bounded(&fq[slot], (it >> 1) & 1, spins);
    ok = ok && mbar_wait_bounded(fu, it & 1, spins);
    const Ctx& m = *reinterpret_cast<const Ctx*>(d + P::OFF_C);
    const int e0 = m.e0;
    const int cn = ok ? m.n : 0;
    const bool active = mine && s < cn;
    const TQ* tq = reinterpret_cast<const TQ*>(d + tile_shift(e0, sizeof(TQ) * NP));
    const uint32_t shv = tile_shift(e0, sizeof(TV) * NP);
    const TV* tu = reinterpret_cast<const TV*>(smem + P::OFF_U + shv);
    TV* sv = reinterpret_cast<TV*>(smem + P::OFF_V + shv) + s * NP;
    const TV* sw = reinterpret_cast<const TV*>(smem + P::OFF_W + shv) + s * NP;
    const TQ* sq = tq + s * NP;
    const TC* es = reinterpret_cast<const TC*>(d + P::OFF_E + tile_shift(e0, sizeof(TC) * 3)) + 3 * s;
    const TC* fs = reinterpret_cast<const TC*>(d + P::OFF_F + tile_shift(e0, sizeof(TC) * 6)) + 6 * s;
    TC* Se = S + s * NP;
    V2* Xe = X + s * NQ2;

    // ---- x-line (j,k) = (a,b) ---------------------------------------------------
    if (active) {
      TC F[NQ], q0e, q1e, u0e, u1e;
      {
        TQ ql[NQ];
        TV ul[NQ];
        LineIO<NQ, TQ>::load(sq + NQ * n, ql);
        LineIO<NQ, TV>::load(tu + s * NP + NQ * n, ul);
        q0e = static_cast<TC>(ql[0]);
        q1e = static_cast<TC>(ql[NQ - 1]);
        u0e = ul[0];
        u1e = ul[NQ - 1];
#pragma unroll
        for (int l = 0; l < NQ; ++l) F[l] = AR::mul(static_cast<TC>(ql[l]), ul[l]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (in_x[x] >= 0) {  // neighbour's i = 0 (+x) or Nq - 1 (-x)
          const int nn = in_x[x] + NQ * n + (x == 0 ? 0 : NQ - 1);
          qP[x == 0 ? 1 : 3] = static_cast<TC>(tq[nn]);
          vP[x == 0 ? 1 : 3] = tu[nn];
        }
      const TC f2 = upwind_flux<AR, TC>(q1e, u1e, qP[1], vP[1], TC(1), fs[1]);
      const TC f4 = upwind_flux<AR, TC>(q0e, u0e, qP[3], vP[3], TC(-1), fs[3]);
      // S and the x fluxes: once the tile before is done with them.
      TC r[NQ];
      if constexpr (P::STORE_EACH) {
        if (it > 0) ok = mbar_wait_bounded(done, (it - 1) & 1, spins) && ok;
      }
#pragma unroll
      for (int i = 0; i < NQ; ++i) {
        r[i] = contract<NQ, ORDER, AR, TC>([&](int l) { return D.d[i * NQ + l]; },
                                           [&](int l) { return F[l]; });
        if constexpr (P::STORE_EACH) {
          TC* o = Se + NQ * n + i;
          if constexpr (NQ % 2 != 0) *o = r[i];
          else if (i & 1) *reinterpret_cast<V2*>(o - 1) = V2{r[i - 1], r[i]};
        }
      }
      if constexpr (!P::STORE_EACH) {
        if (it > 0) ok = mbar_wait_bounded(done, (it - 1) & 1, spins) && ok;
        LineIO<NQ, TC>::store(Se + NQ * n, r);
      }
      Xe[n] = V2{f2, f4};
    }
    ok = ok && mbar_wait_bounded(fv, it & 1, spins);
    if (!bar_and_warps(1, P::CTHREADS, ok)) {
      if (t == 0) {
        atomicExch(A.status, kStatusWaitTimeout);
        mbar_wait_bounded(&fq[slot], (it >> 1) & 1, spins);
        mbar_wait_bounded(fu, it & 1, spins);
        mbar_wait_bounded(fv, it & 1, spins);
        mbar_wait_bounded(fw, it & 1, spins);
        if (more) mbar_wait_bounded(&fq[slot ^ 1], ((it + 1) >> 1) & 1, spins);
      }
      return;
    }
    if (t == 0) mbar_arrive(eu);

    const TC e1 = es[0], e2 = es[1], e3 = es[2];
    // ---- y-line (i,k) = (a,b) ---------------------------------------------------
    if (active) {
      const int y0 = a + NQ2 * b;
      TC F[NQ], q0e, q1e, v0e, v1e;
#pragma unroll
      for (int l = 0; l < NQ; ++l) {
        const TC qv = static_cast<TC>(sq[y0 + NQ * l]);
        const TC vv = sv[y0 + NQ * l];
        if (l == 0) { q0e = qv; v0e = vv; }
        if (l == NQ - 1) { q1e = qv; v1e = vv; }
        F[l] = AR::mul(qv, vv);
      }
      const TC f1 = upwind_flux<AR, TC>(q0e, v0e, qP[0], vP[0], TC(-1), fs[0]);
      const TC f3 = upwind_flux<AR, TC>(q1e, v1e, qP[2], vP[2], TC(1), fs[2]);
      [[maybe_unused]] TC lx2, lx4;
      if constexpr (!EXACT) {
        lx2 = ldro(A.lift + NP + a);
        lx4 = ldro(A.lift + 3 * NP + a);
      }
#pragma unroll
      for (int j = 0; j < NQ; ++j) {
        const TC y = contract<NQ, ORDER, AR, TC>([&](int l) { return F[l]; },
                                                 [&](int l) { return D.d[j * NQ + l]; });
        const int nd = y0 + NQ * j;
        Se[nd] = AR::mad(e2, y, AR::mul(e1, Se[nd]));
        TC L[4];
        if constexpr (!EXACT) {
          L[0] = D.ly[j];
          L[1] = lx2;
          L[2] = D.ly[NQ + j];
          L[3] = lx4;
        } else {
#pragma unroll
          for (int f = 0; f < 4; ++f) L[f] = ldro(A.lift + nd + NP * f);
        }
        // tensorprod_Lift_hexahedral (kern:278-283), faces 1..4.
        const V2 f24 = Xe[j + NQ * b];
        TC lf = AR::mul(L[0], f1);
        lf = AR::mad(L[1], f24.x, lf);
        lf = AR::mad(L[2], f3, lf);
        lf = AR::mad(L[3], f24.y, lf);
        sv[nd] = lf;
      }
    }
    const double* q0p = nullptr;
    TO* out = nullptr;
    double dt = 0.0;
    if constexpr (BATCH) {
      q0p = m.q0;
      out = m.out;
      dt = m.dt;
    } else {
      q0p = A.q0;
      out = A.out;
      dt = A.dt;
    }
    const long base = static_cast<long>(e0 + s) * NP + n;
    // q0 (in L2 since the tile's copies), on its way across the barrier.
    const bool use_q0 = STAGE && A.rk_a != 0.0;
    double q0r[STAGE ? NQ : 1];
    if constexpr (STAGE) {
      if (use_q0 && active) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) q0r[k] = ld_stream(q0p + base + NQ2 * k);
      }
    }
    ok = mbar_wait_bounded(fw, it & 1, spins);
    if (!bar_and_warps(1, P::CTHREADS, ok)) {
      if (t == 0) {
        atomicExch(A.status, kStatusWaitTimeout);
        mbar_wait_bounded(fw, it & 1, spins);
        if (more) {
          mbar_wait_bounded(&fq[slot ^ 1], ((it + 1) >> 1) & 1, spins);
          mbar_wait_bounded(fu, (it + 1) & 1, spins);
        }
      }
      return;
    }

    // ---- column (i,j) = (a,b) -----------------------------------------------------
    // Long FP64 columns leave S, the lift and q in shared memory until the node
    // is updated (they would spill); the others free them first.
    constexpr int NL = P::LATE ? 1 : NQ;
    TC fz[NQ], acc[NL], lf[NL], f5 = TC(0), f6 = TC(0);
    TQ qc[NL];
    if (active) {
      TC wlo = TC(0), whi = TC(0), qlo = TC(0), qhi = TC(0);
#pragma unroll
      for (int l = 0; l < NQ; ++l) {
        const TQ q1 = sq[n + NQ2 * l];
        const TC wv = sw[n + NQ2 * l];
        const TC qv = static_cast<TC>(q1);
        if (l == 0) { qlo = qv; wlo = wv; }
        if (l == NQ - 1) { qhi = qv; whi = wv; }
        fz[l] = AR::mul(qv, wv);
        if constexpr (!P::LATE) {
          qc[l] = q1;
          acc[l] = Se[n + NQ2 * l];
          lf[l] = sv[n + NQ2 * l];
        }
      }
      f5 = upwind_flux<AR, TC>(qlo, wlo, qP[4], vP[4], TC(-1), fs[4]);
      f6 = upwind_flux<AR, TC>(qhi, whi, qP[5], vP[5], TC(1), fs[5]);
    }
    // Generic writes (the lift over v) come before the copies that follow.
    auto release = [&]() {
      fence_proxy_async_smem();
      __syncwarp();
      if ((t & 31) == 0) mbar_arrive(done);
    };
    if constexpr (!P::LATE) release();
    if (more) {
      if (!mbar_wait_bounded(&fq[slot ^ 1], ((it + 1) >> 1) & 1, spins))
        atomicExch(A.status, kStatusWaitTimeout);
      else
        gather(slot ^ 1);
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < NQ; ++k) {
        const TC dz = contract<NQ, ORDER, AR, TC>([&](int l) { return fz[l]; },
                                                  [&](int l) { return D.d[k * NQ + l]; });
        TC L4, L5;
        if constexpr (!EXACT) {
          L4 = D.lz[k];
          L5 = D.lz[NQ + k];
        } else {
          L4 = ldro(A.lift + n + NQ2 * k + NP * 4);
          L5 = ldro(A.lift + n + NQ2 * k + NP * 5);
        }
        TC lk, ak;
        TQ qk;
        if constexpr (P::LATE) {
          lk = sv[n + NQ2 * k];
          ak = Se[n + NQ2 * k];
          qk = sq[n + NQ2 * k];
        } else {
          lk = lf[k];
          ak = acc[k];
          qk = qc[k];
        }
        TC f = AR::mad(L4, f5, lk);
        f = AR::mad(L5, f6, f);
        // dqdt = -(Escale1*DxF + Escale2*DyF + Escale3*DzF + Lift), eq:194-198.
        const TC dqdt = -AR::add(AR::mad(e3, dz, ak), f);
        const long o = base + NQ2 * k;
        if constexpr (!STAGE) {
          out[o] = static_cast<TO>(dqdt);
        } else {
          // q = rk_a*q0 + rk_b*(q + dt*dqdt), main.f90:70-71, in FP64.
          using AD = Ar<double, EXACT>;
          double r = AD::mul(A.rk_b, AD::mad(dt, static_cast<double>(dqdt),
                                             static_cast<double>(qk)));
          if (use_q0) r = AD::mad(A.rk_a, q0r[k], r);
          out[o] = static_cast<TO>(r);
        }
      }
    }
    if constexpr (P::LATE) release();
  }
}

}  // namespace sdg
