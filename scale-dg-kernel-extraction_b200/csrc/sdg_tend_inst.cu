// Instantiates the fused tendency kernel for one polynomial order.
// Compiled once per NQ = p+1 (2..16) with -DSDG_NQ=<NQ>, so the fifteen
// fully unrolled variants build in parallel.
#include <stdint.h>

#include <algorithm>
#include <cstring>

#include "sdg_launch.h"
#include "sdg_tend.cuh"
#include "sdg_tend_pipe.cuh"
#include "sdg_tend_split.cuh"
#include "sdg_tend_line.cuh"
#include "sdg_tend_warp.cuh"
#include "sdg_tend_warp32.cuh"

#ifndef SDG_NQ
#error "SDG_NQ must be defined"
#endif

namespace sdg {
namespace {

constexpr int NQ = SDG_NQ;

// kern<<<grid, threads, smem, s.stream>>>(args...), as a programmatic dependent
// launch where the spec asks for one and the kernel takes part.
template <typename... KArgs, typename... Args>
int launch_kernel(void (*kern)(KArgs...), int grid, int threads, size_t smem,
                  const LaunchSpec& s, bool pdl, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = s.pdl && pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) cudaGetLastError();  // returned here, not by a later launch's check
  return static_cast<int>(e);
}

// Launches a persistent pipelined kernel: attribute and occupancy set-up on
// the first call of each instantiation (a call with no tiles only primes
// it, e.g. before a stream capture), then one block per resident slot.  The
// kernel is a template argument so that the set-up state belongs to that
// kernel: kernels of one signature (tendency and stage forms) differ in
// their shared-memory plans.
// floor_blocks: resident blocks per SM to launch at least (the occupancy
// query reports one block per SM for kernels that allocate tensor memory,
// whose shared memory, registers and 32 TMEM columns allow more).
template <auto KERN, int THREADS = PipeGeo<NQ>::THREADS, typename Args, typename Dm>
int launch_pipe(size_t smem, int ntiles, const LaunchSpec& s, const Args& a, const Dm& d,
                int floor_blocks = 0, bool pdl = false) {
  constexpr auto kern = KERN;
  static DeviceSetup setup;  // blocks per SM, per kernel and device
  const int dev = setup_device();
  if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
  int blocks_per_sm = setup.slot[dev].load(std::memory_order_relaxed);
  if (blocks_per_sm == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    int nb = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, THREADS, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    blocks_per_sm = std::max(nb > 0 ? nb : 1, floor_blocks);
    setup.slot[dev].store(blocks_per_sm, std::memory_order_relaxed);
  }
  if (ntiles <= 0) return 0;
  const int grid = std::min(ntiles, blocks_per_sm * (s.num_sms > 0 ? s.num_sms : 148));
  return launch_kernel(kern, grid, THREADS, smem, s, pdl, a, d);
}

// Launches the warp-per-element kernel with H warps an element and tiles of E
// elements, or fewer where that leaves an SM without one: one block per SM, or
// one per tile where there are fewer.  Chained stages of one warp an element keep
// full tiles, which leave SMs to other handles (warp_form).
template <bool STAGE, bool BATCH, bool VEC, int H, int E, typename Args, typename Dm>
int launch_warp(const LaunchSpec& s, Args& a, const Dm& d) {
  constexpr auto kern = tend_warp_kernel<STAGE, BATCH, VEC, H, E>;
  using P = WarpPlan<H, E>;
  static DeviceSetup setup;  // per kernel and device
  const int dev = setup_device();
  if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
  if (setup.slot[dev].load(std::memory_order_relaxed) == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(P::BYTES));
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    setup.slot[dev].store(1, std::memory_order_relaxed);
  }
  const int sms = s.num_sms > 0 ? s.num_sms : 148;
  a.tile_elems =
      s.pdl && H == 1 ? E : std::max(1, std::min(E, (s.nelem + sms - 1) / sms));
  const int ntiles = BATCH ? s.batch_ntiles : (s.nelem + a.tile_elems - 1) / a.tile_elems;
  if (ntiles <= 0) return 0;
  return launch_kernel(kern, std::min(ntiles, sms), P::THREADS, P::BYTES, s, true, a, d);
}

// The mixed form's warp-per-element kernel: tiles of the most elements a slot
// holds, or fewer where that leaves an SM without one.
template <auto KERN, typename TQ, typename Args, typename Dm>
int launch_warp32(const LaunchSpec& s, Args& a, const Dm& d, const FieldMaps& m) {
  constexpr auto kern = KERN;
  using P = Warp32Plan<TQ>;
  static DeviceSetup setup;  // per kernel and device
  const int dev = setup_device();
  if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
  if (setup.slot[dev].load(std::memory_order_relaxed) == 0) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(P::BYTES));
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    setup.slot[dev].store(1, std::memory_order_relaxed);
  }
  const int sms = s.num_sms > 0 ? s.num_sms : 148;
  a.tile_elems = std::max(1, std::min(P::ELEMS, (s.nelem + sms - 1) / sms));
  const int ntiles = s.batch_tiles ? s.batch_ntiles
                                   : (s.nelem + a.tile_elems - 1) / a.tile_elems;
  if (ntiles <= 0) return 0;
  return launch_kernel(kern, std::min(ntiles, sms), P::THREADS, P::BYTES, s, true, a, d, m);
}

// Warps per element of the warp-per-element kernel and elements per tile for a
// mesh of `per_sm` elements per SM: the split forms while one round of their tiles
// holds it, and two rounds of four elements where a round of seven would be
// followed by one of one.  us per single stage / per chained one, with (warps,
// elements) = (4,1) 64 elements 3.96 / 2.63; (4,2) 64 4.41 / 3.19, 252 4.64 / 3.53;
// (2,3) 252 5.11 / 3.86, 392 5.10 / 3.95; (2,4) 392 5.59 / 4.47, 576 5.62 / 4.62, 1100
// 8.64 / 7.29; (1,7) 576 6.38 / 5.23, 729 6.47 / 5.36, 1100 10.14 / 8.25.  (Nine
// warps leave a thread 168 registers instead of 255.)
//
// Chained stages, of which a program may have several handles' in flight, split only
// where the blocks of a few handles still fit side by side: a split element takes
// two to three times the SM time.  us per step of one handle / of four, this rule /
// split forms: 64 elements 8.2 / 3.9, 125 14.4 / 4.0 and 9.4 / 7.3, 343 14.1 / 5.2 and
// 12.7 / 9.0 (the pipelined kernel of this form before: 17.0 / 5.1, 19.1 / 6.9).
enum class WarpForm { k41, k42, k23, k24, k17 };
inline WarpForm warp_form(long n, long sms, bool chained) {
  if (chained) return 2 * n <= sms ? WarpForm::k41 : WarpForm::k17;
  const long per_sm = (n + sms - 1) / sms;
  return per_sm <= 1   ? WarpForm::k41
         : per_sm == 2 ? WarpForm::k42
         : per_sm == 3 ? WarpForm::k23
         : per_sm == 4 || per_sm == 8 ? WarpForm::k24
                                      : WarpForm::k17;
}

// Mixed form at Nq = 8: whether a launch of n elements stays with the pipelined
// kernel.  Its 64 threads an element have a shorter way from the first copy to the
// store than one warp, its rounds of two elements a block fill the SMs better than
// rounds of eleven where there are few, and its blocks leave room for other handles'
// where a block of eleven warps takes an SM.  us per single stage, warp / pipelined:
// 64 elements 4.42 / 3.60, 810 5.87 / 4.96, 1872 10.04 / 8.17, 4096 13.85 / 14.32; per
// step of one handle / of four: 343 12.4 / 8.4 and 12.7 / 4.0, 1331 16.8 / 15.4 and 18.2 /
// 13.2, 4096 40.8 / 42.7 and 44.4 / 39.5, 8000 69.0 / 70.4 and 78.3 / 66.2, 13824 119.6 /
// 109.9 and 129.1 / 115.6.
inline bool warp32_few(long n, long sms) { return n > 0 && n <= 64 * sms; }

// Chained launches of the pipelined kernel: up to this many nodes.  Starting early
// saves about a microsecond a launch, which small meshes feel; but the blocks that
// wait hold their SMs, which other handles' launches feel (three handles, us per
// call: FP64 27,000 elements p = 2, ten steps 356 chained, 353 not; mixed p = 2 414,504
// elements, two steps 835 and 823).
constexpr long kChainNodes = 500000;

template <typename TQ, typename TV, typename TO, typename TC, bool EXACT,
          int ORDER, bool STAGE>
int run(const LaunchSpec& s) {
  using G = Geo<NQ>;
  TendArgs<TQ, TV, TO, TC> a;
  a.q = static_cast<const TQ*>(s.q);
  a.u = static_cast<const TV*>(s.u);
  a.v = static_cast<const TV*>(s.v);
  a.w = static_cast<const TV*>(s.w);
  a.q0 = s.q0;
  a.out = static_cast<TO*>(s.out);
  a.lift = static_cast<const TC*>(s.lift);
  a.pbase = s.pbase;
  a.escale = static_cast<const TC*>(s.escale);
  a.fscale = static_cast<const TC*>(s.fscale);
  a.Ne = s.Ne;
  a.elem0 = s.elem0;
  a.nelem = s.nelem;
  a.rk_a = s.rk_a;
  a.rk_b = s.rk_b;
  a.dt = s.dt;
  a.status = s.status;
  a.wait_spins = s.wait_spins ? s.wait_spins : kWaitSpins;
  a.inject_skip = s.inject_skip;
  a.prefetch_dist = 0;
  a.tile_elems = 0;
  a.chained = s.pdl;
  a.insts = static_cast<const BatchInst*>(s.batch_insts);
  a.tiles = static_cast<const BatchTile*>(s.batch_tiles);
  a.ntiles = s.batch_ntiles;
  DMat<NQ, TC> d;
  for (int i = 0; i < NQ * NQ; ++i) d.d[i] = static_cast<TC>(s.D[i]);
  for (int i = 0; i < 2 * NQ; ++i) {
    d.lz[i] = s.lift_z ? static_cast<TC>(s.lift_z[i]) : TC(0);
    d.lx[i] = s.lift_z ? static_cast<TC>(s.lift_z[2 * NQ + i]) : TC(0);
    d.ly[i] = s.lift_z ? static_cast<TC>(s.lift_z[4 * NQ + i]) : TC(0);
  }
  using P = PipePlan<NQ, TQ, TV, TC, STAGE>;
  using PB = PipePlan<NQ, TQ, TV, TC, STAGE, false, true>;  // batched launches
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool batch = s.batch_tiles != nullptr;
  // Batched arrays are allocated 256-byte aligned by the batch itself.  The
  // fast pipelined kernels need the factored lift; with a verbatim table a
  // fast launch takes the one-tile-per-block kernel.
  const size_t pipe_bytes = batch ? PB::BYTES : P::BYTES;
  constexpr bool WARP = kWarpKernel<NQ, TC, EXACT>;
  const bool can_pipe = !WARP && pipe_bytes <= kPipeMaxSmem && pipe_bytes <= device_smem_optin() &&
                        (EXACT || s.lift_z != nullptr) &&
                        (batch || (aligned(s.q) && aligned(s.u) && aligned(s.v) &&
                                   aligned(s.w) && aligned(s.escale) && aligned(s.fscale)));
  // The one-tile-per-block kernels, asked for.
  const bool block = !batch && (s.variant == kVariantBlock || s.variant == kVariantBlockOcc);
  // Fast FP64 at Nq = 8 with a factored lift: one warp per element (bulk copies
  // where the arrays are aligned), which is also this form's pipelined kernel.
  if constexpr (WARP) {
    if (s.lift_z != nullptr && !block && WarpPlan<1, kWarpElems>::BYTES <= device_smem_optin()) {
      const bool vec = batch || (aligned(s.q) && aligned(s.u) && aligned(s.v) && aligned(s.w) &&
                                 aligned(s.out) && (s.q0 == nullptr || aligned(s.q0)));
      if (batch) return launch_warp<STAGE, true, true, 1, kWarpElems>(s, a, d);
      if (!vec) return launch_warp<STAGE, false, false, 1, kWarpElems>(s, a, d);
      const int sms = s.num_sms > 0 ? s.num_sms : 148;
      const WarpForm form = warp_form(s.nelem, sms, s.pdl);
      const bool prime = s.nelem <= 0;  // a call without elements primes every form
      int rc = 0;
      auto take = [&](WarpForm f, auto launch) {
        if (rc == 0 && (prime || form == f)) rc = launch();
      };
      take(WarpForm::k41, [&] { return launch_warp<STAGE, false, true, 4, 1>(s, a, d); });
      take(WarpForm::k42, [&] { return launch_warp<STAGE, false, true, 4, 2>(s, a, d); });
      take(WarpForm::k23, [&] { return launch_warp<STAGE, false, true, 2, 3>(s, a, d); });
      take(WarpForm::k24, [&] { return launch_warp<STAGE, false, true, 2, 4>(s, a, d); });
      take(WarpForm::k17, [&] { return launch_warp<STAGE, false, true, 1, kWarpElems>(s, a, d); });
      return rc;
    }
  }
  // The mixed form at Nq = 8, likewise, where no other kernel is asked for.
  if constexpr (STAGE && kWarp32Kernel<NQ, TC, EXACT>) {
    if (s.lift_z != nullptr &&
        (batch || (s.field_maps != nullptr && s.variant == kVariantAuto &&
                   !warp32_few(s.nelem, s.num_sms > 0 ? s.num_sms : 148))) &&
        Warp32Plan<TQ>::BYTES <= device_smem_optin()) {
      FieldMaps m;
      std::memset(&m, 0, sizeof(m));
      if (batch) return launch_warp32<tend_warp32_kernel<TQ, TO, true>, TQ>(s, a, d, m);
      std::memcpy(&m, s.field_maps, sizeof(m));
      const int rc = launch_warp32<tend_warp32_kernel<TQ, TO, false>, TQ>(s, a, d, m);
      if (rc != 0 || s.nelem > 0) return rc;
      // (A call without elements primes this kernel and the one of warp32_few.)
    }
  }
  // The line kernel.
  if constexpr (kLineAuto<NQ, TC, EXACT> && !WARP && !(STAGE && kWarp32Kernel<NQ, TC, EXACT>)) {
    using LP = LinePlan<NQ, TQ, TV, TC>;
    static_assert(LP::BYTES <= kPipeMaxSmem, "line kernel: shared memory");
    const bool can = LP::BYTES <= device_smem_optin() && (EXACT || s.lift_z != nullptr) &&
                     (batch || (aligned(s.q) && aligned(s.u) && aligned(s.v) && aligned(s.w) &&
                                aligned(s.escale) && aligned(s.fscale) && aligned(s.pbase) &&
                                (s.q0 == nullptr || aligned(s.q0))));
    const int sms = s.num_sms > 0 ? s.num_sms : 148;
    const bool prime = s.nelem <= 0 && !batch;
    const bool few = !batch && (prime ? kLineFew<NQ, EXACT>
                                      : line_few<NQ, TC, EXACT, STAGE>(s.nelem, sms, s.pdl,
                                                                       s.nelem < s.Ne));
    if (can && (s.variant == kVariantLine || (s.variant == kVariantAuto && !batch))) {
      // Shorter tiles where the longest would leave a block without one; not at Nq = 2,
      // whose elements are small: blocks of a few elements fill the SMs without using
      // them, and stages of other handles wait.  us per step of one handle / of four
      // side by side, tiles spread / full: 1,000 elements 7.3 / 3.0 and 8.1 / 2.4, 4,046
      // 8.6 / 7.5 and 9.3 / 2.9, 8,000 9.0 / 7.6 and 10.3 / 4.0 (the kernel before 14.7 / 5.4).
      const int slots = LineTile<NQ, TC>::BLOCKS * sms;
      a.tile_elems =
          NQ == 2 ? LP::E : std::max(1, std::min(LP::E, (s.nelem + slots - 1) / slots));
      const int ntiles = batch ? s.batch_ntiles : (s.nelem + a.tile_elems - 1) / a.tile_elems;
      if (batch)
        return launch_pipe<tend_line_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, true>,
                           LP::THREADS>(LP::BYTES, ntiles, s, a, d, 0, true);
      // (A call without elements primes this kernel and the one
      // that launches of few elements take.)
      if (!few || prime) {
        const int rc =
            launch_pipe<tend_line_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, false>,
                        LP::THREADS>(LP::BYTES, ntiles, s, a, d, 0, true);
        if (rc != 0 || !few) return rc;
      }
    }
  }
  // The split-column kernel: orders with one element per tile.
  if constexpr (NQ >= 9) {
    constexpr int H = kSplitH<NQ>;
    using SP = SplitPlan<NQ, H, TQ, TV, TC, STAGE>;
    const bool can_split = SP::BYTES <= kPipeMaxSmem && SP::BYTES <= device_smem_optin() &&
                           (EXACT || s.lift_z != nullptr) &&
                           (batch || (aligned(s.q) && aligned(s.u) && aligned(s.v) &&
                                      aligned(s.w) && aligned(s.escale) &&
                                      aligned(s.fscale) && aligned(s.pbase) &&
                                      (s.q0 == nullptr || aligned(s.q0))));
    const bool want_split =
        s.variant == kVariantSplit ||
        (s.variant == kVariantAuto && !batch && kSplitAuto<NQ, TC, EXACT>);
    if (want_split) {
      if (!can_split) {
        if (batch) return static_cast<int>(cudaErrorNotSupported);
      } else {
        constexpr int T = SplitGeo<NQ, H>::THREADS;
        const int ntiles = batch ? s.batch_ntiles : s.nelem;
        if (batch)
          return launch_pipe<tend_split_kernel<NQ, H, TQ, TV, TO, TC, EXACT, ORDER, STAGE, true>,
                             T>(SP::BYTES, ntiles, s, a, d);
        return launch_pipe<tend_split_kernel<NQ, H, TQ, TV, TO, TC, EXACT, ORDER, STAGE, false>,
                           T>(SP::BYTES, ntiles, s, a, d);
      }
    }
  }
  // Tensor-core lines (mixed form, Nq = 8, single instance).
  if constexpr (NQ == 8 && sizeof(TC) == 4 && !EXACT && STAGE) {
    using TP = PipePlan<NQ, TQ, TV, TC, STAGE, true>;
    if (s.variant == kVariantTensor && !batch && can_pipe && TP::BYTES <= device_smem_optin()) {
      const int ntiles = (s.nelem + PipeGeo<NQ>::EPB - 1) / PipeGeo<NQ>::EPB;
      // Blocks per SM of the plan and the launch bounds: 4 x 32 TMEM columns
      // of the SM's 512.
      constexpr int fb = pipe_min_blocks<NQ, TQ, TV, TC, EXACT, STAGE, true>();
      return launch_pipe<tend_pipe_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, false, true>>(
          TP::BYTES, ntiles, s, a, d, fb);
    }
  }
  if (batch && !can_pipe) return static_cast<int>(cudaErrorNotSupported);
  const bool pipe =
      batch || ((s.variant == kVariantPipe || s.variant == kVariantAuto ||
                 s.variant == kVariantSplit || s.variant == kVariantTensor) && can_pipe);
  if constexpr (!WARP) if (pipe) {
    const int ntiles =
        batch ? s.batch_ntiles : (s.nelem + PipeGeo<NQ>::EPB - 1) / PipeGeo<NQ>::EPB;
    constexpr bool PDL = STAGE && kPdl<NQ>;
    if constexpr (!(STAGE && kWarp32Kernel<NQ, TC, EXACT>)) {
      if (batch)
        return launch_pipe<
            tend_pipe_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, true, false, PDL>>(
            PB::BYTES, ntiles, s, a, d, 0, PDL);
    }
    // Chained launches have a kernel of their own: what they add costs the others
    // 2-4 % (mixed p = 5, 256,000 nodes 4.60 -> 4.80 us).  (A call without
    // elements primes both.)
    if constexpr (PDL) {
      const bool chain = s.pdl && static_cast<long>(s.nelem) * G::NP <= kChainNodes;
      if (chain || s.nelem <= 0) {
        const int rc = launch_pipe<
            tend_pipe_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, false, false, true>>(
            P::BYTES, ntiles, s, a, d, 0, true);
        if (rc != 0 || s.nelem > 0) return rc;
      }
    }
    return launch_pipe<tend_pipe_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, false>>(
        P::BYTES, ntiles, s, a, d);
  }

  const size_t smem = SmemLayout<NQ, TC>::BYTES;
  if constexpr (NQ >= 4 && NQ <= 8) {
    // One tile per block, built for 8 resident 128-thread blocks per SM
    // (64 registers per thread) with the largest shared-memory carveout.
    if (s.variant == kVariantBlockOcc) {
      auto kern = tend_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, 8>;
      static DeviceSetup carve;  // per device
      const int dev = setup_device();
      if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
      if (carve.slot[dev].load(std::memory_order_relaxed) == 0) {
        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        carve.slot[dev].store(1, std::memory_order_relaxed);
      }
      if (s.nelem <= 0) return 0;
      a.prefetch_dist = 8 * (s.num_sms > 0 ? s.num_sms : 148);
      const int blocks = (s.nelem + G::EPB - 1) / G::EPB;
      kern<<<blocks, G::THREADS, smem, s.stream>>>(a, d);
      return static_cast<int>(cudaGetLastError());
    }
  }
  // The fast FP64 kernels with columns of 12 or more nodes are built for two
  // resident blocks: left free they take 160-254 registers, one block of
  // 144-256 threads per SM; capped they spill but measured 1.1-1.6x faster
  // (p = 11: 29.5 -> 48.5 G DOF-updates/s, p = 15: 47.5 -> 53.0).
  constexpr int MB = (!EXACT && NQ >= 12) ? 2 : 1;
  auto kern = tend_kernel<NQ, TQ, TV, TO, TC, EXACT, ORDER, STAGE, MB>;
  static DeviceSetup setup;  // blocks per SM, per instantiation and device
  const int dev = setup_device();
  if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
  int resident = setup.slot[dev].load(std::memory_order_relaxed);
  if (resident == 0) {
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(
          kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    int nb = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, G::THREADS, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    resident = nb > 0 ? nb : 1;
    setup.slot[dev].store(resident, std::memory_order_relaxed);
  }
  if (s.nelem <= 0) return 0;
  a.prefetch_dist = resident * (s.num_sms > 0 ? s.num_sms : 148);
  const int blocks = (s.nelem + G::EPB - 1) / G::EPB;
  return launch_kernel(kern, blocks, G::THREADS, smem, s, kPdl<NQ>, a, d);
}

}  // namespace

#define SDG_CAT2(a, b) a##b
#define SDG_CAT(a, b) SDG_CAT2(a, b)

// Which persistent plans fit both the build's limit and the current
// device's per-block opt-in: bit 0 the pipelined kernel, bit 1 the
// split-column kernel (orders with one element per tile), bit 2 the
// warp-per-element kernel of the fast FP64 form, bits 3 and 4 the line kernel
// of the fast and the exact forms with its elements per tile from bit 8 up.
template <typename TQ, typename TV, typename TC, bool STAGE>
int pipe_fits() {
  const size_t optin = device_smem_optin();
  // Batched plans (the ensemble asks): the tile context travels in the slot.
  constexpr size_t bytes = PipePlan<NQ, TQ, TV, TC, STAGE, false, true>::BYTES;
  int r = (bytes <= kPipeMaxSmem && bytes <= optin) ? 1 : 0;
  if constexpr (NQ >= 9) {
    constexpr size_t sb = SplitPlan<NQ, kSplitH<NQ>, TQ, TV, TC, STAGE>::BYTES;
    if (sb <= kPipeMaxSmem && sb <= optin) r |= 2;
  }
  if constexpr (kWarpKernel<NQ, TC, false>) {
    if (WarpPlan<1, kWarpElems>::BYTES <= optin) r |= 4;
  }
  if constexpr (STAGE && kWarp32Kernel<NQ, TC, false>) {
    if (Warp32Plan<TQ>::BYTES <= optin) r |= 4;
  }
  if constexpr (kLineAuto<NQ, TC, false> || kLineAuto<NQ, TC, true>) {
    if (LinePlan<NQ, TQ, TV, TC>::BYTES <= optin)
      r |= (kLineAuto<NQ, TC, false> ? 8 : 0) | (kLineAuto<NQ, TC, true> ? 16 : 0) |
           LineTile<NQ, TC>::E << 8;
  }
  return r;
}

// Pipelined-kernel facts for this order: elements per tile, and whether the
// shared-memory plan of each kind fits.
int SDG_CAT(pipe_info_nq, SDG_NQ)(int kind, int* epb) {
  *epb = PipeGeo<NQ>::EPB;
  switch (kind) {
    case kTendF64: return pipe_fits<double, double, double, false>();
    case kStageF64: return pipe_fits<double, double, double, true>();
    case kStageMixed1: return pipe_fits<double, float, float, true>();
    case kStageMixed2: return pipe_fits<float, float, float, true>();
    case kStageMixed3: return pipe_fits<float, float, float, true>();
    default: return 0;
  }
}

int SDG_CAT(launch_tend_nq, SDG_NQ)(const LaunchSpec& s) {
  if (s.nq != NQ) return -1;
  // Orders only differ for NQ > 8; below that both map to one variant.
  const bool gen = (NQ > 8) && s.order == kOrderGeneral;
  switch (s.kind) {
    case kTendF64:
      if (!s.exact) return run<double, double, double, double, false, kOrderOpt1, false>(s);
      if (gen) return run<double, double, double, double, true, kOrderGeneral, false>(s);
      return run<double, double, double, double, true, kOrderOpt1, false>(s);
    case kStageF64:
      if (!s.exact) return run<double, double, double, double, false, kOrderOpt1, true>(s);
      if (gen) return run<double, double, double, double, true, kOrderGeneral, true>(s);
      return run<double, double, double, double, true, kOrderOpt1, true>(s);
    case kStageMixed1:
      return run<double, float, float, float, false, kOrderOpt1, true>(s);
    case kStageMixed2:
      return run<float, float, float, float, false, kOrderOpt1, true>(s);
    case kStageMixed3:
      return run<float, float, double, float, false, kOrderOpt1, true>(s);
    default:
      return static_cast<int>(cudaErrorInvalidValue);
  }
}

}  // namespace sdg
