// lbm_pair.cuh -- the even and the odd step of an AA pair in one launch, the
// odd step trailing the even one closely enough that it finds the PDFs in L2
// (the list rows in FP64 and reduced storage, and the full-array row).
//
// What bounds the two-launch pair: each step streams all PDFs through HBM
// (304 B per FP64 node and step). The odd step of a tile needs the even step
// of the tiles its links reach and of no others: with the x-y-z numbering
// these lie within one x plane on either side. So block k of the fused launch
// runs the even step of tile k and then the odd step of a tile about two
// planes back, whose PDFs the even step wrote a few microseconds earlier: HBM
// is read once and written once per pair.
//
// Order and waiting. Even steps wait for nothing. An odd step waits until the
// groups of even tiles its links reach are complete (counters in device
// memory, release/acquire at GPU scope). The hardware starts the blocks of a
// one-dimensional grid in index order, and item k only depends on the even
// tiles of blocks at least `margin` less one group below k, so the blocks that
// a waiting one depends on have always started and, waiting for nothing before their even
// tile is counted, always finish it. The wait is bounded all the same: it
// gives up after kPairSpinLimit polls, or as soon as another block has, and
// sets the error word.
//
// Work split of a block: 8 compute warps (one thread per node) and one
// service warp that fetches the item and the tile's run record, polls the
// counters while the compute warps run the even step, and counts the even
// tile once they are done. The release then costs the compute warps nothing
// (waiting for a tile's stores to reach L2 takes 3-6 us under load; done by
// a compute warp the 256^3 packing's pair was slower by 7 %), and there is no
// block-wide barrier between the two steps.
#pragma once
#include <cstdint>

#include "lbm_bulk.cuh"
#include "lbm_chain.cuh"
#include "lbm_kernels.cuh"

namespace lbm {

constexpr int kPairThreads = kListTile + 32;
constexpr uint32_t kPairSpinLimit = 1u << 20;      // polls before giving up
constexpr uint32_t kResidentSpinLimit = 1u << 22;  // the same between resident blocks

// Cache hints. A slot written by the even step is read back by the odd step
// soon, one written by the odd step not before the next pair: even loads and
// odd stores stream (evict first), so that finished tiles do not push waiting
// ones out of L2, and FP64 even stores ask to be kept (256^3 packing, FP64,
// groups of 8 tiles: 0.298 -> 0.275 ms per step; the reduced storage takes a third or less of the
// room and does without the policy's registers).
__device__ __forceinline__ uint64_t l2_keep_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void st_keep(double* a, double v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(a), "d"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// What a block shares: what its odd item stages (kWords words), the item, and
// the hand-overs between the service warp and the compute warps.
template <int R, int kWords>
struct PairShared {
  alignas(128) uint32_t run[kWords];
  alignas(16) PairRec<R> item;
  alignas(8) uint64_t named;  // the item is here (and the first tile's run record)
  alignas(8) uint64_t go;     // the odd step may start: dependencies met, staged data here
  alignas(8) uint64_t even;   // every compute warp has stored its even nodes
};
using ListPairShared = PairShared<3, kRunTileWords>;

template <int R, int kWords>
__device__ __forceinline__ void pair_init(PairShared<R, kWords>* sh) {
  if (threadIdx.x == kListTile) {
    mbar_init(&sh->named, 1);
    mbar_init(&sh->go, 1);
    mbar_init(&sh->even, kListTile / 32);
  }
  __syncthreads();
  chain_next();
}

// One look (by the whole warp) at the even groups the item depends on:
// whether all are complete in launch number `launch` (from 1). Counters and
// targets are compared modulo 2^32.
template <int R>
__device__ __forceinline__ bool pair_ready(const PairRec<R>& it, const PairArgs<R>& p, uint32_t launch) {
  uint32_t all = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) all += it.n[r];
  bool good = true;
  for (uint32_t i = threadIdx.x & 31; i < all; i += 32) {
    uint32_t g = 0, j = i;
    bool found = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!found && j < it.n[r]) {
        g = it.lo[r] + j;
        found = true;
      }
      j -= it.n[r];
    }
    const uint32_t size = min(p.nTiles - (g << p.shift), 1u << p.shift);
    good = static_cast<int32_t>(ld_acquire(p.count + g) - launch * size) >= 0 && good;
  }
  return __all_sync(0xffffffffu, good);
}

// The service warp of block k (see above); runs(item), called by the whole warp:
// the array that the item's staged data lies in.
// first: where the run record of the item's first tile goes (two-grid lists),
// or null.
template <int R, int kWords, class Runs>
__device__ __forceinline__ void pair_serve(PairShared<R, kWords>* sh, const PairArgs<R>& p, Runs runs, int* err,
                                           uint32_t k, uint32_t* second = nullptr, uint32_t* first = nullptr) {
  constexpr int kItemWords = static_cast<int>(sizeof(PairRec<R>) / 4);
  static_assert(kItemWords <= 32, "one item word per lane");
  const int lane = threadIdx.x - kListTile;
  const bool even = k < p.nTiles;
  if (lane < kItemWords)
    reinterpret_cast<uint32_t*>(&sh->item)[lane] = __ldg(reinterpret_cast<const uint32_t*>(p.items + k) + lane);
  __syncwarp();
  const PairRec<R>& it = sh->item;
  const char* const base = static_cast<const char*>(runs(it));
  if (lane == 0) {
    if (first && it.firstRun16) {
      mbar_expect_tx(&sh->named, it.firstRun16 * 16u);
      bulk_g2s(first, base + static_cast<size_t>(it.firstRun) * 16, it.firstRun16 * 16u, &sh->named);
    }
    mbar_arrive(&sh->named);
    if (it.tile != kPairNone && it.run16) {
      mbar_expect_tx(&sh->go, it.run16 * 16u);
      bulk_g2s(second ? second : sh->run, base + static_cast<size_t>(it.run) * 16, it.run16 * 16u, &sh->go);
    }
    if (p.prefetch) {
      // the staged data and the item of blocks that have not started yet, into L2
      if (it.aheadRun16) bulk_prefetch_l2(base + static_cast<size_t>(it.aheadRun) * 16, it.aheadRun16 * 16u);
      if (k + 2 * kPairAhead < p.nItems) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.items + k + 2 * kPairAhead));
    }
  }
  chain_wait();
  // the launch counts itself: its arguments never change, so that a captured
  // launch can be replayed
  const uint32_t launch = ld_relaxed(p.launches) + 1u;
  const bool ready = it.tile == kPairNone || pair_ready(it, p, launch);
  __syncwarp();  // the vote orders nothing: what every lane acquired comes before lane 0's arrival
  if (ready && lane == 0) mbar_arrive(&sh->go);
  if (even) {
    if (!mbar_wait_bounded(&sh->even, 0)) atomicOr(err, 1);
    if (lane == 0) red_release(p.count + (k >> p.shift), 1u);
  }
  // the last block to have read the launch number moves it on
  if (lane == 0 && atomicInc(p.launches + 1, p.nItems - 1u) == p.nItems - 1u) atomicAdd(p.launches, 1u);
  if (!ready) {
    for (uint32_t spin = 0; !pair_ready(it, p, launch); ++spin) {
      const bool stop = spin >= kPairSpinLimit || ((spin & 255u) == 255u && *reinterpret_cast<volatile int*>(err) != 0);
      if (__any_sync(0xffffffffu, stop)) {
        if (lane == 0) atomicOr(err, 1);
        break;
      }
    }
    __syncwarp();  // as above
    if (lane == 0) mbar_arrive(&sh->go);
  }
}

template <int R, int kWords>
__device__ __forceinline__ void pair_service(PairShared<R, kWords>* sh, const PairArgs<R>& p, const void* runs,
                                             int* err, uint32_t k, uint32_t* second = nullptr,
                                             uint32_t* first = nullptr) {
  pair_serve(sh, p, [&](const PairRec<R>&) { return runs; }, err, k, second, first);
}

// Compute warps: their even nodes are stored.
template <class Sh>
__device__ __forceinline__ void pair_even_done(Sh* sh) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(&sh->even);
}

// Compute warps: waits for the item and the run record of its first tile;
// false if they did not come.
template <class Sh>
__device__ __forceinline__ bool pair_named(Sh* sh, int* err) {
  if (mbar_wait_bounded(&sh->named, 0)) return true;
  atomicOr(err, 1);
  return false;
}

// Compute warps: waits for the item; false if it names no odd step.
template <class Sh>
__device__ __forceinline__ bool pair_odd_named(Sh* sh, int* err) {
  return pair_named(sh, err) && sh->item.tile != kPairNone;
}

// Compute warps: waits for the odd step's turn; false if there is none.
template <class Sh>
__device__ __forceinline__ bool pair_odd_turn(Sh* sh, int* err) {
  if (!mbar_wait_bounded(&sh->go, 0)) {
    atomicOr(err, 1);
    return false;
  }
  return sh->item.tile != kPairNone;
}

// ---------------------------------------------------------------------------
// Small domains: all tiles resident, many pairs in one launch.
//
// A domain of few tiles takes many pairs in one cooperative launch, block b on
// tile b throughout: the run record is staged once, and between the half steps
// the blocks meet at a counter instead of ending and starting again. What
// bounds such a domain is that chain of latencies: 48^3 packing (172 tiles),
// FP64, 13.5 us per pair as two launches, 10.4 as one, 8.7 here; 32^3 fluid
// box 12.3, 8.3, 6.0.

// Meeting n (from 1) of the 2 * pairs that the blocks of the (cooperative)
// grid hold. Nobody waits at the last one, which only clears the counter for
// the next launch. False when the bounded wait ran out; every thread of the
// block returns the same.
__device__ __forceinline__ bool resident_meet(const ResidentArgs& r, uint32_t n, int* err, int* shOk) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t want = n * gridDim.x, last = 2u * static_cast<uint32_t>(r.pairs) * gridDim.x;
    int ok = 0;
    if (want == last) {
      if (atomicAdd(r.meet, 1u) == last - 1u) atomicExch(r.meet, 0u);
      ok = 1;
    } else {
      red_release(r.meet, 1u);
      for (uint32_t spin = 0; spin < kResidentSpinLimit && !ok; ++spin) ok = ld_acquire(r.meet) >= want;
      if (!ok) atomicOr(err, 1);
    }
    *shOk = ok;
  }
  __syncthreads();
  return *shOk != 0;
}

}  // namespace lbm
